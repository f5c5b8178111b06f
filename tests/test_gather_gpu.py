"""K/V rows that are not consecutive, on the tcgen05 kernel: groups of four rows through the TMA unit, odd rows and
padding with 16-byte copies, and the layouts that have no 2-D descriptor.  The arithmetic does not depend on how a tile
reached shared memory, so the outputs are compared bit for bit with those of the same plan on consecutive rows."""
import pytest
import torch

import gpu_utils
from test_decode_gpu import adhoc

from ft_b200 import engine, lib

pytestmark = pytest.mark.gpu


def _pool(t, slot_of, slots, layout):
    """t's rows at slots slot_of, every other element NaN: rows outermost, heads outermost (rows of the 2-D view would
    overlap) or rows with a gap between heads."""
    rows, heads, d = t.shape
    nan = dict(fill_value=float("nan"), dtype=t.dtype)
    if layout == "head_major":
        pool = torch.full((heads, slots, d), **nan).permute(1, 0, 2)
    elif layout == "gaps":
        pool = torch.full((slots, heads, d + 8), **nan)[:, :, :d]
    else:
        pool = torch.full((slots, heads, d), **nan)
    dev = torch.empty_strided(pool.shape, pool.stride(), dtype=t.dtype, device="cuda")
    dev.copy_(pool)
    dev[slot_of.cuda()] = t.cuda()
    return dev


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("layout", ["rows", "gaps", "head_major"])
@pytest.mark.parametrize("length", [1, 3, 4, 61, 62, 63, 64, 65, 130, 200])   # every remainder of 4 and of the tile
def test_scattered_rows_give_the_same_bits(d, layout, length):
    c = adhoc([1, 9], [length, 5], 16, 4, d, torch.float16, seed=3, q_scale=0.5)
    run = gpu_utils.EngineRun(c["nodes"], c["ptrs"], c["batch"], c["q"], c["k"], c["v"], c["hq"], c["hkv"], d, c["tsq"])
    want = run.decode(path="tcgen05")
    rows = c["k"].shape[0]
    slots = rows + 11
    slot_of = torch.randperm(slots, generator=torch.Generator().manual_seed(length))[:rows]
    entries = run.aux[0].cpu()
    table = torch.where(entries >= 0, slot_of[entries.clamp(min=0).long()].to(torch.int32), entries).cuda()
    o = torch.full_like(run.q, float("nan"))
    engine.decode(run.q, _pool(c["k"], slot_of, slots, layout), _pool(c["v"], slot_of, slots, layout), o, table,
                  *run.aux[1:], run.tiles[0], run.tiles[1], run.scale, path="tcgen05")
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    assert torch.equal(o.float().cpu(), want)
