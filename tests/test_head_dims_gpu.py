"""The tcgen05 kernel at head_dim 64 and 256 (its shared-memory blocks, gathers, tensor-memory columns and epilogue all
follow head_dim), against the CPU oracle.  Tolerances as in test_decode_gpu.py."""
import pytest
import torch

import cases
import gpu_utils
from test_decode_gpu import ATOL16, adhoc
from oracle import ref_attention

from ft_b200 import engine, lib

pytestmark = pytest.mark.gpu

SHAPES = [
    # (level sizes, level lens, hq, hkv)
    ([1], [1], 4, 4),                    # one row, one token
    ([1, 5], [63, 65], 8, 2),            # tile -+ 1, few rows
    ([1, 15], [200, 7], 32, 8),          # 60 rows: the last row block is ragged
    ([1, 9], [150, 33], 24, 8),          # G=3: Q is gathered with 16-byte copies, not boxes
    ([1, 2], [700, 20], 128, 1),         # G=128: one request fills the row tile
    ([1, 48], [320, 129], 32, 8),        # two row tiles, exact tiles and remainders
    ([1, 3, 24], [30, 129, 31], 16, 16),
]


@pytest.mark.parametrize("d", [64, 256])
@pytest.mark.parametrize("spec", SHAPES, ids=lambda s: "n%s_h%d-%d" % ("-".join(map(str, s[0])), s[2], s[3]))
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
def test_head_dims_against_oracle(d, spec, dtype):
    sizes, lens, hq, hkv = spec
    c = adhoc(sizes, lens, hq, hkv, d, dtype, seed=4, q_scale=0.5)
    truth, truth_lse = ref_attention.per_leaf_attention(c["nodes"], c["ptrs"], c["q"], c["k"], c["v"], d ** -0.5)
    tol = ATOL16 + (float(truth.abs().max()) * 2 ** -8 if dtype == torch.bfloat16 else 0.0)
    for planner in ("reference", "b200"):
        for path in ("tcgen05", "auto"):
            run, out = gpu_utils.run_case(c, planner=planner, path=path)
            assert lib.read_device_status() == 0
            assert (out - truth).abs().max().item() <= tol, (planner, path)
            torch.testing.assert_close(run.o_lse.cpu(), truth_lse, rtol=1e-4, atol=2e-5)


@pytest.mark.parametrize("d", [64, 256])
def test_head_dims_with_scattered_rows_and_row_ranges(d):
    """Every K/V tile gathered row by row; then the same plan with each row narrowed to part of its chunk, and with one
    row id out of range, which is skipped and reported."""
    c = adhoc([1, 15], [200, 70], 32, 8, d, torch.float16, seed=9, q_scale=0.5)
    run = gpu_utils.EngineRun(c["nodes"], c["ptrs"], c["batch"], c["q"], c["k"], c["v"], c["hq"], c["hkv"], d, c["tsq"])
    want = run.decode(path="tcgen05")
    rows = c["k"].shape[0]
    slot_of = torch.randperm(rows + 37, generator=torch.Generator().manual_seed(5))[:rows]
    pools = []
    for t in (c["k"], c["v"]):
        pool = torch.full((rows + 37,) + tuple(t.shape[1:]), float("nan"), dtype=t.dtype)
        pool[slot_of] = t
        pools.append(pool.cuda())
    entries = run.aux[0].cpu()
    table = torch.where(entries >= 0, slot_of[entries.clamp(min=0)].to(torch.int32), entries).cuda()
    o = torch.full_like(run.q, float("nan"))
    args = (run.q, *pools, o, table, *run.aux[1:], run.tiles[0], run.tiles[1], run.scale)
    engine.decode(*args, path="tcgen05")
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    assert torch.equal(o.float().cpu(), want)
    # row ranges: row r of its vnode sees tokens [r, r + 50) of the chunk
    tabs = [t.cpu().numpy() for t in run.aux[:6]]
    n = run.mid_o.shape[0]
    begin = torch.arange(n, dtype=torch.int32) % 13
    ranges = torch.stack([begin, begin + 50], dim=1).contiguous()
    mid_o, mid_lse = ref_attention.stage1_partials(c["q"], c["k"], c["v"], *tabs, run.scale, q_ranges=ranges.numpy())
    engine.stage1(*args, path="tcgen05", row_ranges=ranges.cuda())
    torch.cuda.synchronize()
    torch.testing.assert_close(run.mid_lse.cpu(), mid_lse, rtol=1e-4, atol=2e-5)
    assert (run.mid_o.cpu() - mid_o).abs().max().item() <= ATOL16
    table[3] = 10 ** 8
    engine.decode(*args, path="tcgen05")
    assert lib.read_device_status() & lib.FT_DEV_BAD_KV_INDEX


@pytest.mark.parametrize("d", [64, 256])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("spec", [([1, 16, 256], [64, 32, 16], 32, 8), ([1, 3, 50], [100, 1, 40], 16, 1),
                                  ([1, 40], [10, 20], 8, 8)], ids=["g4", "g16", "g1"])
def test_groups_of_short_nodes(d, dtype, spec):
    """Leaves grouped into many-row tasks with token ranges, through every kernel family that takes the head size."""
    sizes, lens, hq, hkv = spec
    c = adhoc(sizes, lens, hq, hkv, d, dtype, seed=6, q_scale=0.5)
    truth, truth_lse = ref_attention.per_leaf_attention(c["nodes"], c["ptrs"], c["q"], c["k"], c["v"], d ** -0.5)
    tol = ATOL16 + (float(truth.abs().max()) * 2 ** -8 if dtype == torch.bfloat16 else 0.0)
    for path in ("auto", "tcgen05", "generic") + (("mma", "mma_wide", "stream") if d == 64 else ()):
        run, out = gpu_utils.run_case(c, planner="b200", path=path, tell_dtype=True)
        assert run.aux[3].numel() > 2 * run.mid_o.shape[0]       # the plan carries token ranges
        assert lib.read_device_status() == 0
        assert (out - truth).abs().max().item() <= tol, path
        torch.testing.assert_close(run.o_lse.cpu(), truth_lse, rtol=1e-4, atol=2e-5)
