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


@pytest.mark.parametrize("group", [3, 5, 6, 7, 8, 12, 24, 48, 100, 128])
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("rows_per_task", [128, 384])      # one pass; passes that start inside a request
def test_query_tiles_of_any_group_size(group, d, rows_per_task):
    """Q by whole-tile boxes (requests in order), by one box per request (ids shuffled) and row by row (a pass that
    starts inside a request): the same partial rows."""
    import fasttree
    from ft_b200.planner import B200Model
    from oracle import ref_attention
    c = adhoc([1, max(2, 300 // group)], [130, 9], 2 * group, 2, d, torch.bfloat16, seed=2, q_scale=0.5)
    params = gpu_utils.make_params(c["hq"], c["hkv"], c["tsq"], "b200")
    params.b200_model = B200Model(rows_per_cta=rows_per_task)
    tree = gpu_utils.product_tree(c["nodes"])
    aux, _ = fasttree.fasttree_preparation(tree, c["ptrs"], c["batch"], c["hq"], c["hkv"], d, [1024, 128], [132, 528],
                                           [132, 132], params, device="cuda")
    n = aux[9].shape[0]
    req = aux[3][:n].clone()
    ranges = aux[3][n:3 * n].reshape(n, 2).contiguous() if aux[3].numel() > 2 * n else None
    k, v = c["k"].cuda(), c["v"].cuda()
    tabs = [t.cpu().numpy() for t in aux[:6]]
    tabs[3] = tabs[3][:n]
    want_o, want_lse = ref_attention.stage1_partials(c["q"], c["k"], c["v"], *tabs, d ** -0.5,
                                                     q_ranges=None if ranges is None else ranges.cpu().numpy())
    perm = torch.randperm(c["batch"], generator=torch.Generator().manual_seed(1))
    shuffled = torch.empty_like(c["q"])
    shuffled[perm] = c["q"]
    got = []
    for q, entries in ((c["q"], req), (shuffled, perm.cuda()[req.long()].to(torch.int32))):
        q = q.cuda()
        aux[9].fill_(float("nan"))
        engine.stage1(q, k, v, torch.empty_like(q), *aux[:3], entries, *aux[4:], list(params.TSQs), list(params.TSKs),
                      d ** -0.5, path="tcgen05", row_ranges=ranges)
        torch.cuda.synchronize()
        assert lib.read_device_status() == 0
        got.append(aux[9].clone())
        torch.testing.assert_close(aux[10].cpu(), want_lse, rtol=1e-4, atol=2e-5)
        assert (aux[9].cpu() - want_o).abs().max().item() <= 2e-3 + 2 ** -8 * want_o.abs().max().item()
    assert torch.equal(*got)
