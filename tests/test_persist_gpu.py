"""The plan-independent kernel: few-row tasks on its memory-bound body (at most eight rows), on the tensor cores (more
rows, or token ranges that narrow a row), and plans with one phase empty, against the CPU oracle's partials."""
import pytest
import torch

import gpu_utils
from test_decode_gpu import ATOL16, adhoc
from oracle import ref_attention

from ft_b200 import engine, lib

pytestmark = pytest.mark.gpu

SHAPES = [
    ([1, 20], [300, 200], 8, 4),      # 40 rows on the root, leaves of 2 rows
    ([1, 3], [700, 130], 8, 4),       # few-row tasks only, 6 and 2 rows
    ([1, 6], [64, 129], 16, 1),       # leaves of 16 rows
    ([1, 40], [200, 3], 8, 8),        # groups of short leaves: many-row tasks only
    ([1, 700], [10, 150], 4, 4),      # thousands of one-row tasks: several per CTA
]


@pytest.mark.parametrize("narrow", [False, True], ids=["whole_chunks", "row_ranges"])
@pytest.mark.parametrize("spec", SHAPES, ids=lambda s: "n%s_h%d-%d" % ("-".join(map(str, s[0])), s[2], s[3]))
def test_persistent_kernel_partials(spec, narrow):
    sizes, lens, hq, hkv = spec
    c = adhoc(sizes, lens, hq, hkv, 128, torch.float16, seed=8, q_scale=0.5)
    run = gpu_utils.EngineRun(c["nodes"], c["ptrs"], c["batch"], c["q"], c["k"], c["v"], hq, hkv, 128, c["tsq"])
    n = run.mid_o.shape[0]
    args = (run.q, run.k, run.v, run.o, *run.aux[:3], run.aux[3][:n].contiguous(), *run.aux[4:], run.tiles[0], run.tiles[1],
            run.scale)
    tabs = [t.cpu().numpy() for t in run.aux[:6]]
    tabs[3] = tabs[3][:n]
    ranges = None
    if narrow:     # every third row loses its first tokens, every third its last ones
        begin = torch.where(torch.arange(n) % 3 == 1, 2, 0)
        ranges = torch.stack([begin, torch.where(torch.arange(n) % 3 == 2, 60, 1 << 30)], dim=1).to(torch.int32).contiguous()
    elif run.aux[3].numel() >= 3 * n:      # the plan's own ranges ride behind the request ids
        ranges = run.aux[3][n:3 * n].reshape(n, 2).cpu().contiguous()
    mid_o, mid_lse = ref_attention.stage1_partials(c["q"], c["k"], c["v"], *tabs, run.scale,
                                                   q_ranges=None if ranges is None else ranges.numpy())
    engine.stage1(*args, path="persist", row_ranges=None if ranges is None else ranges.cuda())
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    torch.testing.assert_close(run.mid_lse.cpu(), mid_lse, rtol=1e-4, atol=2e-5)
    assert (run.mid_o.cpu() - mid_o).abs().max().item() <= ATOL16


@pytest.mark.parametrize("d,path", [(128, "persist"), (128, "tcgen05"), (64, "tcgen05"), (256, "tcgen05")])
def test_empty_chunks_between_others(d, path):
    """Every third task has query rows but no tokens: its partial rows are zero with an LSE of -inf, and the tasks that
    the same CTA runs before and after it are untouched."""
    c = adhoc([1, 150], [300, 130], 64, 4, d, torch.float16, seed=13, q_scale=0.5)      # 16 rows and more per task
    run = gpu_utils.EngineRun(c["nodes"], c["ptrs"], c["batch"], c["q"], c["k"], c["v"], 64, 4, d, c["tsq"])
    n = run.mid_o.shape[0]
    lens = run.aux[2].clone()
    lens[1::3] = 0
    tabs = [t.cpu().numpy() for t in run.aux[:6]]
    tabs[2], tabs[3] = lens.cpu().numpy(), tabs[3][:n]
    mid_o, mid_lse = ref_attention.stage1_partials(c["q"], c["k"], c["v"], *tabs, run.scale)
    mid_o, mid_lse = torch.nan_to_num(mid_o, nan=0.0), torch.nan_to_num(mid_lse, nan=float("-inf"), neginf=float("-inf"))
    assert int((tabs[2] == 0).sum()) * 4 > 148 and bool(mid_lse.isinf().any())
    for _ in range(3):
        run.mid_o.fill_(float("nan"))
        run.mid_lse.fill_(float("nan"))
        engine.stage1(run.q, run.k, run.v, run.o, *run.aux[:2], lens, run.aux[3][:n].contiguous(), *run.aux[4:], run.tiles[0],
                      run.tiles[1], run.scale, path=path, row_ranges=None)
        torch.cuda.synchronize()
        assert lib.read_device_status() == 0
        torch.testing.assert_close(run.mid_lse.cpu(), mid_lse, rtol=1e-4, atol=2e-5)
        assert (run.mid_o.cpu() - mid_o).abs().max().item() <= ATOL16


@pytest.mark.parametrize("d,path", [(128, "persist"), (128, "tcgen05"), (64, "tcgen05"), (256, "tcgen05")])
@pytest.mark.parametrize("rows", [132, 256, 260, 384])      # packed rows of the root's tasks: two and three passes
def test_tasks_of_several_passes(rows, d, path):
    """Tasks of more than 128 query rows: the passes of a task reuse the buffers their predecessor staged its output in,
    and the looping kernel claims its next task on the last pass."""
    import fasttree
    from ft_b200.planner import B200Model
    c = adhoc([1, rows // 4], [1500, 40], 32, 8, d, torch.float16, seed=14, q_scale=0.5)
    params = gpu_utils.make_params(32, 8, c["tsq"], "b200")
    params.b200_model = B200Model(rows_per_cta=384, min_chunk=64, group_member_tokens=0)
    aux, _ = fasttree.fasttree_preparation(gpu_utils.product_tree(c["nodes"]), c["ptrs"], c["batch"], 32, 8, d, [1024, 128],
                                           [132, 528], [132, 132], params, device="cuda")
    tabs = [t.cpu().numpy() for t in aux[:6]]
    assert int(tabs[5].max()) * 4 == rows
    mid_o, mid_lse = ref_attention.stage1_partials(c["q"], c["k"], c["v"], *tabs, d ** -0.5)
    q, k, v = c["q"].cuda(), c["k"].cuda(), c["v"].cuda()
    for _ in range(3):
        aux[9].fill_(float("nan"))
        engine.stage1(q, k, v, torch.empty_like(q), *aux, list(params.TSQs), list(params.TSKs), d ** -0.5, path=path)
        torch.cuda.synchronize()
        assert lib.read_device_status() == 0
        torch.testing.assert_close(aux[10].cpu(), mid_lse, rtol=1e-4, atol=2e-5)
        assert (aux[9].cpu() - mid_o).abs().max().item() <= ATOL16
