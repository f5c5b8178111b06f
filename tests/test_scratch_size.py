"""Scratch buffers that hold more rows than the plan: the merge is chosen by the plan's rows."""
import pytest
import torch

import fasttree
import gpu_utils
import kv_tree_simple
import sglang_standin
import tree_generation
from ft_b200 import engine

sglang_standin.install()

import plugin_cases  # noqa: E402
from fasttree_sglang_plugin_v0_2_13 import metadata, schedule  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,lens,hq,hkv,dtype", [
    ([1, 16], [60, 40], 32, 8, torch.float32), ([1, 16], [60, 40], 32, 8, torch.float16), ([1, 4], [512, 64], 8, 2, torch.float32),
    ([1, 40], [300, 30], 32, 8, torch.float32), ([1, 6], [3000, 90], 16, 1, torch.bfloat16), ([1, 300], [200, 20], 32, 8, torch.float32),
])
def test_spare_rows_change_nothing(sizes, lens, hq, hkv, dtype):
    nodes = kv_tree_simple.tree_from_rows(tree_generation.generate_tree(sizes, lens))
    batch, ptrs = kv_tree_simple.assign_requests(nodes)
    params = gpu_utils.make_params(hq, hkv, [max(1, 64 * hkv // hq), max(1, 16 * hkv // hq)], "b200")
    params.set_kv_dtype(dtype)
    aux, _ = fasttree.fasttree_preparation(nodes, ptrs, batch, hq, hkv, 128, [1024, 128], [132, 528], [132, 132], params)
    gen = torch.Generator(device="cuda").manual_seed(batch)
    draw = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").to(dtype)
    q, k, v = draw(batch, hq, 128), draw(ptrs[-1], hkv, 128), draw(ptrs[-1], hkv, 128)
    rows, ranges = engine.split_q_entries(aux[3])
    spare = 8192 - rows
    q_entries = torch.cat([aux[3].view(-1)[:rows], torch.zeros(spare, dtype=torch.int32, device="cuda")])
    if ranges is not None:
        ranges = torch.cat([ranges, torch.zeros(spare, 2, dtype=torch.int32, device="cuda")])
    kv_lens = aux[2].clone()
    kv_lens.task_sizes = (*aux[2].task_sizes, rows)
    large = (*aux[:2], kv_lens, q_entries, *aux[4:9], torch.empty(8192, hq, 128, device="cuda"), torch.empty(8192, hq, device="cuda"))
    exact, spared = torch.empty_like(q), torch.empty_like(q)
    rest = (*aux[11:], params.TSQs, params.TSKs, 128 ** -0.5)
    engine.decode(q, k, v, exact, *aux[:11], *rest)
    engine.decode(q, k, v, spared, *large, *rest, row_ranges=ranges)
    assert torch.equal(exact, spared)
    assert engine.build_args(q, k, v, spared, *large, *rest, row_ranges=ranges).plan_rows == rows
    assert engine.build_args(q, k, v, exact, *aux[:11], *rest).plan_rows == 0


@pytest.mark.parametrize("planner,graph_safe", [("b200", False), ("reference", False), ("b200", True)])
def test_a_serving_plan_states_its_rows(planner, graph_safe):
    """... and six per request where the launch is captured for all plans, not the buffers' capacity."""
    for name in sorted(plugin_cases.CASES):
        batch, _rows, hq, hkv = plugin_cases.build(name)
        md = metadata.FastTreeMetadata(hq, hkv, 128, "cpu", max_vnodes=4096, max_vnode_to_q_entries=8192, max_batch_size=512,
                                       planner=planner, graph_safe=graph_safe)
        schedule.prepare_for_fasttree_meta(batch, md)
        assert md.num_partial_rows < md.mid_o.shape[0]
        assert md.vnode_to_kv_lens.task_sizes[4:] == ((6 * len(batch.reqs),) if graph_safe else (md.num_partial_rows,))
