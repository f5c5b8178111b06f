"""The size of the groups of short nodes: the number of rounds in serving plans, the share of a task in the others."""
import numpy as np
import pytest
import torch

import fasttree
import kv_tree_simple
import tree_generation
from ft_b200 import lib, planner


def _burst(requests, prompts, prompt_tokens, tail_tokens, spread):
    """Shared prompts, then one private tail per request with room to grow, as the serving path hands them over."""
    per = -(-requests // prompts)
    nodes = []
    for p in range(prompts):
        ids = np.arange(p * per, min((p + 1) * per, requests), dtype=np.int32)
        nodes.append(planner.VirtualNode([(1000 * p, 1000 * p + prompt_tokens)], ids, q_tile=32, kv_split=512))
    for r in range(requests):
        n = tail_tokens + r % (spread + 1)
        nodes.append(planner.VirtualNode([(10 ** 6 + 300 * r, 10 ** 6 + 300 * r + n)], np.array([r], dtype=np.int32), q_tile=32,
                                         kv_split=128, room=12))
    return nodes


@pytest.mark.parametrize("requests,prompts,prompt_tokens,tail_tokens,spread", [
    (512, 4, 420, 36, 7), (300, 8, 300, 90, 9), (192, 4, 39, 65, 3), (209, 11, 262, 27, 5), (400, 2, 800, 12, 5), (150, 1, 64, 100, 0),
])
def test_another_number_of_rounds_only_where_its_schedule_ends_sooner(monkeypatch, requests, prompts, prompt_tokens, tail_tokens, spread):
    m = planner.B200Model(rows_per_cta=128, group_min_members=4)
    nodes = _burst(requests, prompts, prompt_tokens, tail_tokens, spread)
    slots = m.num_sms * m.ctas_per_sm // 8

    def grouped(rounds):
        monkeypatch.setattr(planner, "GROUP_ROUNDS", rounds)
        out = planner.b200_group_short_nodes(nodes, 32, 4, m, 0, direct=True, num_kv_heads=8)
        # every request's tokens are still met exactly once, whatever the grouping
        tails = sorted((r, e - b) for v in out for r, (b, e) in
                       (zip(v.requests.tolist(), v.row_ranges) if v.row_ranges is not None else
                        ((r, (0, sum(y - x for x, y in v.kv_ranges))) for r in v.requests.tolist() if len(v.requests) == 1)))
        assert tails == sorted((int(v.requests[0]), v.kv_ranges[0][1] - v.kv_ranges[0][0]) for v in nodes if len(v.requests) == 1)
        return planner.b200_simulated_schedule(out, 32, 4, m, slots)[0]

    every = planner.GROUP_ROUNDS
    ends = [grouped((q,)) for q in every]
    chosen = grouped(every)
    assert every[0] == 8 and chosen == min(ends) <= ends[0]


@pytest.mark.parametrize("sizes,lens,hq,hkv", [
    ([1, 9, 162], [1274, 157, 33], 64, 8), ([1, 14, 168], [500, 134, 14], 64, 8), ([1, 18, 216], [1990, 191, 43], 32, 4),
    ([1, 65], [150, 9], 8, 2),
])
def test_another_group_size_needs_no_more_scratch_than_there_is(monkeypatch, sizes, lens, hq, hkv):
    nodes = kv_tree_simple.tree_from_rows(tree_generation.generate_tree(sizes, lens))
    batch, ptrs = kv_tree_simple.assign_requests(nodes)

    def plan(make):
        params = fasttree.FastTreeParams()
        params.set_kv_group_num(hq // hkv)
        params.set_kv_dtype(torch.bfloat16)
        return make(nodes, ptrs, batch, hq, hkv, 128, params)

    spec, native = plan(planner.plan_b200), plan(planner.plan_b200_native)
    for name in ("vnode_to_q_entries", "vnode_to_q_offs", "vnode_to_kv_offs", "vnode_to_kv_lens", "req_to_vnode_entries"):
        np.testing.assert_array_equal(getattr(spec, name), getattr(native, name))
    monkeypatch.setattr(planner, "GROUP_CAPS", (4,))
    first = plan(planner.plan_b200)
    scratch_rows = lib.FT_STATIC_SCRATCH_BYTES // (4 * hq * 129)
    assert len(spec.vnode_to_q_entries) <= max(len(first.vnode_to_q_entries), scratch_rows)


@pytest.mark.parametrize("sizes,lens,hq,hkv,d,quarters", [
    # sizes that a schedule of equal tiles called quicker, and what they took of the first size's time
    ([1, 1, 50, 75, 301], [1993, 46, 10, 10, 32], 4, 1, 128, 4),      # 1.33: longer groups
    ([1, 2, 5, 24, 29], [300, 1178, 253, 16, 23], 32, 8, 256, 4),     # 1.22
    ([1, 343, 408], [9116, 40, 12], 24, 8, 128, 2),                   # 1.14 (the half as long ones 0.93)
    ([1, 4, 199], [590, 144, 54], 24, 8, 64, 4),                      # 1.13
    ([1, 2, 4, 8, 26], [61, 244, 25, 8, 59], 32, 8, 256, 4),          # 1.11
    ([1, 179], [740, 9], 16, 16, 128, 4),                             # 1.11
    ([1, 2, 25], [1218, 63, 9], 64, 8, 128, 4),                       # 1.07: half as many rows again for the merge
])
def test_a_group_size_that_runs_slower_is_not_taken(monkeypatch, sizes, lens, hq, hkv, d, quarters):
    nodes = kv_tree_simple.tree_from_rows(tree_generation.generate_tree(sizes, lens))
    batch, ptrs = kv_tree_simple.assign_requests(nodes)

    def tables(make):
        params = fasttree.FastTreeParams()
        params.set_kv_group_num(hq // hkv)
        params.set_kv_dtype(torch.bfloat16)
        plan = make(nodes, ptrs, batch, hq, hkv, d, params)
        return [plan.vnode_to_kv_lens, plan.vnode_to_q_lens, plan.vnode_to_q_entries]

    chosen, native = tables(planner.plan_b200), tables(planner.plan_b200_native)
    monkeypatch.setattr(planner, "GROUP_CAPS", (quarters,))
    for a, b, c in zip(chosen, native, tables(planner.plan_b200)):
        np.testing.assert_array_equal(a, c)
        np.testing.assert_array_equal(b, c)


def test_a_burst_without_groups_at_two_rounds_keeps_its_tails_apart():
    """168 tails of one or two tiles under 7 prompts at 64/8 heads: two rounds leave them alone, and so they run quickest
    (30.5 us per decode call; grouped 33.0 to 41.0)."""
    m = planner.B200Model(rows_per_cta=128, group_min_members=4)
    nodes = _burst(168, 7, 213, 82, 1)
    out = planner.b200_group_short_nodes(nodes, 16, 2, m, 0, direct=True, num_kv_heads=8)
    assert len(out) == len(nodes) and all(v.row_ranges is None for v in out)
