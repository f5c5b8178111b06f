"""Few-row tasks two to a CTA (and, at head_dim 256, one by eight warps), on their own and beside many-row tasks in one grid,
against the CPU oracle's partials; and which plans take them.  Chunk lengths around the slabs of 16 tokens and the 64 or 128
tokens that a body's warps take per turn; consecutive rows, scattered rows and both in one chunk; 1 to 16 query rows, so
that at head_dim 256 a body runs one pass and two.  The task sizes a plan states choose the form and nothing else: each case
states what brings its form about and asserts it.  Tolerances as in test_decode_gpu.py."""
import numpy as np
import pytest
import torch

import fasttree
import gpu_utils
import kv_tree_simple
import tree_generation
from oracle import ref_attention
from test_decode_gpu import ATOL16

from ft_b200 import engine, lib

pytestmark = pytest.mark.gpu

LENS = [1, 2, 15, 16, 17, 31, 33, 47, 48, 49, 63, 64, 65, 112, 113, 127, 128, 129, 191, 193, 255, 256, 257, 320, 400]
FEW = 31
SIZES = {"one": (0, 0, 0, 0), "pair": (10 ** 9, 1, 0, 0), "eight": (1, 1, 1, 0)}


def _plan(few, many, group, seed):
    """Tables of `many` 40-request nodes and `few` nodes of 1 to 16 / group requests; row ids in runs, shuffled, or half-half."""
    rng = np.random.default_rng(seed)
    lens = [70 + 13 * i for i in range(many)] + [LENS[i % len(LENS)] for i in range(few)]
    qs = [40] * many + [1 + i % max(1, 16 // group) for i in range(few)]
    rows = sum(lens) + 50
    entries, at = [], 7
    for i, n in enumerate(lens):
        ids = np.arange(at, at + n)
        at += n
        if i % 3 == 1:
            rng.shuffle(ids)
        elif i % 3 == 2:
            rng.shuffle(ids[n // 2:])
        entries.append(ids)
    off = lambda x: np.concatenate([[0], np.cumsum(x)[:-1]])
    q_entries = np.concatenate([rng.permutation(64)[:n] for n in qs])
    return rows, [np.concatenate(entries), off(lens), np.array(lens), q_entries, off(qs), np.array(qs)]


@pytest.mark.parametrize("d,form", [(64, "pair"), (128, "pair"), (256, "pair"), (256, "eight")])
@pytest.mark.parametrize("many", [0, 2])
@pytest.mark.parametrize("group,hkv,dtype", [(1, 8, torch.bfloat16), (4, 8, torch.float16), (7, 8, torch.float16)])
@pytest.mark.parametrize("extra", ["", "ranges", "bad_id"])
def test_few_row_tasks(d, form, many, group, hkv, dtype, extra):
    rows, tabs = _plan(FEW, many, group, seed=d + group)
    gen = torch.Generator().manual_seed(group)
    k, v = (torch.randn(rows, hkv, d, generator=gen).to(dtype) for _ in range(2))
    q = (torch.randn(64, hkv * group, d, generator=gen) * 0.5).to(dtype)
    parts = tabs[3].size
    ranges = None
    if extra == "ranges":      # every other row loses its first tokens, its last ones, or all
        ranges = np.stack([np.arange(parts) % 5, np.full(parts, 1000)], axis=1)
        ranges[::4, 1] = 20
    dev = [torch.from_numpy(t.astype(np.int32)).cuda() for t in tabs]
    if extra == "bad_id":      # reported, read as zeros; its node's rows are not compared
        dev[0][int(tabs[1][many + 13]) + 3] = rows + 5
    mid_o, mid_lse = torch.full((parts, hkv * group, d), float("nan"), device="cuda"), torch.empty(parts, hkv * group, device="cuda")
    none = torch.zeros(64, dtype=torch.int32, device="cuda")
    qd = q.cuda()
    dev[2].task_sizes = SIZES[form]
    args = (qd, k.cuda(), v.cuda(), torch.empty_like(qd), *dev, none, none, none, mid_o, mid_lse, [many, FEW], [0, many],
            [40, max(1, 16 // group)], [64, 64], d ** -0.5)
    assert engine.stage1_path_name(*args) == (f"stage1_fused_kernel/{form}" if many or d == 256 else "stage1_pair_kernel")
    engine.stage1(*args, row_ranges=None if ranges is None else torch.from_numpy(ranges.astype(np.int32)).cuda())
    torch.cuda.synchronize()
    assert lib.read_device_status() == (lib.FT_DEV_BAD_KV_INDEX if extra == "bad_id" else 0)
    want_o, want_lse = ref_attention.stage1_partials(q, k, v, *tabs, d ** -0.5, q_ranges=ranges)
    if extra == "bad_id":
        at, n = int(tabs[4][many + 13]), int(tabs[5][many + 13])
        mid_o[at:at + n], mid_lse[at:at + n] = want_o[at:at + n].cuda(), want_lse[at:at + n].cuda()
    tol = ATOL16 + (float(want_o.abs().max()) * 2 ** -8 if dtype == torch.bfloat16 else 0.0)
    torch.testing.assert_close(mid_lse.cpu(), want_lse, rtol=1e-4, atol=2e-5)
    assert (mid_o.cpu() - want_o).abs().max().item() <= tol


ONE, PAIR, EIGHT, TC = "stage1_fused_kernel", "stage1_fused_kernel/pair", "stage1_fused_kernel/eight", "stage1_tc_kernel"


@pytest.mark.parametrize("tree,hq,hkv,d,want", [
    (("1,64", "4096,256"), 32, 8, 128, PAIR),            # even leaves in two rounds, whatever the prefix's length
    (("1,64", "8192,256"), 32, 8, 128, PAIR),
    (("1,8", "4096,256"), 32, 8, 128, ONE),              # too few
    (("1,74", "1000,400"), 32, 8, 128, ONE),             # too few for their length
    (("1,90", "1000,400"), 32, 8, 128, PAIR),
    ((5, 51848), 64, 8, 128, ONE),                       # ragged and long, 2.7 rounds
    ((4, 28143), 32, 8, 64, ONE),
    (("1,10,322", "7998,1052,233"), 64, 8, 64, ONE),     # the step waits for many-row chunks of 7998 tokens
    (("1,59,448", "16,59,142"), 16, 16, 64, PAIR),
    (("1,64", "4096,256"), 16, 8, 256, PAIR),
    (("1,47", "930,280"), 24, 8, 256, EIGHT),            # one of the tasks has 15 rows: two passes for eight, one on tcgen05
    (("1,12,24,48", "2000,400,300,200"), 64, 8, 256, EIGHT),
    (("1,18", "1000,400"), 16, 8, 256, PAIR),
    (("1,16", "1000,400"), 16, 8, 256, TC),              # one round
    (("1,21", "123,60"), 32, 32, 256, TC),               # the step waits for groups of 17 leaves
    (("1,26", "3441,314"), 32, 8, 256, TC),              # beside many-row tasks, and not short
    (("1,9", "11165,203"), 32, 8, 256, TC),              # a round and a quarter, most of it many-row
    (("1,2,4", "16011,518,10"), 32, 8, 256, TC),         # long tasks
], ids=lambda x: "-".join(map(str, x)).replace(",", ".") if isinstance(x, tuple) else str(x).replace("stage1_", ""))
def test_which_plans_take_two_tasks_per_cta(tree, hq, hkv, d, want):
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148
    if isinstance(tree[0], int):
        rows = tree_generation.generate_random_tree(*tree)
    else:
        rows = tree_generation.generate_tree(*([int(x) for x in t.split(",")] for t in tree))
    nodes = kv_tree_simple.tree_from_rows(rows)
    batch, ptrs = kv_tree_simple.assign_requests(nodes)
    params = gpu_utils.make_params(hq, hkv, [max(1, 64 * hkv // hq), max(1, 16 * hkv // hq)], "b200")
    params.set_kv_dtype(torch.float16)
    aux, _ = fasttree.fasttree_preparation(nodes, ptrs, batch, hq, hkv, d, [1024, 128], [132, 528], [132, 132], params)
    q = torch.zeros(batch, hq, d, dtype=torch.float16, device="cuda")
    kv = torch.zeros(ptrs[-1], hkv, d, dtype=torch.float16, device="cuda")
    name = lambda aux: engine.stage1_path_name(q, kv, kv, torch.empty_like(q), *aux, params.TSQs, params.TSKs, d ** -0.5)
    assert type(aux[11]) is list and name(aux) == want
    # a plan that does not state its sizes, as one made by hand: nothing is assumed
    assert name(aux[:2] + (aux[2].clone(),) + aux[3:]) == (TC if d == 256 else ONE)


@pytest.mark.parametrize("d,want", [(256, TC), (128, "stage1_narrow_kernel+stage1_tc_kernel")])
def test_a_few_row_phase_in_front_of_a_many_row_one(d, want):
    """At head_dim 256 both go to the tcgen05 kernel in one launch."""
    q = torch.zeros(64, 32, d, dtype=torch.float16, device="cuda")
    kv = torch.zeros(64, 8, d, dtype=torch.float16, device="cuda")
    ints = lambda n: torch.zeros(n, dtype=torch.int32, device="cuda")
    name = engine.stage1_path_name(q, kv, kv, torch.empty_like(q), ints(900), *[ints(50)] * 2, ints(64), *[ints(50)] * 2,
                                   ints(64), ints(64), ints(64), torch.zeros(64, 32, d, device="cuda"),
                                   torch.zeros(64, 32, device="cuda"), [40, 10], [0, 40], [4, 32], [64, 64], 0.1)
    assert name == want
