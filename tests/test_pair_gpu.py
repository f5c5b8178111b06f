"""Few-row tasks two to a CTA (and, at head_dim 256, one by eight warps), on their own and beside many-row tasks in one grid,
against the CPU oracle's partials.  Chunk lengths around the slabs of 16 tokens and the 64 or 128 tokens that a body's warps
take per turn; consecutive rows, scattered rows and both in one chunk; 1 to 16 query rows.  Tolerances as in
test_decode_gpu.py."""
import numpy as np
import pytest
import torch

from oracle import ref_attention
from test_decode_gpu import ATOL16

from ft_b200 import engine, lib

pytestmark = pytest.mark.gpu

LENS = [1, 2, 15, 16, 17, 31, 33, 47, 48, 49, 63, 64, 65, 112, 113, 127, 128, 129, 191, 193, 255, 256, 257, 320, 400]


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


@pytest.mark.parametrize("d,few", [(64, 130), (128, 130), (256, 130), (256, 31)], ids=["64", "128", "256", "256-eight"])
@pytest.mark.parametrize("many", [0, 2])
@pytest.mark.parametrize("group,hkv,dtype", [(1, 8, torch.bfloat16), (4, 8, torch.float16), (7, 8, torch.float16)])
@pytest.mark.parametrize("extra", ["", "ranges", "bad_id"])
def test_few_row_tasks(d, few, many, group, hkv, dtype, extra):
    if few == 130 and (few * hkv // 2) * 5 < 8 * 296:
        hkv = 8 * -(-8 * 296 // (5 * few * 4))
    rows, tabs = _plan(few, many, group, seed=d + group)
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
    engine.stage1(qd, k.cuda(), v.cuda(), torch.empty_like(qd), *dev, none, none, none, mid_o, mid_lse, [many, few], [0, many],
                  [40, max(1, 16 // group)], [64, 64], d ** -0.5,
                  row_ranges=None if ranges is None else torch.from_numpy(ranges.astype(np.int32)).cuda())
    torch.cuda.synchronize()
    assert lib.read_device_status() == (lib.FT_DEV_BAD_KV_INDEX if extra == "bad_id" else 0)
    want_o, want_lse = ref_attention.stage1_partials(q, k, v, *tabs, d ** -0.5, q_ranges=ranges)
    if extra == "bad_id":
        at, n = int(tabs[4][many + 13]), int(tabs[5][many + 13])
        mid_o[at:at + n], mid_lse[at:at + n] = want_o[at:at + n].cuda(), want_lse[at:at + n].cuda()
    tol = ATOL16 + (float(want_o.abs().max()) * 2 ** -8 if dtype == torch.bfloat16 else 0.0)
    torch.testing.assert_close(mid_lse.cpu(), want_lse, rtol=1e-4, atol=2e-5)
    assert (mid_o.cpu() - want_o).abs().max().item() <= tol
