"""Stage 2 alone against an fp64 merge: every form of the kernel, ragged row counts, empty partials."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _merge(mid_o, mid_lse, entries, offs, lens):
    """fp64 log-sum-exp merge and its LSE, request by request."""
    out, lse = [], []
    for b in range(offs.numel()):
        rows = entries[int(offs[b]):int(offs[b]) + int(lens[b])].long()
        l, x = mid_lse[rows].double(), mid_o[rows].double()          # [n, heads], [n, heads, d]
        top = l.max(dim=0).values if rows.numel() else torch.full(mid_lse.shape[1:], -float("inf"), dtype=torch.float64, device=mid_o.device)
        w = torch.where(l > -float("inf"), (l - top.clamp(min=-1e300)).exp(), torch.zeros_like(l))
        total = w.sum(dim=0)
        x = torch.where(w[..., None] > 0, x, torch.zeros_like(x))    # an empty partial's row may hold anything
        out.append((w[..., None] * x).sum(dim=0) / total.clamp(min=1e-300)[:, None])
        lse.append(torch.where(total > 0, top + total.log(), torch.full_like(total, -float("inf"))))
    return torch.stack(out), torch.stack(lse)


# items = batch x heads x head_dim / 128; mean rows: four-warp forms (fewer and more than 12 rows), one round with and
# without shared weights, many rounds with shared weights, per-lane weights, two float4s per lane; head sizes from 16 on
@pytest.mark.parametrize("batch,heads,d,most,dtype", [
    (3, 5, 128, 40, torch.float16), (7, 8, 64, 13, torch.bfloat16), (1, 1, 16, 30, torch.float32), (9, 3, 32, 9, torch.float16),
    (50, 32, 128, 13, torch.float16), (33, 24, 256, 9, torch.bfloat16), (300, 28, 128, 20, torch.float16),
    (130, 32, 128, 4, torch.float16), (600, 16, 64, 3, torch.float32), (700, 32, 128, 3, torch.bfloat16), (70, 6, 256, 70, torch.float32),
])
def test_merge_forms_match_fp64(batch, heads, d, most, dtype):
    from ft_b200 import engine
    gen = torch.Generator().manual_seed(batch * 131 + heads)
    lens = torch.randint(1, most + 1, (batch,), generator=gen)
    lens[0] = most
    if batch > 2:
        lens[1] = 0                                   # a request without partial rows: zeros, LSE -inf
    offs = torch.cumsum(lens, 0) - lens
    total = int(lens.sum())
    entries = torch.randperm(total, generator=gen)
    mid_o = torch.randn(total, heads, d, generator=gen)
    mid_lse = torch.randn(total, heads, generator=gen) * 8
    empty = torch.rand(total, heads, generator=gen) < 0.1
    mid_lse[empty] = -float("inf")
    mid_o[empty] = float("nan")                       # never read into the result
    dev = [t.to(torch.int32).cuda() for t in (entries, offs, lens)]
    mid_o, mid_lse = mid_o.cuda(), mid_lse.cuda()
    q = torch.zeros(batch, heads, d, dtype=dtype, device="cuda")
    o = torch.full_like(q, 7.0)
    o_lse = torch.zeros(batch, heads, device="cuda")
    k = torch.zeros(1, heads, d, dtype=dtype, device="cuda")
    z = torch.zeros(1, dtype=torch.int32, device="cuda")
    rows = torch.zeros(total, dtype=torch.int32, device="cuda")
    engine.stage2(q, k, k, o, z, z, z, rows, z, z, *dev, mid_o, mid_lse, [1, 0], [0, 1], [16, 4], [64, 64], 0.1, o_lse=o_lse)
    want, want_lse = _merge(mid_o, mid_lse, *dev)
    # the sum of at most 70 products in fp32, its weights to 2^-21 each, then one rounding to the output's type
    eps = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    assert ((o.double() - want).abs() <= 1e-5 + eps * want.abs()).all()
    assert torch.equal(o_lse.isinf(), want_lse.isinf())
    fin = want_lse.isfinite()
    assert ((o_lse.double() - want_lse)[fin].abs() <= 1e-5 * want_lse[fin].abs().clamp(min=1.0)).all()
