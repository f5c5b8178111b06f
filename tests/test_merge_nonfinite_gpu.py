"""Stage 2 on partial rows with infinities and NaN: what counts is the row's weight, not where the row stands or which
kernel meets it."""
import pytest
import torch

from ft_b200 import engine, lib

pytestmark = pytest.mark.gpu


def _merge(rows, mid_o, mid_lse, dtype, batch, heads, d):
    dev = torch.device("cuda")
    offs = torch.arange(batch, dtype=torch.int32, device=dev) * rows
    lens = torch.full((batch,), rows, dtype=torch.int32, device=dev)
    entries = torch.arange(batch * rows, dtype=torch.int32, device=dev)
    q = torch.zeros(batch, heads, d, dtype=dtype, device=dev)
    o, o_lse = torch.full_like(q, 7.0), torch.zeros(batch, heads, device=dev)
    k = torch.zeros(1, heads, d, dtype=dtype, device=dev)
    z = torch.zeros(1, dtype=torch.int32, device=dev)
    q_entries = torch.zeros(batch * rows, dtype=torch.int32, device=dev)
    engine.stage2(q, k, k, o, z, z, z, q_entries, z, z, entries, offs, lens, mid_o, mid_lse, [1, 0], [0, 1], [16, 4], [64, 64],
                  0.1, o_lse=o_lse)
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    return o, o_lse


# forms: four warps per piece (both depths), pieces one per warp, two per warp, one warp per head (one round, several, 256)
@pytest.mark.parametrize("rows,batch,heads,d,dtype", [
    (14, 3, 8, 128, torch.float16), (40, 5, 4, 64, torch.float32), (7, 4, 6, 128, torch.bfloat16), (6, 2, 3, 32, torch.float16),
    (3, 40, 32, 128, torch.float16), (5, 700, 32, 64, torch.bfloat16), (2, 5600, 3, 128, torch.float16),
    (9, 64, 32, 128, torch.float16), (40, 64, 24, 128, torch.float16), (70, 150, 32, 128, torch.float32), (9, 70, 16, 256, torch.bfloat16),
])
def test_rows_of_no_weight_may_hold_anything(rows, batch, heads, d, dtype):
    gen = torch.Generator(device="cuda").manual_seed(rows * 31 + heads)
    at = torch.randint(0, rows, (batch, heads), generator=gen, device="cuda")       # per request and head: the one row that counts
    mid_lse = -300.0 + 20.0 * torch.rand(batch, rows, heads, generator=gen, device="cuda")
    mid_lse.scatter_(1, at[:, None], 5.0)                                            # e^-285 is 0 in fp32
    mid_o = torch.randn(batch, rows, heads, d, generator=gen, device="cuda")
    kept = mid_o.gather(1, at[:, None, :, None].expand(-1, -1, -1, d)).squeeze(1)
    for bad in (float("inf"), float("-inf"), float("nan")):
        x = torch.where(mid_lse[..., None] < 0, torch.full_like(mid_o, bad), mid_o)
        o, o_lse = _merge(rows, x.view(-1, heads, d), mid_lse.view(-1, heads).contiguous(), dtype, batch, heads, d)
        assert torch.equal(o, kept.to(dtype))
        assert (o_lse - 5.0).abs().max() <= 1e-6
    # a row that counts keeps what it holds: one infinite element, the others of its head as before
    x = mid_o.clone()
    x[:, rows // 2, 0, 1] = float("inf")
    lse = torch.zeros_like(mid_lse)
    o, _ = _merge(rows, x.view(-1, heads, d), lse.view(-1, heads).contiguous(), dtype, batch, heads, d)
    assert torch.isposinf(o[:, 0, 1]).all()
    o[:, 0, 1] = 0
    assert torch.isfinite(o).all()
