"""Stage 2 alone against an fp64 merge where the forms that take pieces of a row end: rows that are no whole number of
pieces, strided buffers, outputs without vector stores; and an infinite LSE."""
import pytest
import torch

from ft_b200 import engine, lib
from test_merge_gpu import _merge

pytestmark = pytest.mark.gpu


def _strided(x, inner):
    """``x`` in a buffer with ``inner`` spare elements per innermost row and a spare row per request."""
    buf = torch.full((x.shape[0], x.shape[1] + 1, x.shape[2] + inner), float("nan"), dtype=x.dtype, device=x.device)
    view = buf[:, :x.shape[1], :x.shape[2]]
    view.copy_(x)
    return view


# (4 floats are the buffers' alignment; an output row of d + 1 or d + 3 elements allows no vector store)
@pytest.mark.parametrize("batch,heads,d,most,dtype,spare_o,strided_mid", [
    (9, 3, 32, 24, torch.float16, 0, False),        # four warps on a piece that three heads fill to three quarters
    (40, 5, 16, 16, torch.bfloat16, 0, True),       # ... on the quarter that the last head leaves, rows in strides
    (9, 3, 256, 26, torch.float16, 1, True),        # four warps, a head in two pieces
    (40, 5, 256, 3, torch.float32, 0, False),       # a warp per piece at head_dim 256
    (50, 9, 256, 2, torch.bfloat16, 3, True),
    (50, 7, 64, 5, torch.float16, 1, True),         # a warp per piece, the last one half full
    (6000, 3, 128, 3, torch.float16, 0, False),     # two float4s per lane, the last piece without its second one
    (6700, 5, 64, 3, torch.bfloat16, 1, True),      # ... the last piece a quarter full
    (60, 6, 128, 14, torch.float16, 3, True),       # a warp per head, scalar stores and strided rows
    (1030, 17, 256, 2, torch.float32, 3, False),    # ... at head_dim 256
    (70, 6, 256, 12, torch.bfloat16, 1, True),
])
def test_merge_at_ragged_pieces_and_strides(batch, heads, d, most, dtype, spare_o, strided_mid):
    gen = torch.Generator(device="cuda").manual_seed(batch * 17 + d)
    lens = torch.randint(1, most + 1, (batch,), generator=gen, device="cuda")
    lens[0] = most
    offs = torch.cumsum(lens, 0) - lens
    total = int(lens.sum())
    entries = torch.randperm(total, generator=gen, device="cuda")
    mid_o = torch.randn(total, heads, d, generator=gen, device="cuda")
    mid_lse = torch.randn(total, heads, generator=gen, device="cuda") * 8
    dev = [t.to(torch.int32) for t in (entries, offs, lens)]
    want, want_lse = _merge(mid_o.cpu(), mid_lse.cpu(), *[t.cpu() for t in dev])
    if strided_mid:
        mid_o, mid_lse = _strided(mid_o, 4), _strided(mid_lse[..., None], 0)[..., 0]
    q = torch.zeros(batch, heads, d, dtype=dtype, device="cuda")
    o = _strided(torch.full_like(q, 7.0), spare_o)
    outside = o._base if o._base is not None else o
    o_lse = torch.zeros(batch, heads, device="cuda")
    k = torch.zeros(1, heads, d, dtype=dtype, device="cuda")
    z = torch.zeros(1, dtype=torch.int32, device="cuda")
    rows = torch.zeros(total, dtype=torch.int32, device="cuda")
    engine.stage2(q, k, k, o, z, z, z, rows, z, z, *dev, mid_o, mid_lse, [1, 0], [0, 1], [16, 4], [64, 64], 0.1, o_lse=o_lse)
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    # the sum of at most 26 products in fp32, its weights to 2^-21 each, then one rounding to the output's type
    eps = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    assert ((o.cpu().double() - want).abs() <= 1e-5 + eps * want.abs()).all()
    assert ((o_lse.cpu().double() - want_lse).abs() <= 1e-5 * want_lse.abs().clamp(min=1.0)).all()
    assert int(outside.isnan().sum()) == outside.numel() - o.numel()      # nothing beside the output is written


# forms as above: four warps per piece, a warp per piece, two pieces per warp, a warp per head
@pytest.mark.parametrize("rows,batch,heads,d", [(14, 3, 8, 128), (3, 40, 32, 128), (2, 5600, 3, 128), (9, 64, 32, 128), (9, 70, 16, 256)])
def test_an_infinite_lse_stays_with_its_head(rows, batch, heads, d):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    mid_o = torch.randn(batch * rows, heads, d, generator=gen, device="cuda")
    mid_lse = torch.randn(batch * rows, heads, generator=gen, device="cuda")
    mid_lse[rows // 2::rows, 1] = float("inf")       # one row of every request, one head: a softmax of NaN
    offs = torch.arange(batch, dtype=torch.int32, device="cuda") * rows
    lens = torch.full((batch,), rows, dtype=torch.int32, device="cuda")
    entries = torch.arange(batch * rows, dtype=torch.int32, device="cuda")
    q = torch.zeros(batch, heads, d, device="cuda")
    o = torch.full_like(q, 7.0)
    k = torch.zeros(1, heads, d, device="cuda")
    z = torch.zeros(1, dtype=torch.int32, device="cuda")
    engine.stage2(q, k, k, o, z, z, z, torch.zeros(batch * rows, dtype=torch.int32, device="cuda"), z, z, entries, offs, lens,
                  mid_o, mid_lse, [1, 0], [0, 1], [16, 4], [64, 64], 0.1)
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    assert o[:, 1].isnan().all()
    others = [h for h in range(heads) if h != 1]
    x, w = mid_o.view(batch, rows, heads, d)[:, :, others].double(), torch.softmax(mid_lse.view(batch, rows, heads)[:, :, others].double(), 1)
    assert ((o[:, others].double() - (w[..., None] * x).sum(1)).abs() <= 1e-5).all()
