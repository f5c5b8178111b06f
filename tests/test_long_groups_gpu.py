"""Groups of short nodes of more than 16 KV tiles, which the splitter takes where their schedule ends sooner, at every
head_dim whose kernel honours row ranges."""
import pytest
import torch

import gpu_utils
from ft_b200 import engine, lib
from oracle import ref_attention
from test_decode_gpu import ATOL16, adhoc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,lens,hq,hkv,d", [
    ([1, 235], [2430, 110], 28, 4, 64), ([1, 1, 186, 311], [32, 34, 91, 14], 64, 8, 64), ([1, 166], [1899, 44], 32, 8, 256),
    ([1, 156], [1976, 41], 24, 8, 256),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
def test_groups_of_more_than_sixteen_tiles(sizes, lens, hq, hkv, d, dtype):
    c = adhoc(sizes, lens, hq, hkv, d, dtype, seed=6, q_scale=0.5)
    run = gpu_utils.EngineRun(c["nodes"], c["ptrs"], c["batch"], c["q"], c["k"], c["v"], hq, hkv, d, c["tsq"], tell_dtype=True)
    rows, ranges = engine.split_q_entries(run.aux[3])
    kv_lens, q_offs = run.aux[2].cpu(), run.aux[4].cpu()
    longest = int(kv_lens.argmax())
    first = ranges[int(q_offs[longest])].tolist()
    assert int(kv_lens[longest]) > 16 * 64 and first[1] - first[0] < int(kv_lens[longest])      # the longest task is a group
    truth, truth_lse = ref_attention.per_leaf_attention(c["nodes"], c["ptrs"], c["q"], c["k"], c["v"], d ** -0.5)
    tol = ATOL16 + (float(truth.abs().max()) * 2 ** -8 if dtype == torch.bfloat16 else 0.0)
    out = run.decode()
    assert lib.read_device_status() == 0
    assert (out - truth).abs().max().item() <= tol
    torch.testing.assert_close(run.o_lse.cpu(), truth_lse, rtol=1e-4, atol=2e-5)
