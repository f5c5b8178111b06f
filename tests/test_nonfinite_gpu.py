"""Infinities and NaN in the K/V rows of single requests whose leaves are grouped with others into one task: the requests
they are grouped with get their own attention all the same, through every kernel family that takes the plan."""
import pytest
import torch

import gpu_utils
from test_decode_gpu import adhoc, atol_for
from oracle import ref_attention

from ft_b200 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,dtype", [(64, torch.float16), (64, torch.bfloat16), (128, torch.float16), (128, torch.float32),
                                     (256, torch.bfloat16)], ids=str)
@pytest.mark.parametrize("heads", [(16, 4), (8, 8)], ids=["g4", "g1"])
def test_groups_keep_infinities_apart(d, dtype, heads):
    c = adhoc([1, 40], [70, 20], *heads, d, dtype, seed=12, q_scale=0.5)
    scale = d ** -0.5
    truth, _ = ref_attention.per_leaf_attention(c["nodes"], c["ptrs"], c["q"], c["k"], c["v"], scale)
    leaf = {nd.requests[0]: nd.id for nd in c["nodes"] if nd.num_children == 0}
    for req, what, tensor in ((3, float("inf"), "v"), (17, float("nan"), "v"), (18, float("-inf"), "v"), (30, float("nan"), "k"),
                              (31, float("inf"), "k")):
        c[tensor][c["ptrs"][leaf[req]] + 5] = what
    bad, _ = ref_attention.per_leaf_attention(c["nodes"], c["ptrs"], c["q"], c["k"], c["v"], scale)
    tol = atol_for(dtype) + (float(truth.abs().max()) * 2 ** -8 if dtype == torch.bfloat16 else 0.0)
    clean = [r for r in range(c["batch"]) if r not in (3, 17, 18, 30, 31)]
    paths = {torch.float32: ()}.get(dtype, ("tcgen05",) + (("mma", "mma_wide", "stream") if d < 256 else ()) +
                                    (("persist",) if d == 128 else ()))
    for path in ("auto", "generic") + paths:
        run, out = gpu_utils.run_case(c, planner="b200", path=path, tell_dtype=dtype != torch.float32)
        assert run.aux[3].numel() > 2 * run.mid_o.shape[0]       # the plan carries token ranges
        assert lib.read_device_status() == 0
        assert (out[clean] - truth[clean]).abs().max().item() <= tol, path
        for req in (3, 17, 18):      # a request's own row reaches its result
            assert torch.equal(out[req].isnan(), bad[req].isnan()) and torch.equal(out[req].isinf(), bad[req].isinf()), path
