"""Softmax scales of zero and below: every kernel family against the CPU oracle, on chunks whose last tile is ragged and on
grouped plans, whose rows mask most of their chunk."""
import pytest
import torch

import gpu_utils
from test_decode_gpu import ATOL16, adhoc
from oracle import ref_attention

from ft_b200 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.0, -0.1])
@pytest.mark.parametrize("grouped", [False, True], ids=["ragged", "row_ranges"])
@pytest.mark.parametrize("d", [64, 128, 256])
def test_scales_of_zero_and_below(d, grouped, scale):
    sizes, lens = ([1, 40], [70, 20]) if grouped else ([1, 9], [150, 133])
    c = adhoc(sizes, lens, 16, 4, d, torch.float16, seed=7, q_scale=0.5)
    truth, truth_lse = ref_attention.per_leaf_attention(c["nodes"], c["ptrs"], c["q"], c["k"], c["v"], scale)
    run = gpu_utils.EngineRun(c["nodes"], c["ptrs"], c["batch"], c["q"], c["k"], c["v"], c["hq"], c["hkv"], d, c["tsq"],
                              tell_dtype=True)
    assert (run.aux[3].numel() > 2 * run.mid_o.shape[0]) == grouped       # the plan carries token ranges
    run.scale = scale
    for path in ("auto", "tcgen05", "generic") + (("mma", "mma_wide", "stream") if d < 256 else ()) + (("persist",) if d == 128 else ()):
        out = run.decode(path=path)
        assert lib.read_device_status() == 0
        assert (out - truth).abs().max().item() <= ATOL16, path
        torch.testing.assert_close(run.o_lse.cpu(), truth_lse, rtol=1e-4, atol=2e-5)
