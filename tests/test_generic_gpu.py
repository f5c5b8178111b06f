"""The scalar kernel's grid of row blocks: tasks below, at and above the blocks that the request tile gives, and a request
tile that says nothing about them, against the CPU oracle's partials."""
import pytest
import torch

import gpu_utils
from test_decode_gpu import adhoc, atol_for
from oracle import ref_attention

from ft_b200 import engine, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [None, [0, 0], [1, 1], [300, 300]], ids=["planned", "unknown", "too_small", "large"])
@pytest.mark.parametrize("d,dtype,requests", [(256, torch.float32, 3), (256, torch.float16, 33), (32, torch.float32, 70)], ids=str)
def test_row_blocks_of_the_scalar_kernel(d, dtype, requests, tile):
    c = adhoc([1, requests], [130, 9], 8, 4, d, dtype, seed=15, q_scale=0.5)
    run = gpu_utils.EngineRun(c["nodes"], c["ptrs"], c["batch"], c["q"], c["k"], c["v"], 8, 4, d, c["tsq"])
    tabs = [t.cpu().numpy() for t in run.aux[:6]]
    mid_o, mid_lse = ref_attention.stage1_partials(c["q"], c["k"], c["v"], *tabs, run.scale)
    run.mid_o.fill_(float("nan"))
    engine.stage1(run.q, run.k, run.v, run.o, *run.aux, run.tiles[0] if tile is None else tile, run.tiles[1], run.scale,
                  path="generic")
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    torch.testing.assert_close(run.mid_lse.cpu(), mid_lse, rtol=1e-4, atol=2e-5)
    assert (run.mid_o.cpu() - mid_o).abs().max().item() <= atol_for(dtype)
