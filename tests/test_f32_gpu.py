"""The fp32 stage-1 kernels: what they report for plans that do not hold together."""
import pytest
import torch

import gpu_utils
from ft_b200 import engine, lib
from oracle import ref_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["auto", "generic"])
@pytest.mark.parametrize("d", [64, 128])
def test_each_kind_of_bad_plan_data_is_named_alone(d, path):
    """A partial row that the buffers do not have is no bad request id, and the other way round."""
    nodes = ref_inputs.layered_tree([1, 5], [90, 40])
    q, k, v, ptrs, batch = ref_inputs.draw_qkv(nodes, 8, 2, d, torch.float32, seed=3)
    run = gpu_utils.EngineRun(nodes, ptrs, batch, q, k, v, 8, 2, d, [16, 4], tell_dtype=True)
    rest = (*run.tiles, run.scale)

    def status(aux):
        engine.stage1(run.q, run.k, run.v, run.o, *aux, *rest, path=path)
        torch.cuda.synchronize()
        return lib.read_device_status()

    assert status(run.aux) == 0
    rows = run.mid_o.shape[0]
    assert status(run.aux[:9] + (run.mid_o[:rows - 3], run.mid_lse[:rows - 3]) + run.aux[11:]) == lib.FT_DEV_BAD_ROW_INDEX
    for bad in (batch, -1):
        saved = run.aux[3][0].item()
        run.aux[3][0] = bad
        assert status(run.aux) == lib.FT_DEV_BAD_Q_INDEX
        run.aux[3][0] = saved
    assert status(run.aux) == 0
