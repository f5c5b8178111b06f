"""The fp32 stage-1 kernels: chunk lengths around their tile, what they report for plans that do not hold together."""
import numpy as np
import pytest
import torch

import gpu_utils
from ft_b200 import engine, lib
from oracle import ref_attention, ref_inputs

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


@pytest.mark.parametrize("d,hkv,group", [(64, 2, 3), (128, 2, 4), (128, 3, 1)])
def test_every_row_of_a_tile_is_met(d, hkv, group):
    """Chunks that end anywhere in a 32-token tile, their rows scattered over the buffers."""
    lens = np.array([0, 1, 2, 3, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 48, 63, 64, 65, 97])
    reqs = 1 + np.arange(lens.size) % 4
    rng = np.random.RandomState(d + group)
    rows = int(lens.sum())
    ids = rng.permutation(rows)
    off = lambda x: np.concatenate([[0], np.cumsum(x)[:-1]])
    q_entries = np.concatenate([rng.permutation(5)[:n] for n in reqs])
    tabs = [ids, off(lens), lens, q_entries, off(reqs), reqs]
    gen = torch.Generator().manual_seed(d)
    k, v = (torch.randn(rows, hkv, d, generator=gen) for _ in range(2))
    q = torch.randn(5, hkv * group, d, generator=gen)
    dev = [torch.from_numpy(x.astype(np.int32)).cuda() for x in tabs]
    parts = q_entries.size
    mid_o = torch.full((parts, hkv * group, d), float("nan"), device="cuda")
    mid_lse = torch.empty(parts, hkv * group, device="cuda")
    none = torch.zeros(5, dtype=torch.int32, device="cuda")
    qd = q.cuda()
    args = (qd, k.cuda(), v.cuda(), torch.empty_like(qd), *dev, none, none, none, mid_o, mid_lse, [0, lens.size], [0, 0],
            [16, 4], [64, 64], d ** -0.5)
    assert engine.stage1_path_name(*args) == "stage1_f32_kernel"
    engine.stage1(*args, row_ranges=None)
    torch.cuda.synchronize()
    assert lib.read_device_status() == 0
    want_o, want_lse = ref_attention.stage1_partials(q, k, v, *tabs, d ** -0.5)
    want_o[0], want_lse[0] = 0.0, -float("inf")      # the empty chunk's row, which the reference leaves out
    # sums of at most 97 products of order one in fp32, the reference's in fp32 as well
    torch.testing.assert_close(mid_o.cpu(), want_o.float(), rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(mid_lse.cpu(), want_lse.float(), rtol=1e-5, atol=1e-5)
