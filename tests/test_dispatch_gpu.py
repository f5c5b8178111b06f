"""Which few-row kernel a launch takes: the rule sees an upper bound of the few-row tasks' tokens, never their number of
many-row neighbours."""
import pytest
import torch

from ft_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("few,table,want", [(740, 740 * 80, "stream"), (740, 740 * 80 + 1, "narrow"), (739, 739 * 64, "narrow"),
                                            (740, 740 * 64 + 32000, "narrow")])
@pytest.mark.parametrize("many", [0, 500])
def test_workers_only_where_the_row_id_table_proves_the_tasks_short(few, table, want, many):
    """740 nodes x 8 KV heads are 20 tasks for each of 296 slots; the many-row phase, launched on its own, changes nothing."""
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148
    nodes, d = few + many + 1, 128              # a gap between the phases keeps them in separate launches
    q = torch.zeros(2, 32, d, dtype=torch.float16, device="cuda")
    kv = torch.zeros(64, 8, d, dtype=torch.float16, device="cuda")
    ints = lambda n: torch.zeros(n, dtype=torch.int32, device="cuda")
    name = engine.stage1_path_name(q, kv, kv, torch.empty_like(q), ints(table), *[ints(nodes)] * 2, ints(nodes + 1), *[ints(nodes)] * 2,
                                   ints(4), ints(2), ints(2), torch.zeros(nodes, 32, d, device="cuda"),
                                   torch.zeros(nodes, 32, device="cuda"), [many, few], [0, many + 1], [32, 4], [64, 64], 0.1)
    kernels = ["stage1_tc_kernel"] * (many > 0) + ["stage1_%s_kernel" % want]
    assert name == "+".join(kernels)
