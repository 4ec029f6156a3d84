"""ss_get_stats after FP32 steps that nothing has waited for: it waits for the
default stream, so that its status covers those steps."""
import pytest

from smokesim_b200 import abi, scene
from test_gpu_parity import make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("checked", [False, True])
def test_stats_wait_for_an_unchecked_fp32_solve(checked):
    import torch
    g, _ = make_pair(3, (64, 64, 64), 1, 1, seed=71, min_coarse=8)
    p = scene.workload_params(ref_quirks=0, collect_stats=0)
    for _ in range(3):
        g.step(p)
    torch.cuda.synchronize()
    g.stats()
    done = torch.cuda.Event()

    def busy():
        torch.cuda._sleep(1_000_000_000)     # some 0.5 s on the default stream
        done.record()
        assert not done.query()

    g.step(p)
    if checked:
        g.get_field(abi.FIELD_PRESSURE)
    busy()
    g.stats()
    assert done.query() != checked
    torch.cuda.synchronize()
    busy()
    g.stats()          # nothing unchecked any more: host values, no wait
    assert not done.query()
    torch.cuda.synchronize()
