"""Solve graphs on the legacy default stream (recorded on the simulation's own
stream, launched on the caller's) and their recording on the second solve of a
kind: the oracle's fields on every step, while the schedule changes between
steps and back."""
import pytest

from smokesim_b200 import abi, scene
from test_gpu_device_loop import _step_both
from test_gpu_parity import assert_same, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("prec,tol", [(abi.PREC_FP32, 0.0), (abi.PREC_FP32, 1e-3), (abi.PREC_MIXED, 0.0), (abi.PREC_MIXED, 1e-6)])
def test_graph_recording_bitwise(own, prec, tol):
    import torch
    st = torch.cuda.Stream()
    g, o = make_pair(3, (32, 24, 20), 1, 1, seed=51, min_coarse=4, stream=st.cuda_stream if own else None)
    for k, n_pre in enumerate([2, 2, 2, 1, 2, 1, 1, 2, 2]):
        p = scene.workload_params(ref_quirks=0, precision=prec, tol=tol, n_vcycles=12 if tol else 2, n_coarse=12, n_pre=n_pre)
        code = _step_both(g, o, p)
        assert_same(g, o, 3, f"step {k}")
        assert g.stats().vcycles == o.stats().vcycles
        assert code == (0 if o.stats().converged or tol == 0.0 else abi.SS_E_NOT_CONVERGED)
