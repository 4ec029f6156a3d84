"""Level-0 half-sweeps with four cells a thread, warps filled across rows, and
quotients by table: rows of one, three and five quads, a last block with threads
to spare, dividends so small that the table's steps are not exact, and zeros.
Bit for bit against the FP32 oracle."""
import numpy as np
import pytest

from smokesim_b200 import abi, scene
from test_gpu_parity import make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,enc", [(2, (8, 19, 1), 1), (2, (40, 103, 1), 0), (3, (8, 9, 11), 0), (3, (24, 13, 9), 1),
                                       (3, (40, 64, 33), 1)])
@pytest.mark.parametrize("scale", [1.0, 1e-37, 3e-42, 0.0])
def test_level0_sweeps_bitwise(dim, n, enc, scale):
    g, o = make_pair(dim, n, 1, enc, seed=71, min_coarse=4)
    for f in (abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ, abi.FIELD_PRESSURE):
        if f == abi.FIELD_VZ and dim == 2:
            continue
        a = (g.get_field(f).astype(np.float64) * scale).astype(np.float32)
        g.set_field(f, a)
        o.set_field(f, a)
    p = scene.workload_params(ref_quirks=0, n_pre=3, n_post=2, n_coarse=5)
    for _ in range(2):
        g.v_cycle(p, 0)
        o.v_cycle(0, p)
    assert np.array_equal(g.get_level(0, abi.LEVEL_PRESSURE), o.get_level(0, abi.LEVEL_PRESSURE))
