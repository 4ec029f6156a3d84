"""Advection of velocities and smoke and the projection update, where one thread per
cell takes the faces around it: grids thinner than a block, one cell past a block's edge, wind at the
low face of every axis, traces that end exactly on the last cell or far outside.
Bit for bit against the FP32 oracle."""
import numpy as np
import pytest

from conftest import max_abs
from smokesim_b200 import abi, scene
from test_gpu_parity import assert_same, make_pair

pytestmark = pytest.mark.gpu

THIN = [
    ("2d_thin", 2, (65, 9, 1), 3, 0),
    ("2d_low", 2, (9, 33, 1), 1, 1),
    ("3d_thin", 3, (33, 9, 9), 1, 0),
    ("3d_flat", 3, (31, 12, 7), 3, 0),
    ("3d_edge", 3, (64, 16, 8), 1, 1),
]


@pytest.mark.parametrize("name,dim,n,nch,enc", THIN)
@pytest.mark.parametrize("mask", [abi.STAGE_ADVECT_VELOCITIES, abi.STAGE_ADVECT_VELOCITIES | abi.STAGE_APPLY_BUOYANCY,
                                  abi.STAGE_ADVECT_SMOKE, abi.STAGE_UPDATE_VELOCITIES])
@pytest.mark.parametrize("vel", ["random", "integer", "far"])
def test_transport_edges_bitwise(name, dim, n, nch, enc, mask, vel):
    g, o = make_pair(dim, n, nch, enc, seed=61, min_coarse=3, t_amb=0.5)
    if vel != "random":
        # whole displacements of -2..2 cells at dt = 0.125 end on cells and faces, the last ones included
        rng = np.random.default_rng(7)
        for f in (abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ)[:dim]:
            a = (8.0 * rng.integers(-2, 3, g.get_field(f).shape)).astype(np.float32)
            if vel == "far":
                a[rng.random(a.shape) < 0.5] *= np.float32(1e30)
            g.set_field(f, a)
            o.set_field(f, a)
    p = scene.workload_params(stage_mask=mask, dt=0.125, wind=(0.3, -0.2, 0.4 if dim == 3 else 0.0), t_ambient=0.5)
    for k in range(2):
        g.step(p)
        o.step(p)
        assert_same(g, o, dim, f"{name} {vel} step {k}")
        assert max_abs(g.get_field(abi.FIELD_TEMPERATURE), o.get_field(abi.FIELD_TEMPERATURE)) == 0.0
