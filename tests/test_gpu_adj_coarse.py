"""The transpose of the lower V-cycle in one cluster launch against its per-level
launches (SMOKESIM_CLUSTER=0), on levels in one and two planes a CTA, odd sizes,
partial slabs, 2D, a level that one CTA takes alone, and with the coarsest sweeps
transposed one by one.

Both take the same sums in FP32, in another order in the prolongation's and the
product's adjoint.  A gradient passes through at most a few thousand additions, a
relative 6e-8 each: 1e-4 of its norm bounds the difference."""
import numpy as np
import pytest

from conftest import rel_l2
from smokesim_b200 import abi, scene

pytestmark = pytest.mark.gpu

GRIDS = [
    ("3d_cube", 3, (64, 64, 64), 1, 8),
    ("3d_odd_open", 3, (97, 75, 61), 0, 8),
    ("3d_tall", 3, (66, 34, 130), 1, 8),
    ("3d_small", 3, (24, 20, 18), 0, 4),
    ("2d_odd_open", 2, (300, 173, 1), 0, 4),
    ("2d_square", 2, (256, 256, 1), 1, 8),
]


@pytest.mark.parametrize("name,dim,n,enc,mc", GRIDS)
@pytest.mark.parametrize("sweeps", ["0", "1"])
def test_adjoint_coarse_levels(monkeypatch, name, dim, n, enc, mc, sweeps):
    import torch
    from smokesim_b200 import Sim
    from smokesim_b200.adjoint import Rollout
    from test_gpu_parity import _scene_for
    monkeypatch.setenv("SMOKESIM_ADJ_COARSE_SWEEPS", sweeps)
    p = scene.workload_params(ref_quirks=0, n_pre=2, n_post=1, n_coarse=6, n_vcycles=2,
                              stage_mask=abi.STAGE_RESOLVE_PRESSURE | abi.STAGE_UPDATE_VELOCITIES)
    vel = [abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ][:dim]

    def run(cluster):
        monkeypatch.setenv("SMOKESIM_CLUSTER", cluster)
        g = Sim(abi.make_desc(dim, n, cell_size=1.0, density_channels=1, enclosed=enc, min_coarse=mc))
        rng = scene.Rng(81)
        g.set_scene(*_scene_for(dim, n, rng))
        for k, a in scene.random_state(rng, dim, n, 1).items():
            g.set_field(k, a[: int(np.prod(g.shape(k)))])
        ro = Rollout(g, 1, 1, deterministic=True)
        ro.forward(p, None)
        r = np.random.default_rng(5)
        gv = [torch.from_numpy(r.standard_normal(int(np.prod(g.shape(f)))).astype(np.float32)).cuda() for f in vel]
        torch.cuda.synchronize()
        ro.backward(p, grad_velocity=[t.data_ptr() for t in gv])
        out = [ro.grad(f).copy() for f in vel]
        ro.close()
        g.close()
        return out

    for f, a, b in zip(vel, run("1"), run("0")):
        assert np.isfinite(b).all() and np.abs(b).max() > 0
        assert rel_l2(a, b) <= 1e-4, (f, rel_l2(a, b))
