"""Infinities and NaN in the lower V-cycle's one launch (k_coarse): a cell outside
the grid counts as a pressure of 0, so they reach the cells that the operator
connects and no others, and every other cell keeps the oracle's bits."""
import numpy as np
import pytest

from smokesim_b200 import abi, scene
from test_gpu_parity import make_pair

pytestmark = pytest.mark.gpu

GRIDS = [
    # (dim, n, enclosed, smallest level side, level): one level on several CTAs,
    # one on one CTA, in 3D and 2D, and two levels
    (3, (97, 75, 61), 0, 8, 2),
    (3, (64, 64, 64), 1, 8, 3),
    (3, (64, 64, 64), 1, 8, 2),
    (2, (300, 173, 1), 0, 4, 5),
    (2, (256, 256, 1), 1, 64, 2),
    (2, (256, 256, 1), 1, 8, 4),
]


@pytest.mark.parametrize("dim,n,enc,mc,L", GRIDS)
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("quirks", [1, 0])
def test_nonfinite_stays_with_its_neighbours(dim, n, enc, mc, L, value, quirks):
    g, o = make_pair(dim, n, 1, enc, seed=61, min_coarse=mc, state=False)
    assert 1 <= L < g.levels
    o.restrict_solid_all()
    nx, ny, nz = g.level_sizes[L]
    r = np.random.default_rng(7)
    # black cells (read by the red half-sweep before they are written) at the ends of
    # a row, of a plane and of the march axis, where the next cell of the packed
    # order is no neighbour
    mid = lambda n, odd: n // 2 - ((n // 2 + odd + 1) & 1)  # noqa: E731  near the middle, odd + mid odd
    at = {(x, mid(ny, x + nz // 2), nz // 2) for x in (0, nx - 1)}
    at |= {(mid(nx, y + z), y, z) for y, z in ((ny - 1, nz // 2), (0, nz // 2), (ny // 2, nz - 1), (ny // 2, 0))}
    for x, y, z in sorted(at):
        assert (x + y + z) % 2 == 1
        p0 = r.standard_normal((nz, ny, nx)).astype(np.float32)
        p0[z, y, x] = value
        r0 = r.standard_normal((nz, ny, nx)).astype(np.float32)
        for s in (g, o):
            s.set_level(L, abi.LEVEL_PRESSURE, p0)
            s.set_level(L, abi.LEVEL_RESIDUAL, r0)
        p = scene.workload_params(ref_quirks=quirks, n_pre=1, n_post=1, n_coarse=1)
        g.v_cycle(p, L)
        o.v_cycle(L, p)
        a, b = g.get_level(L, abi.LEVEL_PRESSURE), o.get_level(L, abi.LEVEL_PRESSURE).reshape(nz, ny, nx)
        if L == g.levels - 1:
            assert np.isfinite(b).any() and not np.isfinite(b).all()
        assert np.array_equal(np.isnan(a), np.isnan(b)), (x, y, z, np.isnan(a).sum(), np.isnan(b).sum())
        assert np.array_equal(a, b, equal_nan=True), (x, y, z)
