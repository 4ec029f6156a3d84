"""The lower V-cycle in one cluster launch (k_coarse) against the FP32 oracle,
bit for bit, where its shapes can go wrong: slabs of one, two and several planes,
a partial last slab, one and two cells of each colour per thread, levels that
one CTA takes alone, 2D, and one CTA for everything (SMOKESIM_CLUSTER=0).
Reference: v_cycle (common/physics/grid.c:177-209)."""
import numpy as np
import pytest

from smokesim_b200 import abi, scene
from test_gpu_parity import make_pair

pytestmark = pytest.mark.gpu

COARSE_GRIDS = [
    # (levels below the first): 32^3 in slabs of two planes and two cells a
    # thread, 16^3 in slabs of one plane, 8^3 on one CTA
    ("3d_cube", 3, (64, 64, 64), 1, 8),
    # 48x37x30 as launches, the coarsest 24x18x15 in fifteen slabs of one plane
    ("3d_odd_open", 3, (97, 75, 61), 0, 8),
    # 33x17x65 -> 16x8x32: slabs of five and of two planes, the last ones partial
    ("3d_tall", 3, (66, 34, 130), 1, 8),
    # 150x86 in slabs of six rows (the last partial), 75x43 in slabs of three, 37x21 alone
    ("2d_odd_open", 2, (300, 173, 1), 0, 4),
    ("2d_square", 2, (256, 256, 1), 1, 8),
]


@pytest.mark.parametrize("name,dim,n,enc,mc", COARSE_GRIDS)
@pytest.mark.parametrize("quirks", [1, 0])
@pytest.mark.parametrize("cluster", ["1", "0"])
def test_coarse_levels_bitwise(monkeypatch, name, dim, n, enc, mc, quirks, cluster):
    monkeypatch.setenv("SMOKESIM_CLUSTER", cluster)
    g, o = make_pair(dim, n, 1, enc, seed=41, min_coarse=mc)
    p = scene.workload_params(ref_quirks=quirks, n_pre=2, n_post=1, n_coarse=9)
    for _ in range(2):
        g.v_cycle(p, 0)
        o.v_cycle(0, p)
    for L in range(g.levels):
        assert np.array_equal(g.get_level(L, abi.LEVEL_PRESSURE), o.get_level(L, abi.LEVEL_PRESSURE)), f"p L{L}"
        assert np.array_equal(g.get_level(L, abi.LEVEL_RESIDUAL), o.get_level(L, abi.LEVEL_RESIDUAL)) or L == 0, f"r L{L}"


@pytest.mark.parametrize("scale", [1e-28, 1e28])
def test_coarse_levels_out_of_reciprocal_range_bitwise(scale):
    """Dividends outside the range of the reciprocal form take IEEE division:
    on the shared levels cell by cell, on one CTA's by running again."""
    g, o = make_pair(3, (64, 64, 64), 1, 1, seed=43, min_coarse=8)
    for f in (abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ, abi.FIELD_PRESSURE):
        a = g.get_field(f) * np.float32(scale)
        g.set_field(f, a)
        o.set_field(f, a)
    p = scene.workload_params(ref_quirks=0, n_pre=1, n_post=1, n_coarse=6)
    g.v_cycle(p, 0)
    o.v_cycle(0, p)
    for L in range(g.levels):
        assert np.array_equal(g.get_level(L, abi.LEVEL_PRESSURE), o.get_level(L, abi.LEVEL_PRESSURE)), f"p L{L}"


@pytest.mark.parametrize("prec", [abi.PREC_MIXED, abi.PREC_MIXED_BF16])
@pytest.mark.parametrize("cluster", ["1", "0"])
def test_coarse_levels_mixed_bitwise(monkeypatch, prec, cluster):
    monkeypatch.setenv("SMOKESIM_CLUSTER", cluster)
    g, o = make_pair(3, (64, 48, 80), 1, 1, seed=47, min_coarse=8)
    p = scene.workload_params(ref_quirks=0, precision=prec, n_vcycles=2, n_coarse=11)
    for _ in range(2):
        g.step(p)
        o.step(p)
    for f in (abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ, abi.FIELD_PRESSURE):
        assert np.array_equal(g.get_field(f), o.get_field(f)), f"field {f}"
