"""The lower V-cycle's one launch (k_coarse) and its transpose (k_adj_coarse) on the
ways a level can be cut: slabs of several planes with a partial last one that hand
over to a further level, one and two cells of each colour a thread, slabs after
slabs, levels that one CTA takes alone after slabs and after one another.

Each grid states the levels' slabs: (planes a CTA, one CTA alone).  The test works
them out again from the rule (the smallest cluster on which no thread has more than
one cell of each colour of the first level, else the largest that holds it with
two), and the launches of a solve show the level at which the launch begins."""
import numpy as np
import pytest

from smokesim_b200 import abi, scene
from test_gpu_parity import make_pair

pytestmark = pytest.mark.gpu

THREADS = 512
GRIDS = [
    # name, dim, n, enclosed, smallest side, first level, CTAs, slabs
    ("two_cells_then_slabs", 3, (38, 26, 124), 1, 4, 1, 16, [(4, False), (2, False)]),
    ("two_cells_then_solo", 3, (42, 50, 34), 0, 6, 1, 16, [(2, False), (8, True)]),
    ("odd_two_cells", 3, (75, 18, 68), 1, 4, 1, 16, [(3, False), (2, False)]),
    ("four_planes_then_slabs", 3, (22, 24, 118), 0, 5, 1, 16, [(4, False), (2, False)]),
    ("second_level", 3, (60, 64, 139), 1, 5, 2, 16, [(3, False), (2, False)]),
    ("solo_after_solo", 3, (44, 38, 34), 1, 4, 1, 16, [(2, False), (8, True), (4, True)]),
    ("two_ctas", 3, (18, 26, 19), 0, 4, 1, 2, [(5, False), (4, True)]),
    ("2d_one_cell", 2, (300, 173, 1), 0, 4, 1, 16, [(6, False), (3, False), (21, True), (10, True), (5, True)]),
    ("2d_two_cells", 2, (131, 610, 1), 1, 4, 1, 16, [(20, False), (10, False), (5, False), (38, True), (19, True)]),
]
IDS = [g[0] for g in GRIDS]


def pairs(n, dim):
    """cells of a colour in one plane, planes"""
    return ((n[0] + 1) // 2 * n[1], n[2]) if dim == 3 else ((n[0] + 1) // 2, n[1])


def slab(n, dim, ctas):
    per, planes = pairs(n, dim)
    solo = ctas == 1 or per * planes <= THREADS
    return (planes if solo else -(-planes // ctas)), solo


def check_plan(g, dim, first, ctas, slabs):
    levels = g.level_sizes[first:]
    assert [slab(n, dim, ctas) for n in levels] == slabs
    per = slab(levels[0], dim, ctas)[0] * pairs(levels[0], dim)[0]
    assert THREADS < per <= 2 * THREADS if ctas == 16 and per > THREADS else per <= THREADS
    if ctas > 1:
        assert slab(levels[0], dim, ctas // 2)[0] * pairs(levels[0], dim)[0] > THREADS
    # the first level's last slab is partial
    assert slabs[0][1] or pairs(levels[0], dim)[1] % slabs[0][0] != 0
    # the level above would not fit
    if first > 1:
        n = g.level_sizes[first - 1]
        assert slab(n, dim, 16)[0] * pairs(n, dim)[0] > 2 * THREADS


def check_first_level(g, first, **kw):
    """A sweep more before restriction is two launches more on every level above the
    first; sweeps on the coarsest level are none."""
    count = {}
    for pre, coarse in ((2, 9), (2, 9), (3, 9), (2, 11)):
        g.step(scene.workload_params(ref_quirks=0, n_vcycles=1, n_pre=pre, n_post=1, n_coarse=coarse,
                                     stage_mask=abi.STAGE_RESOLVE_PRESSURE, **kw))
        count[pre, coarse] = g.stats().kernel_launches
    assert count[3, 9] - count[2, 9] == 2 * first
    # (the mixed solve's response matrix is made again: one check, one response)
    assert count[2, 11] - count[2, 9] in (0, 2)


@pytest.mark.parametrize("name,dim,n,enc,mc,first,ctas,slabs", GRIDS, ids=IDS)
@pytest.mark.parametrize("quirks", [1, 0])
def test_slabs_bitwise(name, dim, n, enc, mc, first, ctas, slabs, quirks):
    g, o = make_pair(dim, n, 1, enc, seed=91, min_coarse=mc)
    check_plan(g, dim, first, ctas, slabs)
    p = scene.workload_params(ref_quirks=quirks, n_pre=2, n_post=1, n_coarse=9)
    for _ in range(2):
        g.v_cycle(p, 0)
        o.v_cycle(0, p)
    for L in range(g.levels):
        assert np.array_equal(g.get_level(L, abi.LEVEL_PRESSURE), o.get_level(L, abi.LEVEL_PRESSURE)), f"p L{L}"
        assert np.array_equal(g.get_level(L, abi.LEVEL_RESIDUAL), o.get_level(L, abi.LEVEL_RESIDUAL)) or L == 0, f"r L{L}"
    check_first_level(g, first)


@pytest.mark.parametrize("name,dim,n,enc,mc,first,ctas,slabs", [g for g in GRIDS if g[2][0] % 2 == 0],
                         ids=[g[0] for g in GRIDS if g[2][0] % 2 == 0])
@pytest.mark.parametrize("prec", [abi.PREC_MIXED, abi.PREC_MIXED_BF16])
@pytest.mark.parametrize("sweeps", ["0", "1"])
def test_slabs_mixed_bitwise(monkeypatch, name, dim, n, enc, mc, first, ctas, slabs, prec, sweeps):
    monkeypatch.setenv("SMOKESIM_COARSE_SWEEPS", sweeps)
    g, o = make_pair(dim, n, 1, enc, seed=93, min_coarse=mc)
    o.set_coarse_matrix(sweeps == "0")
    p = scene.workload_params(ref_quirks=0, precision=prec, n_vcycles=2, n_coarse=11)
    for _ in range(2):
        g.step(p)
        o.step(p)
    for f in [abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ][:dim] + [abi.FIELD_PRESSURE]:
        assert np.array_equal(g.get_field(f), o.get_field(f)), f"field {f}"
    check_first_level(g, first, precision=prec)


def _smooth_faces(dim, n, comp, seed):
    """a few of the longest waves on the faces of one axis"""
    r = np.random.default_rng(seed)
    shape = [n[d] + (d == comp) for d in range(3)]
    ax = [np.linspace(0.0, np.pi, s) for s in shape]
    out = np.zeros(shape[::-1])
    for _ in range(6):
        k = [int(r.integers(1, 4)) if d < dim else 0 for d in range(3)]
        ph = r.uniform(0, np.pi, 3)
        out += r.standard_normal() * (np.cos(k[2] * ax[2] + ph[2])[:, None, None] * np.cos(k[1] * ax[1] + ph[1])[None, :, None]
                                      * np.cos(k[0] * ax[0] + ph[0])[None, None, :])
    return out.astype(np.float32).ravel()


@pytest.mark.parametrize("name,dim,n,enc,mc,first,ctas,slabs", GRIDS + [
    ("cube", 3, (64, 64, 64), 1, 8, 1, 16, [(2, False), (1, False), (8, True)])], ids=IDS + ["cube"])
@pytest.mark.parametrize("sweeps", ["0", "1"])
def test_transpose_identity(monkeypatch, name, dim, n, enc, mc, first, ctas, slabs, sweeps):
    """<A x, y> = <x, A^T y> for the projection A of one V-cycle from a zero pressure,
    a linear map of the velocities: A from the FP64 oracle, A^T from the reverse pass.

    x and y are long waves, which the levels of the cluster launch carry.  A^T y is a
    sum of FP32 terms, each through at most a few thousand additions of relative 6e-8:
    1e-4 of |x| |A^T y| bounds the difference.  One sweep of the coarsest level fewer,
    in the oracle, has to show."""
    import torch
    from oracle.oracle import OracleSim
    from smokesim_b200 import Sim
    from smokesim_b200.adjoint import Rollout
    from test_gpu_parity import _scene_for
    monkeypatch.setenv("SMOKESIM_ADJ_COARSE_SWEEPS", sweeps)
    desc = abi.make_desc(dim, n, cell_size=1.0, density_channels=1, enclosed=enc, min_coarse=mc)
    em, ob, bx = _scene_for(dim, n, scene.Rng(95))
    vel = [abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ][:dim]
    x = [_smooth_faces(dim, n, d, 11 + d) for d in range(dim)]
    y = [_smooth_faces(dim, n, d, 21 + d) for d in range(dim)]

    def params(n_coarse):
        return scene.workload_params(ref_quirks=0, n_pre=1, n_post=1, n_coarse=n_coarse, n_vcycles=1,
                                     stage_mask=abi.STAGE_RESOLVE_PRESSURE | abi.STAGE_UPDATE_VELOCITIES)

    def oracle(n_coarse):
        o = OracleSim(desc, "f64")
        o.set_scene(em, ob, bx)
        for f, a in zip(vel, x):
            o.set_field_f64(f, a)
        o.step(params(n_coarse))
        out = sum(float(np.dot(o.get_field(f, f64=True).ravel(), b.astype(np.float64))) for f, b in zip(vel, y))
        o.close()
        return out

    g = Sim(desc)
    g.set_scene(em, ob, bx)
    for f, a in zip(vel, x):
        g.set_field(f, a)
    if name != "cube":
        check_plan(g, dim, first, ctas, slabs)
    ro = Rollout(g, 1, 1, deterministic=True)
    ro.forward(params(3), None)
    gy = [torch.from_numpy(b).cuda() for b in y]
    torch.cuda.synchronize()
    ro.backward(params(3), grad_velocity=[t.data_ptr() for t in gy])
    grad = [ro.grad(f).astype(np.float64).ravel() for f in vel]
    ro.close()
    norm = lambda v: float(np.sqrt(sum(np.dot(a.astype(np.float64), a.astype(np.float64)) for a in v)))  # noqa: E731
    got = sum(float(np.dot(a, b.astype(np.float64))) for a, b in zip(grad, x))
    tol = 1e-4 * norm(x) * norm(grad)
    want = oracle(3)
    assert abs(got - want) <= tol, (got, want, tol)
    assert abs(oracle(2) - want) > 3 * tol, (oracle(2), want, tol)
