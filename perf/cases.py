"""Performance cases: the work a user of this package has it do.

`listed()` names the cases, `draw(rng)` makes another one of the same ranges,
`prepare(case, seed)` builds what a program holds before the call (a `Sim` with
its scene and fields on the GPU), `run(state)` is one pass through the public
entry points, `work(case)` the bytes and operations a pass cannot do without
and `exact(case, seed)` the same results from a plain float64 torch model.

Kinds of case:
  frame      one frame of a running simulation (`Sim.run_physics_step`), as a
             viewer or game loop asks for it; the state moves on with each pass
  rollout    `steps` frames from a given state, restored on every pass, as
             planning, fitting and parameter studies do
  solve      the pressure projection alone (`Sim.multigrid_pressure_solve`)
  transport  the stages around the projection, called one by one
  gradient   a checkpointed rollout and its reverse pass (`Rollout`)
  render     a frame of the headless renderer into device memory
"""
import ctypes
import math

import torch

from smokesim_b200 import Sim, abi, scene
from smokesim_b200.adjoint import Rollout

DT, RHO, T_AMB = 0.1, 1.0, 0.0
PREC = {"fp32": abi.PREC_FP32, "fp16": abi.PREC_MIXED, "bf16": abi.PREC_MIXED_BF16}


def _case(name, kind, nx, ny, nz, **kw):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, channels=1, enclosed=True, quirks=True, precision="fp32", pre=2, post=2,
             coarse=80, cycles=4, tol=0.0, warm=False, stats=False, min_coarse=8, own_stream=True, moving=False, steps=1,
             every=1, store=False, width=0, height=0)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the 2D plume workload: the smallest call, a few hundred kilobytes of state
        _case("frame_2d_256", "frame", 256, 256, 0),
        # a 2D window of odd size with RGB smoke, open sides and the
        # reference's default schedule (one V-cycle of 16 + 16 sweeps down to
        # 4 cells), on the default stream as `Sim(desc)` gives it
        _case("frame_2d_rgb_ragged", "frame", 601, 347, 0, channels=3, enclosed=False, pre=16, post=16, cycles=1,
              min_coarse=4, own_stream=False),
        # the small 3D grid of rollouts and previews, corrected operators
        _case("frame_3d_64", "frame", 64, 64, 64, quirks=False),
        # an odd 3D box with RGB smoke, open sides and a falling sphere that is
        # rasterised again every frame, on the default stream
        _case("frame_3d_rgb_ragged", "frame", 97, 75, 61, channels=3, enclosed=False, quirks=False, moving=True,
              own_stream=False),
        # the 128^3 plume workload: FP32 projection, reference boundary rules,
        # the solver's statistics read every frame
        _case("frame_3d_128", "frame", 128, 128, 128, stats=True),
        # the inverse-control forward: mixed-precision projection to 1e-6
        _case("rollout_mixed_128", "rollout", 128, 128, 128, quirks=False, precision="fp16", tol=1e-6, cycles=40, steps=2),
        # the headline workload: 256^3, mixed precision to 1e-6, extrapolated start
        _case("frame_mixed_256", "frame", 256, 256, 256, quirks=False, precision="fp16", tol=1e-6, cycles=40, warm=True),
        # the projection alone on a box that is not a cube
        _case("solve_192x128x160", "solve", 192, 128, 160, quirks=False),
        # the stages around the projection, one call each
        _case("transport_160x192x144", "transport", 160, 192, 144),
        # gradients of a short 64^3 rollout with per-step emitter forces
        _case("gradient_64", "gradient", 64, 64, 64, quirks=False, steps=8, every=4),
        # gradients through the mixed-precision projection, pressures stored
        _case("gradient_mixed_128", "gradient", 128, 128, 128, quirks=False, precision="fp16", steps=4, every=2,
              store=True),
        # a full frame of the ray marcher
        _case("render_1024", "render", 192, 192, 192, width=1024, height=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, cells, even=False):
    while True:
        n = [_log(rng, lo, hi) for _ in range(3)]
        if even:
            n[0] += n[0] & 1
        if n[0] * n[1] * n[2] <= cells:
            return n


def draw(rng):
    kind = rng.choice(["frame2", "frame2", "frame3", "frame3", "rollout", "solve", "transport", "gradient", "render"])
    coin = lambda: rng.random() < 0.5  # noqa: E731
    if kind == "frame2":
        ref = coin()
        return _case(None, "frame", _log(rng, 48, 1100), _log(rng, 48, 1100), 0, channels=rng.choice([1, 3]),
                     enclosed=coin(), pre=16 if ref else 2, post=16 if ref else 2, cycles=1 if ref else 4,
                     min_coarse=4 if ref else 8, own_stream=coin())
    if kind == "frame3":
        n = _box(rng, 20, 220, 5_000_000)
        return _case(None, "frame", *n, channels=rng.choice([1, 1, 3]), enclosed=coin(), quirks=coin(), moving=coin(),
                     own_stream=coin(), stats=coin())
    if kind == "rollout":
        # a tolerance needs grids whose levels halve exactly; others take a fixed count
        if coin():
            n = [32 * rng.randint(1, 7) for _ in range(3)]
            return _case(None, "rollout", *n, quirks=False, precision=rng.choice(["fp16", "bf16"]), tol=1e-6, cycles=40,
                         warm=coin(), steps=rng.randint(1, 3))
        n = _box(rng, 24, 220, 8_000_000, even=True)
        return _case(None, "rollout", *n, enclosed=coin(), quirks=False, precision=rng.choice(["fp16", "bf16"]),
                     steps=rng.randint(1, 3))
    if kind == "solve":
        return _case(None, "solve", *_box(rng, 24, 256, 9_000_000), enclosed=coin(), quirks=coin(), own_stream=coin())
    if kind == "transport":
        return _case(None, "transport", *_box(rng, 24, 256, 9_000_000), channels=rng.choice([1, 1, 3]), enclosed=coin(),
                     own_stream=coin())
    if kind == "gradient":
        n = _box(rng, 20, 112, 700_000, even=True)
        return _case(None, "gradient", *n, enclosed=coin(), quirks=False, precision=rng.choice(["fp32", "fp16"]),
                     steps=rng.randint(2, 8), every=rng.randint(1, 4), store=coin())
    return _case(None, "render", *_box(rng, 32, 224, 9_000_000), channels=rng.choice([1, 3]), width=_log(rng, 200, 1300),
                 height=_log(rng, 200, 1100))


# ------------------------------------------------------------------- inputs
def _size(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case["nz"] else [])


def _params(case):
    return scene.workload_params(ref_quirks=int(case["quirks"]), precision=PREC[case["precision"]], n_pre=case["pre"],
                                 n_post=case["post"], n_coarse=case["coarse"], n_vcycles=case["cycles"], tol=case["tol"],
                                 warm_start=int(case["warm"]), collect_stats=int(case["stats"]))


def _scene(case, seed):
    """Two plumes at the bottom, a sphere in the middle and a block beside it, all
    in proportion to the grid.  Positions off the cell centres."""
    g = torch.Generator().manual_seed(1000003 * int(seed) + 17)
    r = lambda lo, hi: float(lo + (hi - lo) * torch.rand((), generator=g))  # noqa: E731
    n = _size(case)
    m = min(n)
    em = []
    for _ in range(2):
        z = round(r(0.3, 0.7) * n[2]) + 0.25 if len(n) == 3 else 0.0
        em.append(scene.emitter((round(r(0.3, 0.7) * n[0]) + 0.25, round(0.08 * n[1]) + 0.25, z), 0.0625 * m + 1.1,
                                velocity=(0.0, 2.0, 0.0)))
    anchored = 0.0 if case["moving"] else 1.0
    ob = [scene.obstacle((n[0] / 2 + 0.25, n[1] / 2 + 0.25, n[2] / 2 + 0.25 if len(n) == 3 else 0.0), 0.125 * m + 0.1,
                         anchored=anchored)]
    lo = [round(r(0.15, 0.3) * k) for k in n] + [0] * (3 - len(n))
    hi = [lo[d] + max(2, round(0.12 * m)) for d in range(len(n))] + [1] * (3 - len(n))
    return em, ob, [scene.box(tuple(map(float, lo)), tuple(map(float, hi)))]


def _smooth(shape, g, device, sigma):
    """Unit-variance Gaussian random field of correlation length sigma cells."""
    f = torch.randn(shape, generator=g, device=device)
    for d, s in enumerate(shape):
        k = torch.fft.fftfreq(s, device=device)
        w = torch.exp(-2.0 * (math.pi * sigma * k) ** 2)
        f = torch.fft.ifft(torch.fft.fft(f, dim=d) * w.reshape([-1 if i == d else 1 for i in range(len(shape))]), dim=d).real
    return f / f.std().clamp_min(1e-12)


def _fields(case, seed, device):
    """Velocities of unit size, smoke and heat in patches, no pressure yet."""
    g = torch.Generator(device=device).manual_seed(int(seed) * 7919 + 5)
    n = _size(case)
    sigma = min(8.0, min(n) / 8.0)
    cells = n[::-1]
    f = {}
    for d, name in enumerate([abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ][:len(n)]):
        shape = list(cells)
        shape[len(n) - 1 - d] += 1
        f[name] = _smooth(shape, g, device, sigma)
    dens = [torch.relu(_smooth(cells, g, device, sigma)) for _ in range(case["channels"])]
    f[abi.FIELD_DENSITY] = torch.stack(dens)
    f[abi.FIELD_TEMPERATURE] = torch.relu(_smooth(cells, g, device, sigma))
    f[abi.FIELD_PRESSURE] = torch.zeros(cells, device=device)
    return {k: v.contiguous().float() for k, v in f.items()}


_STREAM = []


def _stream():
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


class _View:
    """A device array of the library for torch.as_tensor (no copy); the simulation
    that owns the memory lives as long as the tensor."""

    def __init__(self, sim, ptr, shape):
        self.sim = sim
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": "<f4", "version": 3}


class _State:
    def __init__(self, case, seed):
        self.case = case
        n = _size(case)
        desc = abi.make_desc(len(n), n, cell_size=1.0, density_channels=case["channels"], enclosed=int(case["enclosed"]),
                             min_coarse=case["min_coarse"], t_ambient=T_AMB)
        self.params = _params(case)
        self.sim = Sim(desc, stream=_stream().cuda_stream) if case["own_stream"] else Sim(desc)
        em, ob, bx = _scene(case, seed)
        self.sim.set_scene(em, ob, bx)
        self.names = [abi.FIELD_VX, abi.FIELD_VY] + ([abi.FIELD_VZ] if len(n) == 3 else [])
        self.names += [abi.FIELD_DENSITY, abi.FIELD_TEMPERATURE, abi.FIELD_PRESSURE]
        self.start = _fields(case, seed, "cuda")
        self.seen = {}
        torch.cuda.synchronize()
        self.restore()

    def restore(self, names=None):
        for f in names or self.names:
            t = self.start[f]
            rc = self.sim.L.ss_set_field_device(self.sim.h, f, ctypes.c_void_p(t.data_ptr()), t.numel(), self.sim.stream)
            if rc:
                raise RuntimeError("ss_set_field_device: %d" % rc)

    def field(self, f):
        ptr, _ = self.sim.device_ptr(f)
        t = self.seen.get(ptr)
        if t is None:
            t = self.seen[ptr] = torch.as_tensor(_View(self.sim, ptr, self.sim.shape(f)), device="cuda")
        return t

    def fields(self, names=None):
        return {"f%d" % f: self.field(f) for f in names or self.names}


def prepare(case, seed):
    s = _State(case, seed)
    kind = case["kind"]
    if kind == "render":
        s.sim.run_physics_step(s.params, 12)   # smoke as it looks after some frames
        s.view = s.sim.render_desc(case["width"], case["height"])
        s.image = torch.empty((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
    if kind == "gradient":
        s.rollout = Rollout(s.sim, case["steps"], case["every"], store_pressure=case["store"])
        g = torch.Generator().manual_seed(int(seed) + 3)
        s.forces = (0.1 * torch.randn((case["steps"], 3), generator=g)).numpy()
        cot = torch.Generator(device="cuda").manual_seed(int(seed) + 9)
        s.cotangent = torch.randn(s.start[abi.FIELD_DENSITY].shape, generator=cot, device="cuda")
        s.grads = [torch.empty(s.start[f].numel(), device="cuda") for f in s.names[:s.sim.dim]]
        s.final = torch.empty_like(s.cotangent)
    torch.cuda.synchronize()
    return s


def run(s):
    case, sim, p = s.case, s.sim, s.params
    kind = case["kind"]
    if kind == "frame":
        sim.run_physics_step(p)
        return s.fields()
    if kind == "rollout":
        s.restore()
        sim.run_physics_step(p, case["steps"])
        return s.fields()
    if kind == "solve":
        s.restore([abi.FIELD_PRESSURE])
        sim.multigrid_pressure_solve(p)
        return s.fields([abi.FIELD_PRESSURE])
    if kind == "transport":
        s.restore(s.names[:-1])
        sim.advect_velocities(p)
        sim.apply_buoyancy(p)
        sim.apply_vorticity(p)
        sim.advect_smoke(p)
        return s.fields(s.names[:-1])
    if kind == "gradient":
        s.restore()
        stream = sim.stream.value
        s.rollout.forward(p, s.forces, stream=stream)
        rc = sim.L.ss_get_field_device(sim.h, abi.FIELD_DENSITY, ctypes.c_void_p(s.final.data_ptr()), s.final.numel(),
                                       sim.stream)
        if rc:
            raise RuntimeError("ss_get_field_device: %d" % rc)
        gf = s.rollout.backward(p, grad_density=s.cotangent.data_ptr(), stream=stream)
        for f, g in zip(s.names, s.grads):
            s.rollout.grad_to_device(f, g.data_ptr(), stream=stream)
        return {"forces": gf, "velocity": s.grads, "density": s.final}
    rc = sim.L.ss_render(sim.h, ctypes.byref(s.view), ctypes.c_void_p(s.image.data_ptr()), 1, sim.stream)
    if rc:
        raise RuntimeError("ss_render: %d" % rc)
    return s.image


def work(case):
    n = _size(case)
    cells = math.prod(n)
    d, ch = len(n), case["channels"]
    state = 8 * d + 8 * (ch + 1) + 8 + 1          # velocities, smoke, heat, pressure in and out, solid map
    cycles = 4 if case["tol"] else case["cycles"]
    sweep = 2 * d + 4
    solve = cycles * ((case["pre"] + case["post"]) * sweep + 4 * d + 8) * (2 ** d / (2 ** d - 1))
    advect = d * (40 + 3 * 2 ** d) + (ch + 1) * 3 * 2 ** d + 60
    kind = case["kind"]
    if kind in ("frame", "rollout"):
        return {"bytes": case["steps"] * cells * state, "flops": case["steps"] * cells * (solve + advect)}
    if kind == "solve":
        return {"bytes": cells * (4 * d + 8 + 1), "flops": cells * solve}
    if kind == "transport":
        return {"bytes": cells * (state - 8), "flops": cells * advect}
    if kind == "gradient":
        return {"bytes": 3 * case["steps"] * cells * state, "flops": 3 * case["steps"] * cells * (solve + advect)}
    pixels = case["width"] * case["height"]
    return {"bytes": pixels * 4 + cells * 4 * ch, "flops": pixels * 100 * 7 * 40}


# --------------------------------------------------------- the float64 model
def _axis(a, d):
    return a.dim() - 1 - d


def _shift(a, d, by, fill=0.0):
    """a at index + by (by = -1 or 1) along axis d, `fill` outside."""
    ax = _axis(a, d)
    n = a.shape[ax]
    edge = torch.full_like(a.narrow(ax, 0, 1), fill)
    return torch.cat([a.narrow(ax, 1, n - 1), edge], ax) if by > 0 else torch.cat([edge, a.narrow(ax, 0, n - 1)], ax)


def _grid(shape, device):
    """index of each axis (x first), broadcast to shape"""
    dim = len(shape)
    out = []
    for d in range(dim):
        v = torch.arange(shape[dim - 1 - d], dtype=torch.float64, device=device)
        out.append(v.reshape([-1 if i == dim - 1 - d else 1 for i in range(dim)]).expand(shape))
    return out


def _sample(a, at, border):
    """Multilinear sample of `a` at texel coordinates (x first), `border` outside."""
    dim = a.dim()
    pad = torch.nn.functional.pad(a[None, None], [3, 3] * dim, value=border)[0, 0]
    size = [a.shape[_axis(a, d)] for d in range(dim)]
    stride, acc = [], 1
    for d in range(dim):
        stride.append(acc)
        acc *= size[d] + 6
    base, w = 0, []
    for d in range(dim):
        t = at[d].clamp(-2.0, size[d] + 1.0)
        f = t.detach().floor()
        w.append(t - f)
        base = base + (f.long() + 3) * stride[d]
    flat = pad.reshape(-1)

    def corner(d, off):
        if d < 0:
            return flat[base + off]
        lo, hi = corner(d - 1, off), corner(d - 1, off + stride[d])
        return lo * (1 - w[d]) + hi * w[d]

    return corner(dim - 1, 0)


class _Model:
    """The smoke step in float64 torch operations, differentiable."""

    def __init__(self, case, seed, device):
        self.case, self.device = case, device
        f32 = lambda v: float(torch.tensor(v, dtype=torch.float32))  # noqa: E731
        p = _params(case)
        self.dt, self.alpha, self.beta, self.eps = f32(DT), p.t_weight_coeff, p.t_temp_coeff, p.vorticity_confinement
        self.n = _size(case)
        self.dim = len(self.n)
        self.shape = self.n[::-1]
        em, ob, bx = _scene(case, seed)
        self.emitters = [([float(v) for v in e.pos][:self.dim], float(e.radius), float(e.density[0]),
                          [float(v) for v in e.density], float(e.temperature), [float(v) for v in e.velocity]) for e in em]
        at = _grid(self.shape, device)
        valid = torch.ones(self.shape, dtype=torch.bool, device=device)
        for d in range(self.dim):
            valid = valid & (at[d] > 1) & (at[d] < self.n[d] - 1)
        inside = torch.zeros_like(valid)
        for o in ob:
            d2 = sum((at[d] - float(o.pos[d])) ** 2 for d in range(self.dim))
            inside |= d2.sqrt() < float(o.radius)
        for b in bx:
            q = torch.ones_like(valid)
            for d in range(self.dim):
                q = q & (at[d] >= float(b.lo[d])) & (at[d] < float(b.hi[d]))
            inside |= q
        self.solid = valid & inside
        if case["enclosed"]:
            for d in range(self.dim):
                self.solid = self.solid | (at[d] == 0) | (at[d] == self.n[d] - 1)
        self.fluid = (~self.solid).double()
        self._levels()

    def _levels(self):
        s = self.solid.double()
        self.levels = []
        size, level = list(self.n), 0
        quirks, closed = self.case["quirks"], self.case["enclosed"]
        smooth_wall = 0.0 if quirks else (1.0 if closed else 0.0)
        resid_wall = 1.0 if quirks else (1.0 if closed else 0.0)
        while min(size) >= self.case["min_coarse"]:
            lv = {"alpha": s, "hh": float(4 ** level)}
            for tag, wall in (("s", smooth_wall), ("r", resid_wall)):
                f = [1 - _shift(s, d, by, wall) for d in range(self.dim) for by in (1, -1)]
                lv["f" + tag], lv["sum" + tag] = f, sum(f)
            at = _grid(list(s.shape), self.device)
            odd = (sum(at) % 2) == 1
            live = (s < 1) & (lv["sums"] != 0)
            lv["colour"] = [live & ~odd, live & odd]
            lv["div"] = torch.where(lv["sums"] == 0, torch.ones_like(s), lv["sums"])
            self.levels.append(lv)
            size = [k // 2 for k in size]
            if min(size) < 1:
                break
            m = self._down(s)
            s = torch.where(m >= 0.5, m, torch.zeros_like(m)).half().double()
            level += 1

    def _down(self, a):
        """mean of the 2^dim children (odd leftovers dropped)"""
        for ax in range(self.dim):
            k = a.shape[ax] // 2
            a = a.narrow(ax, 0, 2 * k).unflatten(ax, (k, 2)).mean(ax + 1)
        return a

    def _near(self, p, f):
        return sum(_shift(p, d, by) * w for (d, by), w in zip([(d, by) for d in range(self.dim) for by in (1, -1)], f))

    def _sweeps(self, p, b, lv, count):
        for _ in range(count):
            for live in lv["colour"]:
                p = torch.where(live, (self._near(p, lv["fs"]) - b) / lv["div"], p)
        return p

    def _up(self, coarse, shape):
        """CLAMP_TO_EDGE linear interpolation at the fine cell centres"""
        a = coarse
        for d in range(self.dim):
            ax = _axis(a, d)
            n, c = shape[self.dim - 1 - d], a.shape[ax]
            t = (torch.arange(n, dtype=torch.float64, device=self.device) + 0.5) / n * c - 0.5
            f = t.floor()
            w = (t - f).reshape([-1 if i == ax else 1 for i in range(self.dim)])
            lo, hi = f.long().clamp(0, c - 1), (f.long() + 1).clamp(0, c - 1)
            a = a.index_select(ax, lo) * (1 - w) + a.index_select(ax, hi) * w
        return a

    def _cycle(self, p, b_s, b_r, level=0):
        """One V-cycle: b_s the smoother's right-hand side (times h^2), b_r the residual's."""
        lv = self.levels[level]
        if level == len(self.levels) - 1:
            return self._sweeps(p, b_s, lv, self.case["coarse"])
        p = self._sweeps(p, b_s, lv, self.case["pre"])
        r = (b_r - (self._near(p, lv["fr"]) - lv["sumr"] * p) / lv["hh"]) * (lv["alpha"] < 1)
        if self.case["quirks"] and level > 0:
            b_s = r * lv["hh"]      # the residual overwrites the right-hand side
        rc = self._down(r)
        e = self._cycle(torch.zeros_like(rc), rc * self.levels[level + 1]["hh"], rc, level + 1)
        p = p + self._up(e, list(p.shape))
        return self._sweeps(p, b_s, lv, self.case["post"])

    # ---- stages
    def emit(self, v, dens, temp, force=None):
        at = _grid(self.shape, self.device)
        v = list(v)
        for pos, rad, _, rgb, heat, vel in self.emitters:
            hit = (sum((at[d] - pos[d]) ** 2 for d in range(self.dim)).sqrt() < rad).double()
            dens = torch.stack([dens[c] + hit * (rgb[c] * self.dt) for c in range(dens.shape[0])])
            temp = temp + hit * (heat * self.dt)
        for c in range(self.dim):
            at = _grid(list(v[c].shape), self.device)
            touched = torch.zeros(v[c].shape, dtype=torch.bool, device=self.device)
            for pos, rad, _, _, _, vel in self.emitters:
                hit = sum((at[d] - pos[d]) ** 2 for d in range(self.dim)).sqrt() < rad
                v[c] = torch.where(hit, torch.full_like(v[c], vel[c]), v[c])
                touched |= hit
            if force is not None:
                v[c] = v[c] + touched.double() * (self.dt * force[c])
        return v, dens, temp

    def _faces_solid(self, c, wall):
        """solid at the high and the low side of each face of axis c"""
        s = self.solid.double()
        ax = _axis(s, c)
        edge = torch.full_like(s.narrow(ax, 0, 1), wall)
        return torch.cat([s, edge], ax) > 0, torch.cat([edge, s], ax) > 0

    def advect_velocity(self, v):
        out = []
        for c in range(self.dim):
            g = [x + (0.0 if d == c else 0.5) for d, x in enumerate(_grid(list(v[c].shape), self.device))]
            back = []
            for j in range(self.dim):
                vel = _sample(v[j], [g[d] - (0.0 if d == j else 0.5) for d in range(self.dim)], 0.0)
                back.append(g[j] - vel * self.dt - (0.0 if j == c else 0.5))
            hi, lo = self._faces_solid(c, 1.0)
            out.append(torch.where(hi | lo, torch.zeros_like(v[c]), _sample(v[c], back, 0.0)))
        return out

    def buoyancy(self, v, before, dens, temp):
        """`before`: the y velocities before the advection, kept at faces that touch solid"""
        def mean(a, border):
            ax = _axis(a, 1)
            edge = torch.full_like(a.narrow(ax, 0, 1), border)
            return 0.5 * (torch.cat([a, edge], ax) + torch.cat([edge, a], ax))
        total = sum(mean(d, 0.0) for d in dens)
        lift = -self.alpha * total + self.beta * (mean(temp, T_AMB) - T_AMB)
        hi, lo = self._faces_solid(1, 0.0)
        return [torch.where(hi | lo, before, v[1] + lift * self.dt) if c == 1 else v[c] for c in range(self.dim)]

    @staticmethod
    def _root(q):
        live = q > 0
        return torch.where(live, torch.where(live, q, torch.ones_like(q)).sqrt(), torch.zeros_like(q))

    def vorticity(self, v):
        def centre(c, d, by):   # mean of the two faces of component c at the cell next door (0 outside)
            ax = _axis(v[c], c)
            near = _shift(v[c], d, by)
            return 0.5 * (near.narrow(ax, 0, self.n[c]) + near.narrow(ax, 1, self.n[c]))
        diff = lambda c, d: centre(c, d, 1) - centre(c, d, -1)  # noqa: E731
        if self.dim == 2:
            w = [(diff(1, 0) - diff(0, 1)) / 2 * self.fluid]
            mag = w[0].abs()
        else:
            w = [(diff(2, 1) - diff(1, 2)) / 2 * self.fluid, (diff(0, 2) - diff(2, 0)) / 2 * self.fluid,
                 (diff(1, 0) - diff(0, 1)) / 2 * self.fluid]
            mag = self._root(sum(x * x for x in w))
        g = [(_shift(mag, d, 1) - _shift(mag, d, -1)) / 2 for d in range(self.dim)]
        size = self._root(sum(x * x for x in g)) + 1e-20
        k = [x / size for x in g]
        if self.dim == 2:
            f = [-k[1] * w[0], -k[0] * w[0]]
        else:
            f = [k[1] * w[2] - w[1] * k[2], k[2] * w[0] - w[2] * k[0], k[0] * w[1] - w[0] * k[1]]
        out = []
        for c in range(self.dim):
            ax = _axis(v[c], c)
            term = f[c] * (0.5 * self.eps * self.dt / RHO)
            out.append(v[c] + torch.cat([term, torch.zeros_like(term.narrow(ax, 0, 1))], ax))
        return out

    def divergence(self, v, wall):
        """faces of solid neighbours count 0 (out of grid: where `wall`)"""
        total = 0
        for c in range(self.dim):
            ax = _axis(v[c], c)
            n = self.n[c]
            hi, lo = v[c].narrow(ax, 1, n), v[c].narrow(ax, 0, n)
            s = self.solid.double()
            total = total + hi * (1 - _shift(s, c, 1, wall)) - lo * (1 - _shift(s, c, -1, wall))
        return total * self.fluid

    def project(self, v, p):
        case = self.case
        quirks, closed = case["quirks"], 1.0 if case["enclosed"] else 0.0
        ds, dr = self.divergence(v, 0.0 if quirks else closed), self.divergence(v, 1.0 if quirks else closed)
        b_s, b_r = RHO * ds / self.dt, RHO * dr / self.dt
        lv = self.levels[0]
        for _ in range(60 if case["tol"] else case["cycles"]):
            p = self._cycle(p, b_s, b_r)
            if case["tol"]:
                r = (b_r - (self._near(p, lv["fr"]) - lv["sumr"] * p)) * self.fluid
                if float(r.norm()) <= 1e-11 * float(b_r.norm()):
                    break
        return p

    def update(self, v, p):
        out = []
        for c in range(self.dim):
            ax = _axis(v[c], c)
            edge = torch.zeros_like(p.narrow(ax, 0, 1))
            hi, lo = self._faces_solid(c, 0.0)
            new = v[c] - self.dt / RHO * (torch.cat([p, edge], ax) - torch.cat([edge, p], ax))
            out.append(torch.where(hi | lo, torch.zeros_like(new), new))
        return out

    def advect_smoke(self, v, dens, temp):
        at = _grid(self.shape, self.device)
        back = []
        for c in range(self.dim):
            ax = _axis(v[c], c)
            back.append(at[c] - 0.5 * (v[c].narrow(ax, 0, self.n[c]) + v[c].narrow(ax, 1, self.n[c])) * self.dt)
        out = [torch.where(self.solid, torch.zeros_like(temp), _sample(d, back, 0.0)) for d in dens]
        heat = torch.where(self.solid, torch.full_like(temp, T_AMB), _sample(temp, back, T_AMB))
        return torch.stack(out), heat

    def step(self, v, dens, temp, p, force=None):
        v, dens, temp = self.emit(v, dens, temp, force)
        before = v[1]
        v = self.buoyancy(self.advect_velocity(v), before, dens, temp)
        v = self.vorticity(v)
        p = self.project(v, p)
        v = self.update(v, p)
        dens, temp = self.advect_smoke(v, dens, temp)
        return v, dens, temp, p


def exact(case, seed):
    kind = case["kind"]
    if kind == "render":
        return None   # an image of bytes
    device = "cuda" if torch.cuda.is_available() else "cpu"
    m = _Model(case, seed, device)
    names = [abi.FIELD_VX, abi.FIELD_VY, abi.FIELD_VZ][:m.dim] + [abi.FIELD_DENSITY, abi.FIELD_TEMPERATURE,
                                                                  abi.FIELD_PRESSURE]
    start = {f: t.double() for f, t in _fields(case, seed, device).items()}
    v = [start[f] for f in names[:m.dim]]
    dens, temp, p = (start[f] for f in names[m.dim:])
    if kind == "gradient":
        force = torch.Generator().manual_seed(int(seed) + 3)
        force = (0.1 * torch.randn((case["steps"], 3), generator=force)).double().to(device).requires_grad_(True)
        v = [x.clone().requires_grad_(True) for x in v]
        cot = torch.Generator(device=device).manual_seed(int(seed) + 9)
        cot = torch.randn(list(dens.shape), generator=cot, device=device).double()
        first = list(v)
        for k in range(case["steps"]):
            v, dens, temp, p = m.step(v, dens, temp, p, force[k])
        g = torch.autograd.grad((dens * cot).sum(), [force] + first)
        return {"forces": g[0], "velocity": [x.reshape(-1) for x in g[1:]], "density": _like(dens.detach(), m)}
    with torch.no_grad():
        if kind == "solve":
            return {"f%d" % abi.FIELD_PRESSURE: _like(m.project(v, p), m)}
        if kind == "transport":
            v = m.buoyancy(m.advect_velocity(v), v[1], dens, temp)
            v = m.vorticity(v)
            dens, temp = m.advect_smoke(v, dens, temp)
        else:
            for _ in range(case["steps"]):
                v, dens, temp, p = m.step(v, dens, temp, p)
    out = {"f%d" % f: _like(x, m) for f, x in zip(names, list(v) + [dens, temp])}
    if kind != "transport":
        # to a tolerance the pressure is what the solver stopped at, up to a constant
        out["f%d" % abi.FIELD_PRESSURE] = None if case["tol"] else _like(p, m)
    return out


def _like(a, m):
    """the shape the fields of `run` have (2D fields carry a z axis of one)"""
    if m.dim == 3:
        return a
    return a[:, None] if a.dim() == 3 else a[None]
