"""The work that a user of this framework has it do, as cases that can be timed.

A particle case is the loop of a driver that keeps its particle array on the
host: hand the state over (``Context.update``), advance it a few time steps
(``Context.step``), read it back (``Context.download_state``), all through
page-locked arrays.  A cloud case is one neighbour search with the summation
density, through the context or through the allocation-free entry point on
device pointers.

The start states are dam breaks caught in motion: the lattice of
``titsolver_gb300.scenarios`` with every fluid particle displaced at random
(as moving particles are), a collapsing column's velocity field and the
hydrostatic density.  The launch shape is the library's default.

``exact`` restates the same step and the same sums in 64-bit torch, without
the library: all pairs within the support radius from a cell grid, the wall
extrapolation, the equation of state and the SSPRK stages.
"""

from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from titsolver_gb300 import _abi, physics, scenarios

RHO0 = 1000.0
C2, C4 = _abi.TG_KERNEL_WENDLAND_C2, _abi.TG_KERNEL_WENDLAND_C4


def listed():
    return [
        # The smallest call: the reference's own default physics (C4 kernel,
        # Morris viscosity, shifting after every step) on a coarse column,
        # the host taking every step: launches and latency.
        dict(name="dam2d_f64_small", kind="dam2d", form="f64", terms="reference", kernel=C4,
             shifting=True, nx=20, col=2.0, steps=1),
        # The benchmark's first configuration: 12,800 fluid particles, plain FP64.
        dict(name="dam2d_f64", kind="dam2d", form="f64", terms="baseline", kernel=C2,
             shifting=False, nx=80, col=2.0, steps=10),
        # Its configuration at scale: 1.28M fluid particles, compensated form.
        dict(name="dam2d_f32c_1m", kind="dam2d", form="f32c", terms="baseline", kernel=C2,
             shifting=False, nx=800, col=2.0, steps=8),
        # A ragged mid-size run with shifting in the compensated form: a
        # column whose sides are no round numbers of particles.
        dict(name="dam2d_f32c_shift", kind="dam2d", form="f32c", terms="reference", kernel=C4,
             shifting=True, nx=213, col=1.37, steps=4),
        # The 3D dam break in plain FP64 (250,000 fluid particles).
        dict(name="dam3d_f64", kind="dam3d", form="f64", terms="baseline", kernel=C2,
             shifting=False, nx=50, col=2.0, steps=2),
        # The 3D dam break, compensated form: 2M and 8M fluid particles.
        dict(name="dam3d_f32c_2m", kind="dam3d", form="f32c", terms="baseline", kernel=C2,
             shifting=False, nx=100, col=2.0, steps=8),
        dict(name="dam3d_f32c_8m", kind="dam3d", form="f32c", terms="baseline", kernel=C2,
             shifting=False, nx=160, col=2.0, steps=4),
        # Batches of independent tanks of uneven size in one launch per pass.
        dict(name="tanks2d_f32c", kind="tanks2d", form="f32c", terms="baseline", kernel=C2,
             shifting=False, tanks=512, lo=20, hi=120, steps=4),
        dict(name="tanks3d_f32c", kind="tanks3d", form="f32c", terms="baseline", kernel=C2,
             shifting=False, tanks=24, lo=12, hi=40, steps=4),
        # The reference's scenario with its tessellated pool walls (faces)
        # and shifting, in plain FP64: 12,800 fluid particles.
        dict(name="pool2d_f64", kind="pool2d", form="f64", terms="reference", kernel=C4,
             shifting=True, nx=80, steps=4),
        # The 4M-point cloud: search and summation density, FP32 positions.
        dict(name="cloud3d_f32", kind="cloud3d", form="f32", kernel=C2, n=4_000_000),
        # The allocation-free density on device pointers, near its largest size.
        dict(name="cloud3d_noalloc", kind="noalloc", form="f64", kernel=C2, dim=3, n=60_001),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["dam2d", "dam2d", "dam3d", "dam3d", "tanks2d", "tanks3d", "pool2d",
                       "cloud3d", "noalloc"])
    if kind == "cloud3d":
        return dict(kind=kind, form=rng.choice(["f32", "f32", "f64"]),
                    kernel=rng.choice([C2, C2, C4]), n=_log(rng, 2_000, 700_000))
    if kind == "noalloc":
        return dict(kind=kind, form="f64", kernel=rng.choice([C2, C4]), dim=rng.choice([2, 3]),
                    n=_log(rng, 500, 65_536))
    form = rng.choice(["f64", "f32c", "f32c"])
    terms = rng.choice(["baseline", "baseline", "reference"])
    kernel = rng.choice([C2, C2, C4, C4, rng.randrange(6)])
    shifting = rng.random() < 0.25
    case = dict(kind=kind, form=form, terms=terms, kernel=kernel, shifting=shifting,
                steps=rng.randint(1, 8))
    if kind == "dam2d":
        case |= dict(nx=_log(rng, 12, 700 if form == "f32c" else 240),
                     col=round(rng.uniform(0.6, 2.2), 2))
    elif kind == "dam3d":
        case |= dict(nx=_log(rng, 8, 90 if form == "f32c" else 36),
                     col=round(rng.uniform(0.6, 2.2), 2))
    elif kind == "tanks2d":
        case |= dict(tanks=_log(rng, 2, 200), lo=rng.randint(8, 20), hi=rng.randint(21, 90))
    elif kind == "tanks3d":
        case |= dict(tanks=_log(rng, 2, 16), lo=rng.randint(6, 12), hi=rng.randint(13, 26))
    else:
        case |= dict(nx=_log(rng, 12, 120), terms="reference", kernel=rng.choice([C4, C4, C2]),
                     shifting=rng.random() < 0.75)
    return case


# ---- inputs ---------------------------------------------------------------


@functools.lru_cache(maxsize=1)
def _scenario(kind, **size):
    if kind == "dam2d":
        return scenarios.dam_break_2d(nx_per_H=size["nx"], column=(size["col"], 1.0))
    if kind == "dam3d":
        return scenarios.dam_break_3d(nx_per_H=size["nx"], column=(size["col"], 1.0, 1.0))
    if kind == "tanks2d":
        return scenarios.batched_tanks(n_tanks=size["tanks"], n_range=(size["lo"], size["hi"]))
    if kind == "tanks3d":
        return scenarios.batched_tanks_3d(n_tanks=size["tanks"], n_range=(size["lo"], size["hi"]))
    return scenarios.dam_break_2d_faces(nx_per_H=size["nx"])


def _size(case):
    return {k: case[k] for k in ("nx", "col", "tanks", "lo", "hi") if k in case}


def _particles(case, seed):
    """The scenario with a moving state: r, v, rho, dv (upload order)."""
    scn = _scenario(case["kind"], **_size(case))
    rng = np.random.Generator(np.random.PCG64(seed))
    d, dx = scn["dim"], scn["dx"]
    r, rho = scn["r"].copy(), scn["rho"]
    v, dv = np.zeros_like(r), np.zeros_like(r)
    at = 0
    for t in scn["tanks"]:
        f = slice(at, at + t["n_fluid"])
        at += t["n_fluid"] + t["n_wall"]
        x = r[f]
        height = x[:, 1].max()
        rate = rng.uniform(0.2, 0.8) * math.sqrt(scenarios.G / height)
        v[f, 0] = rate * x[:, 0]
        v[f, 1] = -rate * x[:, 1]
        v[f] += rng.standard_normal((t["n_fluid"], d), dtype=np.float32) * (0.002 * t["cs0"])
        dv[f, 1] = -scenarios.G
        r[f] += (rng.random((t["n_fluid"], d), dtype=np.float32) - 0.5) * (0.2 * dx)
    return scn, r, v, rho, dv


def _cloud(case, seed):
    if case["kind"] == "cloud3d" or case["dim"] == 3:
        return scenarios.cloud_3d(n_total=case["n"], seed=seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    n, dx = case["n"], 1.0 / math.sqrt(case["n"])
    tank = dict(n_fluid=n, n_wall=0, h=2.0 * dx, m=RHO0 * dx * dx, rho0=RHO0, cs0=1.0)
    return dict(dim=2, tanks=[tank], r=rng.random((n, 2)))


def _params(case, dim):
    make = physics.baseline_params if case["terms"] == "baseline" else physics.reference_params
    p = make(dim, _abi.TG_FP32C if case["form"] == "f32c" else _abi.TG_FP64, case["kernel"])
    p.post_integrate = _abi.TG_POST_SHIFTING if case["shifting"] else _abi.TG_POST_PREPARE
    return p


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _pinned_copy(a):
    return _pinned(a.shape).copy_(torch.from_numpy(a)).numpy()


def prepare(case, seed):
    if case["kind"] == "noalloc":
        scn = _cloud(case, seed)
        n = case["n"]
        return dict(case=case, tank=scn["tanks"][0],
                    r=torch.from_numpy(np.ascontiguousarray(scn["r"])).cuda(),
                    rho=torch.empty(n, dtype=torch.float64, device="cuda"),
                    counts=torch.empty(n, dtype=torch.int32, device="cuda"),
                    hashes=torch.empty(n, dtype=torch.int64, device="cuda"))
    if case["kind"] == "cloud3d":
        scn = _cloud(case, seed)
        ctx = _abi.Context(physics.baseline_params(3, _abi.TG_FP64, case["kernel"]))
        ctx.upload(scn["tanks"], scn["r"], scn["v"], scn["rho"])
        n = case["n"]
        return dict(case=case, ctx=ctx, rho=_pinned(n), counts=_pinned(n, torch.int32),
                    hashes=_pinned(n, torch.int64))
    scn, r, v, rho, dv = _particles(case, seed)
    ctx = _abi.Context(_params(case, scn["dim"]))
    ctx.upload(scn["tanks"], r, v, rho)
    for t, faces in enumerate(scn.get("faces", ())):
        ctx.set_faces(t, faces["face_verts"], faces["poly"])
    state = dict(case=case, ctx=ctx, start=[_pinned_copy(a) for a in (r, v, rho, dv)],
                 end=[_pinned(a.shape) for a in (r, v, rho, dv)])
    if case["form"] == "f32c":
        state["single"] = [torch.empty(a.shape, dtype=torch.float32) for a in (v, rho, dv)]
    return state


# ---- one pass ---------------------------------------------------------------


def run(state):
    case = state["case"]
    if case["kind"] == "noalloc":
        t, r = state["tank"], state["r"]
        st = _abi.load().tg_summation_density_noalloc(
            case["dim"], case["kernel"], case["n"], r.data_ptr(), t["h"], t["m"],
            state["rho"].data_ptr(), state["counts"].data_ptr(), state["hashes"].data_ptr(),
            torch.cuda.current_stream().cuda_stream)
        if st != _abi.TG_OK:
            raise RuntimeError(f"tg_summation_density_noalloc: {st}")
        return {k: state[k] for k in ("rho", "counts", "hashes")}
    ctx = state["ctx"]
    if case["kind"] == "cloud3d":
        rho, counts, hashes = (state[k] for k in ("rho", "counts", "hashes"))
        st = ctx.lib.tg_summation_density(
            ctx.handle, _abi.TG_POS_FP32 if case["form"] == "f32" else _abi.TG_POS_FP64,
            *(ctypes.cast(a.data_ptr(), ctypes.POINTER(t)) for a, t in (
                (rho, ctypes.c_double), (counts, ctypes.c_int32), (hashes, ctypes.c_uint64))))
        if st != _abi.TG_OK:
            raise RuntimeError(f"tg_summation_density: {st}")
        # FP32 positions give an FP32 sum.
        out = rho if case["form"] == "f64" else rho.to(torch.float32)
        return dict(rho=out, counts=counts, hashes=hashes)
    ctx.update(*state["start"])
    dt = ctx.step(case["steps"])
    r, v, rho, dv = state["end"]
    ctx.download_state(r=r.numpy(), v=v.numpy(), rho=rho.numpy(), dv_dt=dv.numpy())
    if case["form"] == "f64":
        return dict(r=r, v=v, rho=rho, dv=dv, dt=dt)
    # The compensated form holds everything but the positions and the time
    # in FP32 (the density as its deviation), and a program that runs it
    # keeps them so.
    v32, drho32, dv32 = state["single"]
    v32.copy_(v)
    drho32.copy_(rho.sub_(RHO0))
    dv32.copy_(dv)
    return dict(r=r, v=v32, drho=drho32, dv=dv32, dt=dt.astype(np.float32))


# ---- the work of a pass -------------------------------------------------------


def _neighbours(dim, h_over_dx, kernel):
    radius = {1: 2.5, 2: 3.0}.get(kernel, 2.0) * h_over_dx
    return (math.pi * radius ** 2) if dim == 2 else (4.0 / 3.0 * math.pi * radius ** 3)


def work(case):
    """Bytes: clouds read the positions and write the three results.  A
    particle step reads and writes the state once per stage (a stage's sums
    need the previous stage's state of every neighbour), and the pass moves
    the state in and out once.  Flops: those of the pair terms and of the
    predicate of every neighbour pair, per stage."""
    if case["kind"] in ("cloud3d", "noalloc"):
        dim = case.get("dim", 3)
        pairs = case["n"] * _neighbours(dim, 2.0 if dim == 2 else 1.3, case["kernel"])
        return dict(bytes=case["n"] * (8 * dim + 20), flops=pairs * (3 * dim + 12))
    # Fluid and wall counts from the scenario's own sizes.
    kind, d = case["kind"], 3 if "3d" in case["kind"] else 2
    if kind in ("dam2d", "pool2d"):
        nx, col = case["nx"], case.get("col", 2.0)
        nf = round(col * nx) * nx
        nw = (5.4 + 6.0) * nx * 3 if kind == "dam2d" else 19 * nx
    elif kind == "dam3d":
        nx, col = case["nx"], case["col"]
        nf = round(col * nx) * nx * nx
        nw = 3 * (5.4 + 6.0) * nx * nx + 6 * 5.4 * 3.0 * nx * nx
    else:
        lo, hi = case["lo"], case["hi"]
        mean = (lo + hi) / 2.0
        sq = mean ** 2 + (hi - lo) ** 2 / 12.0
        if d == 2:
            nf, nw = case["tanks"] * 1.25 * sq, case["tanks"] * 34 * mean
        else:
            nf = case["tanks"] * 1.56 * mean * sq
            nw = case["tanks"] * (34 * 1.25 + 97) * sq
    fp32 = case["form"] == "f32c"
    stage = 8 * d + (4 * d + 4 if fp32 else 8 * d + 8)  # r, v, rho
    per_pair = 43 if d == 3 else 38
    pairs = nf * _neighbours(d, 2.0 if d == 2 else 1.3, case["kernel"])
    host = 2 * (nf + nw) * 8 * (3 * d + 1)
    return dict(bytes=host + case["steps"] * 3 * 2 * nf * stage,
                flops=case["steps"] * 3 * pairs * per_pair)


# ---- the same in 64 bits --------------------------------------------------------


def _f(q, on, p):
    return torch.where(q < on, (on - q).clamp_min(0.0) ** p, torch.zeros_like(q))


def _kernel(k, q):
    """Unit value f(q) and derivative f'(q)."""
    t = (1.0 - 0.5 * q).clamp_min(0.0)
    if k == 0:
        return (0.25 * _f(q, 2.0, 3) - _f(q, 1.0, 3),
                -0.75 * _f(q, 2.0, 2) + 3.0 * _f(q, 1.0, 2))
    if k == 1:
        return (_f(q, 2.5, 4) - 5.0 * _f(q, 1.5, 4) + 10.0 * _f(q, 0.5, 4),
                -4.0 * _f(q, 2.5, 3) + 20.0 * _f(q, 1.5, 3) - 40.0 * _f(q, 0.5, 3))
    if k == 2:
        return (_f(q, 3.0, 5) - 6.0 * _f(q, 2.0, 5) + 15.0 * _f(q, 1.0, 5),
                -5.0 * _f(q, 3.0, 4) + 30.0 * _f(q, 2.0, 4) - 75.0 * _f(q, 1.0, 4))
    if k == 3:
        return (1.0 + 2.0 * q) * t ** 4, -5.0 * q * t ** 3
    if k == 4:
        return ((1.0 + 3.0 * q + 35.0 / 12.0 * q * q) * t ** 6,
                -14.0 / 3.0 * q * (1.0 + 2.5 * q) * t ** 5)
    return ((1.0 + 4.0 * q + 6.25 * q * q + 4.0 * q ** 3) * t ** 8,
            -2.75 * q * (2.0 + 7.0 * q + 8.0 * q * q) * t ** 7)


# Kernel weights per dimension: 1 / (unit integral of f), 2D and 3D.
_WEIGHT = [(10.0 / (7.0 * math.pi), 1.0 / math.pi),
           (96.0 / (1199.0 * math.pi), 1.0 / (20.0 * math.pi)),
           (7.0 / (478.0 * math.pi), 1.0 / (120.0 * math.pi)),
           (7.0 / (4.0 * math.pi), 21.0 / (16.0 * math.pi)),
           (9.0 / (4.0 * math.pi), 495.0 / (256.0 * math.pi)),
           (39.0 / (14.0 * math.pi), 1365.0 / (512.0 * math.pi))]


class _Pairs:
    """The pairs (a, b) within the support radius, from a grid of cells one
    radius wide per tank, in chunks of targets."""

    def __init__(self, r, tank, radius, radius2, budget=24_000_000):
        self.r, self.tank, self.radius2 = r, tank, radius2
        d = r.shape[1]
        nt = radius.shape[0]
        lo = torch.full((nt, d), math.inf, dtype=r.dtype, device=r.device)
        lo.scatter_reduce_(0, tank[:, None].expand_as(r), r, "amin")
        cell = ((r - lo[tank]) / (radius[tank] * (1 + 1e-9))[:, None]).floor().long() + 1
        nc = torch.zeros((nt, d), dtype=torch.long, device=r.device)
        nc.scatter_reduce_(0, tank[:, None].expand_as(cell), cell, "amax")
        nc += 2
        total = nc.prod(1)
        off = total.cumsum(0) - total
        key = off[tank] + cell[:, 0] + nc[tank, 0] * cell[:, 1]
        if d == 3:
            key = key + nc[tank, 0] * nc[tank, 1] * cell[:, 2]
        self.keys, self.order = key.sort(stable=True)
        self.key, self.nc, self.d, self.budget = key, nc, d, budget

    def each(self, targets):
        rows = [(y, z) for z in ((-1, 0, 1) if self.d == 3 else (0,)) for y in (-1, 0, 1)]
        key, t = self.key[targets], self.tank[targets]
        start, count = [], []
        for y, z in rows:
            k = key + y * self.nc[t, 0]
            if self.d == 3:
                k = k + z * self.nc[t, 0] * self.nc[t, 1]
            a = torch.searchsorted(self.keys, k - 1)
            start.append(a)
            count.append(torch.searchsorted(self.keys, k + 1, right=True) - a)
        start, count = torch.stack(start, 1), torch.stack(count, 1)
        ends = count.sum(1).cumsum(0)
        at, n = 0, targets.shape[0]
        while at < n:
            done = int(ends[at - 1]) if at else 0
            to = int(torch.searchsorted(ends, torch.tensor(done + self.budget, device=ends.device),
                                        right=True))
            to = min(n, max(to, at + 1))
            s, c = start[at:to].reshape(-1), count[at:to].reshape(-1)
            who = torch.arange(at, to, device=s.device).repeat_interleave(count[at:to].sum(1))
            first = (s - (c.cumsum(0) - c)).repeat_interleave(c)
            b = self.order[first + torch.arange(first.shape[0], device=s.device)]
            a = targets[who]
            d = self.r[a] - self.r[b]
            s2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]
            if self.d == 3:
                s2 = s2 + d[:, 2] * d[:, 2]
            ok = s2 <= self.radius2[self.tank[a]]
            yield a[ok], b[ok], d[ok], s2[ok]
            at = to


def _splitmix(ids):
    def shr(z, k):  # logical shift of a signed 64-bit integer
        return (z >> k) & ((1 << (64 - k)) - 1)

    def signed(c):
        return c - (1 << 64) if c >= 1 << 63 else c

    z = ids + signed(0x9E3779B97F4A7C15)
    z = (z ^ shr(z, 30)) * signed(0xBF58476D1CE4E5B9)
    z = (z ^ shr(z, 27)) * signed(0x94D049BB133111EB)
    return z ^ shr(z, 31)


def _exact_cloud(case, seed, dev):
    scn = _cloud(case, seed)
    t = scn["tanks"][0]
    n, dim = case["n"], scn["dim"]
    r = torch.from_numpy(np.ascontiguousarray(scn["r"])).to(dev)
    f32 = case["form"] == "f32"
    if f32:  # the positions are rounded once; so is the radius
        r = r.float().double()
    R = {1: 2.5, 2: 3.0}.get(case["kernel"], 2.0) * t["h"]
    tank = torch.zeros(n, dtype=torch.long, device=dev)
    one = torch.full((1,), R, dtype=torch.float64, device=dev)
    pairs = _Pairs(r, tank, one, one * one)
    w = _WEIGHT[case["kernel"]][dim - 2] / t["h"] ** dim
    rho = torch.zeros(n, dtype=torch.float64, device=dev)
    counts = torch.zeros(n, dtype=torch.int32, device=dev)
    hashes = torch.zeros(n, dtype=torch.long, device=dev)
    for a, b, _, s2 in pairs.each(torch.arange(n, device=dev)):
        rho.index_add_(0, a, t["m"] * w * _kernel(case["kernel"], s2.sqrt() / t["h"])[0])
        if not f32:
            counts.index_add_(0, a, torch.ones_like(a, dtype=torch.int32))
            hashes.index_add_(0, a, _splitmix(b + 1))
    # The FP32 predicate decides pairs at the radius by FP32 rounding.
    return dict(rho=rho, counts=None if f32 else counts, hashes=None if f32 else hashes)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] in ("cloud3d", "noalloc"):
        return _exact_cloud(case, seed, dev)
    if case["shifting"] or case["kind"] == "pool2d":
        return None  # shifting decides by exact comparisons, faces by closed forms
    scn, r, v, rho, dv = _particles(case, seed)
    P, d, K = _params(case, scn["dim"]), scn["dim"], case["kernel"]
    ten = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    r, v, rho, dv = ten(r), ten(v), ten(rho), ten(dv)
    sizes = [t["n_fluid"] + t["n_wall"] for t in scn["tanks"]]
    tank = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(dev)
    wall = torch.cat([torch.arange(t["n_fluid"] + t["n_wall"]) >= t["n_fluid"]
                      for t in scn["tanks"]]).to(dev)
    per = {k: ten(np.array([t[k] for t in scn["tanks"]])) for k in ("h", "m", "rho0", "cs0")}
    h, m, rho0, cs0 = (per[k][tank] for k in ("h", "m", "rho0", "cs0"))
    radius = {1: 2.5, 2: 3.0}.get(K, 2.0) * per["h"]
    w = _WEIGHT[K][d - 2] / per["h"] ** d
    fluid, walls = (~wall).nonzero()[:, 0], wall.nonzero()[:, 0]

    def extrapolate(r, rho, pairs):
        S, H = torch.zeros_like(rho), torch.zeros_like(rho)
        pot = cs0 * cs0 * ((rho / rho0) ** (P.xi - 1.0) - 1.0) / (P.xi - 1.0)
        for a, b, _, s2 in pairs.each(walls):
            ok = ~wall[b]
            a, b, s2 = a[ok], b[ok], s2[ok]
            VW = m[b] / rho[b] * w[tank[a]] * _kernel(K, s2.sqrt() / h[a])[0]
            S.index_add_(0, a, VW)
            H.index_add_(0, a, VW * pot[b])
        Hs = torch.where(S.abs() <= 6.0554544523933395e-06, torch.zeros_like(S), H / S)
        e = rho0 * (1.0 + (P.xi - 1.0) * Hs / (cs0 * cs0)) ** (1.0 / (P.xi - 1.0))
        return torch.where(wall, e, rho)

    def sums(r, v, rho):
        pairs = _Pairs(r, tank, radius, radius * radius)
        rho = extrapolate(r, rho, pairs)
        x = rho / rho0
        p, c = rho0 * cs0 * cs0 / P.xi * (x ** P.xi - 1.0), cs0 * x ** (0.5 * (P.xi - 1.0))
        drho, acc = torch.zeros_like(rho), torch.zeros_like(r)
        for a, b, rab, s2 in pairs.each(fluid):
            ok = a != b
            a, b, rab, s2 = a[ok], b[ok], rab[ok], s2[ok]
            dist = s2.sqrt()
            F = w[tank[a]] / h[a] * _kernel(K, dist / h[a])[1] / dist
            vd = ((v[a] - v[b]) * rab).sum(1)
            if P.diffusion == _abi.TG_DIFF_FERRARI:
                D = torch.maximum(c[a], c[b]) * (rho[a] - rho[b]) * dist / rho[b]
            else:
                D = 2.0 * P.delta * h[a] * cs0[a] * (rho[a] - rho[b]) / rho[b]
            drho.index_add_(0, a, m[b] * F * (vd + D))
            if P.viscosity == _abi.TG_VISC_MORRIS:
                Pi = 2.0 * P.mu * vd / (rho[a] * rho[b] * s2)
            else:
                Pi = torch.where(vd < 0.0, P.alpha * h[a] * (c[a] + c[b]) * vd /
                                 ((s2 + 0.01 * h[a] * h[a]) * (rho[a] + rho[b])),
                                 torch.zeros_like(vd))
            coef = m[b] * F * (Pi - p[a] / rho[a] ** 2 - p[b] / rho[b] ** 2)
            acc.index_add_(0, a, coef[:, None] * rab)
        acc[fluid, 1] -= P.g
        return rho, c, drho, acc

    for _ in range(case["steps"]):
        c = cs0 * (rho / rho0) ** (0.5 * (P.xi - 1.0))
        lim = torch.minimum(P.cfl * h / (c + v.norm(dim=1)),
                            P.c_force * (h / dv.norm(dim=1).clamp_min(P.g)).sqrt())
        if P.mu > 0.0:
            lim = torch.minimum(lim, P.c_visc * h * h * rho / P.mu)
        dt = torch.full((len(sizes),), math.inf, dtype=torch.float64, device=dev)
        dt.scatter_reduce_(0, tank[fluid], lim[fluid], "amin")
        step = dt[tank]
        r0, v0, rho_0 = r, v, rho
        for weight in (1.0, 0.25, 2.0 / 3.0):
            rho_e, _, drho, dv = sums(r, v, rho)
            mix = lambda old, new: (1.0 - weight) * old + weight * new  # noqa: E731
            r, v = mix(r0, r + step[:, None] * v), mix(v0, v + step[:, None] * dv)
            rho = torch.where(wall, rho_e, mix(rho_0, rho + step * drho))
    rho = extrapolate(r, rho, _Pairs(r, tank, radius, radius * radius))
    if case["form"] == "f64":
        return dict(r=r, v=v, rho=rho, dv=dv, dt=dt)
    return dict(r=r, v=v, drho=rho - RHO0, dv=dv, dt=dt)
