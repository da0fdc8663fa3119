"""Workloads of the time step, through the public entry points of awp_b200.

Each case is one call a user's program makes again and again: some time steps
of a simulation (``Solver.step``, ``Mesh.step``, ``Batch.step``) from a
wavefield that is under way, with the surface output where the program writes
it, or one misfit gradient (``adjoint.misfit`` and its backward pass).  Grids,
media, sources and options follow awp_b200/scenarios.py and bench.py: the
elastic half-space, the anelastic 1-D gradient with smooth perturbations, the
hill, the two-block mesh with plasticity, the ensemble of uneven grids and the
misfit gradient; odd sizes stand beside the round ones.

``exact`` restates the step in float64 with plain torch operations on the
float32 model arrays (material arrays, sponge, relaxation and metric tables
are inputs of the step and carry their float32 rounding).
"""
import math
import os
import tempfile

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from awp_b200 import Solver, adjoint, default_params
from awp_b200.solver import Batch, Mesh

DEV = "cuda"
VP_MAX = 6300.0
FIELDS9 = ("u1", "v1", "w1", "xx", "yy", "zz", "xy", "xz", "yz")
FIELDS15 = FIELDS9 + ("r1", "r2", "r3", "r4", "r5", "r6")
NST = 4096  # source samples (the moment rate stays active over the timed passes)


def listed():
    return [
        # a small verification run: launches and latency are all there is
        dict(name="shot_48", kind="grid", nx=48, ny=40, nz=36, steps=10, q=True, fault=False,
             gather=False),
        # the elastic homogeneous half-space with its surface written after the steps
        dict(name="halfspace_128", kind="grid", nx=128, ny=128, nz=128, steps=10, q=False,
             fault=False, gather=True),
        # an anelastic shot on a grid whose sizes divide nothing
        dict(name="ragged_301", kind="grid", nx=301, ny=223, nz=108, steps=5, q=True, fault=False,
             gather=True),
        # the production size: anelastic, 200 kinematic subfaults
        dict(name="layered_512", kind="grid", nx=512, ny=512, nz=256, steps=2, q=True, fault=True,
             gather=False),
        # curvilinear top grid, anelastic
        dict(name="hill_384", kind="hill", nx=384, ny=384, nz=160, steps=2, q=True),
        # curvilinear top grid, elastic, odd sizes
        dict(name="hill_151", kind="hill", nx=151, ny=131, nz=68, steps=4, q=False),
        # Drucker-Prager plasticity on one grid
        dict(name="plastic_240", kind="plastic", nx=240, ny=237, nz=120, steps=3, q=True),
        # topography + mesh + plasticity + attenuation (the fine block over a 3x coarser one)
        dict(name="mesh_hill_plastic", kind="mesh", nx=100, ny=100, nz=96, nzc=48, steps=3,
             hill=True, plastic=True),
        # a plain two-block mesh, odd sizes
        dict(name="mesh_53", kind="mesh", nx=53, ny=41, nz=60, nzc=36, steps=5, hill=False,
             plastic=False),
        # an ensemble of uneven grids advanced together, as the library starts it ...
        dict(name="ensemble", kind="ensemble", n=21, lo=64, hi=192, steps=2, mode=0, draw=6),
        # ... and as a graph of each instance's own launches
        dict(name="ensemble_graph", kind="ensemble", n=21, lo=64, hi=192, steps=2, mode=1, draw=7),
        # misfit gradient of a shot, model and gradients on the device
        dict(name="gradient_160", kind="gradient", nx=160, ny=144, nz=96, steps=40, q=True,
             nrec=48, nsnap=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("grid", "grid", "grid", "hill", "plastic", "mesh", "ensemble", "gradient"))
    if kind == "grid":
        nx, ny, nz = _log(rng, 24, 512), _log(rng, 24, 512), 4 * _log(rng, 8, 64)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=2 if nx * ny * nz > 3e7 else 6,
                    q=rng.random() < 0.7, fault=rng.random() < 0.4, gather=rng.random() < 0.5)
    if kind == "hill":
        return dict(kind=kind, nx=_log(rng, 32, 400), ny=_log(rng, 32, 400),
                    nz=4 * _log(rng, 8, 48), steps=2, q=rng.random() < 0.7)
    if kind == "plastic":
        return dict(kind=kind, nx=_log(rng, 40, 256), ny=_log(rng, 40, 256),
                    nz=4 * _log(rng, 8, 36), steps=3, q=rng.random() < 0.8)
    if kind == "mesh":
        return dict(kind=kind, nx=_log(rng, 20, 100), ny=_log(rng, 20, 100),
                    nz=4 * _log(rng, 8, 24), nzc=4 * _log(rng, 6, 16), steps=3,
                    hill=rng.random() < 0.5, plastic=rng.random() < 0.5)
    if kind == "ensemble":
        lo = _log(rng, 40, 80)
        return dict(kind=kind, n=rng.randint(2, 21), lo=lo, hi=lo + _log(rng, 30, 120), steps=2,
                    mode=rng.randint(0, 1), draw=rng.randrange(1 << 20))
    return dict(kind=kind, nx=_log(rng, 32, 160), ny=_log(rng, 32, 144), nz=4 * _log(rng, 8, 24),
                steps=rng.randint(12, 40), q=rng.random() < 0.6, nrec=rng.randint(4, 64),
                nsnap=rng.choice((0, 0, 5)))


# --------------------------------------------------------------------------
# inputs, from the seed alone
# --------------------------------------------------------------------------
def _noise(gen, shape, cells=8):
    """Smooth noise of about unit size: a coarse normal grid, interpolated."""
    c, n = shape[0], shape[1:]
    coarse = torch.randn((1, c) + tuple(max(2, m // cells + 2) for m in n), generator=gen,
                         device=DEV)
    return F.interpolate(coarse, size=n, mode="trilinear", align_corners=True)[0]


def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)


def _media(nx, ny, nz, q, seed, salt, z0=0.0, z1=1.0):
    """[nz][ny][nx][5] vp, vs, rho, Qp, Qs, surface first: the anelastic 1-D
    gradient with perturbations, or the elastic half-space (Q <= 0)."""
    if not q:
        m = torch.empty((nz, ny, nx, 5), device=DEV)
        for k, v in enumerate((6000.0, 3464.0, 2700.0, 0.0, 0.0)):
            m[..., k] = v
        # a half-space of its own for each seed
        m[..., :2] *= 0.95 + 0.05 * float(torch.rand((), generator=_gen(seed, salt + 7),
                                                      device=DEV))
        return m
    depth = z0 + (z1 - z0) * (torch.arange(nz, device=DEV) + 0.5) / nz
    pert = (0.05 * _noise(_gen(seed, salt), (1, nz, ny, nx))[0]).clamp_(-0.15, 0.15)
    vs = (1000.0 + 2500.0 * depth)[:, None, None] * (1.0 + pert)
    vp = (1.73 * vs).clamp(max=VP_MAX)
    vs = vp / 1.73
    qs = 0.05 * vs
    # sediments below Qp 190 over a basement above 400: both branches of the
    # Q(f) weight, with no cell at its switch (Q 200), where one rounding
    # would pick the other branch
    qp = torch.where(depth[:, None, None] < 0.5, (2.0 * qs).clamp(max=190.0),
                     (2.0 * qs).clamp(min=400.0))
    return torch.stack([vp, vs, 310.0 * vp ** 0.25, qp, qs], -1).contiguous()


def _wavefield(nx, ny, nz, seed, salt):
    """A wavefield under way: nine smooth interior fields [9][nx][ny][nz] (k up),
    the stresses sized to the velocities by an impedance."""
    f = _noise(_gen(seed, salt), (9, nx, ny, nz))
    f[:3] *= 0.1
    f[3:] *= 7.0e5
    f[7, :, :, -1] = 0.0  # xz, yz vanish at the free surface
    f[8, :, :, -1] = 0.0
    return f


def _place(get, f, nx, ny, nz, surface):
    """Put the interior fields into padded arrays, with the stress images
    above a free surface."""
    for name, x in zip(FIELDS9, f):
        a = get(name)
        a[10:nx + 10, 10:ny + 10, 32:nz + 32] = x.to(a.dtype)
        if surface and name in ("zz", "xz", "yz"):
            t = nz + 31 if name == "zz" else nz + 30
            a[:, :, nz + 32] = -a[:, :, t]
            a[:, :, nz + 33] = -a[:, :, t - 1]


def _sources(nx, ny, nz, fault, seed, salt, dt, h, n=3, near_surface=False):
    """INSRC positions (1-based, z from the surface) and samples."""
    g = np.random.default_rng((int(seed), salt))
    if fault:
        ns = 200
        pos = np.stack([np.full(ns, nx // 2), g.integers(ny // 4, 3 * ny // 4, ns),
                        g.integers(max(3, nz // 16), nz // 2, ns)], 1)
        _, keep = np.unique(pos, axis=0, return_index=True)
        pos = pos[np.sort(keep)].astype(np.int32)
        ns = len(pos)
        data = np.zeros((ns, 2, 6), np.float32)
        data[:, 0, 0] = 1.0
        data[:, 0, 1] = g.uniform(0.5, 1.5, ns)
        data[:, 0, 2] = 0.0
        data[:, 0, 3] = g.uniform(0.3, 1.0, ns)
        data[:, 0, 4] = h * h
        data[:, 1, 0] = g.uniform(-10, 10, ns)
        data[:, 1, 1] = 90.0
        data[:, 1, 2] = 180.0 + g.uniform(-15, 15, ns)
        return pos, data
    hi = max(4, nz // 8) if near_surface else nz - 4
    pos = np.stack([g.integers(nx // 4, 3 * nx // 4 + 1, n), g.integers(ny // 4, 3 * ny // 4 + 1, n),
                    g.integers(2, hi, n)], 1).astype(np.int32)
    pos = pos + np.arange(n, dtype=np.int32)[:, None] * np.array([1, 0, 0], np.int32)
    t = (np.arange(NST) + 1) * dt
    f0 = 2.0 if not near_surface else 0.06 / dt
    data = (1e14 * g.standard_normal((n, 1, 6)) * np.sin(2 * np.pi * f0 * t)[None, :, None])
    return pos, data.astype(np.float32)


def _params(nx, ny, nz, h, dt, fault=False, **kw):
    n = 2 if fault else NST
    return dict(dict(nx=nx, ny=ny, nz=nz, dh=h, dt=dt, nd=min(20, nx // 4, ny // 4), arbc=0.92,
                     npc=0, nve=1, ifault=5 if fault else 1, nst=n, read_step=n, socalq=1), **kw)


def _dt(h):
    return float(np.float32(0.44 * h / VP_MAX))


class _Ptr:
    """A field's device memory; the tensor made of it keeps the solver alive."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f4",
                                             data=(int(ptr), False), version=3)


def _view(solver, name):
    """A field of a solver as a torch tensor over its own memory."""
    return torch.as_tensor(_Ptr(solver, solver.device_ptr(name), solver.shape), device=DEV)


def _elevation(nx, ny, h, seed):
    """A Gaussian hill with smooth roughness, [nx + 16][ny + 16] metres."""
    g = np.random.default_rng((int(seed), 77))
    x = (np.arange(nx + 16) - 8) * h
    y = (np.arange(ny + 16) - 8) * h
    X, Y = np.meshgrid(x, y, indexing="ij")
    width = 0.2 * min(nx, ny) * h
    e = 20 * h * np.exp(-((X - x.mean()) ** 2 + (Y - y.mean()) ** 2) / (2 * width ** 2))
    n = g.standard_normal(X.shape)
    for _ in range(3):
        n = (n + np.roll(n, 1, 0) + np.roll(n, -1, 0) + np.roll(n, 1, 1) + np.roll(n, -1, 1)) / 5
    return (e + 0.5 * h * n / n.std()).astype(np.float32)


def _write_elevation(elev, nx, ny):
    fd, path = tempfile.mkstemp(suffix=".topo")
    with os.fdopen(fd, "wb") as f:
        np.asarray([nx, ny, 8], np.int32).tofile(f)
        elev.tofile(f)
    return path


def _yield_inputs(nx, ny, nz, h, seed, salt):
    """Padded sigma2 (lithostatic), cohesion and friction angle; about a third
    of the cells at yield under the wavefield above."""
    k = torch.arange(nz + 64, device=DEV)
    depth = (nz + 31 - k).clamp(min=0) * h + 0.5 * h
    g = _noise(_gen(seed, salt), (2, nx + 20, ny + 20, nz + 64))
    s2 = (-2300.0 * 9.81 * depth)[None, None, :] * (1.0 + 0.05 * g[0])
    co = 6.0e5 * torch.exp(0.5 * g[1])
    phi = torch.full_like(co, 30.0) + 3.0 * g[0]
    return s2.contiguous(), co.contiguous(), phi.contiguous()


YIELD = dict(fmajor=1.25, fminor=0.75, strike=[40.0, 310.0, 40.0], dip=[0.0, 0.0, 90.0])


def _ensemble_sizes(case):
    g = np.random.default_rng(int(case["draw"]))
    out = []
    for _ in range(case["n"]):
        nx, ny = (int(g.integers(case["lo"], case["hi"] + 1)) for _ in range(2))
        nz = 4 * int(g.integers(case["lo"] // 4, case["hi"] // 6 + 1)) if case["hi"] // 6 >= \
            case["lo"] // 4 else 4 * (case["lo"] // 4)
        out.append((nx, ny, nz))
    return out


def _blocks(case):
    """The blocks of a mesh case, finest first: nx, ny, nz, h, depth range."""
    h = 40.0
    total = case["nz"] * h + case["nzc"] * 3 * h
    cut = case["nz"] * h / total
    return [(3 * case["nx"], 3 * case["ny"], case["nz"], h, 0.0, cut),
            (case["nx"], case["ny"], case["nzc"], 3 * h, cut, 1.0)]


def _one(nx, ny, nz, h, dt, q, seed, salt, fault=False, n=3, **kw):
    """A solver with media, sources and a wavefield under way."""
    s = Solver(default_params(**_params(nx, ny, nz, h, dt, fault, **kw)))
    m = _media(nx, ny, nz, q, seed, salt)
    torch.cuda.current_stream().synchronize()
    s.upload_media_device(m.data_ptr(), 5)
    s.upload_sources(*_sources(nx, ny, nz, fault, seed, salt, dt, h, n))
    _place(lambda f: _view(s, f), _wavefield(nx, ny, nz, seed, salt + 1), nx, ny, nz, True)
    return s


def prepare(case, seed):
    kind, h = case["kind"], 50.0
    dt = _dt(h)
    st = dict(case=case)
    if kind in ("grid", "hill", "plastic"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        s = _one(nx, ny, nz, h, dt, case["q"], seed, 0, case.get("fault", False),
                 nve=3 if kind == "plastic" else 1)
        if kind == "hill":
            path = _write_elevation(_elevation(nx, ny, h, seed), nx, ny)
            s.topography(path)
            os.unlink(path)
        if kind == "plastic":
            s2, co, phi = (x.cpu().numpy() for x in _yield_inputs(nx, ny, nz, h, seed, 3))
            s.upload_plasticity(s2, co, phi, **YIELD)
        names = FIELDS15 if case["q"] else FIELDS9
        if kind == "plastic":
            names = names + ("yldfac", "neta")
        st.update(solver=s, out={f: _view(s, f) for f in names})
        if case.get("gather"):
            st["frame"] = torch.zeros((3, ny, nx), device=DEV)
            st["out"]["frame"] = st["frame"]
    elif kind == "mesh":
        dt = _dt(40.0)
        nve = 3 if case["plastic"] else 1
        bl = _blocks(case)
        mesh = Mesh([default_params(**_params(b[0], b[1], b[2], b[3], dt, nve=nve, grid=p,
                                              ngrids=2, nd=(18 if p == 0 else 6)))
                     for p, b in enumerate(bl)])
        out = {}
        for p, (nx, ny, nz, hp, z0, z1) in enumerate(bl):
            g = mesh.grid(p)
            m = _media(nx, ny, nz, True, seed, 10 * p, z0, z1)
            torch.cuda.current_stream().synchronize()
            g.upload_media_device(m.data_ptr(), 5)
            if p == 0:
                g.upload_sources(*_sources(nx, ny, nz, False, seed, 0, dt, hp))
                if case["hill"]:
                    path = _write_elevation(_elevation(nx, ny, hp, seed), nx, ny)
                    g.topography(path)
                    os.unlink(path)
                    g.set_topo_plasticity(True)
            if nve == 3:
                s2, co, phi = (x.cpu().numpy()
                               for x in _yield_inputs(nx, ny, nz, hp, seed, 10 * p + 3))
                g.upload_plasticity(s2, co, phi, **YIELD)
            _place(lambda f: _view(g, f), _wavefield(nx, ny, nz, seed, 10 * p + 1), nx, ny, nz,
                   p == 0)
            for f in FIELDS15 + (("yldfac", "neta") if nve == 3 else ()):
                out[f"{f}_{p}"] = _view(g, f)
        st.update(mesh=mesh, out=out)
    elif kind == "ensemble":
        h = 100.0
        dt = _dt(h)
        st["solvers"] = [_one(nx, ny, nz, h, dt, True, seed, 100 * i, n=1)
                         for i, (nx, ny, nz) in enumerate(_ensemble_sizes(case))]
        torch.cuda.synchronize()
        st["batch"] = Batch(st["solvers"])
        st["batch"].set_mode(case["mode"])
        st["out"] = [[_view(s, f) for f in FIELDS9[:3]] for s in st["solvers"]]
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        s = Solver(default_params(**_params(nx, ny, nz, h, dt)))
        m = _media(nx, ny, nz, case["q"], seed, 0)
        torch.cuda.current_stream().synchronize()
        s.upload_media_device(m.data_ptr(), 5)
        s.upload_sources(*_sources(nx, ny, nz, False, seed, 0, dt, h, near_surface=True))
        xyz, comp, obs = _receivers(case, seed, dt)
        adjoint.adjoint_reserve(s, case["steps"], case["nsnap"])
        st.update(solver=s, model=[x.requires_grad_() for x in _moduli(case, seed)], xyz=xyz,
                  comp=comp, obs=obs, final=[_view(s, f) for f in FIELDS9])
    torch.cuda.synchronize()
    return st


def _moduli(case, seed):
    """lambda, mu, rho [nz][ny][nx] of the model the gradient is taken at."""
    m = _media(case["nx"], case["ny"], case["nz"], True, seed, 5).double()
    vp, vs, rho = m[..., 0], m[..., 1], m[..., 2]
    return [x.float().contiguous() for x in (rho * (vp * vp - 2 * vs * vs), rho * vs * vs, rho)]


def _receivers(case, seed, dt):
    g = np.random.default_rng((int(seed), 5))
    nx, ny, n = case["nx"], case["ny"], case["nrec"]
    xyz = np.stack([g.integers(nx // 4, 3 * nx // 4, n), g.integers(ny // 4, 3 * ny // 4, n),
                    np.zeros(n, np.int64)], 1).astype(np.int32)
    comp = g.integers(0, 3, n).astype(np.int32)
    t = np.arange(1, case["steps"] + 1) * dt
    obs = 1e-3 * g.standard_normal((1, n)) * np.sin(2 * np.pi * 0.05 / dt * t)[:, None]
    return xyz, comp, obs.astype(np.float32)


def run(st):
    case = st["case"]
    kind, n = case["kind"], case["steps"]
    if kind == "gradient":
        J = adjoint.misfit(*st["model"], st["solver"], n, st["xyz"], st["comp"], st["obs"],
                           case["nsnap"])
        return {"misfit": J.detach(), "grad": list(torch.autograd.grad(J, st["model"])),
                "final": st["final"]}
    if kind == "mesh":
        st["mesh"].step(n)
    elif kind == "ensemble":
        st["batch"].step(n)
    else:
        st["solver"].step(n)
        if "frame" in st:
            b = st["frame"]
            st["solver"].gather(0, case["nx"] - 1, 1, 0, case["ny"] - 1, 1, 0, 0, 1,
                                *(b[q].data_ptr() for q in range(3)))
    return st["out"]


# Bytes a step cannot do without, per cell: each state field read and written
# once, each material read once (elastic 9 + 3, anelastic 15 + 5 float32); the
# plasticity inputs sigma2, cohesion, angle and the yield factor written; the
# flops are those of the update formulas.
def work(case):
    kind, n = case["kind"], case["steps"]
    if kind == "ensemble":
        cells = sum(a * b * c for a, b, c in _ensemble_sizes(case))
        return dict(bytes=140.0 * cells * n, flops=310.0 * cells * n)
    if kind == "mesh":
        cells = sum(b[0] * b[1] * b[2] for b in _blocks(case))
        return dict(bytes=(156.0 if case["plastic"] else 140.0) * cells * n,
                    flops=(560.0 if case["hill"] else 310.0) * cells * n)
    cells = case["nx"] * case["ny"] * case["nz"]
    per = 140.0 if case["q"] else 84.0
    flops = 310.0 if case["q"] else 150.0
    if kind == "plastic":
        per, flops = per + 16.0, flops + 150.0
    if kind == "hill":
        flops += 250.0
    if kind == "gradient":
        # forward step, velocities stored and read back; adjoint state as the
        # forward one
        per, flops = 2 * per + 24.0, 3 * flops
    extra = 24.0 * cells if kind == "gradient" else 0.0
    return dict(bytes=per * cells * n + extra, flops=flops * cells * n)


def tolerance(case):
    if case["kind"] == "gradient":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "plastic" or case.get("plastic"):
        return {"rel": 1e-5, "max": 1e-2}
    return {"rel": 5e-6, "max": 2e-4}


# --------------------------------------------------------------------------
# the step in 64 bits
# --------------------------------------------------------------------------
C1, C2 = 9.0 / 8.0, -1.0 / 24.0
C2 = float(np.float32(C2))


def _f32(x):
    return x.float().double()


# EX = 0: eight relaxation times, weights and the Q(f) polynomial
_W8 = [0.8867, 1.0440, 0.0423, 0.8110, 1.7275, 0.5615, 0.8323, 0.4641]
_C16 = [-27.5089, 7.4177, -82.8803, 13.1952, 72.0312, 0.5298, -34.1779, 6.0293,
        -52.2607, 8.1754, -1.6270, 4.6858, -27.7770, 6.2852, 14.6295, 3.8839]
_ORDER = [0, 4, 2, 6, 1, 5, 3, 7]


def _relaxation(dt):
    """tau, vx1, vx2, wwo [8] and the polynomial [8][2]."""
    f = np.float32
    fac = f(0.005)
    pi = f(4.0 * math.atan(1.0))
    twopi = f(2) * pi
    tmax = f(1.0 / (float(twopi) * 0.01) * 1.0 * float(fac))
    tmin = f(1.0 / (float(twopi) * 10.0) * 0.2 * float(fac))
    prod, ratio = f(tmax * tmin), f(tmax / tmin)
    tau = np.zeros(8, np.float32)
    w = np.zeros(8, np.float32)
    for n, e in enumerate([1, 6, 7, 4, 8, 3, 2, 5]):
        t = f(2.0 * float(f((e - 0.5) / 8.0)) - 1.0)
        tau[_ORDER[n]] = f(math.exp(0.5 * (math.log(prod) + math.log(ratio) * float(t))))
        w[_ORDER[n]] = f(_W8[n])
    v2 = np.array([f(math.exp(float(f(-f(dt) / t)))) for t in tau], np.float32)
    v1 = np.array([f(0.5 * (1.0 - float(x))) for x in v2], np.float32)
    wwo = np.array([f(8.0 * float(x)) for x in w], np.float32)
    c = np.array(_C16, np.float32).reshape(8, 2)
    return tau, w, v1, v2, wwo, c


def _modulus(dd, v, q, tau, w, c, w0):
    """Unrelaxed modulus of one wave type (float64)."""
    m = dd * v * v
    hiq = torch.zeros_like(q)
    acc = torch.zeros(q.shape, dtype=torch.complex128, device=DEV)
    qq = q.clamp(min=1e-30)
    for t in range(8):
        wt = float(w0) * float(tau[t])
        hiq += float(w[t]) / ((wt * wt + 1.0) * qq)
        wl = float(c[t, 0]) / (qq * qq) + float(c[t, 1]) / qq
        acc += 1.0 / (1.0 - wl / complex(1.0, wt))
    low = m / (8.0 * (1.0 / acc).real)
    return torch.where(q > 200.0, m / (1.0 - hiq), torch.where(q > 0, low, m))


def _up(x, nx, ny, nz):
    """[nz][ny][nx], surface first -> [nx][ny][nz], k up."""
    return x.permute(2, 1, 0).flip(2)


class _X:
    """One grid in 64 bits: padded [nx + 20][ny + 20][nz + 64] arrays."""

    def __init__(self, nx, ny, nz, h, dt, q, seed, salt, z=(0.0, 1.0), grid=0, ngrids=1, fault=False,
                 nsrc=3, nd=None, nve=1, wave=True, near_surface=False, sources=True, model=None):
        self.n = (nx, ny, nz)
        self.grid, self.ngrids, self.q, self.nve = grid, ngrids, q, nve
        self.h, self.dt = float(np.float32(h)), float(np.float32(dt))
        self.dth = float(np.float32(np.float32(dt) / np.float32(h)))
        self.dh1 = float(np.float32(1.0 / h))
        self.shape = (nx + 20, ny + 20, nz + 64)
        self.S = {f: self.zeros() for f in FIELDS15}
        self.step_n, self.fault = 0, fault
        nd = min(20, nx // 4, ny // 4) if nd is None else nd
        alpha = np.float32(math.sqrt(-math.log(np.float32(0.92))) / nd)
        self.dcr = []
        for n, lo, hi, off in ((nx, 1, 1, 10), (ny, 1, 1, 10), (nz, grid == ngrids - 1, 0, 32)):
            c = np.ones(n + 2 * off, np.float32)
            for i in range(nd):
                x = np.float32(alpha * np.float32(nd - i))
                e = math.exp(-float(np.float32(x * x)))
                if lo:
                    c[off + i] = np.float32(c[off + i] * e)
                if hi:
                    c[off + n - 1 - i] = np.float32(c[off + n - 1 - i] * e)
            self.dcr.append(torch.tensor(c, dtype=torch.float64, device=DEV))
        self.tau, self.w8, v1, v2, wwo, c = _relaxation(self.dt)
        t8 = lambda a: torch.tensor(a.astype(np.float64), device=DEV)  # noqa: E731
        self.v1, self.v2, self.wwo, self.cc = t8(v1), t8(v2), t8(wwo), t8(c)
        med = _media(nx, ny, nz, q, seed, salt, *z).double()
        w0 = float(np.float32(2) * np.float32(math.pi) * np.float32(2.5))
        vp, vs, dd, qp, qs = (med[..., k] for k in range(5))
        vp, vs = (_f32(torch.sqrt(_modulus(dd, v, a, self.tau, self.w8, c, w0) / dd))
                  for v, a in ((vp, qp), (vs, qs)))
        vs = torch.where(vp / vs < 1.45, _f32(vp / 1.45), vs)
        self.fx = None  # window of a finer grid above (set by a mesh)
        lam, mu = dd * (vp * vp - 2 * vs * vs), dd * vs * vs
        iq = lambda a: torch.where(a > 0, 1.0 / a.clamp(min=1e-30), torch.zeros_like(a))  # noqa: E731
        self.M = {}
        self.set_moduli(lam, mu, dd)
        for f, a in (("qp", qp), ("qs", qs)):
            p = self.zeros()
            p[10:nx + 10, 10:ny + 10, 32:nz + 32] = _f32(_up(iq(a), nx, ny, nz))
            p[10:nx + 10, 10:ny + 10, nz + 32] = p[10:nx + 10, 10:ny + 10, nz + 31]
            self.M[f] = p
        self.src = _sources(nx, ny, nz, fault, seed, salt, dt, h, nsrc, near_surface) if sources \
            else None
        if wave:
            _place(lambda f: self.S[f], _wavefield(nx, ny, nz, seed, salt + 1), nx, ny, nz,
                   grid == 0)
        self.topo = None

    def zeros(self):
        return torch.zeros(self.shape, dtype=torch.float64, device=DEV)

    def set_moduli(self, lam, mu, rho):
        """Kernel arrays 1/lambda, 1/mu, rho with their one-cell border."""
        nx, ny, nz = self.n
        for f, x in (("lam", 1.0 / lam), ("mu", 1.0 / mu), ("d1", rho)):
            x = _up(x + (_f32(x) - x).detach(), nx, ny, nz)
            x = F.pad(x[None, None], (1,) * 6, mode="replicate")[0, 0]
            self.M[f] = F.pad(x, (31, 31, 9, 9, 9, 9))
        t = nz + 31
        il, im = 1.0 / self.M["lam"][10:nx + 10, 10:ny + 10, t], \
            1.0 / self.M["mu"][10:nx + 10, 10:ny + 10, t]
        r = il / (2 * im + il)
        self.lam_mu = r + (_f32(r) - r).detach()

    # views and window updates (inclusive windows i0, i1, j0, j1, k0, k1)
    def g(self, f, w, di=0, dj=0, dk=0):
        return f[w[0] + di:w[1] + 1 + di, w[2] + dj:w[3] + 1 + dj, w[4] + dk:w[5] + 1 + dk]

    def put(self, name, w, val):
        f = self.S[name]
        if torch.is_grad_enabled():
            f = f.clone()
            self.S[name] = f
        f[w[0]:w[1] + 1, w[2]:w[3] + 1, w[4]:w[5] + 1] = val

    def sponge(self, w):
        x, y, z = self.dcr
        return (x[w[0]:w[1] + 1, None, None] * y[None, w[2]:w[3] + 1, None] *
                z[None, None, w[4]:w[5] + 1])

    def table(self, w):
        """Relaxation entry of each cell of the window (parity pattern)."""
        nx, ny, nz = self.n

        def base(di, dj, nyy, nzz, kk):
            pd = di & 1
            pij = ((pd & nyy) + (dj & 1) + 1) & 1
            return 4 * (pd ^ 1) + 2 * pij + (((nzz & pij) + kk) & 1)
        i = torch.arange(w[0], w[1] + 1, device=DEV)[:, None, None]
        j = torch.arange(w[2], w[3] + 1, device=DEV)[None, :, None]
        k = torch.arange(w[4], w[5] + 1, device=DEV)[None, None, :]
        t = base(i - 10, j - 10, ny, nz, k - 32)
        if self.fx:
            lev = k - (32 + nz - 3)
            f = base(3 * (i - 10), 3 * (j - 10) + 1, self.fx[1], self.fx[2], 1 + 3 * lev)
            inside = (lev >= 0) & (lev < 3) & (i >= 10) & (i < 10 + nx) & (j >= 10) & (j < 10 + ny)
            t = torch.where(inside, f, t.expand_as(f))
        return t

    def velocity(self):
        if self.topo:
            return self.topo_velocity()
        nx, ny, nz = self.n
        w = (10, nx + 9, 10, 9 + ny + ny % 2, 35 if self.grid < self.ngrids - 1 else 32, nz + 31)
        if self.grid > 0:
            w = w[:5] + (nz + 29,)
        S, g, d = self.S, self.g, self.M["d1"]

        def d4(f, p, m, ax):  # c1 (f[p] - f[p-1]) + c2 (f[p+1] - f[p-2]) along ax, p = 0 or 1
            o = lambda n: g(S[f], w, *(n if a == ax else 0 for a in range(3)))  # noqa: E731
            return C1 * (o(p) - o(p - 1)) + C2 * (o(p + 1) - o(p - 2))
        rho = lambda a, b: self.dth / (0.25 * (g(d, w) + g(d, w, *a) + g(d, w, *b) +  # noqa: E731
                                               g(d, w, *(x + y for x, y in zip(a, b)))))
        sp = self.sponge(w)
        new = []
        for f, e, fd in (("u1", (("xx", 0), ("xy", 0), ("xz", 0)), ((0, -1, 0), (0, 0, -1))),
                         ("v1", (("xy", 1), ("yy", 1), ("yz", 0)), ((1, 0, 0), (0, 0, -1))),
                         ("w1", (("xz", 1), ("yz", 0), ("zz", 1)), ((1, 0, 0), (0, -1, 0)))):
            s = sum(d4(x, p, 0, ax) for ax, (x, p) in enumerate(e))
            new.append((f, (g(S[f], w) + rho(*fd) * s) * sp))
        for f, v in new:
            self.put(f, w, v)

    def images(self, w):
        """Velocities on the first level above the surface."""
        nx, ny, nz = self.n
        t = nz + 31
        p = (w[0], w[1], w[2], w[3], t, t)
        u, v, ww = self.S["u1"], self.S["v1"], self.S["w1"]
        g = self.g
        i = torch.arange(p[0], p[1] + 1, device=DEV)[:, None, None]
        j = torch.arange(p[2], p[3] + 1, device=DEV)[None, :, None]
        ui = g(u, p) - (g(ww, p) - g(ww, p, -1))
        vi = g(v, p) - (g(ww, p, 0, 1) - g(ww, p))
        s1 = torch.where(i < nx + 9, g(u, p, 1) - (g(ww, p, 1) - g(ww, p)), 0.0)
        s2 = torch.where(j >= 11, g(v, p, 0, -1) - (g(ww, p) - g(ww, p, 0, -1)), 0.0)
        lm = self.lam_mu[p[0] - 10:p[1] - 9, p[2] - 10:p[3] - 9, None]
        wi = g(ww, p, 0, 0, -1) - lm * (s1 - ui + g(u, p, 1) - g(u, p) + vi - s2 + g(v, p) -
                                        g(v, p, 0, -1))
        q = p[:4] + (t + 1, t + 1)
        for f, x in (("u1", ui), ("v1", vi), ("w1", wi)):
            self.put(f, q, x)

    def window(self):
        nx, ny, nz = self.n
        return (10, nx + 9, 10, ny + 9, 35, nz + 31 if self.grid == 0 else nz + 29)

    def rates(self, w):
        S, g = self.S, self.g

        def d4(f, p, ax):
            o = lambda n: g(S[f], w, *(n if a == ax else 0 for a in range(3)))  # noqa: E731
            return C1 * (o(p) - o(p - 1)) + C2 * (o(p + 1) - o(p - 2))
        return [d4("u1", 1, 0), d4("v1", 0, 1), d4("w1", 0, 2), d4("u1", 1, 1) + d4("v1", 0, 0),
                d4("u1", 1, 2) + d4("w1", 0, 0), d4("v1", 1, 2) + d4("w1", 1, 1)]

    def stress_update(self, w, e, interface=False, dth=None, dt=None):
        """dstrqc of the window from its six strain rates."""
        M, g, dt, dth = self.M, self.g, dt or self.dt, dth or self.dth

        def sum8(m):
            return sum(g(m, w, a, b, c) for a in (0, 1) for b in (0, -1) for c in (0, -1))
        pair = lambda m, *o: g(m, w) + g(m, w, *o)  # noqa: E731
        offs = ((0, 0, -1), (0, -1, 0), (1, 0, 0))
        xm = 16.0 / sum8(M["mu"])
        xl = 8.0 / sum8(M["lam"]) + xm
        xmu = [2.0 / pair(M["mu"], *o) for o in offs]
        sp = self.sponge(w)
        S = self.S
        if not self.q:
            self._write(w, S, e, xl * dth, xm * dth, [x * dth for x in xmu], sp)
            return
        t = self.table(w)
        v1, v2, wo = (a[t] for a in (self.v1, self.v2, self.wwo))
        c0, c1 = self.cc[:, 0][t], self.cc[:, 1][t]

        def weight(q):
            x = 2.0 * q
            return torch.where(x >= 0.005, (c0 * x + c1) * x, (1.0 if interface else 2.0) * wo * q) / wo
        hw = -xm * weight(0.0625 * sum8(M["qs"])) * self.dh1 * v1
        qpa = -weight(0.0625 * sum8(M["qp"])) * xl * self.dh1 * v1
        hh = [-xmu[n] * weight(0.25 * pair(M["qs"], *o)) * self.dh1 * v1 for n, o in enumerate(offs)]
        self._write(w, S, e, xl * dth, xm * dth + dt * hw, [x * dth + dt * y for x, y in zip(xmu, hh)],
                    sp, (hw, qpa, hh, v1, v2, wo, dt))

    def _write(self, w, S, e, xl, xm, xmu, sp, an=None):
        g = self.g
        tr = e[0] + e[1] + e[2]
        if an:
            hw, qpa, hh, v1, v2, wo, dt = an
        for n, f in enumerate(("xx", "yy", "zz", "xy", "xz", "yz")):
            if n < 3:
                inc = xl * tr - xm * (tr - e[n])
                if an:
                    inc = inc + dt * qpa * tr
                    fr = qpa * tr - hw * (tr - e[n])
            else:
                inc = xmu[n - 3] * e[n]
                if an:
                    fr = hh[n - 3] * e[n]
            b = g(S[f], w) + inc
            if an:
                r = g(S["r%d" % (n + 1)], w)
                b = b + dt * (v2 * v1 + 1.0) * r
                if n in (1, 2):
                    b = b * sp
                b = (b + dt * (fr * (wo - 1.0) + v2 * r * (1.0 - v1))) * sp
                self.put("r%d" % (n + 1), w, v2 * r + wo * fr)
            else:
                b = b * sp * (sp if n in (1, 2) else 1.0)
            self.put(f, w, b)

    def middle(self):
        """The band of the stress window that waits for the plasticity phase."""
        nx, ny, _ = self.n
        yl, yr = 10, ny + 9
        a = int(yl + (yr - yl) * 0.25)
        a += a % 2
        b = int(yl + (yr - yl) * 0.75)
        b -= 1 - b % 2
        return 12, nx + 7, max(a, yl + 10), min(b, yr - 10)

    def stress(self):
        if self.topo:
            return self.topo_stress()
        w = self.window()
        if self.nve != 3:
            if self.grid == 0:
                self.images(w)
            self.stress_update(w, self.rates(w))
            return
        i0, i1, j0, j1 = self.middle()
        for b in ((i0, i1, w[2], j0 - 1), (i0, i1, j1 + 1, w[3]), (w[0], i0 - 1, w[2], w[3]),
                  (i1 + 1, w[1], w[2], w[3])):
            self._band(b, w)

    def _band(self, b, w):
        if b[1] < b[0] or b[3] < b[2]:
            return
        b = b + w[4:]
        if self.grid == 0:
            self.images(b)
        self.stress_update(b, self.rates(b))

    def add_sources(self, n):
        if self.src is None or not len(self.src[0]):
            return
        nx, ny, nz = self.n
        pos, data = self.src
        vt = float(np.float32(np.float32(self.dt) / np.float32(
            np.float32(np.float32(self.h) * np.float32(self.h)) * np.float32(self.h))))
        data = data.astype(np.float64)
        for s in range(len(pos)):
            p = (int(pos[s, 0]) + 9, int(pos[s, 1]) + 9, nz + 32 - int(pos[s, 2]))
            w = (p[0], p[0], p[1], p[1], p[2], p[2])
            if not self.fault:
                a = dict(zip(("xx", "yy", "zz", "xz", "yz", "xy"), data[s, n]))
            else:
                typ, slip, rup, rise, area = data[s, 0, :5]
                t = self.step_n * self.dt
                if not t > rup:
                    continue
                om = 2 * math.pi / rise
                f = om * om * (t - rup) * math.exp(-om * (t - rup))
                f *= slip * area / float(self.M["mu"][p])
                st, di, ra = (math.radians(v) for v in data[s, 1, :3])
                sn, cs = math.sin, math.cos
                a = dict(
                    yy=-(sn(di) * cs(ra) * sn(2 * st) + sn(2 * di) * sn(ra) * sn(st) ** 2),
                    xy=sn(di) * cs(ra) * cs(2 * st) + 0.5 * sn(2 * di) * sn(ra) * sn(2 * st),
                    yz=cs(di) * cs(ra) * cs(st) + cs(2 * di) * sn(ra) * sn(st),
                    xx=sn(di) * cs(ra) * sn(2 * st) - sn(2 * di) * sn(ra) * cs(st) ** 2,
                    xz=cs(di) * cs(ra) * sn(st) - cs(2 * di) * sn(ra) * cs(st),
                    zz=sn(2 * di) * sn(ra))
                a = {k: f * v for k, v in a.items()}
            for f, v in a.items():
                self.put(f, w, self.g(self.S[f], w) - vt * float(v))

    def begin(self):
        if self.step_n == 0 and not self.fault:
            self.add_sources(0)
        self.step_n += 1

    def sources(self):
        if self.fault or self.step_n < NST:
            self.add_sources(self.step_n)

    def surface(self):
        """Stress images above the free surface."""
        nx, ny, nz = self.n
        t = nz + 31
        w = lambda k: (10, nx + 9, 10, 9 + ny + ny % 2, k, k)  # noqa: E731
        for f, a in (("zz", t), ("xz", t - 1), ("yz", t - 1)):
            x = [self.g(self.S[f], w(a)), self.g(self.S[f], w(a - 1))]
            self.put(f, w(t + 1), -x[0])
            self.put(f, w(t + 2), -x[1])
        for f in ("xz", "yz"):
            self.put(f, w(t), 0.0)

    # ---- plasticity ------------------------------------------------------
    def set_yield(self, s2, co, phi):
        self.s2, self.co, self.phi = s2.double(), co.double(), phi.double()
        self.S["yldfac"] = torch.ones_like(self.s2)
        self.S["neta"] = self.zeros()
        a, b = (np.radians(np.array(YIELD[k])) for k in ("strike", "dip"))
        R = np.stack([np.cos(a) * np.cos(b), np.sin(a) * np.cos(b), np.sin(b)], 1)
        self.R = R.astype(np.float32).astype(np.float64)
        nx, ny, _ = self.n
        m = torch.zeros((nx + 20, ny + 20), dtype=torch.float64, device=DEV)
        xl, xr, yl, yr = 10, nx + 9, 10, ny + 9
        for i0, i1, j0, j1 in ((xl, xr, yl, yl + 8), (xl, xr, yr - 8, yr), (xl, xl + 8, yl, yr),
                               (xr - 8, xr, yl, yr), (xl + 8, xr - 8, yl + 8, yr - 8)):
            m[max(i0, 0):i1 + 1, max(j0, 0):j1 + 1] += 1
        self.mult = m

    def principal(self, I, J, s2, pf):
        s = s2 + pf
        d = (YIELD["fmajor"], 1.0, YIELD["fminor"])
        c = sum(float(self.R[k, I] * d[k] * self.R[k, J]) for k in range(3)) * s
        return c - pf if I == J else c

    def pfluid(self, w, up=0):
        k = torch.arange(w[4], w[5] + 1, device=DEV, dtype=torch.float64)
        d = (self.n[2] + 31 - k + up) * self.h
        return torch.where(d > 0, (d + self.h * 0.5) * 9.81e3, self.h / 2 * 9.81e3)[None, None, :]

    def plasticity(self):
        if self.nve != 3:
            return
        if not self.topo:
            i0, i1, j0, j1 = self.middle()
            self._band((i0, i1, j0, j1), self.window())
        nx, ny, nz = self.n
        w = (10, nx + 9, 10, ny + 9, 32, nz + 31)
        g, S, P = self.g, self.S, self.principal
        pf = self.pfluid(w)
        a, b = g(self.s2, w), g(self.s2, w, 1)
        ii = {c: 0.5 * (P(*c, a, pf) + P(*c, b, pf)) for c in
              ((0, 0), (1, 1), (2, 2), (0, 2), (1, 2), (0, 1))}
        o = lambda f, *d: g(S[f], w, *d)  # noqa: E731
        xx, yy, zz = o("xx") + ii[0, 0], o("yy") + ii[1, 1], o("zz") + ii[2, 2]
        xz = 0.25 * (o("xz") + o("xz", 1) + o("xz", 0, 0, -1) + o("xz", 1, 0, -1)) + ii[0, 2]
        yz = 0.25 * (o("yz") + o("yz", 0, -1) + o("yz", 0, 0, -1) + o("yz", 0, -1, -1)) + ii[1, 2]
        xy = 0.25 * (o("xy") + o("xy", 1) + o("xy", 0, -1) + o("xy", 1, -1)) + ii[0, 1]
        mu, mup, d1 = g(self.M["mu"], w), g(self.M["mu"], w, 1), g(self.M["d1"], w)
        Tv = self.h / torch.sqrt(1.0 / (mu * d1))
        rphi = g(self.phi, w) * (math.pi / 180)
        sm = (xx + yy + zz) / 3
        dx, dy, dz = xx - sm, yy - sm, zz - sm
        sec = torch.sqrt(0.5 * (dx * dx + dy * dy + dz * dz) + xz * xz + xy * xy + yz * yz)
        lim = (g(self.co, w) * torch.cos(rphi) - (sm + pf) * torch.sin(rphi)).clamp(min=0)
        y = torch.where(sec > lim, lim / sec + (1 - lim / sec) * torch.exp(-self.dt / Tv), 1.0)
        xm = 2.0 / (mu + mup)
        dep = torch.sqrt(0.5 * sum(((v - sm) * y + sm - v) ** 2 for v in (xx, yy, zz)) +
                         2.0 * sum((v * y - v) ** 2 for v in (xy, xz, yz))) / xm
        m = self.mult[w[0]:w[1] + 1, w[2]:w[3] + 1, None]
        self.put("neta", w, torch.where(y < 1, g(S["neta"], w) + m * dep, g(S["neta"], w)))
        self.put("yldfac", w, y)
        w = (10, nx + 9, 10, 9 + ny + ny % 2, 32, nz + 31)
        pf, pfu = self.pfluid(w), self.pfluid(w, 1)
        s = lambda *d: g(self.s2, w, *d)  # noqa: E731
        yl = lambda *d: g(self.S["yldfac"], w, *d)  # noqa: E731
        n = {}
        y = yl()
        ii = {c: 0.5 * (P(c, c, s(), pf) + P(c, c, s(1), pfu)) for c in range(3)}
        full = [o2 + ii[c] for c, o2 in enumerate((g(S["xx"], w), g(S["yy"], w), g(S["zz"], w)))]
        sm = sum(full) / 3
        for c, f in enumerate(("xx", "yy", "zz")):
            n[f] = torch.where(y < 1, (full[c] - sm) * y + sm - ii[c], g(S[f], w))
        it = {"xz": 0.5 * (P(0, 2, s(), pf) + P(0, 2, s(0, 0, 1), pfu)),
              "yz": 0.125 * sum(P(1, 2, s(a, b, c), pfu if c else pf)
                                for a in (0, 1) for b in (0, 1) for c in (0, 1)),
              "xy": 0.5 * (P(0, 1, s(), pf) + P(0, 1, s(0, 1), pf))}
        ya = {"xz": 0.25 * (yl(-1) + y + yl(-1, 0, 1) + yl(0, 0, 1)),
              "yz": 0.25 * (y + yl(0, 1) + yl(0, 1, 1) + yl(0, 0, 1)),
              "xy": 0.25 * (y + yl(0, 1) + yl(-1) + yl(-1, 1))}
        for f in it:
            n[f] = torch.where(ya[f] < 1, (g(S[f], w) + it[f]) * ya[f] - it[f], g(S[f], w))
        for f, v in n.items():
            self.put(f, w, v)

    # ---- curvilinear operators -------------------------------------------
    def set_topo(self, elev):
        self.topo = _metrics(elev, *self.n, self.h)
        nu = np.float32(np.float32(self.dt) / np.float32(self.h))
        self.tdt = np.float32(nu * np.float32(self.h))
        self.tdth = float(np.float32(self.tdt / np.float32(self.h)))
        self.tdt = float(self.tdt)

    def _vertical(self, v, w, tab, kind):
        """Vertical operator at levels w[4]..w[5] of a column array v that
        holds every level: 7-point (kind 7) or 4-point at the half (h) or node
        (n) points, with the closure rows of the top six levels."""
        t = torch.tensor(tab, dtype=torch.float64, device=DEV)
        o = lambda d: v[..., w[4] + d:w[5] + 1 + d]  # noqa: E731
        if kind == 7:
            a, b, c = (float(np.float32(x)) for x in (-0.0026041666666667, 0.09375, -0.6796875))
            s = a * (o(-3) - o(3)) + b * (o(-2) - o(2)) + c * (o(-1) - o(1))
        else:
            a = -2 if kind == "h" else -1
            s = _D0 * (o(a) - o(a + 3)) + _D1 * (o(a + 1) - o(a + 2))
        top = v[..., self.n[2] + 32 - t.shape[1]:self.n[2] + 32].flip(-1)
        s = s.clone()
        s[..., -6:] = (top @ t.T).flip(-1)
        return s

    def topo_velocity(self):
        nx, ny, nz = self.n
        w = (10, nx + 9, 10, ny + 9, 35, nz + 31)
        z = (10, nx + 9, 10, ny + 9, 0, nz + 63)  # whole columns
        S, T, g, d = self.S, self.topo, self.g, self.M["d1"]
        k = slice(w[4], w[5] + 1)
        m = lambda f, a=0, b=0: T[f][w[0] + a:w[1] + 1 + a, w[2] + b + 32:w[3] + 1 + b + 32, None]  # noqa: E731
        g3c, g3 = T["g3_c"][k], T["g3"][k]
        gcf, ggf = T["g_c"], T["g"]
        o = lambda f, a=0, b=0: g(S[f], w, a, b)  # noqa: E731
        c = lambda f, a=0, b=0: g(S[f], z, a, b)  # noqa: E731
        V = self._vertical
        r = lambda *q: 0.25 * sum(g(d, w, *x) for x in q)  # noqa: E731
        rho = (r((0, 0, -1), (0, -1, -1), (0, 0, 0), (0, -1, 0)),
               r((0, 0, -1), (-1, 0, -1), (0, 0, 0), (-1, 0, 0)),
               r((0, 0, 0), (-1, 0, 0), (0, -1, 0), (-1, -1, 0)))
        nu = self.dth
        A = (nu / (m("f_1") * g3c * rho[0]), nu / (m("f_2") * g3c * rho[1]),
             nu / (m("f_c") * g3 * rho[2]))

        def dif(metric, f, ax, a):  # difference of metric * f, points a .. a+3
            at = lambda n: (n, 0) if ax == 0 else (0, n)  # noqa: E731
            return sum(q * m(metric, *at(a + n)) * o(f, *at(a + n))
                       for n, q in enumerate((_D0, _D1, -_D1, -_D0)))

        def itp(f, ax, a):
            at = lambda n: (n, 0) if ax == 0 else (0, n)  # noqa: E731
            return sum(q * c(f, *at(a + n)) for n, q in enumerate((-0.0625, 0.5625, 0.5625, -0.0625)))
        s1 = g3c * (dif("f_c", "xx", 0, -2) + dif("f", "xy", 1, -2)) + V(c("xz"), w, _VDHZ, "h") - \
            m("f1_1") * V(gcf * itp("xx", 0, -2), w, _VDHPZ, 7) - \
            m("f2_1") * V(gcf * itp("xy", 1, -2), w, _VDHPZ, 7)
        s2 = V(c("yz"), w, _VDHZ, "h") + g3c * (dif("f", "xy", 0, -1) + dif("f_c", "yy", 1, -1)) - \
            m("f1_2") * V(gcf * itp("xy", 0, -1), w, _VDHPZ, 7) - \
            m("f2_2") * V(gcf * itp("yy", 1, -1), w, _VDHPZ, 7)
        s3 = g3 * (dif("f_2", "yz", 1, -2) + dif("f_1", "xz", 0, -1)) + \
            V(c("zz"), w, _VDZ, "n") - \
            m("f1_c") * V(ggf * itp("xz", 0, -1), w, _VDPHZ, 7) - \
            m("f2_c") * V(ggf * itp("yz", 1, -2), w, _VDPHZ, 7)
        sp = self.sponge(w)
        new = [(f, (o(f) + a * s) * sp) for f, a, s in zip(("u1", "v1", "w1"), A, (s1, s2, s3))]
        for f, v in new:
            self.put(f, w, v)

    def topo_stress(self):
        nx, ny, nz = self.n
        w = (14, nx + 5, 14, ny + 5, 35, nz + 31)
        z = w[:4] + (0, nz + 63)
        S, T, g = self.S, self.topo, self.g
        k = slice(w[4], w[5] + 1)
        m = lambda f, a=0, b=0: T[f][w[0] + a:w[1] + 1 + a, w[2] + b + 32:w[3] + 1 + b + 32, None]  # noqa: E731
        c = lambda f, a=0, b=0: g(S[f], z, a, b)  # noqa: E731
        V = self._vertical
        J = 1.0 / (m("f_c") * T["g3_c"][k])
        kk = torch.arange(w[4], w[5] + 1, device=DEV)
        J12 = 1.0 / (m("f") * T["g3_c"][torch.where(kk < nz + 26, kk + 6, kk)])
        J13, J23 = 1.0 / (m("f_1") * T["g3"][k]), 1.0 / (m("f_2") * T["g3"][k])
        gc, gg = T["g_c"][k], T["g"][k]
        at = lambda ax, n: (n, 0) if ax == 0 else (0, n)  # noqa: E731

        def dif(f, ax, a):
            return sum(q * g(S[f], w, *at(ax, a + n)) for n, q in enumerate((_D0, _D1, -_D1, -_D0)))

        def itp(metric, f, ax, a):
            return sum(q * m(metric, *at(ax, a + n)) * c(f, *at(ax, a + n))
                       for n, q in enumerate((-0.0625, 0.5625, 0.5625, -0.0625)))
        e = [dif("u1", 0, -1) - J * gc * V(itp("f1_1", "u1", 0, -1), w, _SPHDZ, 7),
             dif("v1", 1, -2) - J * gc * V(itp("f2_2", "v1", 1, -2), w, _SPHDZ, 7),
             J * V(c("w1"), w, _SDHZ, "h"),
             dif("u1", 1, -1) - J12 * gc * V(itp("f2_1", "u1", 1, -1), w, _SPHDZ, 7) +
             dif("v1", 0, -2) - J12 * gc * V(itp("f1_2", "v1", 0, -2), w, _SPHDZ, 7),
             J13 * V(c("u1"), w, _SDZ, "n") +
             dif("w1", 0, -2) - J13 * gg * V(itp("f1_c", "w1", 0, -2), w, _SPDHZ, 7),
             J23 * V(c("v1"), w, _SDZ, "n") +
             dif("w1", 1, -1) - J23 * gg * V(itp("f2_c", "w1", 1, -1), w, _SPDHZ, 7)]
        self.stress_update(w, e, dth=self.tdth, dt=self.tdt)

    def step(self):
        self.begin()
        self.velocity()
        self.stress()
        self.sources()
        self.plasticity()
        self.surface()


# ---- two blocks --------------------------------------------------------------
def _interface(hi, lo):
    """Coarse to fine (bilinear), then fine to coarse (5 x 5 x 5 tent)."""
    nx, ny, nz = lo.n
    k = nz + 29
    wt = (1.0, float(np.float32(2 / 3)), float(np.float32(1 / 3)), 0.0)
    for f, oi, oj in (("xz", 0, 0), ("yz", 1, 1), ("w1", 1, 0), ("xx", 1, 0), ("yy", 1, 0),
                      ("zz", 1, 0), ("u1", 0, 0), ("v1", 1, 1), ("xy", 0, 1)):
        L, H = lo.S[f], hi.S[f]
        a = lambda di, dj: L[8 + di:nx + 12 + di, 8 + dj:ny + 12 + dj, k]  # noqa: E731
        for ii in range(4):
            for jj in range(4):
                v = (a(0, 0) * wt[ii] * wt[jj] + a(1, 0) * wt[3 - ii] * wt[jj] +
                     a(0, 1) * wt[ii] * wt[3 - jj] + a(1, 1) * wt[3 - ii] * wt[3 - jj])
                i0, j0 = 4 + ii + oi, 4 + jj + oj
                H[i0:i0 + 3 * (nx + 3) + 1:3, j0:j0 + 3 * (ny + 3) + 1:3, 33] = v
    tent = (1.0, 2.0, 3.0, 2.0, 1.0)
    for f, di, dj, k0 in (("u1", 0, 0, 3), ("v1", 1, 1, 3), ("xy", 0, 1, 3), ("xx", 1, 0, 3),
                          ("yy", 1, 0, 3), ("zz", 1, 0, 3), ("xz", 0, 0, 4), ("w1", 1, 0, 4),
                          ("yz", 1, 1, 4)):
        for lev, kh in ((0, k0), (1, 6)):
            if lev and k0 == 4:
                continue
            H = hi.S[f]
            s = sum(tent[c] * H[:, :, 32 + kh + c - 2] for c in range(5))
            n = 3 * (nx + 4) + 1
            s = sum(tent[c] * s[2 + di + c:2 + di + c + n:3] for c in range(5))
            n = 3 * (ny + 4) + 1
            s = sum(tent[c] * s[:, 2 + dj + c:2 + dj + c + n:3] for c in range(5))
            lo.S[f][8:nx + 13, 8:ny + 13, 32 + nz - 2 + lev] = s / 729.0


def _layer_velocity(x):
    nx, ny, _ = x.n
    w = (10, nx + 9, 10, ny + 9, 34, 34)
    S, g, d = x.S, x.g, x.M["d1"]
    o = lambda f, *a: g(S[f], w, *a)  # noqa: E731
    rho = lambda *q: x.dth / (0.25 * sum(g(d, w, *a) for a in q))  # noqa: E731
    sp = x.sponge(w)
    n = {"w1": (o("w1") + rho((0, 0, 0), (1, 0, 0), (0, -1, 0), (1, -1, 0)) *
                (o("xz", 1) - o("xz") + o("yz") - o("yz", 0, -1) + o("zz", 0, 0, 1) - o("zz"))) * sp,
         "u1": (o("u1") + rho((0, 0, 0), (0, -1, 0), (0, 0, -1), (0, -1, -1)) *
                (o("xx") - o("xx", -1) + o("xy") - o("xy", 0, -1) + o("xz") - o("xz", 0, 0, -1))) * sp,
         "v1": (o("v1") + rho((0, 0, 0), (1, 0, 0), (0, 0, -1), (1, 0, -1)) *
                (o("xy", 1) - o("xy") + o("yy", 0, 1) - o("yy") + o("yz") - o("yz", 0, 0, -1))) * sp}
    for f, v in n.items():
        x.put(f, w, v)


def _layer_stress(x):
    nx, ny, _ = x.n
    w = (10, nx + 9, 10, ny + 9, 34, 34)
    o = lambda f, *a: x.g(x.S[f], w, *a)  # noqa: E731
    e = [o("u1", 1) - o("u1"), o("v1") - o("v1", 0, -1), o("w1") - o("w1", 0, 0, -1),
         o("u1", 0, 1) - o("u1") + o("v1") - o("v1", -1),
         o("u1", 0, 0, 1) - o("u1") + o("w1") - o("w1", -1),
         o("v1", 0, 0, 1) - o("v1") + o("w1", 0, 1) - o("w1")]
    x.stress_update(w, e, interface=True)


def _mesh_step(hi, lo):
    for x in (hi, lo):
        x.begin()
    for x in (hi, lo):
        x.velocity()
    _layer_velocity(hi)
    _interface(hi, lo)
    for x in (hi, lo):
        x.stress()
    _layer_stress(hi)
    for x in (hi, lo):
        x.sources()
    _interface(hi, lo)
    for x in (hi, lo):
        x.plasticity()
    hi.surface()


# ---- metrics of the curvilinear grid (float32, as the model set-up forms them) ---
_D0 = float(np.float32(0.0416666666666667))
_D1 = -1.125


def _rows(n, *rows):
    out = np.zeros((6, n), np.float32)
    for i, r in enumerate(rows):
        out[i, :len(r)] = np.asarray(r, np.float64).astype(np.float32)
    return out.astype(np.float64)


_Z7 = (-0.6796875, 0.09375, -0.0026041666666667)
_VDHPZ = _rows(
    9, (-1.5373923010673118, -1.1059180740634813, -0.2134752473866528, -0.0352027995732726,
        -0.0075022330101095, -0.0027918394266035),
    (0.8139439685257414, 0.1273679143938725, -1.1932750007455710, 0.1475120181828087,
     0.1125814499297686, -0.0081303502866204),
    (0.1639182541610305, 0.3113839909089030, -0.0536007135209480, -0.3910958927076030,
     -0.0401741813821989, 0.0095685425408165),
    (0.0171478318814576, -0.0916600077207278, 0.7187220404622645, -0.1434031863528334,
     -0.5827389738506837, 0.0847863081664324, -0.0028540125859095),
    (-0.0579176640853654, 0.0022069616616207, 0.0108792602269819, 0.6803612607837533,
     -0.0530169938441240, -0.6736586580761996) + _Z7[1:],
    (0.0020323834153791, 0.0002106933140862, -0.0013351454085978, -0.0938400881871787,
     0.6816971139746001, -0.0002232904416222) + _Z7)
_SPHDZ = _rows(
    9, (1.5373923010673116, -1.0330083346742178, -0.6211677623382129, -0.0454110758451345,
        0.1680934225988761, -0.0058985508086226),
    (0.8713921425924012, -0.1273679143938725, -0.9297550647681331, 0.1912595577524762,
     -0.0050469052908678, -0.0004818158920039),
    (0.0563333965151294, 0.3996393739211770, 0.0536007135209481, -0.5022638816465500,
     -0.0083321572725344, 0.0010225549618299),
    (0.0132930497153990, -0.0706942590708847, 0.5596445380498726, 0.1434031863528334,
     -0.7456356868769503, 0.1028431844156395, -0.0028540125859095),
    (0.0025849423769932, -0.0492307522105194, 0.0524552477068130, 0.5317248489238559,
     0.0530169938441240, -0.6816971139746001) + _Z7[1:],
    (0.0009619461344193, 0.0035553215968974, -0.0124936029037323, -0.0773639466787397,
     0.6736586580761996, 0.0002232904416222) + _Z7)
_VDPHZ = _rows(
    9, (),
    (0.0, -1.5886075042755421, -2.4835574634505861, 0.0421173406787286, 0.4968761536590695,
     -0.0228264197210198),
    (0.0, 0.4428256655817484, -0.0574614517751294, -0.2022259589759502, -0.1944663890497050,
     0.0113281342190362),
    (0.0, -0.3360140866060758, 1.2113298407847195, -0.3111668377093505, -0.6714462506479002,
     0.1111440843153523, -0.0038467501367455),
    (0.0, 0.0338560531369653, -0.0409943223643902, 0.5284757132923059, 0.0115571196122084,
     -0.6162252315536446, 0.0857115441015996, -0.0023808762250444),
    (0.0, -0.0040378273193044, 0.0064139372778371, -0.0890062133451850, 0.6749219241340761,
     0.0002498459192428) + _Z7)
_SPDHZ = _rows(
    9, (),
    (0.0, 1.5886075042755419, -2.2801810182668114, 0.8088980291471826, -0.1316830205960989,
     0.0143585054401857),
    (0.0, 0.4823226655921295, 0.0574614517751295, -0.5663203488781653, 0.0309656800624243,
     -0.0044294485515179),
    (0.0, -0.0174954311279016, 0.4325508330649349, 0.3111668377093504, -0.8538512002386446,
     0.1314757107290064, -0.0038467501367455),
    (0.0, -0.1277481742492071, 0.2574468839590017, 0.4155794781917712, -0.0115571196122084,
     -0.6170517361659126, 0.0857115441015996, -0.0023808762250444),
    (0.0, 0.0064191319587820, -0.0164033832904366, -0.0752421418813823, 0.6740179057989464,
     -0.0002498459192428) + _Z7)
_H4 = (-0.0416666666666667, 1.125, -1.125, 0.0416666666666667)
_SDHZ = _rows(
    8, (0.0, 1.4511412472637157, -1.8534237417911470, 0.3534237417911469, 0.0488587527362844),
    (0.0, 0.8577143189081458, -0.5731429567244373, -0.4268570432755628, 0.1422856810918542),
    (0.0, 0.1674548505882877, 0.4976354482351368, -0.4976354482351368, -0.1674548505882877),
    (0.0, -0.1027061113405124, 0.2624541326469860, 0.8288742701021167, -1.0342864927831414,
     0.0456642013745513),
    (0.0, 0.0, 0.0) + _H4, (0.0, 0.0, 0.0, 0.0) + _H4)
_VDHZ = _SDHZ.copy()
_VDHZ[0, 1] = -_VDHZ[0, 1]
_SDZ = _rows(
    7, (), (1.7779989465546748, -1.3337480247900155, -0.7775013168066564, 0.3332503950419969),
    (0.4410217341392059, 0.1730842484889890, -0.4487228323259926, -0.1653831503022022),
    (-0.1798793213882701, 0.2757257254150788, 0.9597948548284453, -1.1171892610431817,
     0.0615480021879277),
    (-0.0153911381507088, -0.0568851455503591, 0.1998976464597171, 0.8628231468598346,
     -1.0285385292191949, 0.0380940196007109),
    (0.0, 0.0, 0.0) + _H4)
_VDZ = _SDZ.copy()
_VDZ[1, 0] = -_VDZ[1, 0]
_GI = _rows(
    7, (0.8338228784688313, 0.1775123316429260, 0.1435067013076542, -0.1548419114194114),
    (0.1813404047323969, 1.1246711188154426, -0.2933634518280757, -0.0126480717197637),
    (-0.1331142706282399, 0.7930714675884345, 0.3131998767078508, 0.0268429263319546),
    (0.0969078556633046, -0.1539344946680898, 0.4486491202844389, 0.6768738207821733,
     -0.0684963020618270),
    (0.0, 0.0, -0.0625, 0.5625, 0.5625, -0.0625),
    (0.0, 0.0, 0.0, -0.0625, 0.5625, 0.5625, -0.0625))


def _metrics(elev, nx, ny, nz, h):
    """f and its interpolants and derivatives [nx + 20][ny + 84], the vertical
    g, g_c, g3, g3_c [nz + 64]; every operation rounds to float32."""
    c = np.float32
    P = [c(-0.0625), c(0.5625), c(0.5625), c(-0.0625)]
    D = [c(_D0), c(-1.125), c(1.125), c(-_D0)]
    hi = c(1.0 / h)
    T = {n: np.zeros((nx + 20, ny + 84), c) for n in
         ("f", "f_1", "f_2", "f_c", "f1_1", "f1_2", "f1_c", "f2_1", "f2_2", "f2_c")}
    norm = c(1.0 / h / (nz - 2))
    T["f"][2:nx + 18, 34:ny + 50] = (1.0 + (elev * norm).astype(np.float64)).astype(c)
    wi, wj = slice(4, nx + 16), slice(36, ny + 48)

    def at(a, di, dj):
        return a[4 + di:nx + 16 + di, 36 + dj:ny + 48 + dj]

    def four(a, k, axis, first):
        s = None
        for n in range(4):
            v = k[n] * (at(a, first + n, 0) if axis == 0 else at(a, 0, first + n))
            s = v if s is None else s + v
        return s
    f = T["f"]
    T["f_1"][wi, wj] = four(f, P, 1, -2)
    T["f_2"][wi, wj] = four(f, P, 0, -1)
    row = np.zeros_like(f)  # interpolated along x, on every column
    row[4:nx + 16] = P[0] * f[3:nx + 15] + P[1] * f[4:nx + 16] + P[2] * f[5:nx + 17] + \
        P[3] * f[6:nx + 18]
    T["f_c"][wi, wj] = four(row, P, 1, -2)
    for out, src, axis, first in (("f1_1", "f_c", 0, -2), ("f1_2", "f", 0, -1),
                                  ("f1_c", "f_1", 0, -1), ("f2_1", "f", 1, -2),
                                  ("f2_2", "f_c", 1, -1), ("f2_c", "f_2", 1, -2)):
        T[out][wi, wj] = hi * four(T[src], D, axis, first)
    hg = c(1.0 / float(hi))
    g, gc, g3, g3c = (np.zeros(nz + 64, c) for _ in range(4))
    A, B = 32, 32 + nz  # levels A .. B - 1
    g[A:B] = (float(hg) * np.arange(nz)).astype(c)
    g[B - 1] = 0.0

    def row_sum(k, v, up):
        if up:
            s = k[0] * v[0]
            for n in range(1, len(k)):
                s = c(s + c(k[n] * v[n]))
        else:  # from the far end
            s = k[-1] * v[-1]
            for n in range(len(k) - 2, -1, -1):
                s = c(s + c(k[n] * v[n]))
        return c(s)

    def mid(k, a, first, n=nz - 12):
        s = None
        for q in range(4):
            v = k[q] * a[A + 6 + first + q:A + 6 + first + q + n]
            s = v if s is None else s + v
        return s
    gi, dz, dh = (x.astype(c) for x in (_GI, _SDZ, _SDHZ))
    gir = np.concatenate([np.zeros((6, 1), c), gi], 1)
    # left closures: the right ones mirrored
    dzl = np.zeros((6, 8), c)
    dzl[:5, :7] = -dz[1:]
    dzl[5, 4:] = D
    dhl = -dh[:, 1:]
    for k in range(6):
        gc[A + k] = row_sum(gi[k], g[A:A + 7], True)
        gc[B - 1 - k] = row_sum(gir[k], g[B - 8:B][::-1], False)
    gc[A + 6:B - 6] = mid(P, g, -2)
    for k in range(6):
        g3[A + k] = hi * row_sum(dzl[k], gc[A:A + 8], True)
        g3[B - 1 - k] = hi * row_sum(dz[k], gc[B - 7:B][::-1], False)
        g3c[A + k] = hi * row_sum(dhl[k], g[A:A + 7], True)
        g3c[B - 1 - k] = hi * row_sum(dh[k], g[B - 8:B][::-1], False)
    g3[A + 6:B - 6] = hi * mid(D, gc, -1)
    g3c[A + 6:B - 6] = hi * mid(D, g, -2)
    g3[B - 1] = 1.0
    T.update(g=g, g_c=gc, g3=g3, g3_c=g3c)
    return {n: torch.tensor(a.astype(np.float64), device=DEV) for n, a in T.items()}


def exact(case, seed):
    kind, h, n = case["kind"], 50.0, case["steps"]
    dt = _dt(h)
    if kind == "gradient":
        return _exact_gradient(case, seed, h, dt)
    with torch.no_grad():
        if kind == "ensemble":
            h = 100.0
            out = []
            for i, (nx, ny, nz) in enumerate(_ensemble_sizes(case)):
                x = _X(nx, ny, nz, h, _dt(h), True, seed, 100 * i, nsrc=1)
                for _ in range(n):
                    x.step()
                out.append([x.S[f] for f in FIELDS9[:3]])
            return out
        if kind == "mesh":
            dt = _dt(40.0)
            nve = 3 if case["plastic"] else 1
            xs = []
            for p, (nx, ny, nz, hp, z0, z1) in enumerate(_blocks(case)):
                x = _X(nx, ny, nz, hp, dt, True, seed, 10 * p, (z0, z1), p, 2, nve=nve,
                       nd=18 if p == 0 else 6, sources=p == 0)
                if nve == 3:
                    x.set_yield(*_yield_inputs(nx, ny, nz, hp, seed, 10 * p + 3))
                xs.append(x)
            hi, lo = xs
            lo.src = None
            if case["hill"]:
                hi.set_topo(_elevation(*hi.n[:2], hi.h, seed))
            lo.fx = hi.n
            nx, ny, nz = lo.n
            for f in lo.M:  # the coarse block's top three levels take the fine block's media
                for lev in range(3):
                    lo.M[f][10:nx + 10, 10:ny + 10, 32 + nz - 3 + lev] = \
                        hi.M[f][10:10 + 3 * nx:3, 11:11 + 3 * ny:3, 33 + 3 * lev]
            for _ in range(n):
                _mesh_step(hi, lo)
            names = FIELDS15 + (("yldfac", "neta") if nve == 3 else ())
            return {f"{f}_{p}": x.S[f] for p, x in enumerate(xs) for f in names}
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        x = _X(nx, ny, nz, h, dt, case["q"], seed, 0, fault=case.get("fault", False),
               nve=3 if kind == "plastic" else 1)
        if kind == "hill":
            x.set_topo(_elevation(nx, ny, h, seed))
        names = FIELDS15 if case["q"] else FIELDS9
        if kind == "plastic":
            x.set_yield(*_yield_inputs(nx, ny, nz, h, seed, 3))
            names = names + ("yldfac", "neta")
        for _ in range(n):
            x.step()
        out = {f: x.S[f] for f in names}
        if case.get("gather"):
            t = nz + 31
            out["frame"] = torch.stack([x.S[f][10:nx + 10, 10:ny + 10, t - (f == "w1")].T
                                        for f in FIELDS9[:3]])
        return out


def _exact_gradient(case, seed, h, dt):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    with torch.no_grad():
        x = _X(nx, ny, nz, h, dt, case["q"], seed, 0, wave=False, near_surface=True)
    model = [m.double().requires_grad_() for m in _moduli(case, seed)]
    xyz, comp, obs = _receivers(case, seed, dt)
    xyz = torch.tensor(xyz.astype(np.int64), device=DEV)
    comp = torch.tensor(comp.astype(np.int64), device=DEV)
    obs = torch.tensor(obs.astype(np.float64), device=DEV)
    names = FIELDS15 if case["q"] else FIELDS9
    J = torch.zeros((), dtype=torch.float64, device=DEV)

    def one(n, *t):
        x.S = dict(zip(names, t[3:]))
        x.set_moduli(*t[:3])
        x.step_n = n
        if n == 0:
            x.add_sources(0)
        x.step_n = n + 1
        x.velocity()
        x.stress()
        x.sources()
        x.surface()
        v = torch.stack([x.S[f][xyz[:, 0] + 10, xyz[:, 1] + 10, nz + 31 - xyz[:, 2]]
                         for f in FIELDS9[:3]])
        r = v.gather(0, comp[None])[0] - obs[n]
        return (0.5 * (r * r).sum(),) + tuple(x.S[f] for f in names)
    with torch.enable_grad():
        state = tuple(x.zeros() for _ in names)
        for n in range(case["steps"]):
            j, *state = checkpoint(one, n, *model, *state, use_reentrant=False,
                                   preserve_rng_state=False)
            J = J + j
        grad = torch.autograd.grad(J, model)
    return {"misfit": J.detach(), "grad": list(grad), "final": [t.detach() for t in state[:9]]}
