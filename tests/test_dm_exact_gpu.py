"""The mesh-interface launchers of the reference ABI against float64, value by
value: no partial cancellation may cost more than the float operations that
follow it, and a level outside a window must not reach its average."""
import ctypes
from ctypes import c_float, c_int

import numpy as np
import pytest
import torch

from awp_b200 import _lib

pytestmark = pytest.mark.gpu

NGSL, ALIGN = 8, 32
EPS = 2.0 ** -24  # half an ulp, relative
F = ctypes.POINTER(c_float)


def grid_constants(lib, dims, dh, dt):
    n = len(dims)
    arr = [(c_int * n)(*(d[q] for d in dims)) for q in range(3)]
    zero = (c_float * 9)()
    lib.SetDeviceConstValue((c_float * n)(*dh), dt, *arr, n, 1.0, 1.0, zero, zero)


def padded(d):
    return d[0] + 4 + 2 * NGSL, d[1] + 4 + 2 * NGSL, d[2] + 2 * ALIGN


def pointer(t):
    return ctypes.c_void_p(t.data_ptr())


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def test_dstrqc2_memory_variables_match_float64():
    """From a state at rest but for u1, the shear memory variables are wwo *
    h * (difference of u1): products only, apart from the Q(f) polynomial,
    whose two terms nearly cancel for the Q drawn here.  Roundings along the way:
    the pair sum, quotient, polynomial, 1/wwo (2 ulp), dh1*vx1, the weight, h,
    the difference, its product and wwo's: 14 half ulps."""
    lib = _lib.load()
    nx, ny, nz = 37, 41, 12
    dh, dt = 40.0, 0.005
    grid_constants(lib, [(3 * nx, 3 * ny, 16), (nx, ny, nz)], [dh / 3, dh], dt)
    shape = padded((nx, ny, nz))
    g = np.random.default_rng(3)
    w, c, tau = np.zeros(8, np.float32), np.zeros(16, np.float32), np.zeros(8, np.float32)
    hi, lo = c_float(), c_float()
    assert lib.awp_q_weights(0.6, 1.0, w.ctypes.data_as(F), c.ctypes.data_as(F)) == 0
    assert lib.awp_q_tau(0.6, 1.0, ctypes.byref(hi), ctypes.byref(lo), tau.ctypes.data_as(F)) == 0
    assert (w > 0).all()
    e = g.integers(0, 8, shape)
    vx1 = (0.5 * (1 - np.exp(-dt / tau.astype(float)))).astype(np.float32)[e]
    wwo = (8 * w.astype(np.float64)).astype(np.float32)[e]
    # half of the pair means near the polynomial's zero of the cell's entry
    zero = np.where((c[0::2] * c[1::2] < 0) & (-c[1::2] > 0.005 * c[0::2]),
                    -c[1::2] / np.where(c[0::2] == 0, 1, c[0::2]), 0.01)[e]
    zero = np.clip(zero, 0.006, 0.1)
    qs = np.where(g.random(shape) < 0.5, zero * (1 + 1e-3 * g.standard_normal(shape)),
                  np.exp(g.uniform(np.log(1e-3), np.log(0.1), shape))).astype(np.float32)
    mu = (1 / g.uniform(5e9, 4e10, shape)).astype(np.float32)
    names = ["xx", "yy", "zz", "xy", "xz", "yz", "r1", "r2", "r3", "r4", "r5", "r6", "u1", "v1",
             "w1"]
    f = {n: torch.zeros(shape, device="cuda") for n in names}
    u = g.standard_normal(shape).astype(np.float32)
    f["u1"] = dev(u)
    one = torch.ones(max(shape), device="cuda")
    m = {n: dev(a) for n, a in dict(lam=mu, mu=mu, qp=qs, qs=qs).items()}
    k = {n: dev(a) for n, a in dict(vx1=vx1, vx2=np.zeros(shape, np.float32),
                                    ww=(e + 1).astype(np.int32), wwo=wwo, coeff=c).items()}
    s_i, e_i, s_j, e_j = 2 + NGSL, nx + NGSL + 1, 2 + NGSL, ny + NGSL + 1
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    fn = lib.dstrqc2_H
    fn.restype = None
    fn(*(pointer(f[n]) for n in names), *(pointer(m[n]) for n in ("lam", "mu", "qp", "qs")),
       pointer(one), pointer(one), pointer(one), nx, ny, ctypes.c_void_p(st.cuda_stream),
       pointer(k["coeff"]), pointer(k["vx1"]), pointer(k["vx2"]), pointer(k["ww"]),
       pointer(k["wwo"]), s_i, e_i, s_j, e_j, 1)
    st.synchronize()
    kz = ALIGN + 2
    I, J = np.meshgrid(np.arange(s_i, e_i + 1), np.arange(s_j, e_j + 1), indexing="ij")
    dh1 = float(np.float32(1.0 / dh))

    def at(a, di=0, dj=0, dk=0):
        return a[I + di, J + dj, kz + dk].astype(np.float64)

    for name, (di, dj, dk), du in (("r4", (0, 0, -1), at(u, dj=1) - at(u)),
                                   ("r5", (0, -1, 0), at(u, dk=1) - at(u))):
        q = (0.25 * (at(qs) + at(qs, di, dj, dk)).astype(np.float32)).astype(np.float64)
        x = 2 * q
        c0, c1 = (c[2 * e + n][I, J, kz].astype(float) for n in (0, 1))
        w0 = at(wwo)
        weight = np.where(1 / x <= 200, c0 * x * x + c1 * x, w0 * q)
        h = weight / w0 * -dh1 * at(vx1) * 2 / (at(mu) + at(mu, di, dj, dk))
        want = w0 * h * du
        got = f[name].cpu().numpy()[I, J, kz].astype(np.float64)
        assert float(np.median(np.abs(want))) > 0
        err = np.abs(got - want) / np.abs(want)
        assert float(err.max()) <= 14 * EPS, (name, err.max() / EPS)


FIELDS = ["xx", "yy", "zz", "xy", "xz", "yz", "u1", "v1", "w1"]
# level of the first window's centre, windows, shift of the fine columns
WINDOW = dict(u1=(3, 2, 0, 0), v1=(3, 2, 1, 1), xy=(3, 2, 0, 1), xx=(3, 2, 1, 0),
              yy=(3, 2, 1, 0), zz=(3, 2, 1, 0), xz=(4, 1, 0, 0), w1=(4, 1, 1, 0),
              yz=(4, 1, 1, 1))


def swap(lib, fine, coarse, nx, ny):
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    fn = lib.swap_H
    fn.restype = None
    fn(*(pointer(coarse[n]) for n in FIELDS), *(pointer(fine[n]) for n in FIELDS), nx, ny,
       *[None] * 4, -1, ctypes.c_void_p(st.cuda_stream), 0)
    st.synchronize()


def windows(h, nx, ny, kh, di, dj):
    """(terms [125][i][j] in the reference's order, weights) of every coarse column."""
    I, J = np.meshgrid(np.arange(NGSL, nx + NGSL + 5), np.arange(NGSL, ny + NGSL + 5),
                       indexing="ij")
    ci, cj = 3 * (I - 2 - NGSL) + 2 + NGSL + di, 3 * (J - 2 - NGSL) + 2 + NGSL + dj
    r = range(-2, 3)
    t = [((3 - abs(a)) * (3 - abs(b)) * (3 - abs(d)) / 729.0,
          h[ci + a, cj + b, ALIGN + kh + d].astype(np.float64))
         for b in r for a in r for d in r]
    return I, J, t


@pytest.mark.parametrize("nx,ny", [(5, 7), (33, 30)])
def test_swap_windows(nx, ny):
    """Against float64: 13 roundings a term, and no further off than the
    reference's chain of 125 sums; an infinite or undefined level stays in the
    windows that hold it."""
    lib = _lib.load()
    nz, nzf = 12, 16
    grid_constants(lib, [(3 * nx, 3 * ny, nzf), (nx, ny, nz)], [10.0, 30.0], 0.001)
    g = np.random.default_rng(nx)
    host = {n: g.standard_normal(padded((3 * nx, 3 * ny, nzf))).astype(np.float32) for n in FIELDS}
    fine = {n: dev(a) for n, a in host.items()}
    coarse = {n: torch.zeros(padded((nx, ny, nz)), device="cuda") for n in FIELDS}
    swap(lib, fine, coarse, nx, ny)
    for n in FIELDS:
        kh0, nwin, di, dj = WINDOW[n]
        got = coarse[n].cpu().numpy()
        for lev in range(nwin):
            I, J, t = windows(host[n], nx, ny, 6 if lev else kh0, di, dj)
            want = sum(w * h for w, h in t)
            size = sum(w * np.abs(h) for w, h in t)
            chain = np.zeros(want.shape, np.float32)
            for w, h in t:
                chain = (w * h + chain.astype(np.float64)).astype(np.float32)
            err = got[I, J, ALIGN + nz - 2 + lev] - want
            assert (np.abs(err) <= 13 * EPS * size).all(), (n, lev)
            assert np.linalg.norm(err) <= np.linalg.norm(chain - want), (n, lev)
    clean = {n: coarse[n].clone() for n in FIELDS}
    for n in FIELDS:  # outside the first window of every field
        fine[n][:, :, ALIGN + 8] = float("inf")
        if WINDOW[n][0] == 4:
            fine[n][:, :, ALIGN + 1] = float("nan")
    swap(lib, fine, coarse, nx, ny)
    for n in FIELDS:
        level = ALIGN + nz - 2
        assert torch.equal(coarse[n][:, :, level], clean[n][:, :, level]), n
        if WINDOW[n][1] == 2:
            inner = coarse[n][NGSL:nx + NGSL + 5, NGSL:ny + NGSL + 5, level + 1]
            assert bool(torch.isinf(inner).all()), n
