"""Time steps against a float64 restatement, at the sizes where tiles end.

perf/cases.py restates every phase of the step in float64 with plain torch
operations (``exact``); here its inputs are run at sizes around the kernels'
tile edges: z columns of the 32-level Cartesian and the 64/56-level
curvilinear tiles, y rows around 8 and 7, x ranges shorter than a march and
one plane past it.  A float32 step rounds each update a few times; over the
2-3 steps run here the accumulated relative L2 difference is a few 1e-7
(measured 0.5-9e-7 over these cases), so 3e-6 leaves a factor of three."""
import importlib.util
import os

import numpy as np
import pytest
import torch

from awp_b200 import _lib, tune

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def cases():
    spec = importlib.util.spec_from_file_location(
        "perf_cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def leaves(v):
    if isinstance(v, dict):
        for k in sorted(v):
            yield from ((f"{k}.{n}", x) for n, x in leaves(v[k]))
    elif isinstance(v, (list, tuple)):
        for i, x in enumerate(v):
            yield from ((f"{i}.{n}", y) for n, y in leaves(x))
    else:
        yield "", v


def grid(nx, ny, nz, q=True, steps=3, **kw):
    return dict(dict(kind="grid", nx=nx, ny=ny, nz=nz, q=q, steps=steps, fault=False,
                     gather=False), **kw)


CASES = [
    grid(24, 24, 8), grid(25, 31, 32), grid(33, 33, 36, q=False), grid(27, 41, 64, gather=True),
    grid(39, 26, 100, fault=True),
    dict(kind="hill", nx=24, ny=25, nz=12, q=True, steps=2),
    dict(kind="hill", nx=29, ny=31, nz=60, q=False, steps=2),
    dict(kind="hill", nx=26, ny=36, nz=64, q=True, steps=2),
    dict(kind="hill", nx=41, ny=30, nz=68, q=True, steps=2),
    dict(kind="hill", nx=25, ny=28, nz=120, q=False, steps=2),
    dict(kind="hill", nx=37, ny=27, nz=124, q=True, steps=2),
    dict(kind="plastic", nx=41, ny=43, nz=36, q=True, steps=3),
    dict(kind="plastic", nx=44, ny=40, nz=64, q=False, steps=3),
    dict(kind="mesh", nx=20, ny=21, nz=32, nzc=24, steps=3, hill=False, plastic=False),
    dict(kind="mesh", nx=22, ny=20, nz=68, nzc=36, steps=3, hill=True, plastic=True),
    dict(kind="ensemble", n=3, lo=40, hi=70, steps=3, mode=0, draw=3),
    dict(kind="ensemble", n=3, lo=40, hi=70, steps=3, mode=1, draw=4),
    dict(kind="ensemble", n=2, lo=40, hi=50, steps=11, mode=1, draw=5),  # as graphs of 8 and 3
    dict(kind="gradient", nx=36, ny=33, nz=32, steps=14, q=True, nrec=9, nsnap=0),
    dict(kind="gradient", nx=33, ny=36, nz=36, steps=13, q=False, nrec=9, nsnap=3),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c['kind']}-{c.get('nx', c.get('n'))}-"
                         f"{c.get('nz', c.get('mode'))}")
def test_steps_match_float64(case):
    m = cases()
    st = m.prepare(case, 5)
    got = dict(leaves(m.run(st)))
    torch.cuda.synchronize()
    want = dict(leaves(m.exact(case, 5)))
    assert set(got) == set(want)
    for name, x in got.items():
        x, y = torch.as_tensor(x).double(), torch.as_tensor(want[name]).double()
        ref = float(y.norm())
        assert float((x.to(y.device) - y).norm()) <= 3e-6 * ref, (name, ref)


@pytest.mark.parametrize("nx", [40, 45, 47])
def test_plastic_return_of_every_cell(nx):
    """No cohesion and no friction: every cell yields, so the return takes the
    path of a changed cell on whole planes; widths of a multiple of the planes
    a thread reads and of remainders, the stress split's narrow boxes with
    them.  Checked are the fields the return writes (the memory variables'
    increments are differences of neighbouring velocities, in which the
    velocities' rounding of 1e-6 weighs several times as much)."""
    m = cases()
    inputs = m._yield_inputs

    def weak(*args):
        s2, cohes, phi = inputs(*args)
        return s2, 0 * cohes, 0 * phi

    m._yield_inputs = weak
    case = dict(kind="plastic", nx=nx, ny=41, nz=32, q=True, steps=3)
    st = m.prepare(case, 5)
    got = m.run(st)
    torch.cuda.synchronize()
    ny, nz = case["ny"], case["nz"]
    assert int((got["yldfac"] < 1).sum()) > 0.9 * nx * ny * nz
    want = m.exact(case, 5)
    for name in ("xx", "yy", "zz", "xy", "xz", "yz", "yldfac", "neta"):
        x, y = got[name].double(), torch.as_tensor(want[name]).double()
        assert float((x.to(y.device) - y).norm()) <= 3e-6 * float(y.norm()), name


BESIDE = [
    grid(150, 120, 96, steps=6), grid(150, 120, 96, q=False, steps=6),
    dict(kind="hill", nx=120, ny=100, nz=96, q=True, steps=4),
    dict(kind="hill", nx=121, ny=99, nz=68, q=False, steps=4),
    dict(kind="plastic", nx=130, ny=101, nz=64, q=True, steps=4),
    dict(kind="mesh", nx=45, ny=40, nz=64, nzc=48, steps=4, hill=False, plastic=False),
    dict(kind="mesh", nx=40, ny=41, nz=68, nzc=32, steps=4, hill=True, plastic=True),
]


@pytest.mark.parametrize("case", BESIDE, ids=lambda c: f"{c['kind']}-{c['nx']}-{c['nz']}")
def test_marches_beside_another_context(case):
    """Two contexts on their own streams share the SMs; each must leave the
    fields it leaves alone, bit for bit (the producer may refill a slot only
    when every lane has its values, however long its warp waits): every
    variant of the pipelined kernels, the one of several boxes and those that
    take a mesh block's interface layer among them."""
    m = cases()
    alone = m.prepare(case, 1)
    m.run(alone)
    torch.cuda.synchronize()
    want = {f: v.clone() for f, v in alone["out"].items()}
    for _ in range(3):
        a, b = m.prepare(case, 1), m.prepare(case, 2)
        b2 = m.prepare(case, 3)
        m.run(b)
        m.run(a)
        m.run(b2)
        torch.cuda.synchronize()
        for f, v in a["out"].items():
            assert torch.equal(v.view(torch.int32), want[f].view(torch.int32)), f


def test_march_length_does_not_change_curvilinear_fields():
    lib = _lib.load()
    saved = tune.get_tuning(lib)
    m = cases()
    case = dict(kind="hill", nx=45, ny=30, nz=68, q=True, steps=3)
    want = None
    try:
        for ich in (4, 7, 32):
            tune.set_tuning(lib, "ichunk", ich)
            st = m.prepare(case, 2)
            out = m.run(st)
            torch.cuda.synchronize()
            got = {f: v.cpu().numpy().view(np.uint32).copy() for f, v in out.items()}
            if want is None:
                want = got
            for f in got:
                assert np.array_equal(got[f], want[f]), (f, ich)
    finally:
        for k, v in saved.items():
            tune.set_tuning(lib, k, v)


@pytest.mark.parametrize("ny", [12, 19, 20])
def test_overlapping_stress_boxes_follow_one_another(ny):
    """Below 20 rows the boxes around the plasticity band share rows; the TMA
    kernel must update them in the order of the read-only-path family, which
    takes one box a launch, bit for bit."""
    lib = _lib.load()
    saved = tune.get_tuning(lib)
    m = cases()
    case = dict(kind="plastic", nx=41, ny=ny, nz=36, q=True, steps=3)
    got = []
    try:
        for family in (0, 1):
            tune.set_tuning(lib, "tma_str", family)
            st = m.prepare(case, 4)
            out = m.run(st)
            torch.cuda.synchronize()
            got.append({f: v.cpu().numpy().view(np.uint32).copy() for f, v in out.items()})
    finally:
        for k, v in saved.items():
            tune.set_tuning(lib, k, v)
    for f in got[0]:
        assert np.array_equal(got[0][f], got[1][f]), f
