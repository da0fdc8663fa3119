"""The boxes of the NVE = 3 stress split, from the host code compiled alone.

The stress kernel updates the boxes of one launch beside each other, so they
must share no cell; boxes that do (grids of fewer than 20 rows, where the middle
band is empty) have to follow one another in stream order."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "awp_b200", "csrc")
NGSL = 8

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="g++ missing")

SHIM = """
#include "awp_host.h"
extern "C" void split(const int* all, int x0, int nxg, int sub, int* out) {
  AwpBox band, rest[4];
  awp::stress_split({all[0], all[1], all[2], all[3]}, x0, nxg, sub != 0, &band, rest);
  const AwpBox b[5] = {band, rest[0], rest[1], rest[2], rest[3]};
  for (int q = 0; q < 5; ++q) {
    out[4 * q] = b[q].i0; out[4 * q + 1] = b[q].i1;
    out[4 * q + 2] = b[q].j0; out[4 * q + 3] = b[q].j1;
  }
}
extern "C" int run(const int* b, int n) {
  return awp::disjoint_run(reinterpret_cast<const AwpBox*>(b), n);
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "split.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC,
                    str(d / "shim.cpp"), os.path.join(CSRC, "awp_host.cpp"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def boxes(host, all_, x0=0, nxg=0, sub=False):
    out = (ctypes.c_int * 20)()
    host.split((ctypes.c_int * 4)(*all_), x0, nxg, int(sub), out)
    return [tuple(out[4 * q:4 * q + 4]) for q in range(5)]


def cells(b):
    return {(i, j) for i in range(b[0], b[1] + 1) for j in range(b[2], b[3] + 1)}


def launches(host, rest):
    """The runs of boxes that go into one launch each."""
    flat = (ctypes.c_int * 16)(*[v for b in rest for v in b])
    got, q = [], 0
    while q < 4:
        n = host.run(ctypes.byref(flat, 16 * q), 4 - q)
        assert n >= 1
        got.append(rest[q:q + n])
        q += n
    return got


@pytest.mark.parametrize("nx", [4, 9, 33])
@pytest.mark.parametrize("ny", [4, 9, 10, 12, 19, 20, 21, 40, 41])
def test_boxes_of_a_launch_share_no_cell(host, nx, ny):
    all_ = (2 + NGSL, nx + NGSL + 1, 2 + NGSL, ny + NGSL + 1)
    band, *rest = boxes(host, all_, 0, nx)
    runs = launches(host, rest)
    assert [b for r in runs for b in r] == rest
    for r in runs:
        assert sum(len(cells(b)) for b in r) == len(set().union(*map(cells, r)))
    every = [c for b in rest for c in sorted(cells(b))] + sorted(cells(band))
    assert cells(all_) <= set(every)
    if ny >= 20:  # the split itself is a partition, one launch
        assert len(runs) == 1 and len(every) == len(set(every)) == nx * ny
    elif nx > 4:  # front and back rows overlap: the back box comes after
        assert len(runs) == 2 and runs[1][0] == rest[1]


@pytest.mark.parametrize("ny", [12, 24])
def test_parts_split_the_grid_s_boxes(host, ny):
    """A sub-domain's boxes are the grid's, cut at its columns."""
    nxg = 20
    j0, j1 = 2 + NGSL, ny + NGSL + 1
    whole = boxes(host, (2 + NGSL, nxg + NGSL + 1, j0, j1), 0, nxg)
    got = [set() for _ in range(5)]
    for x0, nx in ((0, 4), (4, 9), (13, 7)):
        part = boxes(host, (2 + NGSL, nx + NGSL + 1, j0, j1), x0, nxg, True)
        for r in launches(host, part[1:]):
            assert sum(len(cells(b)) for b in r) == len(set().union(*map(cells, r)))
        for q in range(5):
            got[q] |= {(i + x0, j) for i, j in cells(part[q])}
    assert got == [cells(b) for b in whole]
