"""Kernels launched behind a running predecessor must not name what it writes
``const ... __restrict__``: the qualifiers let the compiler load through the path
for data that stays constant from the launch's start to its end, and such a
launch starts before the predecessor has stored.  Checked in the sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "awp_b200",
                    "csrc")
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?"
                    r"(\w+)\s*\(")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in KERNEL.finditer(text):
            i, depth = text.index("{", m.end()), 0
            for q in range(i, len(text)):
                depth += {"{": 1, "}": -1}.get(text[q], 0)
                if depth == 0:
                    break
            yield m.group(1), text[m.start():q + 1]


def test_overlapped_kernels_load_plainly():
    found = dict(kernels())
    early = {n: t for n, t in found.items() if re.search(r"\bgrid_(start|wait)\(\)", t)}
    assert {"k_pack_vel", "k_adj_stress_gather", "k_addsrc_dev", "k_velocity_tma"} <= set(early)
    bad = [n for n, t in early.items()
           if re.search(r"const\s+\w+\s*\*\s*(const\s+)?__restrict__", t)]
    assert not bad, bad
