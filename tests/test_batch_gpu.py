"""Batched instances (awp_batch_*): many independent simulations of uneven
sizes advanced as parallel branches of their own launches, replayed as CUDA
graphs of up to eight steps.  The batch leaves each instance's arithmetic unchanged, so every field of
every instance must equal, bit for bit, the same run through awp_step."""
import ctypes

import numpy as np
import pytest

from awp_b200 import AwpError, Batch, Solver, _lib, default_params, pointfiles, scenarios, tune

pytestmark = pytest.mark.gpu

F32 = ctypes.POINTER(ctypes.c_float)
FIELDS = ["u1", "v1", "w1", "xx", "yy", "zz", "xy", "xz", "yz", "r1", "r2", "r3", "r4", "r5",
          "r6"]

# (nx, ny, nz, q, ifault, seed): uneven sizes, anelastic and elastic, point
# and kinematic sources
INSTANCES = [(24, 20, 32, True, 1, 3), (40, 28, 16, True, 5, 4), (16, 16, 32, False, 1, 5),
             (32, 24, 24, True, 1, 6), (20, 36, 20, False, 5, 7)]


def make(spec, steps):
    nx, ny, nz, q, ifault, seed = spec
    scn = scenarios.random_small(nx=nx, ny=ny, nz=nz, q=q, ifault=ifault, steps=steps,
                                 seed=seed, nsrc=2)
    s = Solver(default_params(**scn.params))
    s.upload_media(scn.media)
    s.upload_sources(scn.src_pos, scn.src_data)
    return s


# (the tile shape only changes the counts that info reports)
@pytest.mark.parametrize("mode,ty,ichunk,graph,branches",
                         [(0, 8, 16, True, 0), (0, 4, 8, True, 0), (0, 8, 32, False, 0),
                          (1, 8, 16, True, 0), (1, 8, 16, True, 2), (1, 8, 16, True, 1)])
def test_batch_equals_plain_runs(mode, ty, ichunk, graph, branches):
    steps = 12
    plain = [make(sp, steps) for sp in INSTANCES]
    for s in plain:
        s.step(steps)
        s.synchronize()
    want = [{f: s.field(f) for f in FIELDS} for s in plain]
    for s in plain:
        s.close()

    solvers = [make(sp, steps) for sp in INSTANCES]
    b = Batch(solvers)
    b.set_mode(mode)
    b.set_shape(ty, ichunk)
    b.set_graph(graph)
    # mode 1 with fewer branches than instances deals several instances'
    # launches onto one captured branch
    b.set_branches(branches)
    info = b.info()
    assert info["instances"] == len(INSTANCES)
    b.step(5)
    b.step(steps - 5)  # the first five directly, these as a graph
    b.synchronize()
    for n, s in enumerate(solvers):
        assert s.current_step == steps
        for f in FIELDS:
            got = s.field(f)
            assert np.array_equal(got.view(np.uint32), want[n][f].view(np.uint32)), (n, f)
    b.close()
    for s in solvers:
        s.close()


def run_plain(calls, steps):
    """The instances stepped by awp_step through `calls`: step counts, and functions
    of the solvers between them."""
    solvers = [make(sp, steps) for sp in INSTANCES]
    for c in calls:
        if callable(c):
            c(solvers)
        else:
            for s in solvers:
                s.step(c)
    out = []
    for s in solvers:
        s.synchronize()
        out.append({f: s.field(f) for f in FIELDS})
        s.close()
    return out


def run_batch(calls, steps, mode=0, branches=0):
    solvers = [make(sp, steps) for sp in INSTANCES]
    b = Batch(solvers)
    b.set_mode(mode)
    b.set_branches(branches)
    for c in calls:
        c(solvers) if callable(c) else b.step(c)
    b.synchronize()
    out = [{f: s.field(f) for f in FIELDS} for s in solvers]
    b.close()
    for s in solvers:
        s.close()
    return out


def assert_same(got, want):
    for n, (g, w) in enumerate(zip(got, want)):
        for f in FIELDS:
            assert np.array_equal(g[f].view(np.uint32), w[f].view(np.uint32)), (n, f)


@pytest.mark.parametrize("mode,branches", [(0, 0), (0, 2), (1, 0), (1, 1)])
def test_graphs_of_several_steps(mode, branches):
    """A direct call, a graph captured and replayed, a call of whole graphs and
    a remainder, and a replay after it; the point sources end (NST is two steps
    more than the scenario's) inside one of the graphs."""
    calls = [1, 3, 3, 17, 3, 1]
    assert_same(run_batch(calls, 12, mode, branches), run_plain(calls, 12))


@pytest.mark.parametrize("mode", [0, 1])
def test_sources_replaced_between_replays(mode):
    """New sources (another number, so other buffers) and inverse quality
    factors given to instances whose graphs exist: the next call must run with
    them, through graphs of both lengths used before and of one not yet used."""
    def replace(solvers):
        for n in (0, 3):
            nx, ny, nz, q, ifault, seed = INSTANCES[n]
            scn = scenarios.random_small(nx=nx, ny=ny, nz=nz, q=q, ifault=ifault, steps=40,
                                         seed=seed + 50, nsrc=5)
            solvers[n].upload_sources(scn.src_pos, scn.src_data)
        nx, ny, nz = INSTANCES[2][:3]  # elastic until here
        qinv = np.full((nz, ny, nx), 0.01, np.float32)
        s = solvers[2]
        _lib.check(s.lib.awp_set_qinv(s.ctx, qinv.ctypes.data_as(F32),
                                      qinv.ctypes.data_as(F32)), "awp_set_qinv")

    calls = [2, 3, 5, 3, replace, 3, 5, 4]
    assert_same(run_batch(calls, 40, mode), run_plain(calls, 40))


def test_every_graph_keeps_the_tuning_of_the_first_step():
    """Graphs captured later, of other lengths, run the kernel family in force
    at the first step.  With a poll limit of zero the pipelined family gives up
    at once (and says so at the next synchronisation); the read-only-path family
    has no such wait."""
    lib = _lib.load()
    saved = {k: lib.awp_get_tuning(k.encode()) for k in ("tma_vel", "tma_str", "spin_limit")}
    want = run_plain([1, 3, 4], 12)
    try:
        tune.set_tuning(lib, "tma", 0)
        solvers = [make(sp, 12) for sp in INSTANCES]
        b = Batch(solvers)
        b.step(1)
        tune.set_tuning(lib, "tma", 1)
        tune.set_tuning(lib, "spin_limit", 0)
        b.step(3)
        b.step(4)
        b.synchronize()
        tune.set_tuning(lib, "spin_limit", saved["spin_limit"])
        for s in solvers:
            s.synchronize()  # reports a march that gave up
        assert_same([{f: s.field(f) for f in FIELDS} for s in solvers], want)
        b.close()
        for s in solvers:
            s.close()
    finally:
        for k, v in saved.items():
            tune.set_tuning(lib, k, v)


def test_batch_then_plain_steps_continue():
    """Steps through the batch and then through awp_step on an instance agree
    with a run through awp_step alone."""
    spec = INSTANCES[0]
    ref = make(spec, 8)
    ref.step(8)
    ref.synchronize()
    want = ref.field("xx")
    ref.close()
    s = make(spec, 8)
    b = Batch([s])
    b.step(5)
    b.close()
    s.step(3)
    s.synchronize()
    assert np.array_equal(s.field("xx").view(np.uint32), want.view(np.uint32))
    s.close()


def test_batch_refusals(tmp_path):
    a = make(INSTANCES[0], 4)
    c = make(INSTANCES[2], 4)
    path = str(tmp_path / "recv.txt")
    pointfiles.write_input(path, str(tmp_path / "r"), [[800.0, 800.0, -400.0]], [0], degree=1)
    c.receivers(path, 5)
    with pytest.raises(AwpError) as e:
        Batch([a, c])
    assert e.value.status == 7  # AWP_ERR_UNSUPPORTED
    with pytest.raises(AwpError) as e:
        Batch([a, a])
    assert e.value.status == 1
    b = Batch([a])
    a.step(1)  # stepped outside the batch
    with pytest.raises(AwpError) as e:
        b.step(1)
    assert e.value.status == 3
    b.close()
    a.close()
    c.close()
