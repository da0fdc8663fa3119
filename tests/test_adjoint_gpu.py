"""Adjoint gradient of the seismogram misfit (awp_misfit_gradient).

The GPU gradient (hand-written discrete-adjoint kernels, FP32, checkpointed)
is checked along seeded directions dm = (dlambda, dmu, drho) against
  * the FP64 oracle's exact derivative of the same discrete scheme (the oracle
    run on dual numbers: tangent-linear mode, oracle/awp_oracle.cpp), and
  * central finite differences of the FP32 GPU misfit, eps = 1e-3 relative.
Elastic and anelastic (memory variables on) models; receivers at the free
surface and inside."""
import numpy as np
import pytest
import torch

from awp_b200 import Solver, adjoint, default_params, scenarios
from oracle import oracle as orc
from oracle import refbind

pytestmark = pytest.mark.gpu


def moduli(scn):
    m = scn.media
    vp, vs, rho = (m[..., q].astype(np.float64) for q in range(3))
    mu = rho * vs * vs
    lam = rho * (vp * vp - 2 * vs * vs)
    return lam.astype(np.float32), mu.astype(np.float32), rho.astype(np.float32)


def padded(x, p):
    """Interior [nz][ny][nx] (surface first) -> padded kernel layout with the
    one-cell border copy of the media set-up."""
    nx, ny, nz = p["nx"], p["ny"], p["nz"]
    out = np.zeros(refbind.padded_shape(nx, ny, nz), x.dtype)
    core = np.ascontiguousarray(x.transpose(2, 1, 0)[:, :, ::-1])
    out[9:nx + 11, 9:ny + 11, 31:nz + 33] = np.pad(core, 1, mode="edge")
    return out


def receivers(scn):
    p = scn.params
    sx, sy = int(scn.src_pos[0, 0]) - 1, int(scn.src_pos[0, 1]) - 1
    xyz = [(sx + 2, sy, 0), (sx - 3, sy + 2, 0), (sx, sy - 3, 0), (sx + 1, sy + 1, 3),
           (sx - 2, sy - 1, 5), (sx + 3, sy + 3, 2)]
    xyz = [(min(max(x, 0), p["nx"] - 1), min(max(y, 0), p["ny"] - 1), z) for x, y, z in xyz]
    comp = [0, 1, 2, 2, 0, 1]
    return np.asarray(xyz, np.int32), np.asarray(comp, np.int32)


def setup_case(q, seed=11, steps=40, shape=(16, 16, 16)):
    scn = scenarios.random_small(nx=shape[0], ny=shape[1], nz=shape[2], q=q, ifault=1,
                                 steps=steps, seed=seed, nsrc=1)
    s = Solver(default_params(**scn.params))
    s.upload_media(scn.media)
    s.upload_sources(scn.src_pos, scn.src_data)
    lam, mu, rho = moduli(scn)
    rng = np.random.default_rng(seed + 1)
    pert = [(1 + 0.05 * rng.standard_normal(lam.shape)).astype(np.float32) for _ in range(3)]
    xyz, comp = receivers(scn)
    s.set_moduli(lam * pert[0], mu * pert[1], rho * pert[2])
    s.reset()
    d_obs = adjoint.seismograms(s, steps, xyz, comp)
    return scn, s, (lam, mu, rho), xyz, comp, d_obs


def J_at(s, m, steps, xyz, comp, d_obs):
    s.set_moduli(*m)
    s.reset()
    seis = adjoint.seismograms(s, steps, xyz, comp).astype(np.float64)
    return 0.5 * float(np.sum((seis - d_obs) ** 2))


def oracle_directional(scn, m, dm, steps, xyz, comp, d_obs):
    """sum_n sum_r (s - d) ds along dm, by the FP64 dual-number oracle."""
    p = scn.params
    setup = refbind.model_setup(scn)
    o = orc.OracleSim(scn, setup, precision=65)
    lam, mu, rho = (x.astype(np.float64) for x in m)
    dl, dmu, dr = (x.astype(np.float64) for x in dm)
    o.set_field("lam", padded((np.float32(1) / m[0]).astype(np.float32), p))
    o.set_field("mu", padded((np.float32(1) / m[1]).astype(np.float32), p))
    o.set_field("d1", padded(m[2], p))
    o.set_tangent("lam", padded(-dl / (lam * lam), p))
    o.set_tangent("mu", padded(-dmu / (mu * mu), p))
    o.set_tangent("d1", padded(dr, p))
    o.compute_lam_mu()
    names = ["u1", "v1", "w1"]
    idx = [(x + 10, y + 10, p["nz"] + 31 - z) for x, y, z in xyz]
    total = 0.0
    for n in range(steps):
        o.step(1)
        vals = {f: o.field(f, f64=True) for f in set(names[c] for c in comp)}
        tans = {f: o.tangent(f) for f in vals}
        for r, (c, ix) in enumerate(zip(comp, idx)):
            total += (vals[names[c]][ix] - d_obs[n, r]) * tans[names[c]][ix]
    o.close()
    return total


# odd nx and ny: the velocity update covers one row beyond the stress window
# (ny rounded up to even), so the image-adjoint ring row enters the velocity
# transpose there
@pytest.mark.parametrize("q,shape", [(True, (16, 16, 16)), (False, (16, 16, 16)),
                                     (True, (15, 17, 16))])
def test_gradient_matches_oracle_and_finite_differences(q, shape):
    steps = 40
    scn, s, m, xyz, comp, d_obs = setup_case(q, steps=steps, shape=shape)
    s.set_moduli(*m)
    s.reset()
    J, seis, gl, gm, gr = adjoint.misfit_gradient(s, steps, xyz, comp, d_obs)
    assert J > 0 and np.isfinite(J)
    assert s.current_step == steps
    assert np.all(np.isfinite(gl)) and np.all(np.isfinite(gm)) and np.all(np.isfinite(gr))
    rng = np.random.default_rng(5)
    eps = 1e-3
    for d in range(3):
        dm = tuple((x * rng.standard_normal(x.shape)).astype(np.float64) for x in m)
        adj = float(np.sum(gl * dm[0]) + np.sum(gm * dm[1]) + np.sum(gr * dm[2]))
        tan = oracle_directional(scn, m, dm, steps, xyz, comp, d_obs)
        assert abs(adj - tan) <= 1e-3 * abs(tan), (d, adj, tan)
        mp = tuple((x + eps * y).astype(np.float32) for x, y in zip(m, dm))
        mm = tuple((x - eps * y).astype(np.float32) for x, y in zip(m, dm))
        fd = (J_at(s, mp, steps, xyz, comp, d_obs) - J_at(s, mm, steps, xyz, comp, d_obs)) / (2 * eps)
        assert abs(adj - fd) <= 1e-3 * abs(adj), (d, adj, fd)
        print(f"direction {d}: adjoint {adj:.6e}  oracle tangent {tan:.6e}  FD {fd:.6e}")
    s.close()


def test_checkpoint_count_does_not_change_the_gradient():
    steps = 24
    scn, s, m, xyz, comp, d_obs = setup_case(True, seed=21, steps=steps)
    out = []
    for nsnap in (1, 5, 24, 0):  # 0: the velocities of as many last steps as fit are kept
        plan = adjoint.adjoint_plan(s, steps, nsnap)
        adjoint.adjoint_reserve(s, steps, nsnap)  # the call below reuses it
        if nsnap > 0:  # snapshots at the segment starts plus the final state
            assert plan["tail_steps"] == 0
            assert plan["segment_steps"] == -(-steps // nsnap)
            assert plan["snapshots"] == -(-steps // plan["segment_steps"]) + 1
        else:  # a small grid: every step keeps its velocities
            assert plan["tail_steps"] == steps and plan["snapshots"] == 1
        s.set_moduli(*m)
        s.reset()
        out.append(adjoint.misfit_gradient(s, steps, xyz, comp, d_obs, nsnap=nsnap))
    for o in out[1:]:
        assert o[0] == out[0][0]
        for a, b in zip(o[2:], out[0][2:]):
            assert np.array_equal(a, b)
    s.close()


def test_torch_autograd_function():
    steps = 16
    scn, s, m, xyz, comp, d_obs = setup_case(True, seed=31, steps=steps)
    t = [torch.tensor(x, requires_grad=True) for x in m]
    J = adjoint.misfit(*t, s, steps, xyz, comp, d_obs)
    J.backward()
    s.set_moduli(*m)
    s.reset()
    J2, _, gl, gm, gr = adjoint.misfit_gradient(s, steps, xyz, comp, d_obs)
    assert float(J) == J2
    assert np.array_equal(t[0].grad.numpy(), gl)
    assert np.array_equal(t[1].grad.numpy(), gm)
    assert np.array_equal(t[2].grad.numpy(), gr)
    s.close()


def test_multishot_gradient_is_the_sum_of_the_shots():
    steps = 24
    scn, s, m, xyz, comp, _ = setup_case(True, seed=41, steps=steps)
    rng = np.random.default_rng(42)
    shots = []
    for q in range(2):
        pos = scn.src_pos.copy()
        pos[0, 0] = min(max(int(pos[0, 0]) + (3 if q else -3), 2), scn.params["nx"] - 2)
        data = (scn.src_data * (1.0 + 0.5 * q)).astype(np.float32)
        # observed data of the perturbed model for this shot
        s.upload_sources(pos, data)
        pert = [(x * (1 + 0.03 * rng.standard_normal(x.shape))).astype(np.float32) for x in m]
        s.set_moduli(*pert)
        s.reset()
        d_obs = adjoint.seismograms(s, steps, xyz, comp)
        shots.append((pos, data, xyz, comp, d_obs))
    s.set_moduli(*m)
    J, gl, gm, gr = adjoint.misfit_gradient_shots(s, steps, shots)
    Jsum, gsum = 0.0, [np.zeros(x.shape) for x in m]
    for pos, data, rxyz, rcomp, d_obs in shots:
        s.upload_sources(pos, data)
        s.set_moduli(*m)
        s.reset()
        Js, _, a, b, c = adjoint.misfit_gradient(s, steps, rxyz, rcomp, d_obs)
        Jsum += Js
        for acc, x in zip(gsum, (a, b, c)):
            acc += x
    assert J == Jsum
    for x, y in zip((gl, gm, gr), gsum):
        assert np.array_equal(x, y)
    # the summed gradient against central differences of the summed misfit
    dm = tuple((x * rng.standard_normal(x.shape)).astype(np.float64) for x in m)
    adj = float(np.sum(gl * dm[0]) + np.sum(gm * dm[1]) + np.sum(gr * dm[2]))
    eps = 1e-3

    def J_all(mm):
        tot = 0.0
        for pos, data, rxyz, rcomp, d_obs in shots:
            s.upload_sources(pos, data)
            tot += J_at(s, mm, steps, rxyz, rcomp, d_obs)
        return tot
    mp = tuple((x + eps * y).astype(np.float32) for x, y in zip(m, dm))
    mm_ = tuple((x - eps * y).astype(np.float32) for x, y in zip(m, dm))
    fd = (J_all(mp) - J_all(mm_)) / (2 * eps)
    assert abs(adj - fd) <= 1e-3 * abs(adj), (adj, fd)
    s.close()


def interior(x, p):
    """Padded kernel layout -> interior [nz][ny][nx], surface first."""
    nx, ny, nz = p["nx"], p["ny"], p["nz"]
    return np.ascontiguousarray(x[10:nx + 10, 10:ny + 10, 32:nz + 32][:, :, ::-1].transpose(2, 1, 0))


def oracle_directional_q(scn, m, qinv, dq, steps, xyz, comp, d_obs):
    """sum_n sum_r (s - d) ds along a direction dq = (dQp^-1, dQs^-1), by the
    FP64 dual-number oracle (moduli and density held)."""
    p = scn.params
    setup = refbind.model_setup(scn)
    o = orc.OracleSim(scn, setup, precision=65)
    o.set_field("lam", padded((np.float32(1) / m[0]).astype(np.float32), p))
    o.set_field("mu", padded((np.float32(1) / m[1]).astype(np.float32), p))
    o.set_field("d1", padded(m[2], p))
    o.set_field("qp", padded(qinv[0], p))
    o.set_field("qs", padded(qinv[1], p))
    o.set_tangent("qp", padded(dq[0].astype(np.float64), p))
    o.set_tangent("qs", padded(dq[1].astype(np.float64), p))
    o.compute_lam_mu()
    names = ["u1", "v1", "w1"]
    idx = [(x + 10, y + 10, p["nz"] + 31 - z) for x, y, z in xyz]
    total = 0.0
    for n in range(steps):
        o.step(1)
        vals = {f: o.field(f, f64=True) for f in set(names[c] for c in comp)}
        tans = {f: o.tangent(f) for f in vals}
        for r, (c, ix) in enumerate(zip(comp, idx)):
            total += (vals[names[c]][ix] - d_obs[n, r]) * tans[names[c]][ix]
    o.close()
    return total


@pytest.mark.parametrize("shape,qrange", [((16, 16, 16), (20.0, 180.0)),
                                          ((15, 17, 16), (600.0, 2000.0))])
def test_q_gradient_matches_oracle_and_finite_differences(shape, qrange):
    """dJ/dQp^-1 and dJ/dQs^-1 of an anelastic model (awp_misfit_gradient_q):
    along seeded directions, against the FP64 dual oracle's exact derivative
    and five-point central differences (eps = 3e-3 relative).  The Q(f) weight switches
    between its low-Q polynomial and its linear form at Q = 400 (kernel.cu:
    974-1040), where it is not continuous; the derivative holds the branch, so
    the models here sit on one side of the switch: Q in [20, 180] (polynomial
    everywhere) and in [600, 2000] (linear everywhere)."""
    steps = 40
    scn, s, m, xyz, comp, d_obs = setup_case(True, seed=51, steps=steps, shape=shape)
    p = scn.params
    rng = np.random.default_rng(53)
    nq = (p["nz"], p["ny"], p["nx"])
    qinv = tuple((1.0 / rng.uniform(qrange[0], qrange[1], nq)).astype(np.float32)
                 for _ in range(2))
    s.set_qinv(*qinv)
    # the observed data of the perturbed model with these Q
    pert = [(1 + 0.05 * rng.standard_normal(x.shape)).astype(np.float32) for x in m]
    s.set_moduli(*[x * q for x, q in zip(m, pert)])
    s.reset()
    d_obs = adjoint.seismograms(s, steps, xyz, comp)
    s.set_moduli(*m)
    s.reset()
    J, _, gl, gm, gr, gqp, gqs = adjoint.misfit_gradient(s, steps, xyz, comp, d_obs, want_q=True)
    # the lambda / mu / rho gradients are those of the call without Q
    s.reset()
    J0, _, gl0, gm0, gr0 = adjoint.misfit_gradient(s, steps, xyz, comp, d_obs)
    assert J == J0 and np.array_equal(gl, gl0) and np.array_equal(gr, gr0)
    assert np.abs(gqp).max() > 0 and np.abs(gqs).max() > 0
    rng = np.random.default_rng(52)
    # the misfit is far more curved in Q^-1 than in the moduli (the Q(f)
    # weights are quadratic in Q^-1 on the low-Q branch) and its FP32 rounding
    # noise is ~4e-6 J: the two-point central difference is off by ~0.3 % at
    # eps = 1e-3 (curvature) and by ~1.6 % at 1e-4 (noise), so the differences
    # here take the fourth-order five-point stencil at eps = 3e-3, where both
    # stay near 0.1 %
    eps = 3e-3
    for d in range(2):
        dq = tuple((x * rng.standard_normal(x.shape)).astype(np.float64) for x in qinv)
        adj = float(np.sum(gqp * dq[0]) + np.sum(gqs * dq[1]))
        tan = oracle_directional_q(scn, m, qinv, dq, steps, xyz, comp, d_obs)

        def J_q(q):
            s.set_moduli(*m)
            s.set_qinv(*q)
            s.reset()
            seis = adjoint.seismograms(s, steps, xyz, comp).astype(np.float64)
            return 0.5 * float(np.sum((seis - d_obs) ** 2))
        def J_at_q(t):
            return J_q(tuple((x + t * y).astype(np.float32) for x, y in zip(qinv, dq)))
        Jp, Jm = J_at_q(eps), J_at_q(-eps)
        Jp2, Jm2 = J_at_q(2 * eps), J_at_q(-2 * eps)
        fd = (8 * (Jp - Jm) - (Jp2 - Jm2)) / (12 * eps)
        s.set_qinv(*qinv)
        print(f"Q direction {d}: adjoint {adj:.6e}  oracle tangent {tan:.6e}  FD {fd:.6e}  "
              f"(J {J:.6e}, J+ - J- {Jp - Jm:.3e})")
        assert abs(adj - tan) <= 1e-3 * abs(tan), (d, adj, tan, fd)
        # the misfit moves by 2 eps |dJ| between the two runs; where that is
        # within a few 1e-5 of J the FP32 forward runs cannot resolve it, and
        # the exact-derivative check above is the one that holds
        if 2 * eps * abs(adj) > 3e-4 * J:
            assert abs(adj - fd) <= 5e-3 * abs(adj), (d, adj, fd)
    s.close()


def test_torch_autograd_on_device_tensors():
    """The autograd Function passes CUDA tensors to the library by pointer and
    returns the same gradients as the host-array call."""
    steps = 16
    scn, s, m, xyz, comp, d_obs = setup_case(True, seed=61, steps=steps)
    t = [torch.tensor(x, device="cuda", requires_grad=True) for x in m]
    J = adjoint.misfit(*t, s, steps, xyz, comp, d_obs)
    J.backward()
    s.set_moduli(*m)
    s.reset()
    J2, _, gl, gm, gr = adjoint.misfit_gradient(s, steps, xyz, comp, d_obs)
    assert float(J.detach()) == J2
    for tt, g in zip(t, (gl, gm, gr)):
        assert tt.grad.is_cuda
        assert np.array_equal(tt.grad.cpu().numpy(), g)
    s.close()


def test_kept_scratch_does_not_shrink_the_plan():
    """The seismogram scratch of a large call stays with the context; it counts as
    free when the workspace is planned, and it is counted in device_bytes."""
    scn, s, m, xyz, comp, d_obs = setup_case(False, steps=10)
    before = adjoint.adjoint_plan(s, 4_000_000)["tail_steps"]
    held = s.device_bytes
    steps, nrec = 500, 200_000  # 0.4 GB of samples
    rng = np.random.default_rng(0)
    p = scn.params
    pos = np.stack([rng.integers(0, p[n], nrec) for n in ("nx", "ny", "nz")], 1).astype(np.int32)
    adjoint.seismograms(s, steps, pos, np.zeros(nrec, np.int32))
    assert s.device_bytes >= held + 4 * steps * nrec
    after = adjoint.adjoint_plan(s, 4_000_000)["tail_steps"]
    assert 0 < before < 4_000_000  # the plan is limited by the memory
    # a few MB of driver allocations aside: 0.4 GB are some thousand steps here
    assert before - after < 300, (before, after)
    adjoint.adjoint_reserve(s, 200)  # a larger workspace: the scratch is given back
    assert s.device_bytes <= held  # (held: with the small scratch of the set-up's call)
    s.close()
