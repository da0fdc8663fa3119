// Discrete adjoint of the single-grid time step and the material gradient of
// a seismogram misfit.
//
// The forward step (one_step: dvelcx, dstrqc with its free-surface velocity
// images, point sources, fstr) is linear in the wavefield state for fixed
// materials, so its adjoint is the transpose of each map in reverse order:
//
//   fstr^T -> stress^T (memory variables, strain rates, then the images) ->
//   velocity^T
//
// (the fstr transpose is folded into the stress kernel's top three cells; the
// imaged values above the surface are cleared with the velocity images).  The
// free-surface imaging of the rows beyond the stress range (the extra row of
// an odd ny) acts on values that stay zero, so it has no transpose to apply.
//
// The density term needs the stress divergence the velocity update applied;
// it is recovered from the velocities before and after the step
// (fd * D(sigma) = u'/dc - u), so the segment store holds velocities only.
// Every transpose is written in gather form (each thread owns one output
// cell and reads the neighbours whose forward stencils touched it), so no
// atomics are needed and the result is deterministic.  The gradient terms use
// the forward state of the same step (stresses before it for the density
// term, velocities after it for the moduli terms).  Derivation, per map:
//
//   velocity  u' = (u + fd(rho) * D(sigma)) * dc          (dvelcx, kernel.cu:222-253)
//   stress    s' = K (s + P(e) + a r + DT (Q(e)(w-1) + g r)),  r' = b r + w Q(e)
//             (yy, zz carry K twice; dstrqc, kernel.cu:1114-1179)
//   images    u(top+1) = u - (w - w_{i-1}), v(top+1) = v - (w_{j+1} - w),
//             w(top+1) = w(top-1) - lam_mu * Z(u, v, w)     (kernel.cu:1087-1112)
//   fstr      zz(top+1) = -zz(top), ..., xz(top) = yz(top) = 0  (kernel.cu:1616-1647)
#include "awp_adjoint.cuh"

#include "awp_pipe.cuh"
#include "awp_stencil.cuh"

namespace {

enum { LU, LV, LW, LXX, LYY, LZZ, LXY, LXZ, LYZ, LR1, LR2, LR3, LR4, LR5, LR6 };
enum { E1, E2, E3, E4, E5, E6, GL8, GM8, GP1, GP2, GP3, GQP8, GQS8, GQ1, GQ2, GQ3 };

enum { VA, VB, VC, VEA, VEB, VEC };

// Two vertically adjacent cells per thread (the pair starts on an even level,
// so every access is 8-byte aligned), computed with packed arithmetic.
__device__ __forceinline__ float2 ld2(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
__device__ __forceinline__ void st2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
__device__ __forceinline__ void st2(float* p, float2 v, bool ax, bool ay) {
  if (ax && ay) {
    st2(p, v);
  } else {
    if (ax) p[0] = v.x;
    if (ay) p[1] = v.y;
  }
}
// Per-thread asynchronous 8-byte copy global -> shared (cp.async); a thread
// reads back only its own slots, after waiting for its group.
__device__ __forceinline__ void cpa8(float2* s, const float* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(s)),
               "l"(g)
               : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void pre2(const float* p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// Derivative of awp_weight (awp_stencil.cuh) with respect to S, the branch held
// as the forward takes it.
__device__ __forceinline__ float2 dweight(float2 S, const AwpRelax<float2>& t, unsigned thr) {
  const float2 p = vfma(vadd(t.c0, t.c0), S, t.c1);
  return make_float2(__float_as_uint(S.x) >= thr ? p.x : t.c2.x,
                     __float_as_uint(S.y) >= thr ? p.y : t.c2.y);
}

// ---------------------------------------------------------------------------
// stress^T, pointwise part: memory variables and stresses in place, adjoint
// strain rates of the cell into E[], its material weights added to the sums
// in E[].  188 bytes a cell.  A thread marches kSch x planes with the forward
// update's coefficients and register queues for the velocities and media; the
// cell's own adjoint stresses, memory variables and weight sums (read once and
// late) come one plane ahead by cp.async, so a plane's copies are in flight
// while the one before is computed; the next plane's first velocities and media
// are called into L2 at the same time.  Without Q sums 109 us at 160 x 144 x 96
// (0.58 of the copy bandwidth on these bytes): latency at twelve warps an SM.
// Marches of 8 or 16 planes and four CTAs an SM are 5-12 % slower, and without
// the L2 prefetch a whole gradient is 4 % slower.
// ---------------------------------------------------------------------------
constexpr int kSch = 4;

// WANTQ: also accumulate the Q^-1 weights (anelastic runs that ask for the
// Q^-1 gradients); without it the five Q sums are neither read nor written.
template <bool ELASTIC, bool WANTQ>
__global__ void __launch_bounds__(128, 3) k_adj_stress_cell(const __grid_constant__ AdjArgs a) {
  // staged, two planes: 0-5 stresses, 6-10 moduli sums, 11-16 memory
  // variables, 17-21 Q sums
  constexpr int NS = ELASTIC ? 11 : WANTQ ? 22 : 17;
  __shared__ float2 stg[2][NS][128];
  // relaxation constants of the entry pairs (e, e + 1), e even: nine float2
  // per pair in 20 floats (as k_stress_tma)
  __shared__ __align__(16) float tab[4 * 20];
  const int tid = threadIdx.x;
  awp_pipe::grid_go();
  if (!ELASTIC) {
    const float* const src[9] = {a.rel.vx2, a.rel.wwo, a.rel.kv, a.rel.kr, a.rel.kr2,
                                 a.rel.kf,  a.rel.c0,  a.rel.c1, a.rel.c2};
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (tid < 8) tab[(tid >> 1) * 20 + 2 * q + (tid & 1)] = src[q][tid];
    __syncthreads();
  }
  awp_pipe::grid_wait();
  // flat (j, level pair): pairs of levels from the even one at or below sk0
  const int kp0 = a.sk0 & ~1, np = (a.sk1 - kp0) / 2 + 1;
  const int idx = blockIdx.x * 128 + tid;
  const int j = a.sj0 + idx / np, k = kp0 + 2 * (idx % np);
  const int ib = a.si0 + blockIdx.y * kSch, ie = min(ib + kSch - 1, a.si1);
  if (j > a.sj1) return;
  const bool ax = k >= a.sk0, ay = k + 1 <= a.sk1;
  const int S = a.g.slice, Y = a.g.yline;
  const int VS = (int)a.vb.S, VY = (int)a.vb.Y;
  const float c1 = a.c1, c2 = a.c2;
  long long p = (long long)ib * S + (long long)j * Y + k;
  long long pv = (long long)ib * a.vb.S + (long long)j * a.vb.Y + k - a.vb.off;
  auto stage = [&](int b, long long o) {
#pragma unroll
    for (int q = 0; q < 6; ++q) cpa8(&stg[b][q][tid], a.L[LXX + q] + o);
#pragma unroll
    for (int q = 0; q < 5; ++q) cpa8(&stg[b][6 + q][tid], a.E[GL8 + q] + o);
    if (!ELASTIC) {
#pragma unroll
      for (int q = 0; q < 6; ++q) cpa8(&stg[b][11 + q][tid], a.L[LR1 + q] + o);
    }
    if (!ELASTIC && WANTQ) {
#pragma unroll
      for (int q = 0; q < 5; ++q) cpa8(&stg[b][17 + q][tid], a.E[GQP8 + q] + o);
    }
    cpa_commit();
  };
  stage(0, p);
  float2 u_m1, u_0, u_p1, v_m2, v_m1, v_0, w_m2, w_m1, w_0;
  {
    const float *u = a.fu + pv, *v = a.fv + pv, *w = a.fw + pv;
    u_m1 = ld2(u - VS); u_0 = ld2(u); u_p1 = ld2(u + VS);
    v_m2 = ld2(v - 2 * VS); v_m1 = ld2(v - VS); v_0 = ld2(v);
    w_m2 = ld2(w - 2 * VS); w_m1 = ld2(w - VS); w_0 = ld2(w);
  }
  // a media field in one plane (as k_stress_tma)
  struct Mat {
    float2 m, t, q, pk;
  };
  auto mat = [&](const float* f) {
    Mat r;
    r.m = ld2(f);
    const float mk = f[-1];
    r.t = vadd(r.m, ld2(f - Y));
    r.q = awp_quad(r.t, make_float2(vadd(mk, f[-Y - 1]), r.t.x));
    r.pk = vadd(r.m, make_float2(mk, r.m.x));
    return r;
  };
  const float2 zero = make_float2(0.f, 0.f);
  float2 Lq = mat(a.lam + p).q, Pq = zero;
  Mat mc = mat(a.mu + p), rc{zero, zero, zero, zero};
  if (!ELASTIC) {
    Pq = mat(a.qp + p).q;
    rc = mat(a.qs + p);
  }
  const float dcy = a.dcrjy[j];
  const float2 dcz = make_float2(a.dcrjz[k], a.dcrjz[k + 1]);
  const int top = a.g.top();
  const bool tp = k + 1 == top, tp2 = k + 3 == top;  // the pair at the surface, the one below
#pragma unroll 1
  for (int i = ib; i <= ie; ++i) {
    const int buf = (i - ib) & 1;
    if (i < ie) {
      stage(buf ^ 1, p + S);
      // and the next plane's first reads of the velocities and media on their
      // way into L2
      pre2(a.fu + pv + 3 * VS);
      pre2(a.fv + pv + 2 * VS);
      pre2(a.fw + pv + 2 * VS);
      pre2(a.lam + p + 2 * S);
      pre2(a.mu + p + 2 * S);
      if (!ELASTIC) {
        pre2(a.qp + p + 2 * S);
        pre2(a.qs + p + 2 * S);
      }
    }
    // ---- forward strain rates from the velocities after the step ------------
    const float *u = a.fu + pv, *v = a.fv + pv, *w = a.fw + pv;
    const float2 u_p2 = ld2(u + 2 * VS), v_p1 = ld2(v + VS), w_p1 = ld2(w + VS);
    float2 vs1, vs2, vs3, es[3];
    vs1 = awp_d4(c1, c2, u_p1, u_0, u_p2, u_m1);
    vs2 = awp_d4(c1, c2, v_0, ld2(v - VY), ld2(v + VY), ld2(v - 2 * VY));
    es[0] = vadd(awp_d4(c1, c2, ld2(u + VY), u_0, ld2(u + 2 * VY), ld2(u - VY)),
                 awp_d4(c1, c2, v_0, v_m1, v_p1, v_m2));
    {
      const float2 wa = ld2(w - 2), ua = ld2(u + 2), va = ld2(v + 2);
      vs3 = awp_d4(c1, c2, w_0, make_float2(wa.y, w_0.x), make_float2(w_0.y, w[2]), wa);
      es[1] = vadd(awp_d4(c1, c2, make_float2(u_0.y, ua.x), u_0, ua, make_float2(u[-1], u_0.x)),
                   awp_d4(c1, c2, w_0, w_m1, w_p1, w_m2));
      es[2] = vadd(awp_d4(c1, c2, make_float2(v_0.y, va.x), v_0, va, make_float2(v[-1], v_0.x)),
                   awp_d4(c1, c2, ld2(w + VY), w_0, ld2(w + 2 * VY), ld2(w - VY)));
    }
    // ---- materials of the cell (kernel.cu:962-1070) -------------------------
    const float2 Ln = mat(a.lam + p + S).q;
    const Mat mn = mat(a.mu + p + S);
    const float2 L8 = vadd(Lq, Ln), M8 = vadd(mc.q, mn.q);
    const float2 xm_raw = vquot(16.0f, M8), xl_raw = vadd(vquot(8.0f, L8), xm_raw);
    const float2 P[3] = {mc.pk, mc.t, vadd(mc.m, mn.m)};
    const float2 dthv = vset<float2>(a.dth), DT = vset<float2>(a.dt);
    AwpRelax<float2> t{};
    float2 c_h = zero, c_q = zero, c_hh[3] = {zero, zero, zero};
    float2 dqw = zero, dhw = zero, dhh[3] = {zero, zero, zero};
    if (!ELASTIC) {
      const float* e = tab + (awp_tex_index(a.tex, i, j, k) >> 1) * 20;
      const float4* e4 = reinterpret_cast<const float4*>(e);
      const float4 q0 = e4[0], q1 = e4[1], q2 = e4[2], q3 = e4[3];
      t.vx2 = make_float2(q0.x, q0.y); t.wwo = make_float2(q0.z, q0.w);
      t.kv = make_float2(q1.x, q1.y); t.kr = make_float2(q1.z, q1.w);
      t.kr2 = make_float2(q2.x, q2.y); t.kf = make_float2(q2.z, q2.w);
      t.c0 = make_float2(q3.x, q3.y); t.c1 = make_float2(q3.z, q3.w);
      t.c2 = make_float2(e[16], e[17]);
      const float2 pn = mat(a.qp + p + S).q;
      const Mat rn = mat(a.qs + p + S);
      const float2 qs8 = vscale(0.25f, vadd(rc.q, rn.q)), qp8 = vscale(0.25f, vadd(Pq, pn));
      const float2 R[3] = {rc.pk, rc.t, vadd(rc.m, rn.m)};
      c_h = awp_weight(qs8, t.c0, t.c1, t.c2, a.thr);
      c_q = awp_weight(qp8, t.c0, t.c1, t.c2, a.thr);
#pragma unroll
      for (int q = 0; q < 3; ++q) c_hh[q] = awp_weight(R[q], t.c0, t.c1, t.c2, a.thr);
      if (WANTQ) {
        dhw = vscale(0.25f, dweight(qs8, t, a.thr));
        dqw = vscale(0.25f, dweight(qp8, t, a.thr));
#pragma unroll
        for (int q = 0; q < 3; ++q) dhh[q] = dweight(R[q], t, a.thr);
      }
      Pq = pn;
      rc = rn;
    }
    Lq = Ln;
    mc = mn;
    const float2 c_xm = vfma(DT, c_h, dthv);
    const float2 nxm = vmul(vscale(-1.0f, xm_raw), c_xm), nh = vmul(vscale(-1.0f, xm_raw), c_h);
    const float2 xl = vmul(xl_raw, dthv), qpa = vmul(xl_raw, c_q);
    const float2 A = vfma(DT, qpa, xl);
    const float2 K = vscale(a.dcrjx[i] * dcy, dcz);

    // ---- the adjoint state of the cell; fstr^T of the column's top three ----
    // cells (the imaged values above the surface are cleared later, in
    // k_adj_vel_cell): zz(t) += -zz(t+1), zz(t-1) += -zz(t+2), xz/yz(t-1) +=
    // -xz/yz(t+1), xz/yz(t-2) += -xz/yz(t+2), xz/yz(t) after the imaging is zero
    if (i < ie)
      cpa_wait<1>();
    else
      cpa_wait<0>();
    const float2 lx = stg[buf][0][tid], ly = stg[buf][1][tid];
    float2 lz = stg[buf][2][tid], ls[3] = {stg[buf][3][tid], stg[buf][4][tid], stg[buf][5][tid]};
    if (tp) {
      const float2 z = ld2(a.L[LZZ] + p + 2);
      lz.y -= z.x;
      lz.x -= z.y;
      ls[1] = make_float2(ls[1].x - a.L[LXZ][p + 2], 0.f);
      ls[2] = make_float2(ls[2].x - a.L[LYZ][p + 2], 0.f);
    } else if (tp2) {
      ls[1].y -= a.L[LXZ][p + 5];
      ls[2].y -= a.L[LYZ][p + 5];
    }
    float2 rv[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) rv[q] = ELASTIC ? zero : stg[buf][ELASTIC ? 0 : 11 + q][tid];
    // normal components
    const float2 Ky = vmul(K, ly), Kz = vmul(K, lz);
    const float2 PX = vmul(K, lx), PY = vmul(K, Ky), PZ = vmul(K, Kz);
    float2 QX = zero, QY = zero, QZ = zero;
    if (!ELASTIC) {
      QX = vfma(t.kf, PX, vmul(t.wwo, rv[0]));
      QY = vfma(t.kf, Ky, vmul(t.wwo, rv[1]));
      QZ = vfma(t.kf, Kz, vmul(t.wwo, rv[2]));
    }
    const float2 pyz = vadd(PY, PZ), pxz = vadd(PX, PZ), pxy = vadd(PX, PY);
    const float2 qyz = vadd(QY, QZ), qxz = vadd(QX, QZ), qxy = vadd(QX, QY);
    const float2 sP = vadd(pxy, PZ), sQ = vadd(qxy, QZ);
    const float2 s123 = vadd(vadd(vs1, vs2), vs3);
    const float2 v23 = vadd(vs2, vs3), v13 = vadd(vs1, vs3), v12 = vadd(vs1, vs2);
    const float2 G_xl = vmul(s123, sP), G_qpa = vfma(s123, sQ, vmul(DT, G_xl));
    const float2 nG_xm = vfma(v23, PX, vfma(v13, PY, vmul(v12, PZ)));  // minus the derivative
    const float2 nG_h = vfma(v23, QX, vfma(v13, QY, vmul(v12, QZ)));
    const float2 com = vfma(A, sP, vmul(qpa, sQ));
    st2(a.E[E1] + p, vfma(nxm, pyz, vfma(nh, qyz, com)), ax, ay);
    st2(a.E[E2] + p, vfma(nxm, pxz, vfma(nh, qxz, com)), ax, ay);
    st2(a.E[E3] + p, vfma(nxm, pxy, vfma(nh, qxy, com)), ax, ay);
    st2(a.L[LXX] + p, PX, ax, ay);
    st2(a.L[LYY] + p, PY, ax, ay);
    st2(a.L[LZZ] + p, PZ, ax, ay);
    if (!ELASTIC) {
      st2(a.L[LR1] + p, vfma(t.kr, PX, vmul(t.vx2, rv[0])), ax, ay);
      st2(a.L[LR2] + p, vfma(t.kv, PY, vfma(t.kr2, Ky, vmul(t.vx2, rv[1]))), ax, ay);
      st2(a.L[LR3] + p, vfma(t.kv, PZ, vfma(t.kr2, Kz, vmul(t.vx2, rv[2]))), ax, ay);
    }
    // chain to the eight-cell sums.  The derivative of a quotient is one division
    // by the square (2.5 ulp), not the approximate quotient squared (twice its
    // error): it is the same in every step and does not average out of the sum
    // over them.  The time is the same either way.
    const float2 G_xlraw = vfma(G_qpa, c_q, vmul(G_xl, dthv));
    const float2 G_xmraw = vsub(G_xlraw, vfma(nG_xm, c_xm, vmul(nG_h, c_h)));
    st2(a.E[GL8] + p, vfma(vquot(-8.0f, vmul(L8, L8)), G_xlraw, stg[buf][6][tid]), ax, ay);
    st2(a.E[GM8] + p, vfma(vquot(-16.0f, vmul(M8, M8)), G_xmraw, stg[buf][7][tid]), ax, ay);
    if (!ELASTIC && WANTQ) {
      st2(a.E[GQP8] + p, vfma(vmul(G_qpa, xl_raw), dqw, stg[buf][ELASTIC ? 0 : 17][tid]), ax, ay);
      const float2 g = vfma(DT, nG_xm, nG_h);
      st2(a.E[GQS8] + p,
          vfma(vmul(g, vscale(-1.0f, xm_raw)), dhw, stg[buf][WANTQ ? 18 : 0][tid]), ax, ay);
    }
    // shear components
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const float2 mr = vquot(2.0f, P[q]);
      const float2 cm = vfma(DT, c_hh[q], dthv), xmu = vmul(mr, cm), hh = vmul(mr, c_hh[q]);
      const float2 Kl = vmul(K, ls[q]);
      float2 Fq = zero;
      if (!ELASTIC) Fq = vfma(t.kf, Kl, vmul(t.wwo, rv[3 + q]));
      st2(a.L[LXY + q] + p, Kl, ax, ay);
      if (!ELASTIC) st2(a.L[LR4 + q] + p, vfma(t.kr, Kl, vmul(t.vx2, rv[3 + q])), ax, ay);
      st2(a.E[E4 + q] + p, vfma(xmu, Kl, vmul(hh, Fq)), ax, ay);
      const float2 G_xmu = vmul(es[q], Kl), G_hq = vmul(es[q], Fq);
      st2(a.E[GP1 + q] + p,
          vfma(vquot(-2.0f, vmul(P[q], P[q])), vfma(G_hq, c_hh[q], vmul(G_xmu, cm)),
               stg[buf][8 + q][tid]),
          ax, ay);
      if (!ELASTIC && WANTQ)
        st2(a.E[GQ1 + q] + p,
            vfma(vmul(vfma(DT, G_xmu, G_hq), mr), dhh[q], stg[buf][WANTQ ? 19 + q : 0][tid]), ax,
            ay);
    }
    p += S;
    pv += VS;
    u_m1 = u_0; u_0 = u_p1; u_p1 = u_p2;
    v_m2 = v_m1; v_m1 = v_0; v_0 = v_p1;
    w_m2 = w_m1; w_m1 = w_0; w_0 = w_p1;
  }
}

// ---------------------------------------------------------------------------
// stress^T, gather part: adjoint strain rates -> adjoint velocities (images
// and the untouched k = top+2 values included); material weights -> the
// gradients of 1/lambda and 1/mu
// ---------------------------------------------------------------------------
constexpr int kGch = 4;  // x planes a gather thread marches (register queues along x)

// c1*(a - b) + c2*(c - d) added to s
__device__ __forceinline__ float2 add4(float c1, float2 c2, float2 a, float2 b, float2 c, float2 d,
                                       float2 s) {
  return vfma(c2, vsub(c, d), vfma(vset<float2>(c1), vsub(a, b), s));
}

// Level pairs from the even level at or below k0: a pair may reach one level
// past the transpose's range on either side, where E (V) is zero and the sum
// adds nothing.
__global__ void __launch_bounds__(128) k_adj_stress_gather(const __grid_constant__ AdjArgs a) {
  awp_pipe::grid_start();
  const int kp0 = (a.sk0 - 2) & ~1, np = (a.sk1 + 2 - kp0) / 2 + 1;
  const int idx = blockIdx.x * 128 + threadIdx.x;
  const int j = a.sj0 - 2 + idx / np, k = kp0 + 2 * (idx % np);
  const int ib = a.si0 - 2 + blockIdx.y * kGch;
  const int ie = min(ib + kGch - 1, a.si1 + 2);
  if (j > a.sj1 + 2) return;
  const int S = a.g.slice, Y = a.g.yline;
  const long long q = (long long)ib * S + (long long)j * Y + k;
  const float c1 = a.c1;
  const float2 c2 = vset<float2>(a.c2), zero = make_float2(0.f, 0.f);
  // (not const __restrict__: this launch starts before the kernel that writes E
  // ends, so no load of it may take the path for data constant over the launch)
  const float* e1 = a.E[E1] + q;
  const float* e2 = a.E[E2] + q;
  const float* e3 = a.E[E3] + q;
  const float* e4 = a.E[E4] + q;
  const float* e5 = a.E[E5] + q;
  const float* e6 = a.E[E6] + q;
  float* __restrict__ Lu = a.L[LU] + q;
  float* __restrict__ Lv = a.L[LV] + q;
  float* __restrict__ Lw = a.L[LW] + q;
  // x queues: e1 at x-2, x-1, x; e4, e5 at x-1, x, x+1
  float2 e1m2 = ld2(e1 - 2 * S), e1m1 = ld2(e1 - S), e1c = ld2(e1);
  float2 e4m1 = ld2(e4 - S), e4c = ld2(e4), e4p1 = ld2(e4 + S);
  float2 e5m1 = ld2(e5 - S), e5c = ld2(e5), e5p1 = ld2(e5 + S);
#pragma unroll 2
  for (int i = ib; i <= ie; ++i) {
    const float2 lu = ld2(Lu), lv = ld2(Lv), lw = ld2(Lw);
    const float2 e1p1 = ld2(e1 + S), e4p2 = ld2(e4 + 2 * S), e5p2 = ld2(e5 + 2 * S);
    const float2 e4a = ld2(e4 - Y), e4b = ld2(e4 - 2 * Y), e4d = ld2(e4 + Y);
    const float2 e2c = ld2(e2), e2a = ld2(e2 + Y), e2b = ld2(e2 - Y), e2d = ld2(e2 + 2 * Y);
    const float2 e3c = ld2(e3), e3d = ld2(e3 + 2), e5k = ld2(e5 - 2), e6k = ld2(e6 - 2);
    const float2 e6c = ld2(e6), e6a = ld2(e6 - Y), e6b = ld2(e6 - 2 * Y), e6d = ld2(e6 + Y);
    const float e3m = e3[-1], e5p = e5[2], e6p = e6[2];
    float2 s = add4(c1, c2, e1m1, e1c, e1m2, e1p1, zero);
    s = add4(c1, c2, e4a, e4c, e4b, e4d, s);
    s = add4(c1, c2, make_float2(e5k.y, e5c.x), e5c, e5k, make_float2(e5c.y, e5p), s);
    st2(Lu, vadd(lu, s));
    s = add4(c1, c2, e2c, e2a, e2b, e2d, zero);
    s = add4(c1, c2, e4c, e4p1, e4m1, e4p2, s);
    s = add4(c1, c2, make_float2(e6k.y, e6c.x), e6c, e6k, make_float2(e6c.y, e6p), s);
    st2(Lv, vadd(lv, s));
    s = add4(c1, c2, e3c, make_float2(e3c.y, e3d.x), make_float2(e3m, e3c.x), e3d, zero);
    s = add4(c1, c2, e5c, e5p1, e5m1, e5p2, s);
    s = add4(c1, c2, e6a, e6c, e6b, e6d, s);
    st2(Lw, vadd(lw, s));
    e1m2 = e1m1; e1m1 = e1c; e1c = e1p1;
    e4m1 = e4c; e4c = e4p1; e4p1 = e4p2;
    e5m1 = e5c; e5c = e5p1; e5p1 = e5p2;
    e1 += S; e2 += S; e3 += S; e4 += S; e5 += S; e6 += S;
    Lu += S; Lv += S; Lw += S;
  }
}

// ---------------------------------------------------------------------------
// images^T over the imaged columns: the adjoint of the image values (top+1)
// goes to the velocities they were made from, and to lam_mu; the images are
// overwritten each step, so their adjoint is cleared
// ---------------------------------------------------------------------------
// image-adjoint scratch: column (i, j) of the ring-extended surface window
__device__ __forceinline__ long long img_plane(const AdjArgs& a) {
  return (long long)(a.si1 - a.si0 + 3) * (a.sj1 - a.sj0 + 3);
}
__device__ __forceinline__ long long img_index(const AdjArgs& a, int i, int j) {
  return (long long)(i - a.si0 + 1) * (a.sj1 - a.sj0 + 3) + (j - a.sj0 + 1);
}

__global__ void k_adj_images(const AdjArgs a) {
  awp_pipe::grid_start();
  // targets: the imaged columns and the one-column ring the images also read
  const int j = a.sj0 - 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int i = a.si0 - 1 + blockIdx.y;
  if (j > a.sj1 + 1 || i > a.si1 + 1) return;
  const long long S = a.g.slice, Y = a.g.yline;
  const long long p = (long long)i * S + (long long)j * Y + a.g.top();
  const float* Lu = a.L[LU];
  const float* Lv = a.L[LV];
  const float* Lw = a.L[LW];
  // adjoints of the images of column (ii, jj), zero outside the imaged window
  auto win = [&](int ii, int jj) { return ii >= a.si0 && ii <= a.si1 && jj >= a.sj0 && jj <= a.sj1; };
  auto col = [&](int ii, int jj) { return (long long)ii * S + (long long)jj * Y + a.g.top(); };
  auto Au = [&](int ii, int jj) { return win(ii, jj) ? Lu[col(ii, jj) + 1] : 0.f; };
  auto Av = [&](int ii, int jj) { return win(ii, jj) ? Lv[col(ii, jj) + 1] : 0.f; };
  auto Aw = [&](int ii, int jj) { return win(ii, jj) ? Lw[col(ii, jj) + 1] : 0.f; };
  auto lm = [&](int ii, int jj) { return a.lam_mu[(long long)ii * a.lam_mu_ld + jj]; };
  auto m1 = [&](int ii) { return ii < a.gx_lim ? 1.0f : 0.0f; };
  auto m2 = [&](int jj) { return jj >= a.gy_min ? 1.0f : 0.0f; };
  // lZ(ii, jj) = adjoint of Z at column (ii, jj): -lam_mu * A_w
  auto lZ = [&](int ii, int jj) { return win(ii, jj) ? -lm(ii, jj) * Aw(ii, jj) : 0.f; };
  // Z = m1 (u_{i+1} - w_{i+1} + w) - (u - w + w_{i-1}) + (u_{i+1} - u)
  //     + (v - w_{j+1} + w) - m2 (v_{j-1} - w + w_{j-1}) + (v - v_{j-1})
  const float du = Au(i, j) - 2.0f * lZ(i, j) + (m1(i - 1) + 1.0f) * lZ(i - 1, j);
  const float dv = Av(i, j) + 2.0f * lZ(i, j) - (m2(j + 1) + 1.0f) * lZ(i, j + 1);
  const float dw = -Au(i, j) + Au(i + 1, j) + Av(i, j) - Av(i, j - 1) +
                   (m1(i) + 2.0f + m2(j)) * lZ(i, j) - m1(i - 1) * lZ(i - 1, j) -
                   lZ(i + 1, j) - lZ(i, j - 1) - m2(j + 1) * lZ(i, j + 1);
  // lam_mu gradient: d wimg / d lam_mu = -Z
  if (win(i, j)) {
    const float* u = a.fu;
    const float* v = a.fv;
    const float* w = a.fw;
    const long long VS = a.vb.S, VY = a.vb.Y;
    const long long q = (long long)i * VS + (long long)j * VY + a.g.top() - a.vb.off;
    const float Z = m1(i) * (u[q + VS] - w[q + VS] + w[q]) - (u[q] - w[q] + w[q - VS]) +
                    (u[q + VS] - u[q]) + (v[q] - w[q + VY] + w[q]) -
                    m2(j) * (v[q - VY] - w[q] + w[q - VY]) + (v[q] - v[q - VY]);
    a.glm[(long long)i * a.lam_mu_ld + j] += -Z * Aw(i, j);
  }
  // neighbouring columns read this column's image adjoints, so the updates
  // wait for the next kernel (k_adj_vel_cell)
  const long long ip = img_index(a, i, j), np = img_plane(a);
  a.img[ip] = du;
  a.img[ip + np] = dv;
  a.img[ip + 2 * np] = dw;
  a.img[ip + 3 * np] = Aw(i, j);  // to w(top-1)
}


// ---------------------------------------------------------------------------
// velocity^T, pointwise part
// ---------------------------------------------------------------------------
__global__ void k_adj_vel_cell(const AdjArgs a) {
  awp_pipe::grid_start();
  const int k = a.vk0 + blockIdx.x * 32 + threadIdx.x;
  const int j = a.vj0 + blockIdx.y * 4 + threadIdx.y;
  const int i = a.vi0 + blockIdx.z;
  if (k > a.vk1 || j > a.vj1 || i > a.vi1) return;
  const long long S = a.g.slice, Y = a.g.yline;
  const long long p = (long long)i * S + (long long)j * Y + k;
  const float* d = a.d1;
  const float r1 = 0.25f * (d[p] + d[p - Y] + d[p - 1] + d[p - Y - 1]);
  const float r2 = 0.25f * (d[p] + d[p + S] + d[p - 1] + d[p + S - 1]);
  const float r3 = 0.25f * (d[p] + d[p + S] + d[p - Y] + d[p + S - Y]);
  const float fd1 = a.dth / r1, fd2 = a.dth / r2, fd3 = a.dth / r3;
  const float dc = a.dcrjx[i] * a.dcrjy[j] * a.dcrjz[k];
  // fd * D(sigma) * dc of the forward update = u' - dc u
  const long long pv = (long long)i * a.vb.S + (long long)j * a.vb.Y + k - a.vb.off;
  const float su = a.fu[pv] - dc * a.bu[pv];
  const float sv = a.fv[pv] - dc * a.bv[pv];
  const float sw = a.fw[pv] - dc * a.bw[pv];
  float lu = a.L[LU][p], lv = a.L[LV][p], lw = a.L[LW][p];
  const float wa = a.V[VEA][p], wb = a.V[VEB][p], wc = a.V[VEC][p];
  // the image adjoints of the surface columns (k_adj_images) enter here:
  // u, v, w(top) of the window and its ring, w(top-1) of the window; the
  // imaged velocities and stresses above the surface return to zero (fstr
  // and the images rewrite them every step; their transposes went below)
  const int top = a.g.top();
  if (k >= top - 1 && k <= top + 2) {
    const bool ring = i >= a.si0 - 1 && i <= a.si1 + 1 && j >= a.sj0 - 1 && j <= a.sj1 + 1;
    const bool in = i >= a.si0 && i <= a.si1 && j >= a.sj0 && j <= a.sj1;
    if (k == top && ring) {
      const long long ip = img_index(a, i, j), np = img_plane(a);
      lu += a.img[ip];
      lv += a.img[ip + np];
      lw += a.img[ip + 2 * np];
    } else if (k == top - 1 && in) {
      lw += a.img[img_index(a, i, j) + 3 * img_plane(a)];
    } else if (k > top && in) {
      lu = lv = lw = 0.f;
    }
    if (k == top && in) {
      for (int d = 1; d <= 2; ++d) {
        if (top + d > a.vk1) {  // cells no thread of this kernel owns
          a.L[LU][p + d] = 0.f;
          a.L[LV][p + d] = 0.f;
          a.L[LW][p + d] = 0.f;
        }
        a.L[LZZ][p + d] = 0.f;
        a.L[LXZ][p + d] = 0.f;
        a.L[LYZ][p + d] = 0.f;
      }
    }
  }
  a.L[LU][p] = dc * lu;
  a.L[LV][p] = dc * lv;
  a.L[LW][p] = dc * lw;
  a.V[VA][p] = fd1 * dc * lu;
  a.V[VB][p] = fd2 * dc * lv;
  a.V[VC][p] = fd3 * dc * lw;
  // d fd / d rho_avg = -fd / rho_avg, each of the four densities weighs 1/4:
  // d u' / d d(q) = -1/4 * (fd D dc) / rho_avg
  // summed over the time steps (k_adj_material applies their transposes)
  a.V[VEA][p] = wa + -0.25f / r1 * su * lu;
  a.V[VEB][p] = wb + -0.25f / r2 * sv * lv;
  a.V[VEC][p] = wc + -0.25f / r3 * sw * lw;
}

// ---------------------------------------------------------------------------
// velocity^T, gather part: weighted adjoint velocities -> adjoint stresses;
// density weights -> the density gradient
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_adj_vel_gather(const __grid_constant__ AdjArgs a) {
  awp_pipe::grid_start();
  const int kp0 = (a.vk0 - 2) & ~1, np = (a.vk1 + 2 - kp0) / 2 + 1;
  const int idx = blockIdx.x * 128 + threadIdx.x;
  const int j = a.vj0 - 2 + idx / np, k = kp0 + 2 * (idx % np);
  const int ib = a.vi0 - 2 + blockIdx.y * kGch;
  const int ie = min(ib + kGch - 1, a.vi1 + 2);
  if (j > a.vj1 + 2) return;
  const int S = a.g.slice, Y = a.g.yline;
  const long long q = (long long)ib * S + (long long)j * Y + k;
  const float c1 = a.c1;
  const float2 c2 = vset<float2>(a.c2), zero = make_float2(0.f, 0.f);
  // (inputs qualified as in k_adj_stress_gather)
  const float* A = a.V[VA] + q;
  const float* B = a.V[VB] + q;
  const float* C = a.V[VC] + q;
  float* __restrict__ Lxx = a.L[LXX] + q;
  float* __restrict__ Lxy = a.L[LXY] + q;
  float* __restrict__ Lxz = a.L[LXZ] + q;
  float* __restrict__ Lyy = a.L[LYY] + q;
  float* __restrict__ Lyz = a.L[LYZ] + q;
  float* __restrict__ Lzz = a.L[LZZ] + q;
  // x queues: A at x-1, x, x+1; B, C at x-2, x-1, x
  float2 Am1 = ld2(A - S), Ac = ld2(A), Ap1 = ld2(A + S);
  float2 Bm2 = ld2(B - 2 * S), Bm1 = ld2(B - S), Bc = ld2(B);
  float2 Cm2 = ld2(C - 2 * S), Cm1 = ld2(C - S), Cc = ld2(C);
#pragma unroll 2
  for (int i = ib; i <= ie; ++i) {
    const float2 l0 = ld2(Lxx), l1 = ld2(Lxy), l2 = ld2(Lxz), l3 = ld2(Lyy), l4 = ld2(Lyz),
                 l5 = ld2(Lzz);
    const float2 Ap2 = ld2(A + 2 * S), Bp1 = ld2(B + S), Cp1 = ld2(C + S);
    const float2 Aa = ld2(A + Y), Ab = ld2(A - Y), Ad = ld2(A + 2 * Y), Ak = ld2(A + 2);
    const float2 Ba = ld2(B + Y), Bb = ld2(B - Y), Bd = ld2(B - 2 * Y), Bk = ld2(B + 2);
    const float2 Ca = ld2(C + Y), Cb = ld2(C - Y), Cd = ld2(C + 2 * Y), Ck = ld2(C - 2);
    const float Am = A[-1], Bm = B[-1], Cp = C[2];
    st2(Lxx, vadd(l0, add4(c1, c2, Ac, Ap1, Am1, Ap2, zero)));
    st2(Lxy, vadd(l1, add4(c1, c2, Bm1, Bc, Bm2, Bp1, add4(c1, c2, Ac, Aa, Ab, Ad, zero))));
    st2(Lxz, vadd(l2, add4(c1, c2, Cm1, Cc, Cm2, Cp1,
                           add4(c1, c2, Ac, make_float2(Ac.y, Ak.x), make_float2(Am, Ac.x), Ak,
                                zero))));
    st2(Lyy, vadd(l3, add4(c1, c2, Bb, Bc, Bd, Ba, zero)));
    st2(Lyz, vadd(l4, add4(c1, c2, Cc, Ca, Cb, Cd,
                           add4(c1, c2, Bc, make_float2(Bc.y, Bk.x), make_float2(Bm, Bc.x), Bk,
                                zero))));
    st2(Lzz, vadd(l5, add4(c1, c2, make_float2(Ck.y, Cc.x), Cc, Ck, make_float2(Cc.y, Cp), zero)));
    Am1 = Ac; Ac = Ap1; Ap1 = Ap2;
    Bm2 = Bm1; Bm1 = Bc; Bc = Bp1;
    Cm2 = Cm1; Cm1 = Cc; Cc = Cp1;
    A += S; B += S; C += S;
    Lxx += S; Lxy += S; Lxz += S; Lyy += S; Lyz += S; Lzz += S;
  }
}

// ---------------------------------------------------------------------------
// the material weights summed over the steps -> gradients on the padded
// arrays, once per sweep: each cell's weight goes to every material value its
// forward averages read
//   1/lambda, 1/mu : eight-cell sums at the normal-stress node (box8), mu
//                    pairs at the shear nodes (xy: k-1, xz: j-1, yz: i+1)
//   rho            : four-cell averages of the three velocity nodes
// ---------------------------------------------------------------------------
__global__ void k_adj_material(const AdjArgs a, int i0, int j0, int k0, int ni, int nj,
                               int nk) {
  const int k = k0 + blockIdx.x * 32 + threadIdx.x;
  const int j = j0 + blockIdx.y * 4 + threadIdx.y;
  const int i = i0 + blockIdx.z;
  if (k >= k0 + nk || j >= j0 + nj || i >= i0 + ni) return;
  const long long S = a.g.slice, Y = a.g.yline;
  const long long q = (long long)i * S + (long long)j * Y + k;
  // box8(p) = {p, p+S, p-Y, p+S-Y, p-1, p+S-1, p-Y-1, p+S-Y-1} contains q for
  // p in {q, q-S, q+Y, q-S+Y, q+1, q-S+1, q+Y+1, q-S+Y+1}
  auto box = [&](const float* x) {
    return x[q] + x[q - S] + x[q + Y] + x[q - S + Y] + x[q + 1] + x[q - S + 1] + x[q + Y + 1] +
           x[q - S + Y + 1];
  };
  a.glam[q] = box(a.E[GL8]);
  a.gmu[q] = box(a.E[GM8]) + a.E[GP1][q] + a.E[GP1][q + 1] + a.E[GP2][q] + a.E[GP2][q + Y] +
             a.E[GP3][q] + a.E[GP3][q - S];
  if (a.gqp) {  // the inverse quality factors follow the same averages
    a.gqp[q] = box(a.E[GQP8]);
    a.gqs[q] = box(a.E[GQS8]) + a.E[GQ1][q] + a.E[GQ1][q + 1] + a.E[GQ2][q] +
               a.E[GQ2][q + Y] + a.E[GQ3][q] + a.E[GQ3][q - S];
  }
  const float* ea = a.V[VEA];
  const float* eb = a.V[VEB];
  const float* ec = a.V[VEC];
  a.gd[q] = ea[q] + ea[q + Y] + ea[q + 1] + ea[q + Y + 1] + eb[q] + eb[q - S] + eb[q + 1] +
            eb[q - S + 1] + ec[q] + ec[q - S] + ec[q + Y] + ec[q - S + Y];
}

// One thread per distinct (component, cell); receivers sharing a cell are
// added in receiver order (first[c] .. first[c+1] of order[]).
__global__ void k_adj_inject(float* Lu, float* Lv, float* Lw, const long long* idx,
                             const int* comp, const int* first, const int* order, int ncell,
                             const float* res) {
  awp_pipe::grid_start();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const int r0 = order[first[c]];
  float* L = comp[r0] == 0 ? Lu : (comp[r0] == 1 ? Lv : Lw);
  float acc = L[idx[r0]];
  for (int n = first[c]; n < first[c + 1]; ++n) acc += res[order[n]];
  L[idx[r0]] = acc;
}

__global__ void k_sample(const float* u, const float* v, const float* w, const long long* idx,
                         const int* comp, int n, float* out) {
  awp_pipe::grid_start();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const float* f = comp[r] == 0 ? u : (comp[r] == 1 ? v : w);
  out[r] = f[idx[r]];
}

// ---------------------------------------------------------------------------
// gradients on the padded arrays -> interior lambda, mu, rho
// ---------------------------------------------------------------------------
__global__ void k_adj_fold(const AdjArgs a, float* g_lambda, float* g_mu, float* g_rho) {
  const long long n = (long long)a.g.nxt * a.g.nyt * a.g.nzt;
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= n) return;
  const int x = (int)(c % a.g.nxt), y = (int)((c / a.g.nxt) % a.g.nyt),
            z = (int)(c / ((long long)a.g.nxt * a.g.nyt));
  const int lo = 2 + AWP_NGSL, hix = a.g.nxt + 1 + AWP_NGSL, hiy = a.g.nyt + 1 + AWP_NGSL;
  const int kb = AWP_ALIGN, kt = a.g.nzt + AWP_ALIGN - 1;
  const int i = x + lo, j = y + lo, k = kt - z;
  // the border fill copies (i, j, k) into the ghost cells that clamp onto it
  int is[2] = {i, 0}, js[2] = {j, 0}, ks[2] = {k, 0};
  int ni = 1, nj = 1, nk = 1;
  if (i == lo) is[ni++] = lo - 1;
  if (i == hix) is[ni++] = hix + 1;
  if (j == lo) js[nj++] = lo - 1;
  if (j == hiy) js[nj++] = hiy + 1;
  if (k == kb) ks[nk++] = kb - 1;
  if (k == kt) ks[nk++] = kt + 1;
  float gl = 0.f, gm = 0.f, gr = 0.f;
  for (int ii = 0; ii < ni; ++ii)
    for (int jj = 0; jj < nj; ++jj)
      for (int kk = 0; kk < nk; ++kk) {
        const long long p = (long long)is[ii] * a.g.slice + (long long)js[jj] * a.g.yline + ks[kk];
        gl += a.glam[p];
        gm += a.gmu[p];
        gr += a.gd[p];
      }
  const long long p0 = (long long)i * a.g.slice + (long long)j * a.g.yline + k;
  const float il = a.lam[p0], im = a.mu[p0];  // 1/lambda, 1/mu
  float g_l = -il * il * gl;                  // d(1/lambda)/d lambda = -1/lambda^2
  float g_m = -im * im * gm;
  if (k == kt && i >= a.si0 && i <= a.si1 && j >= a.sj0 && j <= a.sj1) {
    // lam_mu = lambda / (lambda + 2 mu)
    const float lm = 1.0f / il, mm = 1.0f / im, den = lm + 2.0f * mm;
    const float glm = a.glm[(long long)i * a.lam_mu_ld + j];
    g_l += glm * 2.0f * mm / (den * den);
    g_m += -glm * 2.0f * lm / (den * den);
  }
  g_lambda[c] = g_l;
  g_mu[c] = g_m;
  g_rho[c] = gr;
}

// padded Qp^-1 / Qs^-1 gradients -> interior cells, border-fill copies folded
__global__ void k_adj_fold_q(const AdjArgs a, float* g_qp, float* g_qs) {
  const long long n = (long long)a.g.nxt * a.g.nyt * a.g.nzt;
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= n) return;
  const int x = (int)(c % a.g.nxt), y = (int)((c / a.g.nxt) % a.g.nyt),
            z = (int)(c / ((long long)a.g.nxt * a.g.nyt));
  const int lo = 2 + AWP_NGSL, hix = a.g.nxt + 1 + AWP_NGSL, hiy = a.g.nyt + 1 + AWP_NGSL;
  const int kb = AWP_ALIGN, kt = a.g.nzt + AWP_ALIGN - 1;
  const int i = x + lo, j = y + lo, k = kt - z;
  int is[2] = {i, 0}, js[2] = {j, 0}, ks[2] = {k, 0};
  int ni = 1, nj = 1, nk = 1;
  if (i == lo) is[ni++] = lo - 1;
  if (i == hix) is[ni++] = hix + 1;
  if (j == lo) js[nj++] = lo - 1;
  if (j == hiy) js[nj++] = hiy + 1;
  if (k == kb) ks[nk++] = kb - 1;
  if (k == kt) ks[nk++] = kt + 1;
  float gp = 0.f, gs = 0.f;
  for (int ii = 0; ii < ni; ++ii)
    for (int jj = 0; jj < nj; ++jj)
      for (int kk = 0; kk < nk; ++kk) {
        const long long p = (long long)is[ii] * a.g.slice + (long long)js[jj] * a.g.yline + ks[kk];
        gp += a.gqp[p];
        gs += a.gqs[p];
      }
  g_qp[c] = gp;
  g_qs[c] = gs;
}

__global__ void k_set_qinv(const float* qpinv, const float* qsinv, float* qp, float* qs,
                           const AwpGeom g) {
  const int lo = 2 + AWP_NGSL, hix = g.nxt + 1 + AWP_NGSL, hiy = g.nyt + 1 + AWP_NGSL;
  const int kb = AWP_ALIGN, kt = g.nzt + AWP_ALIGN - 1;
  const int k = kb - 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = lo - 1 + blockIdx.y;
  const int i = lo - 1 + blockIdx.z;
  if (k > kt + 1 || j > hiy + 1 || i > hix + 1) return;
  const int ci = min(max(i, lo), hix), cj = min(max(j, lo), hiy), ck = min(max(k, kb), kt);
  const long long c = (long long)(kt - ck) * g.nxt * g.nyt + (long long)(cj - lo) * g.nxt + (ci - lo);
  const long long p = (long long)i * g.slice + (long long)j * g.yline + k;
  qp[p] = qpinv[c];
  qs[p] = qsinv[c];
}

__global__ void k_set_moduli(const float* lambda, const float* mu_, const float* rho, float* lam,
                             float* mu, float* d1, const AwpGeom g) {
  // every cell of the one-cell shell around the interior takes the clamped
  // interior value (the border fill of the media set-up)
  const int lo = 2 + AWP_NGSL, hix = g.nxt + 1 + AWP_NGSL, hiy = g.nyt + 1 + AWP_NGSL;
  const int kb = AWP_ALIGN, kt = g.nzt + AWP_ALIGN - 1;
  const int k = kb - 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = lo - 1 + blockIdx.y;
  const int i = lo - 1 + blockIdx.z;
  if (k > kt + 1 || j > hiy + 1 || i > hix + 1) return;
  const int ci = min(max(i, lo), hix), cj = min(max(j, lo), hiy), ck = min(max(k, kb), kt);
  const long long c = (long long)(kt - ck) * g.nxt * g.nyt + (long long)(cj - lo) * g.nxt + (ci - lo);
  const long long p = (long long)i * g.slice + (long long)j * g.yline + k;
  lam[p] = __frcp_rn(lambda[c]);  // correctly rounded (the build divides approximately)
  mu[p] = __frcp_rn(mu_[c]);
  d1[p] = rho[c];
}

// padded velocities -> VelBox rows; rows beyond nk (up to ld) are not read
// level pairs: the box starts on a multiple of four levels
// (inputs qualified as in k_adj_stress_gather)
__global__ void k_pack_vel(const float* u, const float* v, const float* w,
                           float* __restrict__ du, float* __restrict__ dv,
                           float* __restrict__ dw, const VelBox b, long long S, long long Y) {
  awp_pipe::grid_start();
  const int np = (b.nk + 1) / 2, idx = blockIdx.x * 128 + threadIdx.x;
  const int jj = idx / np, kk = 2 * (idx % np), ii = blockIdx.y;
  if (jj >= b.nj) return;
  const long long p = (long long)(b.i0 + ii) * S + (long long)(b.j0 + jj) * Y + b.k0 + kk;
  const long long q = (long long)ii * b.S + (long long)jj * b.Y + kk;
  const float2 x = ld2(u + p), y = ld2(v + p), z = ld2(w + p);
  st2(du + q, x);
  st2(dv + q, y);
  st2(dw + q, z);
}

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

}  // namespace

cudaError_t awp_launch_pack_vel(const float* u, const float* v, const float* w, float* du,
                                float* dv, float* dw, const VelBox& b, const AwpGeom& g,
                                cudaStream_t st) {
  if (b.ni <= 0 || b.nj <= 0 || b.nk <= 0) return cudaSuccess;
  return awp_pipe::launch_after(k_pack_vel, dim3(cdiv((long long)b.nj * ((b.nk + 1) / 2), 128), b.ni), dim3(128), 0, st,  u, v, w, du, dv, dw, b, g.slice, g.yline);
}

cudaError_t awp_launch_adjoint_step(const AdjArgs& a, cudaStream_t st) {
  const int si = a.si1 - a.si0 + 1, sj = a.sj1 - a.sj0 + 1;
  // the imaging (fstr) transpose runs inside k_adj_stress_cell
  auto pairs = [](int k0, int k1) { return (long long)((k1 - (k0 & ~1)) / 2 + 1); };
  const dim3 sgrid(cdiv(sj * pairs(a.sk0, a.sk1), 128), cdiv(si, kSch));
  const auto cell = a.elastic  ? k_adj_stress_cell<true, false>
                    : a.want_q ? k_adj_stress_cell<false, true>
                               : k_adj_stress_cell<false, false>;
  const int vi = a.vi1 - a.vi0 + 1, vj = a.vj1 - a.vj0 + 1, vk = a.vk1 - a.vk0 + 1;
  const dim3 b(128);
  cudaError_t e;
  using awp_pipe::launch_after;
  if ((e = launch_after(cell, sgrid, b, 0, st, a))) return e;
  if ((e = launch_after(k_adj_stress_gather,
                        dim3(cdiv((sj + 4) * pairs(a.sk0 - 2, a.sk1 + 2), 128),
                             cdiv(si + 4, kGch)),
                        b, 0, st, a)))
    return e;
  if ((e = launch_after(k_adj_images, dim3(cdiv(sj + 2, 128), si + 2), b, 0, st, a))) return e;
  if ((e = launch_after(k_adj_vel_cell, dim3(cdiv(vk, 32), cdiv(vj, 4), vi), dim3(32, 4), 0, st,
                        a)))
    return e;
  return launch_after(k_adj_vel_gather,
                      dim3(cdiv((vj + 4) * pairs(a.vk0 - 2, a.vk1 + 2), 128), cdiv(vi + 4, kGch)),
                      b, 0, st, a);
}

cudaError_t awp_launch_adjoint_inject(float* const L[3], const long long* idx, const int* comp,
                                      const int* first, const int* order, int ncell,
                                      const float* res, cudaStream_t st) {
  if (ncell <= 0) return cudaSuccess;
  return awp_pipe::launch_after(k_adj_inject, dim3(cdiv(ncell, 128)), dim3(128), 0, st, L[0], L[1], L[2], idx, comp, first, order, ncell, res);
}

cudaError_t awp_launch_sample(const float* u, const float* v, const float* w,
                              const long long* idx, const int* comp, int nrec, float* out,
                              cudaStream_t st) {
  if (nrec <= 0) return cudaSuccess;
  return awp_pipe::launch_after(k_sample, dim3(cdiv(nrec, 128)), dim3(128), 0, st, u, v, w, idx, comp, nrec, out);
}

cudaError_t awp_launch_adjoint_fold(const AdjArgs& a, float* g_lambda, float* g_mu,
                                    float* g_rho, cudaStream_t st) {
  {
    // every cell a weight can reach: the stress and velocity ranges +-2
    const int i0 = min(a.si0, a.vi0) - 2, i1 = max(a.si1, a.vi1) + 2;
    const int j0 = min(a.sj0, a.vj0) - 2, j1 = max(a.sj1, a.vj1) + 2;
    const int k0 = min(a.sk0, a.vk0) - 2, k1 = max(a.sk1, a.vk1) + 2;
    const int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
    k_adj_material<<<dim3(cdiv(nk, 32), cdiv(nj, 4), ni), dim3(32, 4), 0, st>>>(a, i0, j0, k0,
                                                                                ni, nj, nk);
  }
  const long long n = (long long)a.g.nxt * a.g.nyt * a.g.nzt;
  k_adj_fold<<<cdiv(n, 256), 256, 0, st>>>(a, g_lambda, g_mu, g_rho);
  return cudaGetLastError();
}

cudaError_t awp_launch_set_moduli(const float* lambda, const float* mu_, const float* rho,
                                  float* lam, float* mu, float* d1, const AwpGeom& g,
                                  cudaStream_t st) {
  const dim3 grid(cdiv(g.nzt + 2, 64), g.nyt + 2, g.nxt + 2);
  k_set_moduli<<<grid, 64, 0, st>>>(lambda, mu_, rho, lam, mu, d1, g);
  return cudaGetLastError();
}

cudaError_t awp_launch_adjoint_fold_q(const AdjArgs& a, float* g_qpinv, float* g_qsinv,
                                      cudaStream_t st) {
  if (!a.gqp || !a.gqs) return cudaErrorInvalidValue;
  const long long n = (long long)a.g.nxt * a.g.nyt * a.g.nzt;
  k_adj_fold_q<<<cdiv(n, 256), 256, 0, st>>>(a, g_qpinv, g_qsinv);
  return cudaGetLastError();
}

cudaError_t awp_launch_set_qinv(const float* qpinv, const float* qsinv, float* qp, float* qs,
                                const AwpGeom& g, cudaStream_t st) {
  const dim3 grid(cdiv(g.nzt + 2, 64), g.nyt + 2, g.nxt + 2);
  k_set_qinv<<<grid, 64, 0, st>>>(qpinv, qsinv, qp, qs, g);
  return cudaGetLastError();
}
