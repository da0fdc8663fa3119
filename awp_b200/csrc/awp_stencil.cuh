// Per-cell arithmetic shared by the stencil kernels (awp_kernels.cu, awp_tma.cu).
#pragma once

#include <math.h>

#include "awp_common.h"
#include "awp_f2.cuh"

// ---------------------------------------------------------------------------
// Rounding discipline.  The per-cell arithmetic below is written with explicit
// rounding (intrinsics, or the packed instructions of awp_f2.cuh that round
// each lane alike), so every kernel family that calls it -- one level per
// thread or two, read-only path or TMA-pipelined -- produces the same bits:
// left to the compiler, the contraction of a*b + c into an FMA is chosen per
// kernel and differs between kernels that spell the same expression.
// V is float (one level) or float2 (two adjacent levels).
// ---------------------------------------------------------------------------

// c1*(a - b) + c2*(c - d): one 4th-order staggered difference.
template <class V>
__device__ __forceinline__ V awp_d4(float c1, float c2, V a, V b, V c, V d) {
  return vfma(vset<V>(c2), vsub(c, d), vscale(c1, vsub(a, b)));
}

// The same with a pair of weights per level.
__device__ __forceinline__ float2 awp_d4(float2 c1, float2 c2, float2 a, float2 b, float2 c,
                                         float2 d) {
  return vfma(c2, vsub(c, d), vmul(c1, vsub(a, b)));
}

// Velocity update of dvelcx (kernel.cu:222-253):
// (v + fd*(c1*x0 + c2*x1 + c1*y0 + c2*y1 + c1*z0 + c2*z1)) * dcrj, where
// x0..z1 are the six differences of the three stress derivatives.
template <class V>
__device__ __forceinline__ V awp_vel_update(V v, V fd, V k1, V k2, V x0, V x1, V y0, V y1, V z0,
                                            V z1, V dcrj) {
  V s = vmul(k1, x0);
  s = vfma(k2, x1, s);
  s = vfma(k1, y0, s);
  s = vfma(k2, y1, s);
  s = vfma(k1, z0, s);
  s = vfma(k2, z1, s);
  return vmul(vfma(fd, s, v), dcrj);
}

// dth / (0.25 * (a + b + c + d)) from the two pair sums a + b and c + d: the
// density-averaged velocity factor (kernel.cu:218-221).
template <class V>
__device__ __forceinline__ V awp_vel_factor(float dth, V ab, V cd) {
  return vquot(dth, vscale(0.25f, vadd(ab, cd)));
}

// Sum of the four values of a field around an edge in one x plane, from the
// sums over j and j-1 at k and at k-1; two of these make the eight-cell sums.
template <class V>
__device__ __forceinline__ V awp_quad(V tk, V tkm1) {
  return vadd(tk, tkm1);
}

// Relaxation constants of the memory-variable update of a cell.  The
// reference's update of one component (kernel.cu:1116-1124),
//   t     = base + vx1c*r,          vx1c = DT*(1 + vx2*vx1)
//   r'    = vx2*r + wwo*f
//   f'    = f*(wwo - 1) + vx2*r*(1 - vx1)
//   sigma = (t [* dcrj] + DT*f') * dcrj,
// is linear in r and f, and the Q(f) weight only enters scaled by
// -vx1/(wwo*h), so every product of the step's constants is formed once on
// the host (in double, rounded once) instead of in each cell:
//   sigma = (base + kr*r + kf*f) * dcrj           (kr = kv + kr2)
//         = ((base + kv*r)*dcrj + kr2*r + kf*f) * dcrj   (the twice-damped yy, zz)
// and c0..c2 give weight * (-vx1/h) of a pair sum S of Q^-1: (c0*S + c1)*S on
// the low-Q branch of kernel.cu:974-1040, c2*S otherwise.
template <class V>
struct AwpRelax {
  V vx2, wwo, kv, kr, kr2, kf, c0, c1, c2;
};

__device__ __forceinline__ AwpRelax<float> awp_relax_at(const AwpRelaxTab& t, int e) {
  return {t.vx2[e], t.wwo[e], t.kv[e], t.kr[e], t.kr2[e], t.kf[e], t.c0[e], t.c1[e], t.c2[e]};
}

// The same constants from explicit arrays (vx1, vx2, wwo) of a caller.
__device__ __forceinline__ AwpRelax<float> awp_relax_from(float vx1, float vx2, float wwo, float c0,
                                                          float c1, float DT, float dh1,
                                                          float* l0 = nullptr,
                                                          float* l1 = nullptr) {
  AwpRelax<float> r;
  const float K = -__fmul_rn(dh1, vx1);
  r.vx2 = vx2;
  r.wwo = wwo;
  r.kv = __fmul_rn(DT, __fmaf_rn(vx2, vx1, 1.0f));
  r.kr2 = __fmul_rn(DT, __fmul_rn(vx2, __fsub_rn(1.0f, vx1)));
  r.kr = __fadd_rn(r.kv, r.kr2);
  r.kf = __fmul_rn(DT, __fsub_rn(wwo, 1.0f));
  // c0*S + c1 cancels in part: the two share the factor K/wwo and its error,
  // and have one rounding each of their own
  const float g = __fdividef(K, wwo);
  r.c0 = __fmul_rn(0.25f * c0, g);
  r.c1 = __fmul_rn(0.5f * c1, g);
  if (l0) {
    *l0 = __fmaf_rn(0.25f * c0, g, -r.c0);
    *l1 = __fmaf_rn(0.5f * c1, g, -r.c1);
  }
  r.c2 = 0.5f * K;
  return r;
}

// Q(f) weight times -vx1/h of a pair sum S (four times this for an eight-cell
// sum: pass 0.25*S8).  The reference switches on 1./(q*2.0) <= 200.0 in
// double, q = S/4: for float S that is S >= 2*qthr for positive S, true for
// negative S and -0, false for +0; as bit patterns one unsigned compare, the
// negative values lying above every positive one.
__device__ __forceinline__ float awp_weight(float S, float c0, float c1, float c2, unsigned thr) {
  const float s = __float_as_uint(S) >= thr ? __fmaf_rn(c0, S, c1) : c2;
  return __fmul_rn(s, S);
}
__device__ __forceinline__ float2 awp_weight(float2 S, float2 c0, float2 c1, float2 c2,
                                             unsigned thr) {
  const float2 p = vfma(c0, S, c1);
  const float2 s = make_float2(__float_as_uint(S.x) >= thr ? p.x : c2.x,
                               __float_as_uint(S.y) >= thr ? p.y : c2.y);
  return vmul(s, S);
}

// Quotient and Q(f) weight of a stress cell's coefficients (awp_stress_coef).
struct AwpCellOps {
  template <class V>
  __device__ __forceinline__ V quot(float n, V d) const { return vquot(n, d); }
  template <class V>
  __device__ __forceinline__ V weight(V S, const AwpRelax<V>& t, unsigned thr) const {
    return awp_weight(S, t.c0, t.c1, t.c2, thr);
  }
  template <class V>
  __device__ __forceinline__ V weight_p(V S, const AwpRelax<V>& t, unsigned thr) const {
    return awp_weight(S, t.c0, t.c1, t.c2, thr);
  }
};

// The same where the first level is a mesh block's interface layer (dstrqc2,
// kernel.cu:2564-2767), at the precision of the reference, which divides and
// evaluates the low-Q polynomial in double there: a quotient by the hardware
// reciprocal is corrected by its remainder (half an ulp then), and c0*S + c1,
// whose terms may cancel, takes what rounding left of its constants (l0, l1).
// The switch 1/(2q) <= 200 is in double for Qs, in float for Qp.  The caller
// halves t.c2: the high-Q branch is wwo*q here where dstrqc has 2*wwo*q.
struct AwpLayerOps {
  bool on;
  float l0, l1;  // zero where off
  // n a power of two
  __device__ __forceinline__ float quot(float n, float d) const {
    const float q = __fdividef(n, d);
    const float c = __fmaf_rn(__fmaf_rn(-q, d, n), q * (1.0f / n), q);
    return on && c == c ? c : q;  // d zero or infinite: no remainder
  }
  __device__ __forceinline__ float2 quot(float n, float2 d) const {
    return make_float2(quot(n, d.x), __fdividef(n, d.y));
  }
  __device__ __forceinline__ float poly(float S, float c0, float c1) const {
    return __fadd_rn(__fmaf_rn(c0, S, c1), __fmaf_rn(l0, S, l1));
  }
  __device__ __forceinline__ float low(float S, float c0, float c1, float c2, bool b) const {
    return __fmul_rn(b ? poly(S, c0, c1) : c2, S);
  }
  __device__ __forceinline__ float weight(float S, const AwpRelax<float>& t, unsigned thr) const {
    return low(S, t.c0, t.c1, t.c2, __float_as_uint(S) >= thr);
  }
  __device__ __forceinline__ float weight_p(float S, const AwpRelax<float>& t, unsigned) const {
    return low(S, t.c0, t.c1, t.c2, __fdividef(1.0f, 0.5f * S) <= 200.0f);
  }
  __device__ __forceinline__ float2 both(float2 S, const AwpRelax<float2>& t, bool x,
                                         unsigned thr) const {
    const float y = __float_as_uint(S.y) >= thr ? __fmaf_rn(t.c0.y, S.y, t.c1.y) : t.c2.y;
    return make_float2(low(S.x, t.c0.x, t.c1.x, t.c2.x, x), __fmul_rn(y, S.y));
  }
  __device__ __forceinline__ float2 weight(float2 S, const AwpRelax<float2>& t,
                                           unsigned thr) const {
    return both(S, t, __float_as_uint(S.x) >= thr, thr);
  }
  __device__ __forceinline__ float2 weight_p(float2 S, const AwpRelax<float2>& t,
                                             unsigned thr) const {
    return both(S, t, on ? __fdividef(1.0f, 0.5f * S.x) <= 200.0f : __float_as_uint(S.x) >= thr,
                thr);
  }
};

// Coefficients of one stress cell (kernel.cu:962-1070): with e_n the strain
// rates and tr their trace, the elastic increments are A*tr + nxm*(tr - e_n)
// (normal) and m*e (shear), the memory variables' forcing Q*tr + nh*(tr - e_n)
// and h*e.
template <class V>
struct AwpStrCoef {
  V A, Q, nxm, nh, m[3], h[3];
};

// L8, M8, QP8, QS8: the eight-cell sums of lam, mu, qp, qs; P and R: mu's and
// qs's pair sums with k-1, j-1 and i+1.  The reference divides in double
// ((float)(8.0/(double)x)); here the five quotients use the hardware
// reciprocal (within two ulp), which keeps the update off the division slow
// path; the parity tests hold the result to the reference build at relative
// L2 1e-5.
template <bool ELASTIC, class V, class Ops = AwpCellOps>
__device__ __forceinline__ AwpStrCoef<V> awp_stress_coef(V L8, V M8, const V (&P)[3], V QP8, V QS8,
                                                         const V (&R)[3], const AwpRelax<V>& t,
                                                         unsigned thr, V dth, V DT,
                                                         const Ops& ops = Ops()) {
  AwpStrCoef<V> r;
  const V nxm = ops.quot(-16.0f, M8);
  const V xl = vsub(ops.quot(8.0f, L8), nxm);
  if (ELASTIC) {
    r.nxm = vmul(dth, nxm);
    r.A = vmul(dth, xl);
    r.Q = r.nh = vset<V>(0.f);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      r.m[q] = vmul(dth, ops.quot(2.0f, P[q]));
      r.h[q] = vset<V>(0.f);
    }
    return r;
  }
  const V hw = ops.weight(vscale(0.25f, QS8), t, thr);
  const V qw = ops.weight_p(vscale(0.25f, QP8), t, thr);
  r.nh = vmul(nxm, hw);
  r.nxm = vmul(nxm, vfma(DT, hw, dth));
  r.Q = vmul(xl, qw);
  r.A = vmul(xl, vfma(DT, qw, dth));
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const V m = ops.quot(2.0f, P[q]);
    const V w = ops.weight(R[q], t, thr);
    r.h[q] = vmul(m, w);
    r.m[q] = vmul(m, vfma(DT, w, dth));
  }
  return r;
}

// Memory-variable step of one component (see AwpRelax); r is advanced.
template <class V>
__device__ __forceinline__ V awp_mem_step(V base, V& r, V f, const AwpRelax<V>& t, V dcrj,
                                          bool twice) {
  const V r0 = r;
  r = vfma(t.wwo, f, vmul(t.vx2, r0));
  if (!twice) return vmul(vfma(t.kf, f, vfma(t.kr, r0, base)), dcrj);
  const V b = vmul(vfma(t.kv, r0, base), dcrj);
  return vmul(vfma(t.kf, f, vfma(t.kr2, r0, b)), dcrj);
}

// One stress/memory-variable update of a cell (dstrqc, kernel.cu:1114-1179),
// the state passed in and out through registers.
//   sg: xx yy zz xy xz yz; rr: r1..r6
//   d:  vs1 vs2 vs3 (normal strain rates), then the xy, xz, yz difference pairs
template <bool ELASTIC, class V>
__device__ __forceinline__ void awp_stress_update(V (&sg)[6], V (&rr)[6], const AwpStrCoef<V>& q,
                                                  const AwpRelax<V>& t, V dcrj, const V (&d)[9]) {
  const V s23 = vadd(d[1], d[2]), s13 = vadd(d[0], d[2]), s12 = vadd(d[0], d[1]);
  const V tr = vadd(s12, d[2]);
  const V e[3] = {vadd(d[3], d[4]), vadd(d[5], d[6]), vadd(d[7], d[8])};
  const V o[3] = {s23, s13, s12};
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    // (a packed product added to a packed sum may be contracted by the
    // assembler: the fused form is spelled out instead)
    const V b = vfma(q.nxm, o[n], vfma(q.A, tr, sg[n]));
    if (ELASTIC) {
      // the reference multiplies yy and zz by the sponge factor twice (kernel.cu:1130-1150)
      sg[n] = vmul(b, dcrj);
      if (n > 0) sg[n] = vmul(sg[n], dcrj);
    } else {
      sg[n] = awp_mem_step(b, rr[n], vfma(q.nh, o[n], vmul(q.Q, tr)), t, dcrj, n > 0);
    }
  }
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    const V b = vfma(q.m[n], e[n], sg[3 + n]);
    if (ELASTIC)
      sg[3 + n] = vmul(b, dcrj);
    else
      sg[3 + n] = awp_mem_step(b, rr[3 + n], vmul(q.h[n], e[n]), t, dcrj, false);
  }
}
