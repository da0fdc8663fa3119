// TMA-pipelined stencil kernels for the context API (sm_100a).
//
// Each CTA owns a tile of 32 k (one 128-byte line) x 8 j and marches a chunk of
// x planes.  A producer warp issues cp.async.bulk.tensor loads of each plane's
// tiles (with the j/k halo the stencil needs) into shared-memory rings, one
// or two planes ahead of the arithmetic; four consumer warps compute, each
// thread two vertically adjacent cells with packed arithmetic (awp_f2.cuh).
// What the x stencil needs of a cell's own column travels in registers, so a
// tile stays in shared memory only while its neighbours in j and k are read.
// Results are stored straight from registers, one full 128-byte line per half
// warp.
//
// Measured at 512 x 512 x 256, anelastic (us per launch, share of the measured
// copy bandwidth on the algorithmic bytes), against the form before (256
// threads, one cell each, every x neighbour from shared memory, one barrier of
// the CTA per plane, 554 thread instructions a cell in the stress update):
//   velocity  800 -> 545 (0.66 -> 0.96),  stress 1815 -> 1388 (0.70 -> 0.92).
//
// Tile boxes (x = k fastest, y = j, z = i), all 16-byte aligned in x:
//   halo   : 40 x 11 floats, k in [kb-4, kb+36), j from jb-1 or jb-2
//   media  : 36 x  9 floats, k in [kb-4, kb+32), j in [jb-1, jb+8)
//   own    : 32 x  8 floats; with a j halo 32 x 11, with a k halo 40 x 8
//
// Synchronisation: a full mbarrier per ring stage (the copies' bytes), and a
// ring of "step done" mbarriers on which the consumer warps arrive and the
// producer waits before it refills what that step read last; no barrier of
// the whole CTA in the march.  Every wait is bounded; a wait that runs out
// sets the context's error word, its warp leaves the march, the others follow
// when their own waits run out, and the producer drains the copies in flight
// before the CTA ends.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "awp_kernels.cuh"
#include "awp_pipe.cuh"
#include "awp_stencil.cuh"
#include "awp_tma.cuh"

#define LDG(p) __ldg(p)

using namespace awp_pipe;

namespace {

constexpr int TZ = 32, TY = 8;
constexpr int NC = TZ * TY / 2;       // consumer threads (two cells each)
constexpr int NT = NC + 32;           // and the producer warp
constexpr int HX = 40, HY = 11;       // halo box
constexpr int HTILE = 448;            // its slot (floats, a multiple of 128 B)
constexpr int MX = 36, MY = 9, MTILE = 352;  // media box and slot
constexpr int OTILE = TZ * TY;        // own box and slot
constexpr int JTILE = TZ * HY;        // j-halo box (32 x 11) and slot (352)
constexpr int KTILE = HX * TY;        // k-halo box (40 x 8) and slot (320)
// ===========================================================================
// Stress + memory variables (dstrqc, kernel.cu:880-1197), same bits as
// k_stress in awp_kernels.cu (see there for the term-by-term citation).
//
// Bound by DRAM: 124 bytes a cell and the halo.  Halo/media stages run two
// planes ahead, the cell's own twelve fields one: 63 KB of rings, three CTAs
// (twelve computing warps) per SM.
// ===========================================================================
template <bool ELASTIC>
struct StrCfg {
  static constexpr int NM = ELASTIC ? 2 : 4;   // lam, mu (, qp, qs)
  static constexpr int NO_ = ELASTIC ? 6 : 12;  // xx..yz (, r1..r6)
  static constexpr int LH = 2, LO = 1;         // planes ahead
  static constexpr int NH = 1 + LH, NO = 1 + LO;
  static constexpr int DU = 3 + LH;            // u: planes i .. i+2 and the ones ahead
  static constexpr int DV = 2 + LH;            // v, w: planes i, i+1 and the ones ahead
  static constexpr int F_U = 0, F_V = F_U + DU * HTILE, F_W = F_V + DV * HTILE,
                       F_M = F_W + DV * HTILE, F_O = F_M + NH * NM * MTILE,
                       F_T = F_O + NO * NO_ * OTILE;  // relaxation table
  static constexpr int kTab = ELASTIC ? 0 : 4 * 20;
  static constexpr size_t bytes = sizeof(float) * (F_T + kTab) + sizeof(Pipe<NH, NO, NC / 32>);
};

// The boxes of a launch: one, on the grid's three axes, or several with their
// CTAs in a row, box by box, in the same order (levels, then j, then chunks).
// Separate launches for the four boxes around a plasticity section's middle band
// each end in a wave that is nearly empty and two of them are a few planes wide
// (240 x 237 x 120: 116 -> 98 us a step).
struct StrBoxes {
  AwpBox box[AWP_MAXBOX];
  int first[AWP_MAXBOX], nj[AWP_MAXBOX];  // first CTA / nk, tiles in j
  int n, nk;                              // boxes, tiles in k
};

// LAYER: the launch takes a mesh block's interface layer too (StrArgs::layer).
template <bool ELASTIC, bool LAYER>
__global__ void __launch_bounds__(NT, ELASTIC ? 4 : 3)
    k_stress_tma(const __grid_constant__ StrArgs a, const __grid_constant__ TmaMaps tm,
                 const __grid_constant__ StrBoxes bx, const int ichunk, int* err,
                 const unsigned spin) {
  using C = StrCfg<ELASTIC>;
  constexpr int NM = C::NM, NO = C::NO_;
  extern __shared__ __align__(128) float smem[];
  auto& pipe = *reinterpret_cast<Pipe<C::NH, C::NO, NC / 32>*>(smem + C::F_T + C::kTab);
  const int tid = threadIdx.x;
  int kt = blockIdx.x, jt = blockIdx.y, it = blockIdx.z, q = 0;
  if (bx.n > 1) {
    it = kt / bx.nk;
    kt -= it * bx.nk;
    while (q + 1 < bx.n && it >= bx.first[q + 1]) ++q;
    jt = it - bx.first[q];
    it = jt / bx.nj[q];
    jt -= it * bx.nj[q];
  }
  const int kb = AWP_ALIGN + kt * TZ, jb = bx.box[q].j0 + jt * TY;
  const int ib = bx.box[q].i0 + it * ichunk, je = bx.box[q].j1;
  const int n = min(ichunk, bx.box[q].i1 - ib + 1);

  grid_go();
  if (tid == 0) pipe.init();
  if (!ELASTIC) {
    // relaxation constants of the entry pairs (e, e + 1), e even, that two
    // adjacent levels take: nine float2 per pair in 20 floats
    float* tab = smem + C::F_T;
    const float* const src[9] = {a.rel.vx2, a.rel.wwo, a.rel.kv, a.rel.kr, a.rel.kr2,
                                 a.rel.kf,  a.rel.c0,  a.rel.c1, a.rel.c2};
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (tid < 8) tab[(tid >> 1) * 20 + 2 * q + (tid & 1)] = src[q][tid];
  }
  __syncthreads();
  grid_wait();

  if (tid >= NC) {  // producer warp
    if (tid == NC) {
      pipe.produce(
          n,
          [&](int s, uint64_t* b) {
            // the first stage also brings the planes the later ones find there
            const int u0 = s == 0 ? 0 : s + 2, v0 = s == 0 ? 0 : s + 1;
            mbar_expect_tx(b, ((s + 2 - u0 + 1) + 2 * (s + 1 - v0 + 1)) * HX * HY * 4 +
                                  NM * MX * MY * 4);
            for (int p = u0; p <= s + 2; ++p)
              tma_load3(smem + C::F_U + (p % C::DU) * HTILE, &tm.halo[0], b, kb - 4, jb - 1,
                        ib + p);
            for (int p = v0; p <= s + 1; ++p) {
              tma_load3(smem + C::F_V + (p % C::DV) * HTILE, &tm.halo[1], b, kb - 4, jb - 2,
                        ib + p);
              tma_load3(smem + C::F_W + (p % C::DV) * HTILE, &tm.halo[2], b, kb - 4, jb - 1,
                        ib + p);
            }
            float* m = smem + C::F_M + (s % C::NH) * NM * MTILE;
            for (int f = 0; f < NM; ++f)
              tma_load3(m + f * MTILE, &tm.media[f], b, kb - 4, jb - 1, ib + s + 1);
          },
          [&](int s, uint64_t* b) {
            mbar_expect_tx(b, NO * OTILE * 4);
            float* o = smem + C::F_O + (s % C::NO) * NO * OTILE;
            for (int f = 0; f < NO; ++f)
              tma_load3(o + f * OTILE, &tm.own[f], b, kb, jb, ib + s);
          },
          err, spin);
    }
    return;
  }

  const int row = tid >> 4, kp = (tid & 15) * 2;
  const int k = kb + kp, j = jb + row;
  const bool jin = j <= je;
  // the interface layer of a mesh block: second order, weights (1, 0)
  const bool layer = LAYER && k + 1 == a.k0;
  const bool ax = jin && ((k >= a.k0 && k <= a.k1) || layer),
             ay = jin && k + 1 >= a.k0 && k + 1 <= a.k1;
  const int S = a.slice, Y = a.yline;
  const float2 c1 = make_float2(layer ? 1.0f : a.c1, a.c1),
               c2 = make_float2(layer ? 0.0f : a.c2, a.c2);
  const long long col = (long long)j * Y + k;
  const float dcy = LDG(a.dcrjy + min(j, je));
  const float2 dcz = ldg2(a.dcrjz + k);
  // the pair (ktop - 1, ktop): nzt is even, so the surface is a second level
  const bool top = a.fs && (k + 1 == a.ktop);
  float* __restrict__ SG[6] = {a.xx, a.yy, a.zz, a.xy, a.xz, a.yz};
  float* __restrict__ RR[6] = {a.r1, a.r2, a.r3, a.r4, a.r5, a.r6};
  // texture entries of the two levels at even and odd steps
  int e0[2], e1[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    e0[q] = awp_tex_index(a.tex, ib + q, j, k);
    e1[q] = awp_tex_index(a.tex, ib + q, j, k + 1);
  }

  // own-column values of the planes before the ones the tiles bring, and the
  // media sums of the first plane, straight from global memory
  long long o = (long long)ib * S + col;
  float2 u_m1, u_0, u_p1, v_m2, v_m1, v_0, w_m2, w_m1, w_0;
  {
    const float *U = a.u1 + o, *V = a.v1 + o, *W = a.w1 + o;
    u_m1 = ldg2(U - S); u_0 = ldg2(U); u_p1 = ldg2(U + S);
    v_m2 = ldg2(V - 2 * (long long)S); v_m1 = ldg2(V - S); v_0 = ldg2(V);
    w_m2 = ldg2(W - 2 * (long long)S); w_m1 = ldg2(W - S); w_0 = ldg2(W);
  }
  // one media field in one plane: value, sum with j-1, that sum plus the one a
  // level below, and the pair sum with the level below
  struct Mat {
    float2 m, t, q, pk;
  };
  auto mat = [&](float2 A, float Ak, float2 B, float Bk) {  // rows j, j-1; k-1 values
    Mat r;
    r.m = A;
    r.t = vadd(A, B);
    const float tk = vadd(Ak, Bk);
    r.q = awp_quad(r.t, make_float2(tk, r.t.x));
    r.pk = vadd(A, make_float2(Ak, A.x));
    return r;
  };
  auto mat_g = [&](const float* p) { return mat(ldg2(p), p[-1], ldg2(p - Y), p[-Y - 1]); };
  auto mat_s = [&](const float* p) { return mat(lds2(p), p[-1], lds2(p - MX), p[-MX - 1]); };
  float2 Lq, Mq, Mt, Mm, Mk, Pq = {}, Rq = {}, Rt = {}, Rm = {}, Rk = {};
  {
    Lq = mat_g(a.lam + o).q;
    const Mat m = mat_g(a.mu + o);
    Mq = m.q; Mt = m.t; Mm = m.m; Mk = m.pk;
    if (!ELASTIC) {
      Pq = mat_g(a.qp + o).q;
      const Mat r = mat_g(a.qs + o);
      Rq = r.q; Rt = r.t; Rm = r.m; Rk = r.pk;
    }
  }
  const int hu = (row + 1) * HX + kp + 4, hv = (row + 2) * HX + kp + 4;
  const int hm = (row + 1) * MX + kp + 4, ho = row * TZ + kp;

  Cursor<C::NH> ch;
  Cursor<C::NO> co;
  Cursor<awp_pipe::ND> cd;
  int su = 0, su2 = 2, sv = 0, sv1 = 1;  // slots of u planes i, i+2 and v, w planes i, i+1
  bool ok = true;
#pragma unroll 1
  for (int s = 0; s < n; ++s) {
    ok = mbar_wait(pipe.full_h + ch.slot, ch.phase, spin);
    if (!__all_sync(0xffffffffu, ok)) break;
    const float* U0 = smem + C::F_U + su * HTILE + hu;
    const float* V0 = smem + C::F_V + sv * HTILE + hv;
    const float* W0 = smem + C::F_W + sv * HTILE + hu;
    const float2 u_p2 = lds2(smem + C::F_U + su2 * HTILE + hu);
    const float2 v_p1 = lds2(smem + C::F_V + sv1 * HTILE + hv);
    const float2 w_p1 = lds2(smem + C::F_W + sv1 * HTILE + hu);
    const float2 u_jm1 = lds2(U0 - HX), u_jp1 = lds2(U0 + HX), u_jp2 = lds2(U0 + 2 * HX);
    const float2 v_jm2 = lds2(V0 - 2 * HX), v_jm1 = lds2(V0 - HX), v_jp1 = lds2(V0 + HX);
    const float2 w_jm1 = lds2(W0 - HX), w_jp1 = lds2(W0 + HX), w_jp2 = lds2(W0 + 2 * HX);
    // k neighbours: the level below and the pair above (u, v), the pair below
    // and the level above (w)
    const float u_km1 = U0[-1], v_km1 = V0[-1];
    float2 u_kp = lds2(U0 + 2), v_kp = lds2(V0 + 2);
    const float2 w_km = lds2(W0 - 2);
    float w_kp = W0[2];

    // ---- media: sums of plane i + 1, coefficients of plane i ---------------
    const float* M = smem + C::F_M + ch.slot * NM * MTILE + hm;
    AwpRelax<float2> rx{};
    const int odd = s & 1;
    if (!ELASTIC) {
      const float* tab = smem + C::F_T;
      const int ea = odd ? e0[1] : e0[0], eb = odd ? e1[1] : e1[0];
      const float4* t4 = reinterpret_cast<const float4*>(tab + (ea >> 1) * 20);
      const float4 q0 = t4[0], q1 = t4[1], q2 = t4[2], q3 = t4[3];
      const float2 q4 = lds2(tab + (ea >> 1) * 20 + 16);
      rx.vx2 = make_float2(q0.x, q0.y); rx.wwo = make_float2(q0.z, q0.w);
      rx.kv = make_float2(q1.x, q1.y); rx.kr = make_float2(q1.z, q1.w);
      rx.kr2 = make_float2(q2.x, q2.y); rx.kf = make_float2(q2.z, q2.w);
      rx.c0 = make_float2(q3.x, q3.y); rx.c1 = make_float2(q3.z, q3.w);
      rx.c2 = q4;
      if (eb != (ea | 1) || (ea & 1)) {
        // entries that are not an even-odd pair: the level of a mesh's coarse
        // block that takes the finer block's pattern
        auto at = [&](int q) {
          return make_float2(tab[(ea >> 1) * 20 + 2 * q + (ea & 1)],
                             tab[(eb >> 1) * 20 + 2 * q + (eb & 1)]);
        };
        rx = {at(0), at(1), at(2), at(3), at(4), at(5), at(6), at(7), at(8)};
      }
    }
    AwpStrCoef<float2> cf;
    {
      const float2 Ln = mat_s(M).q;
      const Mat mn = mat_s(M + MTILE);
      const float2 P[3] = {Mk, Mt, vadd(Mm, mn.m)};
      float2 QP8 = {}, QS8 = {}, R[3] = {};
      if (!ELASTIC) {
        const float2 pn = mat_s(M + 2 * MTILE).q;
        const Mat rn = mat_s(M + 3 * MTILE);
        QP8 = vadd(Pq, pn);
        QS8 = vadd(Rq, rn.q);
        R[0] = Rk; R[1] = Rt; R[2] = vadd(Rm, rn.m);
        Pq = pn;
        Rq = rn.q; Rt = rn.t; Rm = rn.m; Rk = rn.pk;
      }
      const float2 L8 = vadd(Lq, Ln), M8 = vadd(Mq, mn.q);
      const float2 dth = vset<float2>(a.dth), DT = vset<float2>(a.dt);
      if (LAYER) {
        AwpLayerOps ops{layer, 0.f, 0.f};
        if (layer) {
          const int e = odd ? e0[1] : e0[0];
          ops.l0 = a.lay.l0[e];
          ops.l1 = a.lay.l1[e];
          rx.c2.x *= 0.5f;
        }
        cf = awp_stress_coef<ELASTIC>(L8, M8, P, QP8, QS8, R, rx, a.thr, dth, DT, ops);
      } else {
        cf = awp_stress_coef<ELASTIC>(L8, M8, P, QP8, QS8, R, rx, a.thr, dth, DT);
      }
      Lq = Ln;
      Mq = mn.q; Mt = mn.t; Mm = mn.m; Mk = mn.pk;
    }
    const int i = ib + s;
    const float2 dcrj = vscale(LDG(a.dcrjx + i) * dcy, dcz);

    // ---- free-surface velocity images (kernel.cu:1087-1112) ----------------
    if (top) {
      const float uimg = u_0.y - (w_0.y - w_m1.y);
      const float vimg = v_0.y - (w_jp1.y - w_0.y);
      if (jin) {
        const float vs1 = (i < a.gx_lim) ? u_p1.y - (w_p1.y - w_0.y) : 0.0f;
        const float vs2 = (j >= a.gy_min) ? v_jm1.y - (w_0.y - w_jm1.y) : 0.0f;
        const float wimg = __fmaf_rn(
            -LDG(a.lam_mu + (long long)i * a.lam_mu_ld + j),
            __fadd_rn(__fadd_rn(__fadd_rn(vs1 - uimg, u_p1.y - u_0.y), vimg - vs2),
                      v_0.y - v_jm1.y),
            w_0.x);
        a.u1[o + 2] = uimg;
        a.v1[o + 2] = vimg;
        a.w1[o + 2] = wimg;
        w_kp = wimg;
      }
      u_kp.x = uimg;
      v_kp.x = vimg;
    }

    float2 d[9];
    d[0] = awp_d4(c1, c2, u_p1, u_0, u_p2, u_m1);
    d[1] = awp_d4(c1, c2, v_0, v_jm1, v_jp1, v_jm2);
    d[2] = make_float2(awp_d4(c1.x, c2.x, w_0.x, w_km.y, w_0.y, w_km.x),
                       awp_d4(c1.y, c2.y, w_0.y, w_0.x, w_kp, w_km.y));
    d[3] = awp_d4(c1, c2, u_jp1, u_0, u_jp2, u_jm1);
    d[4] = awp_d4(c1, c2, v_0, v_m1, v_p1, v_m2);
    d[5] = make_float2(awp_d4(c1.x, c2.x, u_0.y, u_0.x, u_kp.x, u_km1),
                       awp_d4(c1.y, c2.y, u_kp.x, u_0.y, u_kp.y, u_0.x));
    d[6] = awp_d4(c1, c2, w_0, w_m1, w_p1, w_m2);
    d[7] = make_float2(awp_d4(c1.x, c2.x, v_0.y, v_0.x, v_kp.x, v_km1),
                       awp_d4(c1.y, c2.y, v_kp.x, v_0.y, v_kp.y, v_0.x));
    d[8] = awp_d4(c1, c2, w_jp1, w_0, w_jp2, w_jm1);

    ok = mbar_wait(pipe.full_o + co.slot, co.phase, spin);
    if (!__all_sync(0xffffffffu, ok)) break;
    const float* O = smem + C::F_O + co.slot * NO * OTILE + ho;
    float2 sg[6], rr[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      sg[q] = lds2(O + q * OTILE);
      if (!ELASTIC) rr[q] = lds2(O + (6 + q) * OTILE);
    }
    awp_stress_update<ELASTIC>(sg, rr, cf, rx, dcrj, d);
    if (ax || ay) {
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        st2(SG[q] + o, sg[q], ax, ay);
        if (!ELASTIC) st2(RR[q] + o, rr[q], ax, ay);
      }
    }
    warp_done(pipe.done + cd.slot, tid & 31);

    o += S;
    u_m1 = u_0; u_0 = u_p1; u_p1 = u_p2;
    v_m2 = v_m1; v_m1 = v_0; v_0 = v_p1;
    w_m2 = w_m1; w_m1 = w_0; w_0 = w_p1;
    ch.next();
    co.next();
    cd.next();
    su = su + 1 == C::DU ? 0 : su + 1;
    su2 = su2 + 1 == C::DU ? 0 : su2 + 1;
    sv = sv1;
    sv1 = sv1 + 1 == C::DV ? 0 : sv1 + 1;
  }
  if (!__all_sync(0xffffffffu, ok) && (tid & 31) == 0) atomicExch(err, 1);
}

// ===========================================================================
// Velocity (dvelcx_opt, kernel.cu:125-268), same bits as k_velocity.  The xx
// tile is read only at the cell's own column, one plane ahead; xy and xz at
// their own column two planes ahead and with their j or k neighbours when the
// march arrives; yy, zz, yz, the density and the velocities once.
// ===========================================================================
struct VelCfg {
  static constexpr int LA = 2;          // planes ahead
  static constexpr int NH = 1 + LA;     // stages
  static constexpr int DS = 3 + LA;     // xy, xz: planes i .. i+2 and the ones ahead
  // one stage: xx(i+1), yy, zz, yz(i), density(i+1), u, v, w(i)
  static constexpr int G_XX = 0, G_YY = OTILE, G_ZZ = G_YY + JTILE, G_YZ = G_ZZ + KTILE,
                       G_D = G_YZ + HTILE, G_O = G_D + MTILE, STAGE = G_O + 3 * OTILE;
  static constexpr int F_XY = 0, F_XZ = F_XY + DS * JTILE, F_S = F_XZ + DS * KTILE,
                       F_END = F_S + NH * STAGE;
  static constexpr size_t bytes = sizeof(float) * F_END + sizeof(Pipe<NH, 0, NC / 32>);
};

template <bool LAYER>
__global__ void __launch_bounds__(NT, 4)
    k_velocity_tma(const VelArgs a, const __grid_constant__ TmaMaps tm, const int ichunk,
                   int* err, const unsigned spin) {
  using C = VelCfg;
  extern __shared__ __align__(128) float smem[];
  auto& pipe = *reinterpret_cast<Pipe<C::NH, 0, NC / 32>*>(smem + C::F_END);
  const int tid = threadIdx.x;
  const int kb = AWP_ALIGN + blockIdx.x * TZ;
  const int jb = a.j0 + blockIdx.y * TY;
  const int ib = a.i0 + blockIdx.z * ichunk;
  const int ie = min(ib + ichunk - 1, a.i1);
  const int n = ie - ib + 1;

  grid_go();
  if (tid == 0) pipe.init();
  __syncthreads();
  grid_wait();

  if (tid >= NC) {  // producer warp
    if (tid == NC) {
      pipe.produce(
          n,
          [&](int s, uint64_t* b) {
            const int p0 = s == 0 ? 0 : s + 2;
            mbar_expect_tx(b, ((s + 2 - p0 + 1) * (JTILE + KTILE) + 4 * OTILE + JTILE + KTILE +
                               HX * HY + MX * MY) * 4);
            for (int p = p0; p <= s + 2; ++p) {
              tma_load3(smem + C::F_XY + (p % C::DS) * JTILE, &tm.halo[3], b, kb, jb - 2, ib + p);
              tma_load3(smem + C::F_XZ + (p % C::DS) * KTILE, &tm.halo[4], b, kb - 4, jb, ib + p);
            }
            float* g = smem + C::F_S + (s % C::NH) * C::STAGE;
            const int i = ib + s;
            tma_load3(g + C::G_XX, &tm.halo[0], b, kb, jb, i + 1);
            tma_load3(g + C::G_YY, &tm.halo[1], b, kb, jb - 1, i);
            tma_load3(g + C::G_ZZ, &tm.halo[2], b, kb - 4, jb, i);
            tma_load3(g + C::G_YZ, &tm.halo[5], b, kb - 4, jb - 2, i);
            tma_load3(g + C::G_D, &tm.media[0], b, kb - 4, jb - 1, i + 1);
            for (int f = 0; f < 3; ++f)
              tma_load3(g + C::G_O + f * OTILE, &tm.own[f], b, kb, jb, i);
          },
          [](int, uint64_t*) {}, err, spin);
    }
    return;
  }

  const int row = tid >> 4, kp = (tid & 15) * 2;
  const int k = kb + kp, j = jb + row;
  const bool jin = j <= a.j1;
  const bool layer = LAYER && k + 1 == a.k0;  // as in k_stress_tma (dvelc2)
  const bool ax = layer ? j <= a.layer_j1 : jin && k >= a.k0 && k <= a.k1,
             ay = jin && k + 1 >= a.k0 && k + 1 <= a.k1;
  const int S = a.slice, Y = a.yline;
  const float2 c1 = make_float2(layer ? 1.0f : a.c1, a.c1),
               c2 = make_float2(layer ? 0.0f : a.c2, a.c2);
  const float dth = a.dth;
  const float dcy = LDG(a.dcrjy + min(j, a.j1));
  const float2 dcz = ldg2(a.dcrjz + k);
  long long o = (long long)ib * S + (long long)j * Y + k;
  float2 xx_m2, xx_m1, xx_0, xy_m1, xy_0, xy_p1, xz_m1, xz_0, xz_p1;
  // density of the current plane: rows j and j-1; the level below and its sum
  // over the two rows (formed in the step that reads them)
  float2 d_0, d_0j;
  float d_0k, d_0s;
  {
    const float *X = a.xx + o, *P = a.xy + o, *Q = a.xz + o, *D = a.d1 + o;
    xx_m2 = ldg2(X - 2 * (long long)S); xx_m1 = ldg2(X - S); xx_0 = ldg2(X);
    xy_m1 = ldg2(P - S); xy_0 = ldg2(P); xy_p1 = ldg2(P + S);
    xz_m1 = ldg2(Q - S); xz_0 = ldg2(Q); xz_p1 = ldg2(Q + S);
    d_0 = ldg2(D); d_0j = ldg2(D - Y); d_0k = D[-1]; d_0s = vadd(d_0k, D[-Y - 1]);
  }
  const int o_own = row * TZ + kp;                    // no halo
  const int o_yy = (row + 1) * TZ + kp;               // j halo from jb - 1
  const int o_xy = (row + 2) * TZ + kp;               // j halo from jb - 2
  const int o_k = row * HX + kp + 4;                  // k halo
  const int o_yz = (row + 2) * HX + kp + 4;           // both, from jb - 2
  const int o_d = (row + 1) * MX + kp + 4;

  Cursor<C::NH> ch;
  Cursor<awp_pipe::ND> cd;
  int ss = 0, ss2 = 2;  // slots of the xy, xz planes i, i+2
  bool ok = true;
#pragma unroll 1
  for (int s = 0; s < n; ++s) {
    ok = mbar_wait(pipe.full_h + ch.slot, ch.phase, spin);
    if (!__all_sync(0xffffffffu, ok)) break;
    const float* G = smem + C::F_S + ch.slot * C::STAGE;
    const float* XY = smem + C::F_XY + ss * JTILE + o_xy;
    const float* XZ = smem + C::F_XZ + ss * KTILE + o_k;
    const float* YY = G + C::G_YY + o_yy;
    const float* ZZ = G + C::G_ZZ + o_k;
    const float* YZ = G + C::G_YZ + o_yz;
    const float* D = G + C::G_D + o_d;
    const float2 xx_p1 = lds2(G + C::G_XX + o_own);
    const float2 xy_p2 = lds2(smem + C::F_XY + ss2 * JTILE + o_xy);
    const float2 xz_p2 = lds2(smem + C::F_XZ + ss2 * KTILE + o_k);
    const float2 xy_jm1 = lds2(XY - TZ), xy_jm2 = lds2(XY - 2 * TZ), xy_jp1 = lds2(XY + TZ);
    const float2 xz_km = lds2(XZ - 2);
    const float xz_kp = XZ[2];
    const float2 yy_0 = lds2(YY), yy_jp1 = lds2(YY + TZ), yy_jp2 = lds2(YY + 2 * TZ),
                 yy_jm1 = lds2(YY - TZ);
    const float2 zz_0 = lds2(ZZ), zz_kp = lds2(ZZ + 2);
    const float zz_km1 = ZZ[-1];
    const float2 yz_0 = lds2(YZ), yz_km = lds2(YZ - 2), yz_jm1 = lds2(YZ - HX),
                 yz_jm2 = lds2(YZ - 2 * HX), yz_jp1 = lds2(YZ + HX);
    const float yz_kp = YZ[2];
    const float2 d_p = lds2(D), d_pj = lds2(D - MX);
    const float d_pk = D[-1], d_ps = vadd(d_pk, D[-MX - 1]);
    const float2 u_old = lds2(G + C::G_O + o_own), v_old = lds2(G + C::G_O + OTILE + o_own),
                 w_old = lds2(G + C::G_O + 2 * OTILE + o_own);

    // density factors: pair sums at the level and at the one below
    const float2 dj = vadd(d_0, d_0j), dx = vadd(d_0, d_p);
    const float2 fd1 = awp_vel_factor(dth, dj, make_float2(d_0s, dj.x));
    const float2 fd2 = awp_vel_factor(dth, dx, make_float2(vadd(d_0k, d_pk), dx.x));
    const float2 fd3 = awp_vel_factor(dth, dx, vadd(d_0j, d_pj));
    const float2 dcrj = vscale(LDG(a.dcrjx + ib + s) * dcy, dcz);

    const float2 u = awp_vel_update(
        u_old, fd1, c1, c2, vsub(xx_0, xx_m1), vsub(xx_p1, xx_m2), vsub(xy_0, xy_jm1),
        vsub(xy_jp1, xy_jm2), make_float2(xz_0.x - xz_km.y, xz_0.y - xz_0.x),
        make_float2(xz_0.y - xz_km.x, xz_kp - xz_km.y), dcrj);
    const float2 v = awp_vel_update(
        v_old, fd2, c1, c2, vsub(xy_p1, xy_0), vsub(xy_p2, xy_m1), vsub(yy_jp1, yy_0),
        vsub(yy_jp2, yy_jm1), make_float2(yz_0.x - yz_km.y, yz_0.y - yz_0.x),
        make_float2(yz_0.y - yz_km.x, yz_kp - yz_km.y), dcrj);
    const float2 w = awp_vel_update(
        w_old, fd3, c1, c2, vsub(xz_p1, xz_0), vsub(xz_p2, xz_m1), vsub(yz_0, yz_jm1),
        vsub(yz_jp1, yz_jm2), make_float2(zz_0.y - zz_0.x, zz_kp.x - zz_0.y),
        make_float2(zz_kp.x - zz_km1, zz_kp.y - zz_0.x), dcrj);
    if (ax || ay) {
      st2(a.u1 + o, u, ax, ay);
      st2(a.v1 + o, v, ax, ay);
      st2(a.w1 + o, w, ax, ay);
    }
    warp_done(pipe.done + cd.slot, tid & 31);
    o += S;
    xx_m2 = xx_m1; xx_m1 = xx_0; xx_0 = xx_p1;
    xy_m1 = xy_0; xy_0 = xy_p1; xy_p1 = xy_p2;
    xz_m1 = xz_0; xz_0 = xz_p1; xz_p1 = xz_p2;
    d_0 = d_p; d_0j = d_pj; d_0k = d_pk; d_0s = d_ps;
    ch.next();
    cd.next();
    ss = ss + 1 == C::DS ? 0 : ss + 1;
    ss2 = ss2 + 1 == C::DS ? 0 : ss2 + 1;
  }
  if (!__all_sync(0xffffffffu, ok) && (tid & 31) == 0) atomicExch(err, 1);
}


PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

}  // namespace

// L2 promotion of the tensor maps' fetches (process-wide; a context encodes
// its maps with the value of the moment and re-encodes them when it changes):
// 0 none, 1 64 B, 2 128 B, 3 256 B.  A column's rows are not multiples of 256
// bytes, so the wide granule fetches padding and rows no box asks for
// (k_stress_tma at 512 x 512 x 256: 1618 us with 256 B, 1515 none or 128 B).
static int g_l2_promotion = 0;

int awp_tma_set_l2_promotion(int mode) {
  if (mode < 0 || mode > 3) return 1;
  g_l2_promotion = mode;
  return 0;
}

int awp_tma_get_l2_promotion() { return g_l2_promotion; }

int awp_tma_encode(CUtensorMap* map, const float* base, const AwpGeom& g, int box_x, int box_y) {
  auto fn = encode_fn();
  if (!fn) return 1;
  // The map ends four levels above the surface (the stencils reach two): of the
  // last tile of a column that is no multiple of 32 levels, the padding beyond
  // is filled in, not read (five steps of 301 x 223 x 108 1585 -> 1537 us, an
  // ensemble of 21 uneven grids 2797 -> 2723).
  const cuuint64_t dims[3] = {(cuuint64_t)std::min<long long>(g.top() + 5, g.nz_pad()),
                              (cuuint64_t)g.ny_pad(), (cuuint64_t)g.nx_pad()};
  const cuuint64_t strides[2] = {(cuuint64_t)g.yline * 4, (cuuint64_t)g.slice * 4};
  const cuuint32_t box[3] = {(cuuint32_t)box_x, (cuuint32_t)box_y, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r =
      fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box,
         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
         g_l2_promotion == 0   ? CU_TENSOR_MAP_L2_PROMOTION_NONE
         : g_l2_promotion == 1 ? CU_TENSOR_MAP_L2_PROMOTION_L2_64B
         : g_l2_promotion == 2 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B
                               : CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 2;
}

int awp_tma_box(int group, int* bx, int* by) {
  switch (group) {
    case 0: *bx = HX; *by = HY; return 0;   // j and k halo
    case 1: *bx = MX; *by = MY; return 0;   // media
    case 2: *bx = TZ; *by = TY; return 0;   // own
    case 3: *bx = TZ; *by = HY; return 0;   // j halo only
    case 4: *bx = HX; *by = TY; return 0;   // k halo only
  }
  return 1;
}

namespace {

Shape g_shape_str[4][kMaxDev], g_shape_vel[2][kMaxDev];
constexpr int kMost = 6;  // planes of a march (march_planes)

}  // namespace

cudaError_t awp_launch_stress_tma(const StrArgs& a, const AwpBox* box, int nbox, const TmaMaps& tm,
                                  bool elastic, int ichunk, int* err, cudaStream_t st) {
  const int nk = a.k1 - AWP_ALIGN + 1;
  StrBoxes bx{};
  int ni = 0;
  for (int q = 0; q < nbox && bx.n < AWP_MAXBOX; ++q) {
    if (box[q].empty()) continue;
    bx.box[bx.n] = box[q];
    bx.nj[bx.n++] = (int)cdiv_u(box[q].j1 - box[q].j0 + 1, TY);
    ni = std::max(ni, box[q].i1 - box[q].i0 + 1);
  }
  if (nk <= 0 || bx.n == 0) return cudaSuccess;
  bx.nk = (int)cdiv_u(nk, TZ);
  auto chunks = [&](int q, int c) {
    return (long long)cdiv_u(bx.box[q].i1 - bx.box[q].i0 + 1, c);
  };
  const size_t sm = elastic ? StrCfg<true>::bytes : StrCfg<false>::bytes;
  const auto f = elastic ? (a.layer ? k_stress_tma<true, true> : k_stress_tma<true, false>)
                         : (a.layer ? k_stress_tma<false, true> : k_stress_tma<false, false>);
  int resident = 0;
  const cudaError_t e = resident_ctas(
      (const void*)f, sm, NT, g_shape_str[(elastic ? 2 : 0) + (a.layer ? 1 : 0)], &resident);
  if (e != cudaSuccess) return e;
  const int c = march_planes(
      [&](int c) {
        long long t = 0;
        for (int q = 0; q < bx.n; ++q) t += chunks(q, c) * bx.nj[q] * bx.nk;
        return t;
      },
      ni, resident, ichunk, kMost);
  dim3 grid(bx.nk, bx.nj[0], (unsigned)chunks(0, c));
  if (bx.n > 1) {
    long long t = 0;
    for (int q = 0; q < bx.n; ++q) {
      bx.first[q] = (int)t;
      t += chunks(q, c) * bx.nj[q];
    }
    grid = dim3((unsigned)(t * bx.nk));
  }
  return launch_after(f, grid, dim3(NT), sm, st, a, tm, bx, c, err, awp_pipe_spin_limit);
}

cudaError_t awp_launch_velocity_tma(const VelArgs& a, const TmaMaps& tm, int ichunk, int* err,
                                    cudaStream_t st) {
  const int nk = a.k1 - AWP_ALIGN + 1, nj = a.j1 - a.j0 + 1, ni = a.i1 - a.i0 + 1;
  if (nk <= 0 || nj <= 0 || ni <= 0) return cudaSuccess;
  const dim3 tile(cdiv_u(nk, TZ), cdiv_u(nj, TY));
  const auto f = a.layer ? k_velocity_tma<true> : k_velocity_tma<false>;
  int resident = 0;
  const cudaError_t e = resident_ctas((const void*)f, VelCfg::bytes, NT,
                                      g_shape_vel[a.layer ? 1 : 0], &resident);
  if (e != cudaSuccess) return e;
  const int c = march_planes((long long)tile.x * tile.y, ni, resident, ichunk, kMost);
  return launch_after(f, dim3(tile.x, tile.y, cdiv_u(ni, c)), dim3(NT), VelCfg::bytes, st,
                      a, tm, c, err, awp_pipe_spin_limit);
}

// the pipeline waits' poll limit
unsigned awp_pipe_spin_limit = kSpinLimit;

int awp_tma_set_spin_limit(long long polls) {
  if (polls < 0 || polls > (1ll << 30)) return 1;
  awp_pipe_spin_limit = (unsigned)polls;
  return 0;
}

long long awp_tma_get_spin_limit() { return awp_pipe_spin_limit; }
