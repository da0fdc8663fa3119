// Curvilinear (topography) velocity and stress half-steps of the top grid.
//
// The reference spells these operators out as generated code, one kernel for
// the interior (k below the top six points) and one for the six boundary rows
// next to the free surface:
//   velocity: dtopo_vel_111_unroll (kernels/velocity_unroll.cu:1-428) and
//             dtopo_vel_112 (kernels/optimized_velocity.cu:1040-1629),
//   stress:   dtopo_str_111 / dtopo_str_112 (kernels/stress_attenuation.cu:73-1415),
// launched by topo_velocity_*_H (velocity.cu) and topo_stress_*_H
// (stress_attenuation.cu).  Here each half-step is one TMA-pipelined kernel
// (awp_pipe.cuh): a CTA marches along x with a tile of 64 levels x kCol
// columns, a producer warp keeping the next planes' tiles in shared memory.
//
// A warp owns the 64 levels of one column, two adjacent levels per lane, and
// computes with packed arithmetic (awp_f2.cuh).  The vertical operators
// (7-point differences of horizontal interpolants, 4-point differences) take
// the neighbouring levels from the neighbouring lanes by warp shuffles: six
// shuffles give a 7-point difference at both of a lane's levels.  Warps
// overlap by two lanes (four levels, the operators reach three) on each side:
// tiles of 56 output levels, the top tile outputting its 60 levels under the
// surface.  The boundary-closure rows r = nz-1-k of the summation-by-parts
// tables (awp_topo_tables.h) read the top levels of the column, which all sit
// in the top tile's last lanes, by broadcast shuffles; each of the lanes 29..31
// keeps its two rows' coefficients in shared memory.
//
// What makes the operators cheap: the vertical differences are linear and the
// surface metrics f do not depend on k, so the x and y terms of a component
// share one difference (three of them for the velocity, five for the stress);
// a column's surface metrics, already multiplied by the operators' weights,
// are formed by the warp's lanes in parallel once per plane and read back as
// broadcasts; the vertical metrics' reciprocals are formed once per march.
//
// Term structure (f = surface function interpolants, g = vertical metric;
// relative indices, k = 0 the bottom point of the grid):
//   u_t = (A / (f g3 rho)) * [ D_x(f g3 sigma_x) + D_y(f g3 sigma_y) + D_z sigma_z
//                              - f1 * Dz(g P_x sigma_x) - f2 * Dz(g P_y sigma_y) ]
//   sigma_t from strain rates  D_x u - J^-1 g P_x(f1 Dz u)  etc.
// and the memory-variable / sponge update shared with the Cartesian kernels
// (awp_stress_coef / awp_stress_update).  The sums are associated differently
// from the reference's, so agreement with it is to rounding; the metric and
// density quotients are products of hardware reciprocals (within two ulp each)
// where the reference rounds one double quotient.  Relative L2 error against
// float64 over three hills and six seeds each: velocities 0.84, 0.62, 1.03e-7
// (0.89, 0.64, 1.06e-7 with correctly rounded quotients and the reference's
// order), stresses 1.04, 0.71, 0.96e-7 (1.11, 0.73, 0.98e-7).
#include "awp_topo_kern.cuh"

#include "awp_pipe.cuh"
#include "awp_stencil.cuh"
#include "awp_topo_tables.h"

using namespace awp_pipe;

namespace {

// interior 4-point interpolation / difference and the 7-point vertical
// difference of the interpolant (the reference's double literals as float)
constexpr float kP0 = (float)-0.0625, kP1 = (float)0.5625;
constexpr float kD0 = (float)0.0416666666666667, kD1 = (float)-1.1250000000000000;
constexpr float kZ0 = (float)-0.0026041666666667, kZ1 = (float)0.0937500000000000,
                kZ2 = (float)-0.6796875000000000;
constexpr unsigned kAll = 0xffffffffu;
constexpr int kSpan = 64;     // levels of a warp
constexpr int kTileOut = 56;  // output levels of a tile below the top one
// Columns (computing warps) of a CTA, and its tiles: own 64 x NC, j halo 64 x
// (NC + 3), media 64 x (NC + 1).  Two CTAs of eight warps with the producer at
// 116-128 registers; the velocity kernel's three CTAs at 80 were slower (433
// -> 462 us at 384 x 384 x 160: spills).
template <int NC>
struct Tile {
  static constexpr int kCol = NC, kThreads = 32 * (NC + 1);
  static constexpr int kOwn = kSpan * NC, kHalo = kSpan * (NC + 3), kMed = kSpan * (NC + 1);
};
using VelTile = Tile<7>;
using StrTile = Tile<7>;
constexpr int kMost = 32;    // planes of a march (march_planes)

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

// Column position of a warp: tile t = 0 holds the top 64 levels, tile t > 0
// the 64 levels starting 56 t lower; lane L holds levels kb + 2L and
// kb + 2L + 1.  A level is output when its lane is not a halo lane (two at
// each end; the top tile has no upper halo) and k >= 3 (the reference leaves
// the three bottom points to the mesh coupling, dm_offset = 3).  Loads from
// global memory read level max(kb + 2L, -32): the levels below the grid are
// padding and only ever feed halo lanes, and the clamp keeps a short grid's
// reads inside it (its tiles' copies are zero-filled there).
struct ColPos2 {
  int k, ld, lane;
  bool top, out0, out1;
  __device__ ColPos2(int nz, int tile) {
    lane = threadIdx.x & 31;
    top = (tile == 0);
    k = nz - kSpan - kTileOut * tile + 2 * lane;
    ld = k < -AWP_ALIGN ? -AWP_ALIGN : k;
    const bool in = lane >= 2 && (top || lane <= 29);
    out0 = in && k >= 3;
    out1 = in && k + 1 >= 3;
  }
};

// Boundary-closure rows of one table for the lanes 29..31 of the top tile:
// c[31 - lane][p] = the coefficients of levels nz-1-2p (x, y) and nz-2-2p (z,
// w) in the rows of the lane's two levels (rows 2(31-lane) + 1 and
// 2(31-lane)).  The shared-memory pipe is the curvilinear kernels' busiest
// (67 %), and the closures were 29 % of the velocity kernel's traffic as
// broadcast shuffles: each lane now takes the top ten levels from lanes 27..31
// as five pairs, and its coefficients four at a time.
struct Closure {
  float4 c[3][5];
};
template <int NT>
__device__ __forceinline__ void closure_load(Closure& cl, const float (&T)[6][NT], int t) {
  if (t < 15) {
    const int q = t / 5, m = 2 * (t % 5);
    cl.c[q][t % 5] = make_float4(m < NT ? T[2 * q + 1][m] : 0.f, m < NT ? T[2 * q][m] : 0.f,
                                 m + 1 < NT ? T[2 * q + 1][m + 1] : 0.f,
                                 m + 1 < NT ? T[2 * q][m + 1] : 0.f);
  }
}
template <int NT>
__device__ __forceinline__ float2 closure(float2 v, const ColPos2& c, const Closure& cl,
                                          float2* top, float2 s) {
  // the warp's own scratch: this column's levels nz-10 .. nz-1
  __syncwarp();
  if (c.lane >= 27) top[31 - c.lane] = v;
  __syncwarp();
  const float4* const k = cl.c[c.lane >= 29 ? 31 - c.lane : 0];
  float2 b = make_float2(0.f, 0.f);
#pragma unroll
  for (int p = (NT + 1) / 2 - 1; p >= 0; --p) {
    const float4 w = k[p];
    const float2 t = top[p];  // levels nz-2-2p, nz-1-2p
    if (2 * p + 1 < NT) b = vfma(make_float2(w.z, w.w), dup(t.x), b);
    b = vfma(make_float2(w.x, w.y), dup(t.y), b);
  }
  return c.lane >= 29 ? b : s;
}

// 7-point vertical difference at the lane's two levels l, l+1 of a value held
// two levels per lane (interior coefficients), or the boundary rows in the
// top tile.
__device__ __forceinline__ float2 zd7(float2 v, const ColPos2& c, const Closure& cl,
                                      float2* top) {
  const float m3 = __shfl_up_sync(kAll, v.y, 2);    // l-3
  const float m2 = __shfl_up_sync(kAll, v.x, 1);    // l-2
  const float m1 = __shfl_up_sync(kAll, v.y, 1);    // l-1
  const float p2 = __shfl_down_sync(kAll, v.x, 1);  // l+2
  const float p3 = __shfl_down_sync(kAll, v.y, 1);  // l+3
  const float p4 = __shfl_down_sync(kAll, v.x, 2);  // l+4
  const float2 a = make_float2(m3 - p3, m2 - p4), b = make_float2(m2 - p2, m1 - p3),
               d = make_float2(m1 - v.y, v.x - p2);
  const float2 s = vfma(dup(kZ0), a, vfma(dup(kZ1), b, vscale(kZ2, d)));
  return c.top ? closure<9>(v, c, cl, top, s) : s;  // warp-uniform branch
}

// 4-point vertical difference: half-point form (k-2..k+1) or node form
// (k-1..k+2), or the boundary rows (NT of them).
template <bool HALF, int NT>
__device__ __forceinline__ float2 zd4(float2 v, const ColPos2& c, const Closure& cl,
                                      float2* top) {
  const float m1 = __shfl_up_sync(kAll, v.y, 1), p2 = __shfl_down_sync(kAll, v.x, 1);
  float2 a, b;
  if (HALF) {
    const float m2 = __shfl_up_sync(kAll, v.x, 1);
    a = make_float2(m2 - v.y, m1 - p2);
    b = make_float2(m1 - v.x, v.x - v.y);
  } else {
    const float p3 = __shfl_down_sync(kAll, v.y, 1);
    a = make_float2(m1 - p2, v.x - p3);
    b = make_float2(v.x - v.y, v.y - p2);
  }
  const float2 s = vfma(dup(kD0), a, vscale(kD1, b));
  return c.top ? closure<NT>(v, c, cl, top, s) : s;
}

// The value at level - 1 of each of a lane's two levels
__device__ __forceinline__ float2 below(float2 v) {
  return make_float2(__shfl_up_sync(kAll, v.y, 1), v.x);
}

// 1-D vertical metric (or sponge) at a lane's two levels
__device__ __forceinline__ float2 gk2(const float* __restrict__ g, int k) {
  return make_float2(__ldg(g + k + AWP_ALIGN), __ldg(g + k + 1 + AWP_ALIGN));
}

// One weight of a column: scale * metric(i + di, j + dj), or scale / metric.
struct Weight {
  const float* p;
  float scale;
  bool inv;
  __device__ float at(long long off) const {
    const float f = __ldg(p + off);
    return inv ? __fdividef(scale, f) : scale * f;
  }
};

// Per-warp table of a plane's weights, duplicated for packed arithmetic, two
// planes deep.
template <int N>
struct Table {
  float2 w[2][N];
};

// kD (difference) and kP (interpolation) weights of a 4-point operator
__device__ __forceinline__ float dw(int q) { return q == 0 ? kD0 : q == 1 ? kD1 : q == 2 ? -kD1 : -kD0; }
__device__ __forceinline__ float pw(int q) { return (q == 0 || q == 3) ? kP0 : kP1; }

__device__ __forceinline__ float2 dot4(const float2* w, float2 a, float2 b, float2 c, float2 d,
                                       float2 s) {
  s = vfma(w[0], a, s);
  s = vfma(w[1], b, s);
  s = vfma(w[2], c, s);
  return vfma(w[3], d, s);
}
__device__ __forceinline__ float2 dot4(const float2* w, float2 a, float2 b, float2 c, float2 d) {
  float2 s = vmul(w[0], a);
  s = vfma(w[1], b, s);
  s = vfma(w[2], c, s);
  return vfma(w[3], d, s);
}
// interior 4-point difference with constant weights
__device__ __forceinline__ float2 diff4(float2 a, float2 b, float2 c, float2 d) {
  return vfma(dup(kD0), vsub(a, d), vscale(kD1, vsub(b, c)));
}
// interpolant P0 (a + d) + P1 (b + c)
__device__ __forceinline__ float2 itp4(float2 a, float2 b, float2 c, float2 d) {
  return vfma(dup(kP0), vadd(a, d), vscale(kP1, vadd(b, c)));
}

// ===========================================================================
// Velocity
// ===========================================================================
// weights of a column: four-point differences of f X, then the slopes of the
// interpolants, then nu / f of the three components
enum VelW { kAx = 0, kAy = 4, kBx = 8, kBy = 12, kCy = 16, kCx = 20, kS = 24, kN = 30, kVelW = 33 };
constexpr int kVelWPad = 40;

struct TopoVelCfg : VelTile {
  static constexpr int LA = 2, NH = 1 + LA, DS = 3 + LA;  // planes ahead, rings
  // one stage: xx(i+1), xz(i+2), yy, yz (j halo), zz, density, u, v, w (i)
  static constexpr int G_XX = 0, G_XZ = kOwn, G_YY = 2 * kOwn, G_YZ = G_YY + kHalo,
                       G_ZZ = G_YZ + kHalo, G_D = G_ZZ + kOwn, G_O = G_D + kMed,
                       STAGE = G_O + 3 * kOwn;
  static constexpr int F_S = DS * kHalo, F_W = F_S + NH * STAGE,
                       F_C = F_W + kCol * 2 * kVelWPad * 2, F_T = F_C + 4 * 60,
                       F_G = F_T + kCol * 5 * 2, F_END = F_G + 7 * 64 + 4;
  static constexpr size_t bytes = sizeof(float) * F_END + sizeof(Pipe<NH, 0, kCol>) + 8;
};

__global__ void __launch_bounds__(VelTile::kThreads, 2)
    k_topo_velocity(const __grid_constant__ TopoArgs a, const __grid_constant__ TmaMaps tm,
                    const int ichunk, int* err, const unsigned spin) {
  using C = TopoVelCfg;
  constexpr int kCol = C::kCol, kOwn = C::kOwn, kHalo = C::kHalo;
  extern __shared__ __align__(128) float smem[];
  Closure* const cl = reinterpret_cast<Closure*>(smem + C::F_C);
  auto& pipe = *reinterpret_cast<Pipe<C::NH, 0, kCol>*>(smem + C::F_END);
  const int tid = threadIdx.x, warp = tid >> 5;
  const ColPos2 c(a.nz, blockIdx.x);
  const int kb = AWP_ALIGN + a.nz - kSpan - kTileOut * (int)blockIdx.x;
  const int j0 = blockIdx.y * kCol, jb = j0 + AWP_NGSL + 2;
  const int i0 = blockIdx.z * ichunk, n = min(ichunk, a.nx - i0), ib = i0 + AWP_NGSL + 2;
  grid_go();
  if (tid == 0) pipe.init();
  closure_load(cl[0], kTopoVelDhpz4r, tid);
  closure_load(cl[1], kTopoVelDphz4r, tid);
  closure_load(cl[2], kTopoVelDhz4r, tid);
  closure_load(cl[3], kTopoVelDz4r, tid);
  // the vertical metrics depend on k alone: one copy for all the columns
  enum { kGc, kGg, kG3c, kG3, kIg3c, kIg3, kDcz };
  float2* const vm = reinterpret_cast<float2*>(smem + C::F_G);
  if (warp == 0) {
    vm[32 * kGc + c.lane] = gk2(a.g_c, c.ld);
    vm[32 * kGg + c.lane] = gk2(a.g, c.ld);
    vm[32 * kG3c + c.lane] = gk2(a.g3_c, c.ld);
    vm[32 * kG3 + c.lane] = gk2(a.g3, c.ld);
    vm[32 * kIg3c + c.lane] = vquot(1.0f, gk2(a.g3_c, c.ld));
    vm[32 * kIg3 + c.lane] = vquot(1.0f, gk2(a.g3, c.ld));
    vm[32 * kDcz + c.lane] = gk2(a.dcrjz, c.ld);
  }
  auto M = [&](int q) { return vm[32 * q + c.lane]; };
  __syncthreads();
  grid_wait();

  if (warp == kCol) {  // producer warp
    if (c.lane == 0) {
      pipe.produce(
          n,
          [&](int s, uint64_t* b) {
            const int p0 = s == 0 ? 0 : s + 2;
            mbar_expect_tx(b, ((s + 2 - p0 + 1) * kHalo + C::STAGE) * 4);
            for (int p = p0; p <= s + 2; ++p)
              tma_load3(smem + (p % C::DS) * kHalo, &tm.halo[3], b, kb, jb - 2, ib + p);
            float* g = smem + C::F_S + (s % C::NH) * C::STAGE;
            const int i = ib + s;
            tma_load3(g + C::G_XX, &tm.halo[0], b, kb, jb, i + 1);
            tma_load3(g + C::G_XZ, &tm.halo[4], b, kb, jb, i + 2);
            tma_load3(g + C::G_YY, &tm.halo[1], b, kb, jb - 1, i);
            tma_load3(g + C::G_YZ, &tm.halo[5], b, kb, jb - 2, i);
            tma_load3(g + C::G_ZZ, &tm.halo[2], b, kb, jb, i);
            tma_load3(g + C::G_D, &tm.media[0], b, kb, jb - 1, i);
            for (int f = 0; f < 3; ++f)
              tma_load3(g + C::G_O + f * kOwn, &tm.own[f], b, kb, jb, i);
          },
          [](int, uint64_t*) {}, err, spin);
    }
    return;
  }

  const int j = j0 + warp;
  const bool jin = j < a.ny;
  const bool o0 = c.out0 && jin, o1 = c.out1 && jin;
  const int S = a.slice, Y = a.yline, FL = a.fld;
  const int ja = jb + warp;  // a warp past the grid computes on its padding
  const int jm = min(j, a.ny - 1);
  // the lowest tile's lane of levels 2 and 3 takes the interface layer
  const bool low = a.layer && blockIdx.x + 1 == gridDim.x;
  const bool lay = low && c.k == 2 && c.lane >= 2 && (c.top || c.lane <= 29) && jin;
  long long o = (long long)ib * S + (long long)ja * Y + (c.ld + AWP_ALIGN);
  // this lane's two weights of the column (weight index lane, lane + 32)
  Table<kVelWPad>& tab = reinterpret_cast<Table<kVelWPad>*>(smem + C::F_W)[warp];
  auto weight = [&](int w) {
    // arrays of the six differences, six slopes and three quotients
    const float* const D[6] = {a.f_c, a.f, a.f, a.f_c, a.f_2, a.f_1};
    const float* const SL[6] = {a.f1_1, a.f2_1, a.f1_2, a.f2_2, a.f1_c, a.f2_c};
    const float* const Q[3] = {a.f_1, a.f_2, a.f_c};
    // first offset and axis (x: true) of the differences, in VelW's order
    constexpr int first[6] = {-2, -2, -1, -1, -2, -1};
    constexpr bool alongx[6] = {true, false, true, false, false, true};
    Weight r{a.f, 0.f, false};
    int di = 0, dj = 0;
    if (w < kS) {
      const int q = w >> 2, m = w & 3;
      r.p = D[q];
      r.scale = dw(m);
      (alongx[q] ? di : dj) = first[q] + m;
    } else if (w < kN) {
      r.p = SL[w - kS];
      r.scale = 1.0f;
    } else if (w < kVelW) {
      r.p = Q[w - kN];
      r.scale = a.nu;
      r.inv = true;
    }
    r.p += (long long)(ib + di) * FL + (jm + dj + AWP_NGSL + 2 + AWP_ALIGN);
    return r;
  };
  const Weight w0 = weight(c.lane), w1 = weight(c.lane + 32);
  float n0 = w0.at(0), n1 = c.lane < 1 ? w1.at(0) : 0.f;

  const float dcy = __ldg(a.dcrjy + ja);
  float2* const top = reinterpret_cast<float2*>(smem + C::F_T) + warp * 5;
  // own-column values of the planes before the ones the tiles bring
  float2 xx_m2, xx_m1, xx_0, xy_m1, xy_0, xy_p1, xz_m1, xz_0, xz_p1, d_m, t_m;
  {
    const float *X = a.xx + o, *P = a.xy + o, *Q = a.xz + o, *D = a.d1 + o - S;
    xx_m2 = ldg2(X - 2 * (long long)S); xx_m1 = ldg2(X - S); xx_0 = ldg2(X);
    xy_m1 = ldg2(P - S); xy_0 = ldg2(P); xy_p1 = ldg2(P + S);
    xz_m1 = ldg2(Q - S); xz_0 = ldg2(Q); xz_p1 = ldg2(Q + S);
    d_m = ldg2(D);
    t_m = vadd(d_m, ldg2(D - Y));
  }
  const int l = 2 * c.lane;
  const int h0 = warp * kSpan + l, h1 = (warp + 1) * kSpan + l, h2 = (warp + 2) * kSpan + l;

  Cursor<C::NH> ch;
  Cursor<awp_pipe::ND> cd;
  int ss = 0, ss2 = 2;
  bool ok = true;
#pragma unroll 1
  for (int s = 0; s < n; ++s) {
    // the plane's weights, then the next plane's loads
    float2* const W = tab.w[s & 1];
    W[c.lane] = dup(n0);
    if (c.lane < 1) W[32] = dup(n1);
    if (s + 1 < n) {
      n0 = w0.at((long long)(s + 1) * FL);
      if (c.lane < 1) n1 = w1.at((long long)(s + 1) * FL);
    }
    const float dcx = __ldg(a.dcrjx + ib + s);
    __syncwarp();
    ok = mbar_wait(pipe.full_h + ch.slot, ch.phase, spin);
    if (!__all_sync(kAll, ok)) break;
    const float* G = smem + C::F_S + ch.slot * C::STAGE;
    const float* XY = smem + ss * kHalo + h2;
    const float* YY = G + C::G_YY + h1;
    const float* YZ = G + C::G_YZ + h2;
    const float2 xx_p1 = lds2(G + C::G_XX + h0), xz_p2 = lds2(G + C::G_XZ + h0);
    const float2 xy_p2 = lds2(smem + ss2 * kHalo + h2);
    const float2 d_0 = lds2(G + C::G_D + h1), t_0 = vadd(d_0, lds2(G + C::G_D + h0));
    const float2 dcrj = vscale(dcx * dcy, M(kDcz));

    // --- u1 -----------------------------------------------------------------
    {
      const float2 y2 = lds2(XY - 2 * kSpan), y1 = lds2(XY - kSpan), yp = lds2(XY + kSpan);
      float2 e = dot4(W + kAx, xx_m2, xx_m1, xx_0, xx_p1);
      e = dot4(W + kAy, y2, y1, xy_0, yp, e);
      e = vfma(M(kG3c), e, zd4<true, 8>(xz_0, c, cl[2], top));
      float2 q = vmul(W[kS], itp4(xx_m2, xx_m1, xx_0, xx_p1));
      q = vfma(W[kS + 1], itp4(y2, y1, xy_0, yp), q);
      e = vsub(e, zd7(vmul(M(kGc), q), c, cl[0], top));
      const float2 ir = vquot(1.0f, vscale(0.25f, vadd(t_0, below(t_0))));
      const float2 A = vmul(vmul(W[kN], M(kIg3c)), ir), u0 = lds2(G + C::G_O + h0);
      float2 u = vmul(vfma(A, e, u0), dcrj);
      if (low) {  // dvelc2 (kernel.cu:2289-2343)
        const float km = __shfl_up_sync(kAll, xz_0.y, 1);
        const float su = (xx_0.x - xx_m1.x) + (xy_0.x - y1.x) + (xz_0.x - km);
        if (lay) u.x = __fmul_rn(__fmaf_rn(a.nu * ir.x, su, u0.x), dcrj.x);
      }
      st2(a.u1 + o, u, o0 || lay, o1);
    }
    const float2 yz_0 = lds2(YZ);
    // --- u2 -----------------------------------------------------------------
    {
      const float2 y0 = lds2(YY), ym = lds2(YY - kSpan), y1 = lds2(YY + kSpan),
                   y2 = lds2(YY + 2 * kSpan);
      float2 e = dot4(W + kBx, xy_m1, xy_0, xy_p1, xy_p2);
      e = dot4(W + kBy, ym, y0, y1, y2, e);
      e = vfma(M(kG3c), e, zd4<true, 8>(yz_0, c, cl[2], top));
      float2 q = vmul(W[kS + 2], itp4(xy_m1, xy_0, xy_p1, xy_p2));
      q = vfma(W[kS + 3], itp4(ym, y0, y1, y2), q);
      e = vsub(e, zd7(vmul(M(kGc), q), c, cl[0], top));
      const float2 x = vadd(d_0, d_m);
      const float2 A = vmul(vmul(W[kN + 1], M(kIg3c)), vquot(1.0f, vscale(0.25f, vadd(x, below(x)))));
      const float2 v0 = lds2(G + C::G_O + kOwn + h0);
      float2 v = vmul(vfma(A, e, v0), dcrj);
      if (low) {
        const float km = __shfl_up_sync(kAll, yz_0.y, 1), dk = __shfl_up_sync(kAll, d_0.y, 1);
        if (lay) {
          const float* D = a.d1 + o + S;
          const float sv = (xy_p1.x - xy_0.x) + (y1.x - y0.x) + (yz_0.x - km);
          const float r = __fmul_rn(0.25f, (d_0.x + D[0]) + (dk + D[-1]));
          v.x = __fmul_rn(__fmaf_rn(__fdividef(a.nu, r), sv, v0.x), dcrj.x);
        }
      }
      st2(a.v1 + o, v, o0 || lay, o1);
    }
    // --- u3 -----------------------------------------------------------------
    {
      const float2 y2 = lds2(YZ - 2 * kSpan), y1 = lds2(YZ - kSpan), yp = lds2(YZ + kSpan);
      float2 e = dot4(W + kCy, y2, y1, yz_0, yp);
      e = dot4(W + kCx, xz_m1, xz_0, xz_p1, xz_p2, e);
      const float2 z = lds2(G + C::G_ZZ + h0);
      e = vfma(M(kG3), e, zd4<false, 7>(z, c, cl[3], top));
      float2 q = vmul(W[kS + 4], itp4(xz_m1, xz_0, xz_p1, xz_p2));
      q = vfma(W[kS + 5], itp4(y2, y1, yz_0, yp), q);
      e = vsub(e, zd7(vmul(M(kGg), q), c, cl[1], top));
      const float2 A = vmul(vmul(W[kN + 2], M(kIg3)), vquot(1.0f, vscale(0.25f, vadd(t_0, t_m))));
      const float2 w0 = lds2(G + C::G_O + 2 * kOwn + h0);
      float2 w = vmul(vfma(A, e, w0), dcrj);
      if (lay) {
        const float* D = a.d1 + o + S;
        const float sw = (xz_p1.x - xz_0.x) + (yz_0.x - y1.x) + (z.y - z.x);
        const float r = __fmul_rn(0.25f, t_0.x + (D[0] + D[-Y]));
        w.x = __fmul_rn(__fmaf_rn(__fdividef(a.nu, r), sw, w0.x), dcrj.x);
      }
      st2(a.w1 + o, w, o0 || lay, o1);
    }
    warp_done(pipe.done + cd.slot, c.lane);

    o += S;
    xx_m2 = xx_m1; xx_m1 = xx_0; xx_0 = xx_p1;
    xy_m1 = xy_0; xy_0 = xy_p1; xy_p1 = xy_p2;
    xz_m1 = xz_0; xz_0 = xz_p1; xz_p1 = xz_p2;
    d_m = d_0; t_m = t_0;
    ch.next();
    cd.next();
    ss = ss + 1 == C::DS ? 0 : ss + 1;
    ss2 = ss2 + 1 == C::DS ? 0 : ss2 + 1;
  }
  if (!__all_sync(kAll, ok) && c.lane == 0) atomicExch(err, 1);
}

// ===========================================================================
// Stress and memory variables
// ===========================================================================
// weights of a column: the interpolants of f-weighted velocities, then 1 / f
enum StrW { kIu = 0, kIv = 4, kJu = 8, kJv = 12, kKw = 16, kLw = 20, kF = 24, kStrW = 28 };

template <bool ELASTIC>
struct TopoStrCfg : StrTile {
  static constexpr int NM = ELASTIC ? 2 : 4, NF = ELASTIC ? 6 : 12;
  static constexpr int LH = 2, LO = 1, NH = 1 + LH, NO = 1 + LO, DU = 3 + LH, DV = 2 + LH;
  static constexpr int F_U = 0, F_V = F_U + DU * kHalo, F_W = F_V + DV * kHalo,
                       F_M = F_W + DV * kHalo, F_O = F_M + NH * NM * kMed,
                       F_T = F_O + NO * NF * kOwn, F_X = F_T + (ELASTIC ? 0 : 80),
                       F_C = F_X + kCol * 2 * 32 * 2, F_L = F_C + 4 * 60,
                       F_G = F_L + kCol * 5 * 2 + 2, F_END = F_G + 6 * 64;  // vertical metrics of the lanes
  static constexpr size_t bytes = sizeof(float) * F_END + sizeof(Pipe<NH, NO, kCol>) + 8;
};

// LAYER: on a block over a coarser one (TopoArgs::layer).
template <bool ELASTIC, bool LAYER>
__global__ void __launch_bounds__(StrTile::kThreads, 2)
    k_topo_stress(const __grid_constant__ TopoArgs a, const __grid_constant__ TmaMaps tm,
                  const int ichunk, int* err, const unsigned spin) {
  using C = TopoStrCfg<ELASTIC>;
  constexpr int NM = C::NM, NF = C::NF;
  constexpr int kCol = C::kCol, kOwn = C::kOwn, kHalo = C::kHalo, kMed = C::kMed;
  extern __shared__ __align__(128) float smem[];
  Closure* const cl = reinterpret_cast<Closure*>(smem + C::F_C);
  auto& pipe = *reinterpret_cast<Pipe<C::NH, C::NO, kCol>*>(smem + C::F_END);
  const int tid = threadIdx.x, warp = tid >> 5;
  const ColPos2 c(a.nz, blockIdx.x);
  const int kb = AWP_ALIGN + a.nz - kSpan - kTileOut * (int)blockIdx.x;
  const int j0 = a.s_j + blockIdx.y * kCol, jb = j0 + AWP_NGSL + 2;
  const int i0 = a.s_i + blockIdx.z * ichunk, n = min(ichunk, a.e_i - i0),
            ib = i0 + AWP_NGSL + 2;
  grid_go();
  if (tid == 0) pipe.init();
  closure_load(cl[0], kTopoStrPhdz4r, tid);
  closure_load(cl[1], kTopoStrPdhz4r, tid);
  closure_load(cl[2], kTopoStrDhz4r, tid);
  closure_load(cl[3], kTopoStrDz4r, tid);
  if (!ELASTIC) {  // relaxation constants of the entry pairs (as k_stress_tma)
    float* t = smem + C::F_T;
    const float* const src[9] = {a.rel.vx2, a.rel.wwo, a.rel.kv, a.rel.kr, a.rel.kr2,
                                 a.rel.kf,  a.rel.c0,  a.rel.c1, a.rel.c2};
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (tid < 8) t[(tid >> 1) * 20 + 2 * q + (tid & 1)] = src[q][tid];
  }
  // the vertical metrics depend on k alone: one copy for all the columns, read
  // where they are used (held in registers they spilled)
  enum { kGc, kGg, kIg3c, kIg3, kIg12, kDcz };
  float2* const vm = reinterpret_cast<float2*>(smem + C::F_G);
  if (warp == 0) {
    vm[32 * kGc + c.lane] = gk2(a.g_c, c.ld);
    vm[32 * kGg + c.lane] = gk2(a.g, c.ld);
    vm[32 * kIg3c + c.lane] = vquot(1.0f, gk2(a.g3_c, c.ld));
    vm[32 * kIg3 + c.lane] = vquot(1.0f, gk2(a.g3, c.ld));
    // the xy Jacobian's interior rows read g3_c six points higher
    // (stress_attenuation.cu:471), the boundary rows at k (:1149)
    vm[32 * kIg12 + c.lane] =
        vquot(1.0f, gk2(a.g3_c, c.top && c.lane >= 29 ? c.ld : c.ld + 6));
    vm[32 * kDcz + c.lane] = gk2(a.dcrjz, c.ld);
  }
  __syncthreads();
  grid_wait();

  if (warp == kCol) {  // producer warp
    if (c.lane == 0) {
      pipe.produce(
          n,
          [&](int s, uint64_t* b) {
            const int u0 = s == 0 ? 0 : s + 2, v0 = s == 0 ? 0 : s + 1;
            mbar_expect_tx(
                b, ((s + 2 - u0 + 1) * kHalo + 2 * (s + 1 - v0 + 1) * kHalo + NM * kMed) * 4);
            for (int p = u0; p <= s + 2; ++p)
              tma_load3(smem + C::F_U + (p % C::DU) * kHalo, &tm.halo[0], b, kb, jb - 1, ib + p);
            for (int p = v0; p <= s + 1; ++p) {
              tma_load3(smem + C::F_V + (p % C::DV) * kHalo, &tm.halo[1], b, kb, jb - 2, ib + p);
              tma_load3(smem + C::F_W + (p % C::DV) * kHalo, &tm.halo[2], b, kb, jb - 1, ib + p);
            }
            float* m = smem + C::F_M + (s % C::NH) * NM * kMed;
            for (int f = 0; f < NM; ++f)
              tma_load3(m + f * kMed, &tm.media[f], b, kb, jb - 1, ib + s + 1);
          },
          [&](int s, uint64_t* b) {
            mbar_expect_tx(b, NF * kOwn * 4);
            float* q = smem + C::F_O + (s % C::NO) * NF * kOwn;
            for (int f = 0; f < NF; ++f)
              tma_load3(q + f * kOwn, &tm.own[f], b, kb, jb, ib + s);
          },
          err, spin);
    }
    return;
  }

  const int j = j0 + warp;
  const bool jin = j < a.e_j;
  const bool o0 = c.out0 && jin, o1 = c.out1 && jin;
  const int S = a.slice, Y = a.yline, FL = a.fld;
  const int ja = jb + warp, jm = min(j, a.ny - 1);
  const bool low = LAYER && blockIdx.x + 1 == gridDim.x;  // as in k_topo_velocity
  const bool lay = low && c.k == 2 && c.lane >= 2 && (c.top || c.lane <= 29) && jin;
  long long o = (long long)ib * S + (long long)ja * Y + (c.ld + AWP_ALIGN);
  float* __restrict__ SG[6] = {a.xx, a.yy, a.zz, a.xy, a.xz, a.yz};
  float* __restrict__ RR[6] = {a.r1, a.r2, a.r3, a.r4, a.r5, a.r6};
  Table<32>& tab = reinterpret_cast<Table<32>*>(smem + C::F_X)[warp];
  Weight wt{a.f, 0.f, false};
  {
    // interpolants: f1_1 u (x), f2_2 v (y), f2_1 u (y), f1_2 v (x), f1_c w (x),
    // f2_c w (y); then 1/f_c, 1/f, 1/f_1, 1/f_2
    const float* const I[6] = {a.f1_1, a.f2_2, a.f2_1, a.f1_2, a.f1_c, a.f2_c};
    const float* const Q[4] = {a.f_c, a.f, a.f_1, a.f_2};
    constexpr int first[6] = {-1, -2, -1, -2, -2, -1};
    constexpr bool alongx[6] = {true, false, false, true, true, false};
    int di = 0, dj = 0;
    if (c.lane < kF) {
      const int q = c.lane >> 2, m = c.lane & 3;
      wt.p = I[q];
      wt.scale = pw(m);
      (alongx[q] ? di : dj) = first[q] + m;
    } else if (c.lane < kStrW) {
      wt.p = Q[c.lane - kF];
      wt.scale = 1.0f;
      wt.inv = true;
    }
    wt.p += (long long)(ib + di) * FL + (jm + dj + AWP_NGSL + 2 + AWP_ALIGN);
  }
  float nw = wt.at(0);

  auto G = [&](int q) { return vm[32 * q + c.lane]; };
  const float dcy = __ldg(a.dcrjy + ja);
  float2* const top = reinterpret_cast<float2*>(smem + C::F_L) + warp * 5;
  // texture entry pairs at even and odd steps (two adjacent levels starting at
  // an even one: entries e, e + 1)
  const int e0 = awp_tex_index(a.tex, ib, ja, c.k + AWP_ALIGN) >> 1,
            e1 = awp_tex_index(a.tex, ib + 1, ja, c.k + AWP_ALIGN) >> 1;
  float2 u_m1, u_0, u_p1, v_m2, v_m1, v_0, w_m2, w_m1, w_0;
  {
    const float *U = a.u1 + o, *V = a.v1 + o, *W = a.w1 + o;
    u_m1 = ldg2(U - S); u_0 = ldg2(U); u_p1 = ldg2(U + S);
    v_m2 = ldg2(V - 2 * (long long)S); v_m1 = ldg2(V - S); v_0 = ldg2(V);
    w_m2 = ldg2(W - 2 * (long long)S); w_m1 = ldg2(W - S); w_0 = ldg2(W);
  }
  // media sums of the current plane: over j, j-1 and the level below
  auto quad = [&](float2 t) { return awp_quad(t, below(t)); };
  float2 Lq, Mq, Mt, Mm, Pq = {}, Rq = {}, Rt = {}, Rm = {};
  {
    auto rows = [&](const float* p, float2& m) {
      m = ldg2(p);
      return vadd(m, ldg2(p - Y));
    };
    float2 m;
    Lq = quad(rows(a.lam + o, m));
    Mt = rows(a.mu + o, Mm);
    Mq = quad(Mt);
    if (!ELASTIC) {
      Pq = quad(rows(a.qp + o, m));
      Rt = rows(a.qs + o, Rm);
      Rq = quad(Rt);
    }
  }
  const int l = 2 * c.lane;
  const int h0 = warp * kSpan + l, h1 = (warp + 1) * kSpan + l, h2 = (warp + 2) * kSpan + l;

  Cursor<C::NH> ch;
  Cursor<C::NO> co;
  Cursor<awp_pipe::ND> cd;
  int su = 0, su2 = 2, sv = 0, sv1 = 1;
  bool ok = true;
#pragma unroll 1
  for (int s = 0; s < n; ++s) {
    float2* const W = tab.w[s & 1];
    W[c.lane] = dup(nw);
    if (s + 1 < n) nw = wt.at((long long)(s + 1) * FL);
    const float dcx = __ldg(a.dcrjx + ib + s);
    __syncwarp();
    ok = mbar_wait(pipe.full_h + ch.slot, ch.phase, spin);
    if (!__all_sync(kAll, ok)) break;
    const float* U0 = smem + C::F_U + su * kHalo + h1;
    const float* V0 = smem + C::F_V + sv * kHalo + h2;
    const float* W0 = smem + C::F_W + sv * kHalo + h1;
    const float2 u_p2 = lds2(smem + C::F_U + su2 * kHalo + h1);
    const float2 v_p1 = lds2(smem + C::F_V + sv1 * kHalo + h2);
    const float2 w_p1 = lds2(smem + C::F_W + sv1 * kHalo + h1);
    const float2 zero = make_float2(0.f, 0.f);

    // ---- strain rates: every vertical difference of a horizontal interpolant
    // is one difference of the interpolated column
    float2 d[9];
    {
      // normal components: Jii = 1 / (f_c g3_c) (stress_attenuation.cu:340-431)
      const float2 J = vmul(W[kF], G(kIg3c)), Jg = vmul(J, G(kGc));
      const float2 v2 = lds2(V0 - 2 * kSpan), v1 = lds2(V0 - kSpan), vp = lds2(V0 + kSpan);
      d[0] = vsub(diff4(u_m1, u_0, u_p1, u_p2),
                  vmul(Jg, zd7(dot4(W + kIu, u_m1, u_0, u_p1, u_p2), c, cl[0], top)));
      d[1] = vsub(diff4(v2, v1, v_0, vp), vmul(Jg, zd7(dot4(W + kIv, v2, v1, v_0, vp), c, cl[0], top)));
      d[2] = vmul(J, zd4<true, 8>(w_0, c, cl[2], top));
      if (low) {  // dstrqc2 (kernel.cu:2564-2767): second-order rates, Cartesian
        const float km = __shfl_up_sync(kAll, w_0.y, 1);
        if (lay) {
          d[0].x = u_p1.x - u_0.x;
          d[1].x = v_0.x - v1.x;
          d[2].x = w_0.x - km;
        }
      }
    }
    {
      // xy: J12i = 1 / (f g3_c)
      const float2 J = vmul(vmul(W[kF + 1], G(kIg12)), G(kGc));
      const float2 um = lds2(U0 - kSpan), u1 = lds2(U0 + kSpan), u2 = lds2(U0 + 2 * kSpan);
      const float2 q = dot4(W + kJv, v_m2, v_m1, v_0, v_p1, dot4(W + kJu, um, u_0, u1, u2));
      d[3] = diff4(um, u_0, u1, u2);
      d[4] = vsub(diff4(v_m2, v_m1, v_0, v_p1), vmul(J, zd7(q, c, cl[0], top)));
      if (lay) {
        d[3].x = u1.x - u_0.x;
        d[4].x = v_0.x - v_m1.x;
      }
    }
    {
      // xz: J13i = 1 / (f_1 g3) (:550-598, :1254-1317)
      const float2 J = vmul(W[kF + 2], G(kIg3));
      const float2 z = zd7(dot4(W + kKw, w_m2, w_m1, w_0, w_p1), c, cl[1], top);
      d[5] = vmul(J, vsub(zd4<false, 7>(u_0, c, cl[3], top), vmul(G(kGg), z)));
      d[6] = diff4(w_m2, w_m1, w_0, w_p1);
      if (lay) {
        d[5].x = u_0.y - u_0.x;
        d[6].x = w_0.x - w_m1.x;
      }
    }
    {
      // yz: J23i = 1 / (f_2 g3) (:600-650, :1319-1380)
      const float2 J = vmul(W[kF + 3], G(kIg3));
      const float2 wm = lds2(W0 - kSpan), w1 = lds2(W0 + kSpan), w2 = lds2(W0 + 2 * kSpan);
      const float2 z = zd7(dot4(W + kLw, wm, w_0, w1, w2), c, cl[1], top);
      d[7] = vmul(J, vsub(zd4<false, 7>(v_0, c, cl[3], top), vmul(G(kGg), z)));
      d[8] = diff4(wm, w_0, w1, w2);
      if (lay) {
        d[7].x = v_0.y - v_0.x;
        d[8].x = w1.x - w_0.x;
      }
    }

    // ---- material coefficients and the update (as the Cartesian dstrqc) -----
    AwpRelax<float2> rx{};
    if (!ELASTIC) {
      const float* t = smem + C::F_T + ((s & 1) ? e1 : e0) * 20;
      const float4* t4 = reinterpret_cast<const float4*>(t);
      const float4 q0 = t4[0], q1 = t4[1], q2 = t4[2], q3 = t4[3];
      rx.vx2 = make_float2(q0.x, q0.y); rx.wwo = make_float2(q0.z, q0.w);
      rx.kv = make_float2(q1.x, q1.y); rx.kr = make_float2(q1.z, q1.w);
      rx.kr2 = make_float2(q2.x, q2.y); rx.kf = make_float2(q2.z, q2.w);
      rx.c0 = make_float2(q3.x, q3.y); rx.c1 = make_float2(q3.z, q3.w);
      rx.c2 = lds2(t + 16);
    }
    AwpStrCoef<float2> cf;
    {
      const float* M = smem + C::F_M + ch.slot * NM * kMed;
      auto rows = [&](int f, float2& m) {
        m = lds2(M + f * kMed + h1);
        return vadd(m, lds2(M + f * kMed + h0));
      };
      float2 m, mm;
      const float2 Ln = quad(rows(0, m)), mt = rows(1, mm), mq = quad(mt);
      const float2 P[3] = {vadd(Mm, below(Mm)), Mt, vadd(Mm, mm)};
      float2 QP8 = zero, QS8 = zero, R[3] = {zero, zero, zero};
      if (!ELASTIC) {
        float2 rm;
        const float2 pq = quad(rows(2, m)), rt = rows(3, rm), rq = quad(rt);
        QP8 = vadd(Pq, pq);
        QS8 = vadd(Rq, rq);
        R[0] = vadd(Rm, below(Rm)); R[1] = Rt; R[2] = vadd(Rm, rm);
        Pq = pq;
        Rq = rq; Rt = rt; Rm = rm;
      }
      const float2 L8 = vadd(Lq, Ln), M8 = vadd(Mq, mq);
      if (LAYER) {
        const int e = 2 * ((s & 1) ? e1 : e0);
        AwpLayerOps ops{lay, 0.f, 0.f};
        float2 dth = dup(a.dth), DT = dup(a.DT);
        if (lay) {
          ops.l0 = a.lay.l0[e];
          ops.l1 = a.lay.l1[e];
          const AwpRelax<float> l = awp_relax_at(a.lay_rel, e);
          rx.kv.x = l.kv; rx.kr.x = l.kr; rx.kr2.x = l.kr2; rx.kf.x = l.kf;
          rx.c2.x *= 0.5f;
          dth.x = a.lay_dth;
          DT.x = a.lay_dt;
        }
        cf = awp_stress_coef<ELASTIC>(L8, M8, P, QP8, QS8, R, rx, a.thr, dth, DT, ops);
      } else {
        cf = awp_stress_coef<ELASTIC>(L8, M8, P, QP8, QS8, R, rx, a.thr, dup(a.dth), dup(a.DT));
      }
      Lq = Ln;
      Mq = mq; Mt = mt; Mm = mm;
    }
    const float2 dcrj = vscale(dcx * dcy, G(kDcz));
    ok = mbar_wait(pipe.full_o + co.slot, co.phase, spin);
    if (!__all_sync(kAll, ok)) break;
    const float* O = smem + C::F_O + co.slot * NF * kOwn + h0;
    float2 sg[6], rr[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      sg[q] = lds2(O + q * kOwn);
      if (!ELASTIC) rr[q] = lds2(O + (6 + q) * kOwn);
    }
    awp_stress_update<ELASTIC>(sg, rr, cf, rx, dcrj, d);
    if (o0 || o1) {  // (lay has o1)
      const bool ox = o0 || lay;
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        st2(SG[q] + o, sg[q], ox, o1);
        if (!ELASTIC) st2(RR[q] + o, rr[q], ox, o1);
      }
    }
    warp_done(pipe.done + cd.slot, c.lane);

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
  if (!__all_sync(kAll, ok) && c.lane == 0) atomicExch(err, 1);
}

// Tiles of a column: the top one (outputs nz-60 .. nz-1), then one per 56
// levels below it until a tile outputs level 3.
unsigned column_tiles(int nz) {
  return 1u + (nz > 63 ? (unsigned)((nz - 63 + kTileOut - 1) / kTileOut) : 0u);
}

Shape g_shape_vel[kMaxDev], g_shape_str[4][kMaxDev];

}  // namespace

int awp_topo_box(int kernel, int group, int* bx, int* by) {
  const int nc = kernel == 0 ? VelTile::kCol : StrTile::kCol;
  *bx = kSpan;
  *by = group == 0 ? nc + 3 : group == 1 ? nc + 1 : nc;
  return 0;
}

cudaError_t awp_launch_topo_velocity(const TopoArgs& a, const TmaMaps& tm, int ichunk, int* err,
                                     cudaStream_t st) {
  if (a.nz < 12 || a.nx < 1 || a.ny < 1) return cudaErrorInvalidValue;
  const dim3 tile(column_tiles(a.nz), cdiv_u(a.ny, VelTile::kCol));
  int resident = 0;
  const cudaError_t e = resident_ctas((const void*)k_topo_velocity, TopoVelCfg::bytes,
                                      VelTile::kThreads,
                                      g_shape_vel, &resident);
  if (e != cudaSuccess) return e;
  const int ch = march_planes((long long)tile.x * tile.y, a.nx, resident, ichunk, kMost);
  return launch_after(k_topo_velocity, dim3(tile.x, tile.y, cdiv_u(a.nx, ch)),
                      dim3(VelTile::kThreads), TopoVelCfg::bytes, st, a, tm, ch, err,
                      awp_pipe_spin_limit);
}

cudaError_t awp_launch_topo_stress(const TopoArgs& a, const TmaMaps& tm, bool elastic, int ichunk,
                                   int* err, cudaStream_t st) {
  if (a.nz < 12) return cudaErrorInvalidValue;
  const int ni = a.e_i - a.s_i, nj = a.e_j - a.s_j;
  if (ni <= 0 || nj <= 0) return cudaSuccess;
  const dim3 tile(column_tiles(a.nz), cdiv_u(nj, StrTile::kCol));
  const size_t sm = elastic ? TopoStrCfg<true>::bytes : TopoStrCfg<false>::bytes;
  const auto f = elastic ? (a.layer ? k_topo_stress<true, true> : k_topo_stress<true, false>)
                         : (a.layer ? k_topo_stress<false, true> : k_topo_stress<false, false>);
  int resident = 0;
  const cudaError_t e =
      resident_ctas((const void*)f, sm, StrTile::kThreads,
                    g_shape_str[(elastic ? 2 : 0) + (a.layer ? 1 : 0)], &resident);
  if (e != cudaSuccess) return e;
  const int ch = march_planes((long long)tile.x * tile.y, ni, resident, ichunk, kMost);
  const dim3 grid(tile.x, tile.y, cdiv_u(ni, ch));
  return launch_after(f, grid, dim3(StrTile::kThreads), sm, st, a, tm, ch, err,
                      awp_pipe_spin_limit);
}
