// Discontinuous-mesh coupling kernels (reference: src/awp/kernel.cu:2289-3234,
// src/awp/mesh.c:1404-1443).  All are 2-D over an interface (a few planes of
// work per step) and bound by the 32-byte sectors their single levels of
// k-contiguous columns touch.
//
// At one rank the reference's swap-area exchanges (swap.c:549-583,
// kernel.cu:3320-3676) return at once and bgcaccess (kernel.cu:2809-2852)
// only ever reads the grid itself: every index swap3 forms lies inside the
// padded fine grid, so the window average reads the fine grid directly.
#include <cuda_runtime.h>

#include "awp_dm.cuh"
#include "awp_pipe.cuh"
#include "awp_stencil.cuh"

namespace {

__device__ __forceinline__ long long at(const DmGrid& g, int i, int j, int k) {
  return (long long)i * g.slice + (long long)j * g.yline + k;
}

// ===========================================================================
// dvelc2 (kernel.cu:2289-2343)
// ===========================================================================
__global__ void k_dvelc2(const DmVel2Args a) {
  awp_pipe::grid_start();
  const int j = 2 + AWP_NGSL + blockIdx.x * blockDim.x + threadIdx.x;
  const int i = 2 + AWP_NGSL + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.g.nxt + 2 + AWP_NGSL || j >= a.g.nyt + 2 + AWP_NGSL) return;
  const int S = a.g.slice, Y = a.g.yline;
  const int k = 2 + AWP_ALIGN;
  const long long pos = at(a.g, i, j, k);
  // every load first (a store could alias a later load, and would make it
  // wait): each of these values is a 32-byte sector of its own column
  const float* d = a.d1 + pos;
  const float *xx = a.g.xx + pos, *yy = a.g.yy + pos, *zz = a.g.zz + pos, *xy = a.g.xy + pos,
              *xz = a.g.xz + pos, *yz = a.g.yz + pos;
  const float d0 = d[0], dk = d[-1], dx = d[S], dxk = d[S - 1], dy = d[-Y], dyk = d[-Y - 1],
              dxy = d[S - Y];
  const float u0 = a.g.u1[pos], v0 = a.g.v1[pos], w0 = a.g.w1[pos];
  const float xx0 = xx[0], xxm = xx[-S], yy0 = yy[0], yyp = yy[Y], zz0 = zz[0], zzp = zz[1];
  const float xy0 = xy[0], xyx = xy[S], xyy = xy[-Y];
  const float xz0 = xz[0], xzx = xz[S], xzk = xz[-1];
  const float yz0 = yz[0], yzy = yz[-Y], yzk = yz[-1];
  const float dcrj = __fmul_rn(__fmul_rn(a.dcrjz[k], a.dcrjx[i]), a.dcrjy[j]);
  auto mean = [](float p, float q, float r, float t) {
    return __fmul_rn(0.25f, __fadd_rn(__fadd_rn(__fadd_rn(p, q), r), t));
  };
  const float fd1 = a.dth / mean(d0, dy, dk, dyk), fd2 = a.dth / mean(d0, dx, dk, dxk),
              fd3 = a.dth / mean(d0, dx, dy, dxy);
  const float sw = __fadd_rn(__fadd_rn(__fsub_rn(xzx, xz0), __fsub_rn(yz0, yzy)),
                             __fsub_rn(zzp, zz0));
  const float su = __fadd_rn(__fadd_rn(__fsub_rn(xx0, xxm), __fsub_rn(xy0, xyy)),
                             __fsub_rn(xz0, xzk));
  const float sv = __fadd_rn(__fadd_rn(__fsub_rn(xyx, xy0), __fsub_rn(yyp, yy0)),
                             __fsub_rn(yz0, yzk));
  a.g.w1[pos] = __fmul_rn(__fmaf_rn(fd3, sw, w0), dcrj);
  a.g.u1[pos] = __fmul_rn(__fmaf_rn(fd1, su, u0), dcrj);
  a.g.v1[pos] = __fmul_rn(__fmaf_rn(fd2, sv, v0), dcrj);
}

// ===========================================================================
// dstrqc2 (kernel.cu:2564-2767), anelastic form (ELA2 undefined)
// ===========================================================================
// Every load is issued before the arithmetic: the kernel's time is the sectors
// of one level of k-contiguous columns, one 32-byte sector per value (300 x
// 300: 58 us), so a mesh block leaves it only the ring outside the exclusion
// rectangle (14 us): inside, the stress kernel that has the lines above in
// shared memory updates the layer too.
__global__ void __launch_bounds__(128) k_dstrqc2(const DmStr2Args a) {
  awp_pipe::grid_start();
  const int j = a.j0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int i = a.i0 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i > a.i1 || j > a.j1) return;
  if (i >= a.ex_i0 && i <= a.ex_i1 && j >= a.ex_j0 && j <= a.ex_j1) return;
  const int S = a.g.slice, Y = a.g.yline;
  const int k = AWP_ALIGN + 2;
  const long long pos = at(a.g, i, j, k);
  const DmGrid& g = a.g;
  float sg[6] = {g.xx[pos], g.yy[pos], g.zz[pos], g.xy[pos], g.xz[pos], g.yz[pos]};
  float rr[6] = {a.r1[pos], a.r2[pos], a.r3[pos], a.r4[pos], a.r5[pos], a.r6[pos]};
  const float *u = g.u1 + pos, *v = g.v1 + pos, *w = g.w1 + pos;
  const float u0 = u[0], ux = u[S], uy = u[Y], uk = u[1];
  const float v0 = v[0], vx = v[-S], vy = v[-Y], vk = v[1];
  const float w0 = w[0], wx = w[-S], wy = w[Y], wk = w[-1];
  // a field's value, its pair sums with k-1, j-1, i+1 and its eight-cell sum
  struct Mat {
    float pk, pj, pi, s8;
  };
  auto mat = [&](const float* f) {
    const float* p = f + pos;
    const float m0 = p[0], mk = p[-1], mj = p[-Y], mjk = p[-Y - 1], mi = p[S], mik = p[S - 1],
                mij = p[S - Y], mijk = p[S - Y - 1];
    return Mat{vadd(m0, mk), vadd(m0, mj), vadd(m0, mi),
               vadd(awp_quad(vadd(m0, mj), vadd(mk, mjk)),
                    awp_quad(vadd(mi, mij), vadd(mik, mijk)))};
  };
  const Mat L = mat(a.lam), M = mat(a.mu), P = mat(a.qp), R = mat(a.qs);
  const float dcrj = __fmul_rn(__fmul_rn(a.dcrjz[k], a.dcrjx[i]), a.dcrjy[j]);
  AwpRelax<float> rx;
  AwpLayerOps ops{true, 0.f, 0.f};
  if (a.vx1) {
    const float vx1 = a.vx1[pos], wwo = a.wwo[pos];
    const float *cf = a.coeff_dev + 2 * a.ww[pos] - 2, c0 = cf[0], c1 = cf[1];
    rx = awp_relax_from(vx1, a.vx2[pos], wwo, c0, c1, a.dt, a.dh1, &ops.l0, &ops.l1);
  } else {
    const int t = awp_tex_index(a.tex, i, j, k);
    rx = awp_relax_at(a.rel, t);
    ops.l0 = a.lay.l0[t];
    ops.l1 = a.lay.l1[t];
  }
  rx.c2 *= 0.5f;
  const float PM[3] = {M.pk, M.pj, M.pi}, PR[3] = {R.pk, R.pj, R.pi};
  const AwpStrCoef<float> cf =
      awp_stress_coef<false>(L.s8, M.s8, PM, P.s8, R.s8, PR, rx, a.thr, a.dth, a.dt, ops);
  const float d[9] = {__fsub_rn(ux, u0), __fsub_rn(v0, vy), __fsub_rn(w0, wk),  // x, y, z
                      __fsub_rn(uy, u0), __fsub_rn(v0, vx),                     // xy pair
                      __fsub_rn(uk, u0), __fsub_rn(w0, wx),                     // xz pair
                      __fsub_rn(vk, v0), __fsub_rn(wy, w0)};                    // yz pair
  awp_stress_update<false>(sg, rr, cf, rx, dcrj, d);
  g.xx[pos] = sg[0]; g.yy[pos] = sg[1]; g.zz[pos] = sg[2];
  g.xy[pos] = sg[3]; g.xz[pos] = sg[4]; g.yz[pos] = sg[5];
  a.r1[pos] = rr[0]; a.r2[pos] = rr[1]; a.r3[pos] = rr[2];
  a.r4[pos] = rr[3]; a.r5[pos] = rr[4]; a.r6[pos] = rr[5];
}

// ===========================================================================
// intp3d (kernel.cu:2359-2561): bilinear weights (1, 2/3, 1/3, 0) spread each
// coarse cell's four corners over a 4 x 4 fine patch at kh = align+1.
// Neighbouring patches share an edge, where the weight is 0 on one side and
// the reference's threads store the same value: a thread stores its patch's
// 3 x 3 cells, the last rows and columns their edge too (each store is a
// sector of its own).
// ===========================================================================
__global__ void k_intp3d(const DmPairArgs a) {
  awp_pipe::grid_start();
  const int j = AWP_NGSL + blockIdx.x * blockDim.x + threadIdx.x;
  const int i = AWP_NGSL + blockIdx.y * blockDim.y + threadIdx.y;
  if (i > a.lo.nxt + 3 + AWP_NGSL || j > a.lo.nyt + 3 + AWP_NGSL) return;
  const float w[4] = {1.0f, (float)(2. / 3.), (float)(1. / 3.), 0.0f};
  const DmGrid &lo = a.lo, &hi = a.hi;
  const long long pl = at(lo, i, j, lo.nzt + AWP_ALIGN - 3);
  const long long pip = pl + lo.slice, pjp = pl + lo.yline, pij = pl + lo.slice + lo.yline;
  const int ih = (i - 2 - AWP_NGSL) * 3 + 2 + AWP_NGSL;
  const int jh = (j - 2 - AWP_NGSL) * 3 + 2 + AWP_NGSL;
  const long long ph = at(hi, ih, jh, AWP_ALIGN + 1);
  // field, its fine patch offset in i and j
  auto patch = [&](const float* L, float* H, int oi, int oj) {
    const float v0 = L[pl], v1 = L[pip], v2 = L[pjp], v3 = L[pij];
    const int nj = j == lo.nyt + 3 + AWP_NGSL ? 4 : 3, ni = i == lo.nxt + 3 + AWP_NGSL ? 4 : 3;
    for (int jj = 1; jj <= nj; ++jj)
      for (int ii = 1; ii <= ni; ++ii) {
        const float wa = w[ii - 1], wb = w[jj - 1], wc = w[4 - ii], wd = w[4 - jj];
        float s = __fmul_rn(__fmul_rn(v0, wa), wb);
        s = __fmaf_rn(__fmul_rn(v1, wc), wb, s);
        s = __fmaf_rn(__fmul_rn(v2, wa), wd, s);
        s = __fmaf_rn(__fmul_rn(v3, wc), wd, s);
        H[ph + (long long)(ii - 1 + oi) * hi.slice + (long long)(jj - 1 + oj) * hi.yline] = s;
      }
  };
  // one field per blockIdx.z (the nine patches of a column are independent):
  // the velocities first
  switch (blockIdx.z + (a.set == AWP_DM_STRESS ? 3 : 0)) {
    case 0: patch(lo.w1, hi.w1, 1, 0); break;
    case 1: patch(lo.u1, hi.u1, 0, 0); break;
    case 2: patch(lo.v1, hi.v1, 1, 1); break;
    case 3: patch(lo.xz, hi.xz, 0, 0); break;
    case 4: patch(lo.yz, hi.yz, 1, 1); break;
    case 5: patch(lo.xx, hi.xx, 1, 0); break;
    case 6: patch(lo.yy, hi.yy, 1, 0); break;
    case 7: patch(lo.zz, hi.zz, 1, 0); break;
    default: patch(lo.xy, hi.xy, 0, 1); break;
  }
}

// ===========================================================================
// swap3 (kernel.cu:3032-3217): tent-weighted 5 x 5 x 5 window average of the
// fine grid (WWL = 2) into the coarse grid's top two layers.
// ===========================================================================
// The tent weight is a product (3-|ii|)(3-|jj|)(3-|kk|) / 729, so a window is
// three five-point sums, one per axis: 5 + 5 + 5 terms a value where the
// reference adds 125 in one float chain (each partial sum rounded; the three
// short sums round less).  A CTA takes 4 (i) x 32 (j) coarse columns of one
// field (blockIdx.z): its fine columns' levels align+1 .. align+8 are summed
// along k as they are read (eight lanes a column: k-contiguous, sector-wide
// loads), then along j and i from shared memory.
// 300 x 300 over 100 x 100, all nine fields: 51 -> 26 us a launch against the chain of 125
// double-precision terms.
constexpr int kSwTI = 4, kSwTJ = 32;
constexpr int kSwBI = 3 * (kSwTI - 1) + 5, kSwBJ = 3 * (kSwTJ - 1) + 5;
constexpr int kSwThreads = 32 * kSwBI;  // a warp per fine row

__global__ void __launch_bounds__(kSwThreads) k_swap3(const DmPairArgs a) {
  awp_pipe::grid_start();
  __shared__ float ks[2][kSwBI][kSwBJ + 1];  // summed along k (two windows)
  __shared__ float js[2][kSwBI][kSwTJ + 1];  // ... and along j
  const DmGrid &lo = a.lo, &hi = a.hi;
  const int tid = threadIdx.x;
  const int i0 = AWP_NGSL + blockIdx.y * kSwTI, j0 = AWP_NGSL + blockIdx.x * kSwTJ;
  const int imax = lo.nxt + AWP_NGSL + 4, jmax = lo.nyt + AWP_NGSL + 4;
  const int nci = min(kSwTI, imax - i0 + 1), ncj = min(kSwTJ, jmax - j0 + 1);
  float* dst;
  const float* src;
  int kh0, nwin, di, dj;  // level-0 window at kh0 (level 1 at 6); shifted fine columns
  switch (blockIdx.z + (a.set == AWP_DM_STRESS ? 3 : 0)) {  // the velocities first
    case 0: dst = lo.u1; src = hi.u1; kh0 = 3; nwin = 2; di = 0; dj = 0; break;
    case 1: dst = lo.v1; src = hi.v1; kh0 = 3; nwin = 2; di = 1; dj = 1; break;
    case 2: dst = lo.w1; src = hi.w1; kh0 = 4; nwin = 1; di = 1; dj = 0; break;
    case 3: dst = lo.xx; src = hi.xx; kh0 = 3; nwin = 2; di = 1; dj = 0; break;
    case 4: dst = lo.yy; src = hi.yy; kh0 = 3; nwin = 2; di = 1; dj = 0; break;
    case 5: dst = lo.zz; src = hi.zz; kh0 = 3; nwin = 2; di = 1; dj = 0; break;
    case 6: dst = lo.xy; src = hi.xy; kh0 = 3; nwin = 2; di = 0; dj = 1; break;
    case 7: dst = lo.xz; src = hi.xz; kh0 = 4; nwin = 1; di = 0; dj = 0; break;
    default: dst = lo.yz; src = hi.yz; kh0 = 4; nwin = 1; di = 1; dj = 1; break;
  }
  // the window of coarse column c centres on fine column 3 (c - 2 - ngsl) + 2 + ngsl + d
  const int fi0 = (i0 - 2 - AWP_NGSL) * 3 + AWP_NGSL + di,
            fj0 = (j0 - 2 - AWP_NGSL) * 3 + AWP_NGSL + dj;
  const int nbi = 3 * (nci - 1) + 5, nbj = 3 * (ncj - 1) + 5;
  // along k: lane kk of eight holds level align+1+kk; its weights in the two
  // windows, centred on levels align + kh0 and align + 6
  {
    const int kk = tid & 7;
    auto tent = [](int d) { return (float)(3 - min(3, d < 0 ? -d : d)); };
    const float w0 = tent(kk + 1 - kh0), w1 = tent(kk + 1 - 6);
    const int warp = tid >> 5, c4 = (tid & 31) >> 3;
    const int bi = warp;
    if (bi < nbi) {
      const float* p = src + at(hi, fi0 + bi, fj0, AWP_ALIGN + 1 + kk);
      constexpr int kFly = 9;  // columns of a lane in flight (latency bound)
      for (int b0 = 0; b0 < nbj; b0 += 4 * kFly) {
        float h[kFly];
#pragma unroll
        for (int q = 0; q < kFly; ++q) {
          const int bj = b0 + 4 * q + c4;
          h[q] = bj < nbj ? p[(long long)bj * hi.yline] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < kFly; ++q) {
          const int bj = b0 + 4 * q + c4;
          // a level outside a window adds nothing to it, whatever it holds
          float s0 = w0 > 0.f ? w0 * h[q] : 0.f, s1 = w1 > 0.f ? w1 * h[q] : 0.f;
#pragma unroll
          for (int m = 4; m >= 1; m >>= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, m);
            s1 += __shfl_xor_sync(0xffffffffu, s1, m);
          }
          if (kk == 0 && bj < nbj) {
            ks[0][bi][bj] = s0;
            ks[1][bi][bj] = s1;
          }
        }
      }
    }
  }
  __syncthreads();
  for (int t = tid; t < nwin * nbi * kSwTJ; t += kSwThreads) {
    const int cj = t & (kSwTJ - 1), r = t / kSwTJ, lev = r >= nbi ? 1 : 0, bi = r - lev * nbi;
    if (cj < ncj) {
      const float* p = &ks[lev][bi][3 * cj];
      js[lev][bi][cj] = (p[0] + p[4]) + 2.f * (p[1] + p[3]) + 3.f * p[2];
    }
  }
  __syncthreads();
  for (int t = tid; t < nwin * kSwTI * kSwTJ; t += kSwThreads) {
    const int cj = t & (kSwTJ - 1), ci = (t / kSwTJ) & (kSwTI - 1), lev = t / (kSwTJ * kSwTI);
    if (ci < nci && cj < ncj) {
      const float(*p)[kSwTJ + 1] = &js[lev][3 * ci];
      const float s = (p[0][cj] + p[4][cj]) + 2.f * (p[1][cj] + p[3][cj]) + 3.f * p[2][cj];
      dst[at(lo, i0 + ci, j0 + cj, AWP_ALIGN + lo.nzt - 2 + lev)] = __fdiv_rn(s, 729.0f);
    }
  }
}

// ===========================================================================
// checkmesh (mesh.c:1404-1443)
// ===========================================================================
__global__ void k_checkmesh(const DmCheckArgs a) {
  const int j = 2 + AWP_NGSL + blockIdx.x * blockDim.x + threadIdx.x;
  const int i = 2 + AWP_NGSL + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.glo.nxt + 2 + AWP_NGSL || j >= a.glo.nyt + 2 + AWP_NGSL) return;
  const int ih = (i - 2 - AWP_NGSL) * 3 + 2 + AWP_NGSL;
  const int jh = (j - 2 - AWP_NGSL) * 3 + 3 + AWP_NGSL;
  for (int l = 0; l < 3; ++l) {
    const long long pl = at(a.glo, i, j, AWP_ALIGN + a.glo.nzt - 3 + l);
    const long long ph = at(a.ghi, ih, jh, AWP_ALIGN + 1 + 3 * l);
    for (int f = 0; f < a.nf; ++f)
      if (a.lo[f][pl] != a.hi[f][ph]) a.lo[f][pl] = a.hi[f][ph];
  }
}

inline unsigned cdiv(int a, int b) { return (unsigned)((a + b - 1) / b); }

unsigned pair_fields(const DmPairArgs& a) {
  return a.set == AWP_DM_ALL ? 9 : a.set == AWP_DM_VELOCITY ? 3 : 6;
}

}  // namespace

cudaError_t awp_launch_dvelc2(const DmVel2Args& a, cudaStream_t st) {
  const dim3 block(32, 4);
  return awp_pipe::launch_after(k_dvelc2, dim3(cdiv(a.g.nyt, 32), cdiv(a.g.nxt, 4)), block, 0, st, a);
}

cudaError_t awp_launch_dstrqc2(const DmStr2Args& a, cudaStream_t st) {
  if (a.i1 < a.i0 || a.j1 < a.j0) return cudaSuccess;
  const dim3 block(32, 4);
  return awp_pipe::launch_after(k_dstrqc2, dim3(cdiv(a.j1 - a.j0 + 1, 32), cdiv(a.i1 - a.i0 + 1, 4)), block, 0, st, a);
}

cudaError_t awp_launch_intp3d(const DmPairArgs& a, cudaStream_t st) {
  const dim3 block(32, 4);
  return awp_pipe::launch_after(k_intp3d, dim3(cdiv(a.lo.nyt + 4, 32), cdiv(a.lo.nxt + 4, 4), pair_fields(a)), block, 0, st, a);
}

cudaError_t awp_launch_swap3(const DmPairArgs& a, cudaStream_t st) {
  // columns ngsl .. n + ngsl + 4 of the coarse block
  return awp_pipe::launch_after(k_swap3, dim3(cdiv(a.lo.nyt + 5, kSwTJ), cdiv(a.lo.nxt + 5, kSwTI), pair_fields(a)), dim3(kSwThreads), 0, st, a);
}

cudaError_t awp_launch_checkmesh(const DmCheckArgs& a, cudaStream_t st) {
  const dim3 block(32, 4);
  k_checkmesh<<<dim3(cdiv(a.glo.nyt, 32), cdiv(a.glo.nxt, 4)), block, 0, st>>>(a);
  return cudaGetLastError();
}
