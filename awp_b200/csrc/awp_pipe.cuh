// Producer / consumer pipeline of the TMA kernels: a producer warp fills rings
// of shared-memory slots with cp.async.bulk.tensor copies, computing warps
// consume them plane by plane (awp_tma.cu, awp_topo_kern.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <utility>

// Poll limit the next launches give their pipeline waits (process-wide;
// awp_tma_set_spin_limit).
extern unsigned awp_pipe_spin_limit;

namespace awp_pipe {

constexpr int ND = 4;  // ring of "step done" barriers
// Poll limit of the pipeline waits: the default, and the one the drain of an
// aborted march always uses (copies already issued must land before the CTA
// releases its shared memory, whatever limit the march itself ran with).
constexpr unsigned kSpinLimit = 1u << 26;

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// One arrival per warp (by its lane 0), for all 32 lanes' reads of a step.  The
// refill is a write of the async proxy, which program order alone does not keep
// behind a lane's plain loads: every lane orders its own with a proxy fence,
// then the warp meets, then lane 0's arrival releases the slot.  (Without the
// order a plane was seen to change under its readers when another context's
// kernels shared the SM.)
__device__ __forceinline__ void warp_done(uint64_t* bar, int lane) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  asm volatile(
      "{\n .reg .pred p;\n setp.eq.s32 p, %1, 0;\n"
      " @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}\n" ::"r"(smem_u32(bar)),
      "r"(lane)
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false when the limit ran out
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity,
                                          unsigned limit = kSpinLimit) {
  for (unsigned n = 0; n < limit; ++n)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load3(void* dst, const CUtensorMap* map, uint64_t* bar,
                                          int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// Programmatic dependent launch: a kernel launched by launch_after may start
// while its predecessor in the stream drains, and must call grid_wait before it
// touches global memory; grid_go (by every CTA) lets the successor start.
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_go() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// both, for kernels with nothing to set up first
__device__ __forceinline__ void grid_start() {
  grid_go();
  grid_wait();
}

// Slot and mbarrier phase of a position that advances through a ring of DEPTH.
template <int DEPTH>
struct Cursor {
  int slot = 0;
  unsigned phase = 0;
  __device__ __forceinline__ void next() {
    if (++slot == DEPTH) {
      slot = 0;
      phase ^= 1u;
    }
  }
};

__device__ __forceinline__ float2 lds2(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
__device__ __forceinline__ float2 ldg2(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
// store a thread's two cells: one 8-byte store where both are in range
__device__ __forceinline__ void st2(float* p, float2 v, bool ax, bool ay) {
  if (ax && ay) {
    *reinterpret_cast<float2*>(p) = v;
  } else {
    if (ax) p[0] = v.x;
    if (ay) p[1] = v.y;
  }
}

// The march's shared bookkeeping: full barriers of the two stage rings (NH
// halo/media stages, NO own stages), the step-done ring of NW computing warps,
// and the producer's protocol.  Step s = 0 .. n-1 is plane ib + s.
template <int NH, int NO, int NW>
struct Pipe {
  uint64_t full_h[NH], full_o[NO > 0 ? NO : 1], done[ND];

  __device__ void init() {
    for (int q = 0; q < NH; ++q) mbar_init(full_h + q, 1);
    for (int q = 0; q < NO; ++q) mbar_init(full_o + q, 1);
    for (int q = 0; q < ND; ++q) mbar_init(done + q, NW);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }

  // One thread: issue the stages of steps 0 .. n-1, each as soon as the step
  // that last read its slots is done (stage s of a ring of N reuses what step
  // s - N read).  On a wait that runs out, wait for the copies issued.
  template <class IH, class IO>
  __device__ void produce(int n, IH&& issue_h, IO&& issue_o, int* err, unsigned spin) {
    int sh = 0, so = NO > 0 ? 0 : n;
    Cursor<NH> ch;
    Cursor<NO> co;
    for (; sh < n && sh < NH; ++sh, ch.next()) issue_h(sh, full_h + ch.slot);
    for (; so < n && so < NO; ++so, co.next()) issue_o(so, full_o + co.slot);
    Cursor<ND> cd;
    for (int s = 0; sh < n || so < n; ++s, cd.next()) {
      if (!mbar_wait(done + cd.slot, cd.phase, spin)) {
        atomicExch(err, 1);
        break;
      }
      if (sh == s + NH && sh < n) {
        issue_h(sh, full_h + ch.slot);
        ++sh;
        ch.next();
      }
      if (so == s + NO && so < n) {
        issue_o(so, full_o + co.slot);
        ++so;
        co.next();
      }
    }
    // the last stages of both rings: in an undisturbed march the consumers
    // wait for them too, after an abort nobody else does
    for (int q = sh > NH ? sh - NH : 0; q < sh; ++q)
      (void)mbar_wait(full_h + q % NH, (q / NH) & 1);
    if (NO > 0)
      for (int q = so > NO ? so - NO : 0; q < so; ++q)
        (void)mbar_wait(full_o + q % (NO > 0 ? NO : 1), (q / (NO > 0 ? NO : 1)) & 1);
  }
};

inline unsigned cdiv_u(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// Launch constants of a kernel on the current device: the shared-memory limit
// raised once, and the CTAs the device holds at a time.
struct Shape {
  std::atomic<int> resident{0};
};
constexpr int kMaxDev = 64;

inline cudaError_t resident_ctas(const void* kernel, size_t smem, int threads,
                                 Shape (&shape)[kMaxDev], int* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  int r = shape[dev].resident.load(std::memory_order_acquire);
  if (r == 0) {
    int sms = 0, per = 0;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)))
      return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem))) return e;
    r = std::max(1, sms * per);
    shape[dev].resident.store(r, std::memory_order_release);
  }
  *out = r;
  return cudaSuccess;
}

// x planes a CTA marches, at most `cap` (the tuning value).  A grid of many
// waves takes `most` (the kernel's): the CTAs in flight then stay within a few
// planes of one another, so the halos of neighbouring tiles and the planes two
// chunks share are found in L2 (k_stress_tma, 512 x 512 x 256: 1385 us at 6
// planes, 1466 at 8 and 1617 at 32 with the wider L2 promotion; the
// curvilinear kernels have a longer prologue and take 32).  A grid of few
// waves, in flight as a whole, takes the chunk with the least waves x (planes
// + fill), of equals the shortest; fill is the planes' worth of time a march
// spends before its first result, mostly hidden behind the SM's other CTAs
// (ten steps of 128 x 128 x 128, 634 us, and five of a 53 x 41 x 60 mesh, 580,
// with chunks up to six planes: 604 and 573 with longer ones, 600 and 597
// with a fill of two planes, 602 and 599 with four; 48 x 40 x 36: 34 -> 9 us
// and 60 -> 13 us for the two kernels against 32 planes throughout; kFill and
// the limit of four waves were set on these grids).
// `ctas(c)`: the grid's CTAs at chunks of c planes, ni its longest extent.
template <class F>
inline int march_planes(F ctas, int ni, int resident, int cap, int most) {
  constexpr int kFill = 1, kLeast = 4;
  cap = std::min(cap, ni);
  if (ctas(std::min(cap, most)) > 4ll * resident) return std::min(cap, most);
  int best = cap;
  long long cost = -1;
  for (int c = cap; c >= std::min(kLeast, cap); --c) {
    const long long w = (long long)cdiv_u(ctas(c), resident) * (c + kFill);
    if (cost < 0 || w <= cost) {
      cost = w;
      best = c;
    }
  }
  return best;
}
inline int march_planes(long long tiles, int ni, int resident, int cap, int most) {
  return march_planes([&](int c) { return tiles * cdiv_u(ni, c); }, ni, resident, cap, most);
}

// Launch a kernel that calls grid_wait: its start-up overlaps the tail of the
// kernel before it in the stream.  The kernels of an ordinary step are launched
// so; receivers, SOURCEFILE and FORCEFILE adds, halo copies, a batch's sources
// near the surface and the read-only-path family are plain launches (ten
// steps of a 48 x 40 x 36 shot: 206 -> 152 us; of a 240 x 237 x 120 grid with
// plasticity 1312 -> 1265 for three); with some of a step's kernels only, a
// plain launch behind an overlapped one waits longer than behind a plain one
// (128 x 128 x 128: 655 us, 696 with fstr alone overlapped).
template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                                cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  if (e != cudaSuccess) (void)cudaGetLastError();  // reported here, once
  return e;
}

}  // namespace awp_pipe
