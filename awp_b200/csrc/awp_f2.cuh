// Arithmetic on one level (float) or on two vertically adjacent levels
// (float2) with the same bits per level.
//
// sm_100a's packed FP32 instructions (add / mul / fma .f32x2) do two lanes of
// IEEE single-precision work in one issue slot.  Measured on a B200 at the
// same number of independent chains: FFMA 3.8 warp instructions per clock and
// SM, packed FFMA 2.0, so the lanes per clock stay the same (36 T per second)
// and every second issue slot is freed for loads and integer work.  The
// stencil kernels issued on 52-76 % of the cycles before and are the ones
// that gain.
#pragma once

__device__ __forceinline__ unsigned long long f2_pack(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}

__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// .ftz as the build's -use_fast_math gives the scalar forms
__device__ __forceinline__ float2 vadd(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_pack(a)), "l"(f2_pack(b)));
  return f2_unpack(r);
}
__device__ __forceinline__ float2 vmul(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_pack(a)), "l"(f2_pack(b)));
  return f2_unpack(r);
}
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(f2_pack(a)), "l"(f2_pack(b)), "l"(f2_pack(c)));
  return f2_unpack(r);
}
// a - b as one packed instruction: fma(b, -1, a) rounds a - b once, as a
// subtraction does
__device__ __forceinline__ float2 vsub(float2 a, float2 b) {
  return vfma(b, make_float2(-1.0f, -1.0f), a);
}

template <class V> __device__ __forceinline__ V vset(float a);
template <> __device__ __forceinline__ float vset<float>(float a) { return a; }
template <> __device__ __forceinline__ float2 vset<float2>(float a) { return make_float2(a, a); }

// s * a, s + a with a scalar
template <class V> __device__ __forceinline__ V vscale(float s, V a) { return vmul(vset<V>(s), a); }

// n / a by the hardware reciprocal (within two ulp of the correctly rounded
// quotient)
__device__ __forceinline__ float vquot(float n, float a) { return __fdividef(n, a); }
__device__ __forceinline__ float2 vquot(float n, float2 a) {
  return make_float2(__fdividef(n, a.x), __fdividef(n, a.y));
}
