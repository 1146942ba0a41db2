// Device helpers shared by the two solver kernels (cg2d_solver.cu, cg2d_team.cu): the solver's arithmetic, its
// row-sum butterflies and small memory operations.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "cg2d_internal.cuh"

namespace cg2d {

// ------------------------------------------------------------------------------------------------
// arithmetic without contraction (the reference rounds every product and every sum)

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }

// apply_operator (cg2d.py:181-188): aW(i)x(i-1) + aW(i+1)x(i+1) + aS(j)x(j-1) + aS(j+1)x(j+1) + aC x
template <class T>
__device__ __forceinline__ T op_A(T aw, T ae, T as, T an, T ac, T vw, T ve, T vs, T vn, T vc) {
  T t = mul(aw, vw);
  t = add(t, mul(ae, ve));
  t = add(t, mul(as, vs));
  t = add(t, mul(an, vn));
  t = add(t, mul(ac, vc));
  return t;
}

// apply_preconditioner (cg2d.py:191-198): pC r + pW(i)r(i-1) + pW(i+1)r(i+1) + pS(j)r(j-1) + pS(j+1)r(j+1)
template <class T>
__device__ __forceinline__ T op_M(T pc, T pw, T pe, T ps, T pn, T vc, T vw, T ve, T vs, T vn) {
  T t = mul(pc, vc);
  t = add(t, mul(pw, vw));
  t = add(t, mul(pe, ve));
  t = add(t, mul(ps, vs));
  t = add(t, mul(pn, vn));
  return t;
}

__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ float ldcg(const float* p) { return __ldcg(p); }
__device__ __forceinline__ void stcg(double* p, double v) { __stcg(p, v); }
__device__ __forceinline__ void stcg(float* p, float v) { __stcg(p, v); }
__device__ __forceinline__ void stcg(float2* p, float2 v) { __stcg(p, v); }
__device__ __forceinline__ void stcg(double2* p, double2 v) { __stcg(p, v); }

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// where a time limit ran out: gs[2] = 1 grid-wide wait, 2 bulk-copy wait, 3 unit-count wait; gs[3] = pass << 16 | CTA
__device__ __forceinline__ void note_timeout(unsigned* gs, unsigned where, unsigned pass) {
  if (atomicCAS(&gs[1], 0u, (unsigned)CG2D_BARRIER_TIMEOUT) == 0u) {
    gs[2] = where;
    gs[3] = (pass << 16) | (blockIdx.x & 0xffffu);
  }
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// compact index -> padded index of the same point
__device__ __forceinline__ long long cmp_to_pad(const TopoDev& tp, int c) {
  const int per = tp.nj * tp.ni;
  const int t = c / per;
  const int rem = c - t * per;
  const int j = rem / tp.ni;
  const int i = rem - j * tp.ni;
  return ((long long)t * tp.npy + (j + tp.OLy)) * tp.npx + (i + tp.OLx);
}

// MIXED fuses the FP32 stencils and vector updates and the FP64 solution update; FP64 rounds every product and every sum
template <bool MIXED> struct Ar;
template <> struct Ar<false> {   // FP64: rounded product, rounded sum (no contraction)
  __device__ static __forceinline__ double madd(double a, double b, double c) { return add(mul(a, b), c); }
  __device__ static __forceinline__ double dot(double a, double b, double c) { return add(c, mul(a, b)); }
};
template <> struct Ar<true> {    // MIXED: FP32 stencils and updates fused; FP64 solution update and dots fused
  __device__ static __forceinline__ float madd(float a, float b, float c) { return __fmaf_rn(a, b, c); }
  __device__ static __forceinline__ double madd(double a, double b, double c) { return __fma_rn(a, b, c); }
  __device__ static __forceinline__ double dot(double a, double b, double c) { return __fma_rn(a, b, c); }
};

// apply_operator / apply_preconditioner with the arithmetic of Ar (same terms in the same order as op_A / op_M)
template <bool MIXED, class T>
__device__ __forceinline__ T stencil5(T c0, T c1, T c2, T c3, T c4, T v0, T v1, T v2, T v3, T v4) {
  using A = Ar<MIXED>;
  T t = mul(c0, v0);
  t = A::madd(c1, v1, t);
  t = A::madd(c2, v2, t);
  t = A::madd(c3, v3, t);
  return A::madd(c4, v4, t);
}

// both right-hand sides of an instance at once (packed FP32): each lane as the scalar operations above
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
// stencil5 (apply_operator / apply_preconditioner terms in the reference's order) on both solves
__device__ __forceinline__ float2 stencil5p(float c0, float c1, float c2, float c3, float c4, float2 v0, float2 v1,
                                           float2 v2, float2 v3, float2 v4) {
  float2 t = mul2(f2(c0), v0);
  t = fma2(f2(c1), v1, t);
  t = fma2(f2(c2), v2, t);
  t = fma2(f2(c3), v3, t);
  return fma2(f2(c4), v4, t);
}
// The row sums of a warp's lane partials: for each sum, the xor butterfly over the 32 lanes (lane l adds the
// partner l ^ o's value for o = 16, 8, 4, 2, 1). With several sums the butterflies share their first levels: at
// level o a lane keeps half of its sums and hands the other half to its partner, which keeps those (the partner of a
// lane that keeps sum q keeps q too, so every addition is the one the sum's own butterfly makes: the results are
// the same bit for bit), so that two sums cost 5 exchanges instead of 10 and four 7 instead of 20 (each exchange of
// a double is two shuffles). Sum q of 2 ends in lanes 16q..16q+15, of 4 in lanes 8q..8q+7.
__device__ __forceinline__ double xchg(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double butterfly(double v) {
  for (int o = 16; o > 0; o >>= 1) v = add(v, xchg(v, o));
  return v;
}
// two sums: the result of a in lanes 0..15, of b in lanes 16..31
__device__ __forceinline__ double butterfly2(double a, double b) {
  const bool lo = (threadIdx.x & 16) == 0;
  double v = add(lo ? a : b, xchg(lo ? b : a, 16));
  for (int o = 8; o > 0; o >>= 1) v = add(v, xchg(v, o));
  return v;
}
// four sums: the result of sum q in lanes 8q..8q+7
__device__ __forceinline__ double butterfly4(double a0, double a1, double a2, double a3) {
  const bool lo16 = (threadIdx.x & 16) == 0, lo8 = (threadIdx.x & 8) == 0;
  const double b0 = add(lo16 ? a0 : a2, xchg(lo16 ? a2 : a0, 16));
  const double b1 = add(lo16 ? a1 : a3, xchg(lo16 ? a3 : a1, 16));
  double v = add(lo8 ? b0 : b1, xchg(lo8 ? b1 : b0, 8));
  for (int o = 4; o > 0; o >>= 1) v = add(v, xchg(v, o));
  return v;
}
}  // namespace cg2d
