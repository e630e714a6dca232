// Shared device helpers of the batched small-matrix kernels (sm_100a): argument
// block, element-type traits, the bit-exact arithmetic building blocks, and copy
// helpers.
//
// Bit-exactness. Every factor element receives exactly the reference's chain of
// operations (TinySolverDx kernels.hpp): LU (kernels.hpp:91-119) a_ij <-
// fma(-l_ik, u_kj, a_ij) in increasing k with l_ik = a_ik / u_kk correctly
// rounded (Markstein-corrected reciprocal below); Cholesky as the reference's
// default simd backend compiles it (kernels.hpp:57-87: fused for n <= 16, product
// rounded before the subtraction for n >= 17, sub_mul below). The pivot search
// compares keys built from |a| so that the reference's tie-breaking (strict '>',
// first maximum wins, NaN never wins unless it sits on the diagonal position) is
// reproduced exactly (seg_argmax below).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tsdx {
namespace dev {

constexpr unsigned kFull = 0xffffffffu;

template <class T> struct KeyT;
template <> struct KeyT<double> { using U = unsigned long long; };
template <> struct KeyT<float> { using U = unsigned; };

__device__ __forceinline__ unsigned long long key_bits(double v) { return (unsigned long long)__double_as_longlong(fabs(v)); }
__device__ __forceinline__ unsigned key_bits(float v) { return __float_as_uint(fabsf(v)); }

__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// s - x*y with the product rounded first (never contracted)
__device__ __forceinline__ double sub_mul(double s, double x, double y) { return __dsub_rn(s, __dmul_rn(x, y)); }
__device__ __forceinline__ float sub_mul(float s, float x, float y) { return __fsub_rn(s, __fmul_rn(x, y)); }
__device__ __forceinline__ double div_(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float div_(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double sqrt_(double a) { return __dsqrt_rn(a); }
__device__ __forceinline__ float sqrt_(float a) { return __fsqrt_rn(a); }

// ---- correctly rounded division by a value whose reciprocal is shared -----------
// Markstein's correction step (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Develop. 34(1), 1990): with
// y = RN(1/b) and q = RN(a*y), the remainder e = a - b*q is exact (one FMA) and
// RN(q + e*y) = RN(a/b) as long as no intermediate underflows or overflows.
// A pivot step divides a whole column by one pivot, so y is computed once
// (__drcp_rn / __frcp_rn, IEEE round-to-nearest) and every quotient costs a
// multiply and two FMAs. A zero numerator is answered by q itself whenever q is
// not NaN: then y is finite, so b is neither zero nor NaN, and a*y is the zero
// with the sign of a XOR the sign of b (RN(1/b) keeps b's sign, also when it
// underflows), which is IEEE's a/b. This case is common, not rare: the rows that
// pad an order up to its kernel's tile are zero left of the diagonal block, so
// each pivot step divides zeros. Other operands outside the safe range
// (subnormals, huge values, Inf, NaN, a zero over a zero or a subnormal divisor)
// take the IEEE division. Checked bit-for-bit against __ddiv_rn / __fdiv_rn by
// tests/test_gpu_parity.py::test_markstein_division.
static __device__ __noinline__ double div_slow(double a, double b) { return __ddiv_rn(a, b); }
static __device__ __noinline__ float div_slow(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double rcp_(double b) { return __drcp_rn(b); }
__device__ __forceinline__ float rcp_(float b) { return __frcp_rn(b); }
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  const double aq = fabs(q), aa = fabs(a);
  if (!(aq >= 0x1p-960 && aq <= 0x1p+960 && aa >= 0x1p-960 && aa <= 0x1p+960)) return (a == 0.0 && q == 0.0) ? q : div_slow(a, b);
  const double e = __fma_rn(-b, q, a);
  return __fma_rn(e, y, q);
}
__device__ __forceinline__ float div_by(float a, float b, float y) {
  const float q = __fmul_rn(a, y);
  const float aq = fabsf(q), aa = fabsf(a);
  if (!(aq >= 0x1p-100f && aq <= 0x1p+100f && aa >= 0x1p-100f && aa <= 0x1p+100f)) return (a == 0.0f && q == 0.0f) ? q : div_slow(a, b);
  const float e = __fmaf_rn(-b, q, a);
  return __fmaf_rn(e, y, q);
}

__device__ __forceinline__ void named_barrier(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// ---- argmax over a lane segment: larger key wins, ties go to the smaller position.
__device__ __forceinline__ int seg_argmax(unsigned mask, unsigned long long key, int pos, unsigned long long* kout) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mhi = __reduce_max_sync(mask, hi);
  const unsigned mlo = __reduce_max_sync(mask, hi == mhi ? lo : 0u);
  const int cand = (hi == mhi && lo == mlo) ? pos : 0x7fffffff;
  *kout = ((unsigned long long)mhi << 32) | mlo;
  return __reduce_min_sync(mask, cand);
}
__device__ __forceinline__ int seg_argmax(unsigned mask, unsigned key, int pos, unsigned* kout) {
  const unsigned mk = __reduce_max_sync(mask, key);
  *kout = mk;
  return __reduce_min_sync(mask, key == mk ? pos : 0x7fffffff);
}

// ---- cp.async (LDGSTS) staging of a global byte range into padded rows --------
template <int VEC>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (VEC == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
  else if constexpr (VEC == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gmem) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <class T>
struct SolveArgs {
  T* A;            // (batch, n, n) row-major; overwritten by the factor
  T* B;            // (batch, n, ldb) row-major; columns [b0, b0 + nrhs) are solved in place
  int* piv;        // (batch, n) LU pivots, 0-based sequential (LU only)
  int* info;       // (batch) or nullptr
  long long batch;
  int n, ldb, b0, nrhs;
  const int* status;   // optional: matrices with status[m] >= 0 are skipped (no reads, no writes)
  int wf;              // 1: A <- factor and piv written (reference semantics); 0: A left untouched
};

}  // namespace dev
}  // namespace tsdx

namespace tsdx {
namespace dev {

// 16-byte shared-memory vector access (2 doubles / 4 floats).
template <class T> struct Vec16;
template <> struct Vec16<double> {
  using type = double2;
  static constexpr int n = 2;
  __device__ static __forceinline__ double get(const double2& v, int i) { return i == 0 ? v.x : v.y; }
  __device__ static __forceinline__ void set(double2& v, int i, double x) { if (i == 0) v.x = x; else v.y = x; }
};
template <> struct Vec16<float> {
  using type = float4;
  static constexpr int n = 4;
  __device__ static __forceinline__ float get(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
  __device__ static __forceinline__ void set(float4& v, int i, float x) {
    if (i == 0) v.x = x; else if (i == 1) v.y = x; else if (i == 2) v.z = x; else v.w = x;
  }
};

// ROWS rows of a row-major matrix from row r0 on, lane c's columns c + 32 s; +0 outside the
// matrix. All loads are in flight together: behind `if (r < n)` and `if (c < n)` each row
// waited for the one before (the tier prediction at order 32, 131,072 matrices 1381 -> 580
// us, the refinement at order 64, 65,536 matrices 4586 -> 2860).
template <int ROWS, int SL>
__device__ __forceinline__ void load_rows(const double* __restrict__ A, int n, int r0, int lane, double (&v)[ROWS][SL]) {
  if (r0 + ROWS <= n && n == 32 * SL) {
    const double* p = A + r0 * n + lane;
#pragma unroll
    for (int j = 0; j < ROWS; ++j)
#pragma unroll
      for (int s = 0; s < SL; ++s) v[j][s] = __ldg(p + j * n + 32 * s);
    return;
  }
#pragma unroll
  for (int j = 0; j < ROWS; ++j)
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      const int r = min(r0 + j, n - 1), c = min(lane + 32 * s, n - 1);
      v[j][s] = __ldg(A + r * n + c);
    }
#pragma unroll
  for (int j = 0; j < ROWS; ++j)
#pragma unroll
    for (int s = 0; s < SL; ++s) v[j][s] = (r0 + j < n && lane + 32 * s < n) ? v[j][s] : 0.0;
}

}  // namespace dev
}  // namespace tsdx
