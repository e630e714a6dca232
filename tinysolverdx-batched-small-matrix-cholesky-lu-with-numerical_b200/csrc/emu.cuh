// Emulated fp16 / bf16 factorizations and solves on the GPU: the reference's
// per-operation-rounding formats (include/tinysolverdx/precision.hpp:41-97), where every
// +, -, *, / and sqrt is computed in float and rounded to the target format with no wide
// accumulator, run by the algorithms of kernels.hpp:18-37, 91-119, 184-227 over those
// values. The reference runs these formats only on the CPU (batched.hpp:130-132); here
// backend "cuda" runs them too, bit-identical to the CPU path (NaN payloads are the
// GPU's): the rounding is the hardware's float -> binary16 / bfloat16 conversion, which
// is precision.hpp's (round to nearest even, subnormals, overflow to infinity), and each
// float operation is an explicitly rounded intrinsic so nothing is contracted.
//
// One warp per matrix, the matrix in shared memory as float (every value of the formats
// is a float). Storage in global memory is float64, float32 or (fp16 alone) binary16 bits;
// every stored value is exactly representable, so the round trip is exact. What bounds it: the
// host copies; the kernel itself is arithmetic in shared memory (one thread per matrix
// over float64 global memory, which this replaces, spent its time on uncoalesced reads).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace tsdx {
namespace dev {

template <int FMT>
struct EmuOps {
  static __device__ __forceinline__ float R(float x) {
    if constexpr (FMT == 0) return __half2float(__float2half_rn(x));
    else return __bfloat162float(__float2bfloat16_rn(x));
  }
  static __device__ __forceinline__ float sub(float a, float b) { return R(__fsub_rn(a, b)); }
  static __device__ __forceinline__ float mul(float a, float b) { return R(__fmul_rn(a, b)); }
  static __device__ __forceinline__ float div(float a, float b) { return R(__fdiv_rn(a, b)); }
  static __device__ __forceinline__ float sqrt_(float a) { return R(__fsqrt_rn(a)); }
  static __device__ __forceinline__ float in(double v) { return R(__double2float_rn(v)); }
  static __device__ __forceinline__ float in(float v) { return R(v); }
  static __device__ __forceinline__ float in(__half v) { return R(__half2float(v)); }
};
__device__ __forceinline__ void emu_out(double* p, float v) { *p = (double)v; }
__device__ __forceinline__ void emu_out(float* p, float v) { *p = v; }
__device__ __forceinline__ void emu_out(__half* p, float v) { *p = __float2half_rn(v); }

// Floats per matrix of order n in shared memory: rows of n + 1 (odd strides for even
// orders; a column read by consecutive lanes then touches different banks).
__host__ __device__ constexpr int emu_stride(int n) { return n | 1; }
__host__ __device__ constexpr int emu_factor_words(int n) { return n * emu_stride(n); }

template <int FMT, class S>
__device__ __forceinline__ void emu_load(float* M, const S* a, int n, int lane) {
  const int st = emu_stride(n);
  int r = lane / n, c = lane - r * n;
  const int dr = 32 / n, dc = 32 - dr * n;
  for (int e = lane; e < n * n; e += 32) {
    M[r * st + c] = EmuOps<FMT>::in(a[e]);
    r += dr;
    c += dc;
    if (c >= n) {
      c -= n;
      ++r;
    }
  }
  __syncwarp();
}
template <class S>
__device__ __forceinline__ void emu_store(const float* M, S* a, int n, int lane) {
  const int st = emu_stride(n);
  int r = lane / n, c = lane - r * n;
  const int dr = 32 / n, dc = 32 - dr * n;
  for (int e = lane; e < n * n; e += 32) {
    emu_out(a + e, M[r * st + c]);
    r += dr;
    c += dc;
    if (c >= n) {
      c -= n;
      ++r;
    }
  }
  __syncwarp();
}

// Row by row, as the reference: row i takes its entries j < i in increasing j, each
// updating the rest of the row. A pivot that is not positive stops there: row i keeps its
// entries j < i, the pivot and the rows after i their rounded input, and the upper
// triangle is left as it is.
template <int FMT, class S>
__global__ void __launch_bounds__(256) emu_cholesky_kernel(S* A, int n, long long batch, int* info) {
  using E = EmuOps<FMT>;
  extern __shared__ float emu_smem[];
  const int wpc = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* M = emu_smem + warp * emu_factor_words(n);
  const int st = emu_stride(n);
  for (long long m = (long long)blockIdx.x * wpc + warp; m < batch; m += (long long)gridDim.x * wpc) {
    S* a = A + m * n * n;
    emu_load<FMT, S>(M, a, n, lane);
    int inf = 0;
    for (int i = 0; i < n; ++i) {
      float* row = M + i * st;
      const int j0 = lane, j1 = lane + 32;
      float s0 = j0 <= i ? row[j0] : 0.f, s1 = j1 <= i ? row[j1] : 0.f;  // entries j0, j1 of row i
      for (int k = 0; k < i; ++k) {
        const float sk = __shfl_sync(kFull, k < 32 ? s0 : s1, k & 31);
        const float l = E::div(sk, M[k * st + k]);
        if (k < 32) s0 = j0 == k ? l : s0;
        else s1 = j1 == k ? l : s1;
        if (j0 > k && j0 < i) s0 = E::sub(s0, E::mul(l, M[j0 * st + k]));
        if (j0 == i) s0 = E::sub(s0, E::mul(l, l));
        if (j1 > k && j1 < i) s1 = E::sub(s1, E::mul(l, M[j1 * st + k]));
        if (j1 == i) s1 = E::sub(s1, E::mul(l, l));
      }
      const float d = __shfl_sync(kFull, i < 32 ? s0 : s1, i & 31);
      if (j0 < i) row[j0] = s0;
      if (j1 < i) row[j1] = s1;
      if (!(d > 0.0f)) {
        inf = i + 1;
        break;
      }
      if (lane == (i & 31)) row[i] = E::sqrt_(d);
      __syncwarp();
    }
    __syncwarp();
    if (!inf)
      for (int i = 0; i < n; ++i)
        for (int j = i + 1 + lane; j < n; j += 32) M[i * st + j] = 0.f;
    __syncwarp();
    emu_store<S>(M, a, n, lane);
    if (lane == 0 && info) info[m] = inf;
  }
}

// Right-looking with physical row swaps; lane l owns columns l and l + 32 of the update
// and rows l and l + 32 of the pivot search and the division.
template <int FMT, class S>
__global__ void __launch_bounds__(256) emu_lu_kernel(S* A, int n, long long batch, int* piv, int* info) {
  using E = EmuOps<FMT>;
  extern __shared__ float emu_smem[];
  const int wpc = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* M = emu_smem + warp * emu_factor_words(n);
  const int st = emu_stride(n);
  for (long long m = (long long)blockIdx.x * wpc + warp; m < batch; m += (long long)gridDim.x * wpc) {
    S* a = A + m * n * n;
    emu_load<FMT, S>(M, a, n, lane);
    int inf = 0;
    for (int k = 0; k < n; ++k) {
      // the first largest |a_ik|; NaN never wins unless it stands at row k
      unsigned key = 0, at = 0xffffffffu;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int i = lane + 32 * s;
        if (i < k || i >= n) continue;
        const unsigned u = __float_as_uint(M[i * st + k]) & 0x7fffffffu;
        const unsigned q = u > 0x7f800000u ? (i == k ? 0xffffffffu : 0u) : u + 1u;
        if (q > key) {
          key = q;
          at = i;
        }
      }
      const unsigned best = __reduce_max_sync(kFull, key);
      const int p = (int)__reduce_min_sync(kFull, key == best ? at : 0xffffffffu);
      if (lane == 0) piv[m * n + k] = p;
      if (p != k)
        for (int j = lane; j < n; j += 32) {
          const float t = M[k * st + j];
          M[k * st + j] = M[p * st + j];
          M[p * st + j] = t;
        }
      __syncwarp();
      const float pk = M[k * st + k];
      if (pk == 0.0f) {
        if (inf == 0) inf = k + 1;
        continue;
      }
      for (int i = k + 1 + lane; i < n; i += 32) M[i * st + k] = E::div(M[i * st + k], pk);
      __syncwarp();
      // the columns right of k, dealt to the lanes; several rows at once where few are left
      const int cols = n - k - 1;
      if (cols > 0) {
        const int per = cols >= 32 ? 1 : 32 / cols, sub = cols >= 32 ? 0 : lane / cols;
        for (int j = k + 1 + (cols >= 32 ? lane : lane - sub * cols); j < n && sub < per; j += 32) {
          const float u = M[k * st + j];
          for (int i = k + 1 + sub; i < n; i += per) M[i * st + j] = E::sub(M[i * st + j], E::mul(M[i * st + k], u));
        }
      }
      __syncwarp();
    }
    emu_store<S>(M, a, n, lane);
    if (lane == 0 && info) info[m] = inf;
  }
}

// B (n x nrhs) <- (L L^T)^{-1} B, or with LU = (P L U): one lane per right-hand side,
// the factor (rounded on entry) in shared memory. The sums run in increasing k in both
// directions, as the reference's.
template <int FMT, bool LU, class S>
__global__ void __launch_bounds__(256) emu_solve_kernel(const S* F, const int* piv, int n, long long batch, S* B, int nrhs) {
  using E = EmuOps<FMT>;
  extern __shared__ float emu_smem[];
  const int wpc = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* M = emu_smem + warp * (emu_factor_words(n) + n * 32);
  float* b = M + emu_factor_words(n) + lane;  // this lane's column, a stride of 32
  const int st = emu_stride(n);
  for (long long m = (long long)blockIdx.x * wpc + warp; m < batch; m += (long long)gridDim.x * wpc) {
    emu_load<FMT, S>(M, F + m * n * n, n, lane);
    for (int c0 = 0; c0 < nrhs; c0 += 32) {
      const int c = c0 + lane;
      if (c < nrhs) {
        S* bg = B + m * (long long)n * nrhs + c;
        for (int i = 0; i < n; ++i) b[i * 32] = E::in(bg[(long long)i * nrhs]);
        if (LU) {
          const int* pv = piv + m * n;
          for (int k = 0; k < n; ++k) {
            const int p = pv[k];
            if (p != k && p >= 0 && p < n) {
              const float t = b[k * 32];
              b[k * 32] = b[p * 32];
              b[p * 32] = t;
            }
          }
        }
        for (int i = 0; i < n; ++i) {
          float s = b[i * 32];
#pragma unroll 4
          for (int k = 0; k < i; ++k) s = E::sub(s, E::mul(M[i * st + k], b[k * 32]));
          b[i * 32] = LU ? s : E::div(s, M[i * st + i]);
        }
        for (int i = n - 1; i >= 0; --i) {
          float s = b[i * 32];
#pragma unroll 4
          for (int k = i + 1; k < n; ++k) s = E::sub(s, E::mul(LU ? M[i * st + k] : M[k * st + i], b[k * 32]));
          b[i * 32] = E::div(s, M[i * st + i]);
        }
        for (int i = 0; i < n; ++i) emu_out(bg + (long long)i * nrhs, b[i * 32]);
      }
    }
    __syncwarp();
  }
}

}  // namespace dev
}  // namespace tsdx
