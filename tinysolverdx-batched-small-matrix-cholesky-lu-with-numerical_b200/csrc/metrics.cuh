// Error metrics on the GPU: the reference's long-double ground-truth metrics
// (src/runtime.cpp:194-242) restated in double-double arithmetic, one or two warps per
// matrix, so that error reports over whole batches need no host round trip.
//
//   chol_backward_error   ||A - L L^T||_F / ||A||_F                  (runtime.cpp:194-206)
//   lu_backward_error     ||P A - L U||_F / ||A||_F, P from the pivots (runtime.cpp:208-228)
//   solve_backward_error  ||b - A x||_2 / (||A||_F ||x||_2 + ||b||_2) (runtime.cpp:230-242)
//
// Double-double (a value is an unevaluated sum hi + lo, |lo| <= ulp(hi)/2) carries
// about 106 significand bits, more than the reference's x87 long double (64), so
// the sums of products here are at least as accurate as the reference's. The
// building blocks are the published error-free transformations: TwoSum (Knuth,
// TAOCP vol. 2, 4.2.2), TwoProduct with a fused multiply-add, and the double-double
// additions of Hida, Li and Bailey ("Algorithms for quad-double precision floating point
// arithmetic", ARITH-15, 2001), in the sums of products too: with the low part a plain
// running sum instead (10 operations a product), the elements of A - L U of order 64 had
// 3.5 times the error.
//
// What bounds them: the factor metrics are FP64 arithmetic (n^3 / 3 products at 19
// operations), the solve metric reads A once. The matrix is staged in shared memory
// (cp.async, coalesced) in rows of an odd number of 16-byte units, so that a lane per row
// reads two columns at a time without bank conflicts.
#pragma once
#include <cuda_runtime.h>

#include "rows.cuh"

namespace tsdx {
namespace dev {

struct DD {
  double hi, lo;
};

__device__ __forceinline__ DD two_sum(double a, double b) {
  const double s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  const double e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
  return {s, e};
}
__device__ __forceinline__ DD fast_two_sum(double a, double b) {  // |a| >= |b|
  const double s = __dadd_rn(a, b);
  return {s, __dsub_rn(b, __dsub_rn(s, a))};
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  DD s = two_sum(a.hi, b.hi);
  const DD t = two_sum(a.lo, b.lo);
  s.lo = __dadd_rn(s.lo, t.hi);
  s = fast_two_sum(s.hi, s.lo);
  s.lo = __dadd_rn(s.lo, t.lo);
  return fast_two_sum(s.hi, s.lo);
}
// a + x y, the product taken exactly (TwoProduct). dd_add without its last renormalisation,
// which does not change the sum.
__device__ __forceinline__ DD dd_fma(DD a, double x, double y) {
  const double p = __dmul_rn(x, y);
  const DD t = two_sum(a.lo, __fma_rn(x, y, -p));
  DD s = two_sum(a.hi, p);
  s = fast_two_sum(s.hi, __dadd_rn(s.lo, t.hi));
  return {s.hi, __dadd_rn(s.lo, t.lo)};
}
__device__ __forceinline__ DD dd_sqr(DD a) {
  const double p = __dmul_rn(a.hi, a.hi);
  return fast_two_sum(p, __fma_rn(__dmul_rn(2.0, a.hi), a.lo, __fma_rn(a.hi, a.hi, -p)));
}
__device__ __forceinline__ DD dd_warp_sum(DD v) {
  for (int o = 16; o > 0; o >>= 1) {
    DD w;
    w.hi = __shfl_xor_sync(0xffffffffu, v.hi, o);
    w.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
    v = dd_add(v, w);
  }
  return v;
}
__device__ __forceinline__ double dd_sqrt(DD a) { return sqrt(__dadd_rn(a.hi, a.lo)); }

// Shared-memory row of an order-n matrix: an odd number of 16-byte units.
__host__ __device__ constexpr int met_row_bytes(int n) { return (((n + 1) / 2) | 1) * 16; }
__host__ __device__ constexpr int met_factor_bytes(int n) { return n * met_row_bytes(n) + 64 * 4 + 32; }  // + pivots, partial sums
__host__ __device__ constexpr int met_solve_bytes(int n) { return n * met_row_bytes(n) + 64 * 8 + 64; }   // + x, partial sums

// Stages an n x n matrix; a last odd column is paired with zero. Two warps take every
// other row.
template <int TW>
__device__ __forceinline__ void met_stage(unsigned char* M, const double* A, int n, int rs, int lane, int w) {
  const int rowb = n * 8;
  const char* src = reinterpret_cast<const char*>(A);
  auto rows = [&](auto vec) {
    constexpr int V = decltype(vec)::value;
    if constexpr (TW == 1) {
      walk_chunks<double, 64, 32, V>(n, lane, [&](int r, int c) { cp_async<V>(M + r * rs + c * V, src + r * rowb + c * V); });
    } else {
      const bool first = lane * V < rowb, second = V == 8 && (lane + 32) * V < rowb;
#pragma unroll 4
      for (int r = w; r < n; r += TW) {
        if (first) cp_async<V>(M + r * rs + lane * V, src + r * rowb + lane * V);
        if (second) cp_async<V>(M + r * rs + (lane + 32) * V, src + r * rowb + (lane + 32) * V);
      }
    }
  };
  if (vec_of<double>(A, n) == 16) rows(std::integral_constant<int, 16>());
  else rows(std::integral_constant<int, 8>());
  cp_async_commit();
  if (n & 1)
    for (int r = lane + 32 * w; r < n; r += 32 * TW) *reinterpret_cast<double*>(M + r * rs + rowb) = 0.0;
}

// ||b - A x|| / (||A||_F ||x|| + ||b||). A row per lane, two warps (TW) above order 32;
// sums over even and odd columns, so that four chains of additions are in flight (order
// 64, 2,000 matrices: one warp, two rows a lane 52 us, this 44).
template <int TW>
__global__ void __launch_bounds__(512, 1) solve_bwd_kernel(const double* __restrict__ A, const double* __restrict__ x,
                                                        const double* __restrict__ b, int n, long long batch,
                                                        double* out) {
  extern __shared__ __align__(16) unsigned char met_smem[];
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int unit = warp / TW, w = warp % TW, units = (blockDim.x >> 5) / TW, i = lane + 32 * w;
  const int rs = met_row_bytes(n);
  unsigned char* M = met_smem + unit * met_solve_bytes(n);
  double* xs = reinterpret_cast<double*>(M + n * rs);
  double* part = xs + 64;
  auto barrier = [&]() {
    if constexpr (TW == 1) __syncwarp();
    else named_barrier(1 + unit, 32 * TW);
  };
  const long long step = (long long)gridDim.x * units;
  for (long long m = (long long)blockIdx.x * units + unit; m < batch; m += step) {
    if (i == 0 && m + step < batch) prefetch_l2(A + (m + step) * n * n, (long long)n * n * 8);
    met_stage<TW>(M, A + m * n * n, n, rs, lane, w);
    const double xi = i < n ? x[m * n + i] : 0.0, bi = i < n ? b[m * n + i] : 0.0;
    xs[i] = xi;  // zero from n on: the partner of a last odd column
    DD num{0, 0}, fa{0, 0}, fx = dd_fma({0, 0}, xi, xi), fb = dd_fma({0, 0}, bi, bi);
    cp_async_wait<0>();
    barrier();
    if (i < n) {
      const unsigned char* row = M + i * rs;
      DD r0{bi, 0}, r1{0, 0}, f0{0, 0}, f1{0, 0};
#pragma unroll 2
      for (int j = 0; j < n; j += 2) {
        const double2 a = *reinterpret_cast<const double2*>(row + j * 8), v = *reinterpret_cast<const double2*>(xs + j);
        r0 = dd_fma(r0, a.x, -v.x);
        r1 = dd_fma(r1, a.y, -v.y);
        f0 = dd_fma(f0, a.x, a.x);
        f1 = dd_fma(f1, a.y, a.y);
      }
      num = dd_sqr(dd_add(r0, r1));
      fa = dd_add(f0, f1);
    }
    DD v[4] = {dd_warp_sum(num), dd_warp_sum(fa), dd_warp_sum(fx), dd_warp_sum(fb)};
    if (TW == 2 && i == 32) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        part[2 * q] = v[q].hi;
        part[2 * q + 1] = v[q].lo;
      }
    }
    barrier();  // the last reads of the matrix are done as well
    if (i == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (TW == 2) v[q] = dd_add(v[q], {part[2 * q], part[2 * q + 1]});
      out[m] = dd_sqrt(v[0]) / (dd_sqrt(v[1]) * dd_sqrt(v[2]) + dd_sqrt(v[3]));
    }
  }
}

// ||P A - L U||_F / ||A||_F (LU packed, unit L) or ||A - L L^T||_F / ||A||_F: the
// factor is staged in shared memory, lane i owns rows i and i + 32 of the product, two
// columns at a time. Products beyond min(i, j) enter with a zero multiplier; both rows
// share a loop over the first 32 columns of the factor, where only the first needs it.
// Orders above 32 take two warps (TW), every other pair of columns each: shared memory
// holds six matrices of order 64, and six warps leave the FP64 pipe half idle (measured
// with cheaper sums, LU of order 64 and its solve metric, 16,384 matrices: one warp and
// row at a time 2855 us, rows sharing a loop 2627, two warps 1877; with these sums LU
// alone 2670, where one warp with uncoalesced reads took 7000).
template <bool CHOL, int TW>
__global__ void __launch_bounds__(512) factor_bwd_kernel(const double* __restrict__ A, const double* __restrict__ F,
                                                         const int* __restrict__ piv, int n, long long batch,
                                                         double* out) {
  extern __shared__ __align__(16) unsigned char met_smem[];
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int unit = warp / TW, w = warp % TW, units = (blockDim.x >> 5) / TW, tid = lane + 32 * w;
  const int rs = met_row_bytes(n);
  unsigned char* M = met_smem + unit * met_factor_bytes(n);
  int* pv = reinterpret_cast<int*>(M + n * rs);
  double* part = reinterpret_cast<double*>(pv + 64);
  auto barrier = [&]() {
    if constexpr (TW == 1) __syncwarp();
    else named_barrier(1 + unit, 32 * TW);
  };
  const long long step = (long long)gridDim.x * units;
  for (long long m = (long long)blockIdx.x * units + unit; m < batch; m += step) {
    const double* a = A + m * n * n;
    if (tid == 0 && m + step < batch) {
      prefetch_l2(F + (m + step) * n * n, (long long)n * n * 8);
      prefetch_l2(A + (m + step) * n * n, (long long)n * n * 8);
    }
    met_stage<TW>(M, F + m * n * n, n, rs, lane, w);
    int src[2] = {lane, lane + 32};  // the row of A behind each row of P A
    if constexpr (!CHOL) {
      for (int k = tid; k < n; k += 32 * TW) pv[k] = piv[m * n + k];
      barrier();
      // the sequential swaps, followed backwards for every row at once
      for (int k = n - 1; k >= 0; --k) {
        const int p = pv[k];
        if (p < 0 || p >= n) continue;
#pragma unroll
        for (int s = 0; s < 2; ++s) src[s] = src[s] == k ? p : (src[s] == p ? k : src[s]);
      }
    }
    cp_async_wait<0>();
    barrier();
    DD num{0, 0}, fa{0, 0};
    const bool v16 = vec_of<double>(A, n) == 16, both = TW == 2;
    const unsigned char* row[2];
    const double* arow[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int i = lane + 32 * s;
      row[s] = M + (i < n ? i : 0) * rs;
      arow[s] = a + (i < n ? src[s] : 0) * n;
    }
    double2 an[2];  // the next two columns of A
    auto fetch = [&](int j) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (s == 1 && !both) break;
        if (v16) an[s] = __ldg(reinterpret_cast<const double2*>(arow[s] + j));
        else an[s] = make_double2(__ldg(arow[s] + j), j + 1 < n ? __ldg(arow[s] + j + 1) : 0.0);
      }
    };
    fetch(2 * w);
#pragma unroll 1
    for (int j = 2 * w; j < n; j += 2 * TW) {
      const bool two = j + 1 < n;
      DD d[2][2];  // the sums of products; then A's elements less these
      double2 av[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (s == 1 && !both) break;
        d[s][0] = d[s][1] = {0, 0};
        av[s] = an[s];
        if (lane + 32 * s < n) {
          fa = dd_fma(fa, av[s].x, av[s].x);
          if (two) fa = dd_fma(fa, av[s].y, av[s].y);
        }
      }
      if (j + 2 * TW < n) fetch(j + 2 * TW);
      // columns k, k + 1 of L against U(k, j ..) and U(k + 1, j ..): rows FROM .. of the two
      // slots, the first of them masked to k < i (k <= i for CHOL); LAST: k = j, where
      // U(j + 1, j) does not exist
      auto pair = [&](int k, auto from, auto to, auto last) {
        constexpr int FROM = decltype(from)::value, TO = decltype(to)::value;
        constexpr bool LAST = decltype(last)::value;
        double2 u0, u1;
        if constexpr (CHOL) {
          const double2 lj = *reinterpret_cast<const double2*>(M + j * rs + k * 8);
          const double2 lj1 = *reinterpret_cast<const double2*>(M + (two ? j + 1 : j) * rs + k * 8);
          u0 = make_double2(lj.x, lj1.x);
          u1 = make_double2(lj.y, lj1.y);
        } else {
          u0 = *reinterpret_cast<const double2*>(M + k * rs + j * 8);
          u1 = *reinterpret_cast<const double2*>(M + (LAST && !two ? k : k + 1) * rs + j * 8);
        }
#pragma unroll
        for (int s = FROM; s < TO; ++s) {
          const int i = lane + 32 * s;
          double2 l = *reinterpret_cast<const double2*>(row[s] + k * 8);
          if (s == FROM) {
            l.x = (CHOL ? k <= i : k < i) ? l.x : 0.0;
            l.y = (CHOL ? k < i : k + 1 < i) ? l.y : 0.0;
          }
          d[s][0] = dd_fma(d[s][0], l.x, u0.x);
          d[s][1] = dd_fma(d[s][1], l.x, u0.y);
          if constexpr (!LAST) d[s][0] = dd_fma(d[s][0], l.y, u1.x);
          d[s][1] = dd_fma(d[s][1], l.y, u1.y);
        }
      };
      using Z = std::integral_constant<int, 0>;
      using O = std::integral_constant<int, 1>;
      using T = std::integral_constant<int, 2>;
      const int low = min(j, 32);
      if (both) {
#pragma unroll 1
        for (int k = 0; k < low; k += 2) pair(k, Z(), T(), std::false_type());
#pragma unroll 2
        for (int k = 32; k < j; k += 2) pair(k, O(), T(), std::false_type());
        if (j < 32) pair(j, Z(), T(), std::true_type());
        else pair(j, O(), T(), std::true_type());
      } else {
#pragma unroll 2
        for (int k = 0; k < low; k += 2) pair(k, Z(), O(), std::false_type());
        pair(j, Z(), O(), std::true_type());
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int i = lane + 32 * s;
        if (i >= n) continue;
        if constexpr (!CHOL) {  // the unit diagonal of L
          const double2 u = *reinterpret_cast<const double2*>(row[s] + j * 8);
          d[s][0] = dd_add(d[s][0], {i <= j ? u.x : 0.0, 0.0});
          d[s][1] = dd_add(d[s][1], {i <= j + 1 ? u.y : 0.0, 0.0});
        }
        num = dd_add(num, dd_sqr(dd_add({av[s].x, 0.0}, {-d[s][0].hi, -d[s][0].lo})));
        if (two) num = dd_add(num, dd_sqr(dd_add({av[s].y, 0.0}, {-d[s][1].hi, -d[s][1].lo})));
      }
    }
    DD sn = dd_warp_sum(num), sa = dd_warp_sum(fa);
    if constexpr (TW == 2) {
      if (tid == 32) {
        part[0] = sn.hi;
        part[1] = sn.lo;
        part[2] = sa.hi;
        part[3] = sa.lo;
      }
    }
    barrier();  // the factor's last reads are done as well
    if (tid == 0) {
      if constexpr (TW == 2) {
        sn = dd_add(sn, {part[0], part[1]});
        sa = dd_add(sa, {part[2], part[3]});
      }
      out[m] = dd_sqrt(sn) / dd_sqrt(sa);
    }
  }
}

}  // namespace dev
}  // namespace tsdx
