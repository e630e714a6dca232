// Shared pieces of the kernels that keep a matrix in shared memory: layout, copies, and
// the back substitution of the two-warp LU kernels (blk2.cuh, blk3.cuh). The matrix and
// its right-hand sides (appended as columns) stand in padded rows. Rows never move in an
// LU: ord[k] records the physical row retired at step k and the factor is written in that
// order, which is where the reference's full-row swaps leave each row
// (TinySolverDx kernels.hpp:91-119). The forward substitution rides along as extra columns
// (the reference's chain, kernels.hpp:184-193 / 214-218); the backward substitution is
// column-oriented with reciprocal diagonals, so X agrees to rounding.
#pragma once
#include "common.cuh"

namespace tsdx {
namespace dev {

// Hint: bring [p, p + bytes) into L2 (one bulk prefetch; the range is trimmed to
// whole 16-byte units, as the instruction requires).
__device__ __forceinline__ void prefetch_l2(const void* p, long long bytes) {
  const unsigned long long a = reinterpret_cast<unsigned long long>(p);
  const unsigned long long lo = (a + 15) & ~15ull, hi = (a + bytes) & ~15ull;
  if (hi > lo)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((unsigned)(hi - lo)) : "memory");
}

// GO overrides the lanes per matrix (32: one matrix per warp for any NP).
template <class T, int NP, int NRHS, int GO = 0>
struct BlkCfg {
  static constexpr int G = GO ? GO : NP <= 4 ? 4 : NP <= 8 ? 8 : NP <= 16 ? 16 : 32;  // lanes per matrix
  static constexpr int S = 32 / G;                                          // matrices per warp
  static constexpr int MR = (NP + G - 1) / G;                               // row slots per lane
  static constexpr int PB = NP < 8 ? NP : 8;                                // panel width
  static constexpr int NC = NP + NRHS;                                      // columns incl. B
  static constexpr int CH = 8;                                              // trailing chunk
  static constexpr int NCP = (NC + CH - 1) / CH * CH;                       // row capacity
  // padded row: an odd number of 16-byte units keeps lane-private row accesses conflict-free
  static constexpr int RS = (NCP * int(sizeof(T)) + 31) / 32 * 32 + 16;
  static constexpr int MAT = NP * RS;
  static constexpr int AUX = 2 * NP * 4;  // ord[NP], piv[NP]
  static constexpr int SEGB = (MAT + AUX + 127) / 128 * 128;
  static constexpr int WARPB = S * SEGB;
  static_assert(NP % PB == 0, "panel width divides the padded order");
  static_assert(MR <= 4, "at most four row slots per lane");
};

// One matrix for one segment. Every pointer may be null when the job is not live.
template <class T>
struct MatJob {
  const T* A;   // n x n row-major input
  T* Aout;      // where the factor goes (nullptr: not written)
  T* B;         // n x ldb right-hand sides, columns [b0, b0 + nrhs) solved in place
  int* piv;     // n pivots (LU) or nullptr
  int* info;    // one info word or nullptr
  int n, ldb, b0, nrhs;
  bool live;
};

struct Seg {
  int lane, lsl, segbase;
  unsigned zrow;  // shared address of a row of zeros (rows.cuh)
};

// Widest copy chunk that keeps every row start aligned.
template <class T> __device__ __forceinline__ int vec_of(const void* p, int n) {
  const unsigned long long a = reinterpret_cast<unsigned long long>(p);
  const int row = n * int(sizeof(T));
  if (row % 16 == 0 && a % 16 == 0) return 16;
  if (row % 8 == 0 && a % 8 == 0) return 8;
  return 4;
}

template <class T, int G, int RS>
__device__ __forceinline__ void seg_copy_in(unsigned char* M, const T* A, int n, int lsl) {
  const int vec = vec_of<T>(A, n);
  const int rc = n * int(sizeof(T)) / vec;
  const char* g = reinterpret_cast<const char*>(A);
  for (int r = 0; r < n; ++r) {
    const char* gr = g + (long long)r * n * int(sizeof(T));
    unsigned char* sr = M + r * RS;
    for (int c = lsl; c < rc; c += G) {
      if (vec == 16) cp_async<16>(sr + c * 16, gr + c * 16);
      else if (vec == 8) cp_async<8>(sr + c * 8, gr + c * 8);
      else cp_async<4>(sr + c * 4, gr + c * 4);
    }
  }
  cp_async_commit();
}

// Copies n rows out of shared memory: output row k <- shared row src[k] (or k).
template <class T, int G, int RS>
__device__ __forceinline__ void seg_copy_out(const unsigned char* M, T* A, int n, int lsl, const int* src) {
  const int vec = vec_of<T>(A, n);
  const int rc = n * int(sizeof(T)) / vec;
  char* g = reinterpret_cast<char*>(A);
  if (vec == 16 && rc <= G && G % rc == 0) {
    // one 16-byte chunk per lane and row, G / rc rows per pass; the passes are
    // independent, so unrolled they keep several loads in flight
    const int rpp = G / rc, c = lsl % rc;
#pragma unroll 4
    for (int k = lsl / rc; k < n; k += rpp) {
      const unsigned char* sr = M + (src ? src[k] : k) * RS;
      *reinterpret_cast<uint4*>(g + (long long)k * n * int(sizeof(T)) + c * 16) =
          *reinterpret_cast<const uint4*>(sr + c * 16);
    }
    return;
  }
  for (int k = 0; k < n; ++k) {
    const unsigned char* sr = M + (src ? src[k] : k) * RS;
    char* gr = g + (long long)k * n * int(sizeof(T));
    for (int c = lsl; c < rc; c += G) {
      if (vec == 16) *reinterpret_cast<uint4*>(gr + c * 16) = *reinterpret_cast<const uint4*>(sr + c * 16);
      else if (vec == 8) *reinterpret_cast<uint2*>(gr + c * 8) = *reinterpret_cast<const uint2*>(sr + c * 8);
      else *reinterpret_cast<unsigned*>(gr + c * 4) = *reinterpret_cast<const unsigned*>(sr + c * 4);
    }
  }
}

// y <- fma(-u, x, y) when p, else y unchanged: one predicated FMA (no select).
__device__ __forceinline__ void fma_if(double& y, bool p, double u, double x) {
  asm("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q fma.rn.f64 %0, %2, %3, %0;\n}"
      : "+d"(y)
      : "r"((int)p), "d"(-u), "d"(x));
}
__device__ __forceinline__ void fma_if(float& y, bool p, float u, float x) {
  asm("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q fma.rn.f32 %0, %2, %3, %0;\n}"
      : "+f"(y)
      : "r"((int)p), "f"(-u), "f"(x));
}

// Column-oriented back substitution with reciprocal diagonals; U(i,k) sits in shared row
// ord[i].
template <class T, int NP, int NRHS, int GO>
__device__ __forceinline__ void seg_backsolve(unsigned char* M, const int* ord, const MatJob<T>& j, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  constexpr int G = C::G, MR = C::MR, RS = C::RS;
  auto at = [&](int r, int c) -> T& { return *reinterpret_cast<T*>(M + r * RS + c * int(sizeof(T))); };
  T yv[MR][NRHS], dv[MR];
  const unsigned char* ubase[MR];  // this lane's rows of U
  constexpr int ustride = int(sizeof(T));
#pragma unroll
  for (int t = 0; t < MR; ++t) {
    const int i = g.lsl + G * t;
    const int ii = i < NP ? i : 0;
    const int pr = ord[ii];
    dv[t] = rcp_(at(pr, ii));
    ubase[t] = M + pr * RS;
#pragma unroll
    for (int c = 0; c < NRHS; ++c) yv[t][c] = at(pr, NP + c);
  }
  // a warp-uniform trip count (segments of one warp may hold different n); the
  // identity-padded positions >= n carry zeros and change nothing. Rows above k take
  // the update as a predicated FMA (U is read for every row; the address is inside
  // the matrix); a row's y is final after its own step, so each row forms its
  // x = y * RN(1/u_ii) once more at the end, the product that was broadcast.
#pragma unroll 4
  for (int k = NP - 1; k >= 0; --k) {
    const int ks = k / G, kl = g.segbase + (k & (G - 1));
    T d = dv[0];
#pragma unroll
    for (int t = 1; t < MR; ++t) d = (ks == t) ? dv[t] : d;
    T x[NRHS];
#pragma unroll
    for (int c = 0; c < NRHS; ++c) {
      T y = yv[0][c];
#pragma unroll
      for (int t = 1; t < MR; ++t) y = (ks == t) ? yv[t][c] : y;
      x[c] = __shfl_sync(kFull, y * d, kl);
    }
#pragma unroll
    for (int t = 0; t < MR; ++t) {
      const bool above = g.lsl + G * t < k;
      const T u = *reinterpret_cast<const T*>(ubase[t] + k * ustride);
#pragma unroll
      for (int c = 0; c < NRHS; ++c) fma_if(yv[t][c], above, u, x[c]);
    }
  }
  if (j.live && j.B) {
#pragma unroll
    for (int t = 0; t < MR; ++t) {
      const int i = g.lsl + G * t;
      if (i >= j.n) continue;
      T* brow = j.B + (long long)i * j.ldb + j.b0;
#pragma unroll
      for (int c = 0; c < NRHS; ++c)
        if (c < j.nrhs) brow[c] = yv[t][c] * dv[t];
    }
  }
}

}  // namespace dev
}  // namespace tsdx
