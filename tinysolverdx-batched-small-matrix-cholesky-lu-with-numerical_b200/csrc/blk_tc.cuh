// float64 LU with partial pivoting, one warp per matrix, the trailing update on the
// FP64 tensor cores (mma.sync.m8n8k4.f64), padded orders 32..64.
//
// Layout: the matrix and its right-hand sides (appended as columns, padded to a
// multiple of 8) in shared memory, one padded row per physical row, as in blk.cuh.
// Per panel of 8 columns (k0 = 0, 8, ...):
//   1. pivot steps in registers (lane l holds rows l and l + 32): argmax of |a| by a
//      warp reduction on the high word of the key (exact tie-break only when two
//      candidates share it), the winner's remaining panel row and reciprocal published
//      in a shared-memory record, multipliers through that correctly rounded reciprocal,
//      rank-1 update of the panel. Positions are not tracked: pivots follow from the
//      order of the winners (position_of, rows.cuh). The reciprocal also stays in the
//      row's padding, for the back substitution;
//   2. U12: the panel's pivot rows on the trailing columns, one lane per column;
//   3. trailing update A22 -= L21 U12 on 8 x 8 tiles: tile (I, J) covers the active rows
//      8I .. 8I + 7 in physical order (gathered through a map of the rows still active)
//      and columns 8J .. 8J + 7, one m8n8k4 MMA per 4 columns of the panel (two per
//      tile).
// The back substitution runs in blocks of 8 rows on the same instruction: the block is
// solved in registers, then the rows above take it by tile products whose fragments count
// the columns downwards, so every element keeps the chain of a column-oriented back
// substitution.
//
// Exactness. mma.sync.m8n8k4 with float64 operands accumulates its four products in
// k order as fused multiply-adds, d = fma(a3, b3, fma(a2, b2, fma(a1, b1,
// fma(a0, b0, c)))); this was checked bit for bit against that chain on B200 over
// 4.2 million elements of wide dynamic range (and matches no other order). With
// a = -l_ik and b = u_kj the two MMAs of a tile apply the reference's chain
// a_ij <- fma(-l_ik, u_kj, a_ij) for k = k0 .. k0 + 7 in increasing order
// (TinySolverDx kernels.hpp:111-116), so factors, pivots and info stay
// bit-identical to the CPU backends. A zero-pivot step enters as a = -0, b = +0,
// and fma(-0, +0, c) = c for every c, which is the reference's skipped column.
#pragma once
#include "rows.cuh"

namespace tsdx {
namespace dev {

// not volatile: the MMA has no effect beyond its outputs, so independent tiles may
// be interleaved by the scheduler
__device__ __forceinline__ void dmma_m8n8k4(double2& c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c.x), "+d"(c.y)
      : "d"(a), "d"(b));
}

template <int NP, int NRHS>
struct TcCfg {
  using B = BlkCfg<double, NP, NRHS, 32>;  // the row layout of blk.cuh
  static constexpr int RS = B::RS, MAT = B::MAT, NC = B::NC, NCP = B::NCP;
  static constexpr int PB = 8;
  static constexpr int MR = B::MR;       // rows per lane
  static constexpr int OFF_RCP = RS - 8;      // in every row's padding: the reciprocal of its pivot
  // ord[NP] (physical row retired at each step); pmap[NP] (the active rows), where the
  // pivot steps keep the winner's record {8 panel columns, reciprocal, row}, two in turns
  static constexpr int REC = 80;
  static constexpr int OFF_ORD = MAT, OFF_MAP = MAT + NP * 4;
  static constexpr int WARPB = OFF_MAP + (2 * REC > NP * 4 ? 2 * REC : NP * 4);
  static_assert(NP % 8 == 0 && NP >= 32 && NP <= 64, "one warp per matrix, two row slots at most");
  static_assert(NCP % 8 == 0 && RS >= NCP * 8 + 8 && MAT % 16 == 0, "columns in tiles of 8");
};

// Column tile J of the trailing update, or J and J + 1:
// every load before the products, every store after them.
template <int NCT, int NTI, int RS>
__device__ __forceinline__ void tc_tile_cols(unsigned char* M, const int (&prow)[NTI], const double (&a0)[NTI],
                                             const double (&a1)[NTI], bool za, bool zc, int ua, int uc, int J, int lane) {
  const int fr = lane >> 2, fq = lane & 3;
  double b0[NCT], b1[NCT];
  double2 c[NCT][NTI];
#pragma unroll
  for (int t = 0; t < NCT; ++t) {
    b0[t] = za ? 0.0 : *reinterpret_cast<const double*>(M + ua + (8 * (J + t) + fr) * 8);
    b1[t] = zc ? 0.0 : *reinterpret_cast<const double*>(M + uc + (8 * (J + t) + fr) * 8);
#pragma unroll
    for (int I = 0; I < NTI; ++I) c[t][I] = *reinterpret_cast<const double2*>(M + prow[I] + (8 * (J + t) + 2 * fq) * 8);
  }
#pragma unroll
  for (int t = 0; t < NCT; ++t)
#pragma unroll
    for (int I = 0; I < NTI; ++I) dmma_m8n8k4(c[t][I], a0[I], b0[t]);
#pragma unroll
  for (int t = 0; t < NCT; ++t)
#pragma unroll
    for (int I = 0; I < NTI; ++I) dmma_m8n8k4(c[t][I], a1[I], b1[t]);
#pragma unroll
  for (int t = 0; t < NCT; ++t)
#pragma unroll
    for (int I = 0; I < NTI; ++I) *reinterpret_cast<double2*>(M + prow[I] + (8 * (J + t) + 2 * fq) * 8) = c[t][I];
}

// Trailing update of one panel: NTI row tiles of 8 active rows (logical positions
// j1 .. NP - 1 through the position map) against the column tiles from j1 on, the
// right-hand-side tile included. A fragment (lane: tile row fr,
// k = fq): -l at panel columns k0 + fq and k0 + 4 + fq; B fragment (k = fq, column fr):
// the pivot rows of those steps (a zero-pivot step: a = -0, b = +0).
template <int NP, int NRHS, int NTI, bool ZB>
__device__ __forceinline__ void tc_tiles(unsigned char* M, const int* ord, const int* pmap, unsigned zb, int k0,
                                         int lane) {
  using C = TcCfg<NP, NRHS>;
  constexpr int RS = C::RS, NCP = C::NCP;
  const int fr = lane >> 2, fq = lane & 3, j1 = k0 + 8;
  const bool za = ZB && ((zb >> fq) & 1u), zc = ZB && ((zb >> (4 + fq)) & 1u);
  int prow[NTI];
  double a0[NTI], a1[NTI];
#pragma unroll
  for (int I = 0; I < NTI; ++I) prow[I] = pmap[j1 + 8 * I + fr] * RS;
  const int ua = ord[k0 + fq] * RS, uc = ord[k0 + 4 + fq] * RS;
#pragma unroll
  for (int I = 0; I < NTI; ++I) {
    const double x = *reinterpret_cast<const double*>(M + prow[I] + (k0 + fq) * 8);
    const double y = *reinterpret_cast<const double*>(M + prow[I] + (k0 + 4 + fq) * 8);
    a0[I] = za ? -0.0 : -x;
    a1[I] = zc ? -0.0 : -y;
  }
  int J = j1 / 8;
#pragma unroll 1
  for (; J + 1 < NCP / 8; J += 2) tc_tile_cols<2, NTI, RS>(M, prow, a0, a1, za, zc, ua, uc, J, lane);
  if (J < NCP / 8) tc_tile_cols<1, NTI, RS>(M, prow, a0, a1, za, zc, ua, uc, J, lane);
}
template <int NP, int NRHS, bool ZB>
__device__ __forceinline__ void tc_all_tiles(unsigned char* M, const int* ord, const int* pmap, unsigned zb, int k0,
                                             int lane) {
  constexpr int MOST = NP / 8 - 1;  // row tiles below the first panel
  switch (MOST - k0 / 8) {  // 0: only right-hand sides are left, and they have no active row
    case 7: if constexpr (MOST >= 7) tc_tiles<NP, NRHS, 7, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 6: if constexpr (MOST >= 6) tc_tiles<NP, NRHS, 6, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 5: if constexpr (MOST >= 5) tc_tiles<NP, NRHS, 5, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 4: if constexpr (MOST >= 4) tc_tiles<NP, NRHS, 4, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 3: tc_tiles<NP, NRHS, 3, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 2: tc_tiles<NP, NRHS, 2, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 1: tc_tiles<NP, NRHS, 1, ZB>(M, ord, pmap, zb, k0, lane); break;
    default: break;
  }
}

// U12, a column per lane: the panel's pivot rows brought up to date by a unit-lower solve
// (ZB: the panel had a zero-pivot step, which enters as fma(-(+0), +0, acc) == acc). All
// loads first: after a store to the column the next load waited for it.
template <int NP, int NRHS, bool ZB>
__device__ __forceinline__ void tc_u12(unsigned char* M, const int* ord, unsigned zb, int k0, int lane) {
  using C = TcCfg<NP, NRHS>;
  constexpr int PB = C::PB, RS = C::RS;
  int prs[PB];
  double l[PB][PB];
#pragma unroll
  for (int i = 0; i < PB; ++i) prs[i] = ord[k0 + i] * RS;
#pragma unroll
  for (int i = 0; i < PB; ++i)
#pragma unroll
    for (int i0 = 0; i0 < i; i0 += 2) {
      const double2 v = *reinterpret_cast<const double2*>(M + prs[i] + (k0 + i0) * 8);
      l[i][i0] = -v.x;
      l[i][i0 + 1] = -v.y;
    }
#pragma unroll 1
  for (int jc = k0 + PB + lane; jc < C::NC; jc += 32) {
    double acc[PB];
#pragma unroll
    for (int i = 0; i < PB; ++i) acc[i] = *reinterpret_cast<const double*>(M + prs[i] + jc * 8);
#pragma unroll
    for (int q = 0; q < PB - 1; ++q) {
      const bool z = ZB && ((zb >> q) & 1u);
      const double u = z ? 0.0 : acc[q];
#pragma unroll
      for (int i = q + 1; i < PB; ++i) acc[i] = fma_(z ? -0.0 : l[i][q], u, acc[i]);
    }
#pragma unroll
    for (int i = 1; i < PB; ++i) *reinterpret_cast<double*>(M + prs[i] + jc * 8) = acc[i];
  }
}

// Back substitution in blocks of 8 positions, from the last one down, on the
// right-hand sides that the factorization left in the augmented columns (a tile of 8,
// zero past NRHS), transposed: lane (fr, fq) holds right-hand side fr of positions 8 I +
// 2 fq, 2 fq + 1 of every block I. The four lanes of a right-hand side gather its 8 values
// and each solves the block, x_k = y_k * RN(1/u_kk) and y <- fma(-u, x_k, y) upwards, in
// registers; the blocks above take the 8 steps as two MMAs with the columns counted
// downwards, the same fused multiply-adds in the same order. One exchange per block:
// with one per position (the right-hand sides along the lanes) order 64 took 15,000
// cycles of a matrix's 64,000.
template <int NP, int NRHS>
__device__ __forceinline__ void tc_backsolve(const unsigned char* M, const int* ord, const MatJob<double>& j, int lane) {
  using C = TcCfg<NP, NRHS>;
  constexpr int RS = C::RS, NB = NP / 8;
  const int fr = lane >> 2, fq = lane & 3;
  auto ld = [&](int off) { return *reinterpret_cast<const double*>(M + off); };
  int row[NB];
  double2 y[NB];
#pragma unroll
  for (int I = 0; I < NB; ++I) {
    row[I] = ord[8 * I + fr] * RS;
    const int2 o = *reinterpret_cast<const int2*>(ord + 8 * I + 2 * fq);
    y[I] = make_double2(ld(o.x * RS + (NP + fr) * 8), ld(o.y * RS + (NP + fr) * 8));
  }
#pragma unroll
  for (int K = NB - 1; K >= 0; --K) {
    int br[8];
    {
      const int4 a = *reinterpret_cast<const int4*>(ord + 8 * K), b = *reinterpret_cast<const int4*>(ord + 8 * K + 4);
      const int o[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int p = 0; p < 8; ++p) br[p] = o[p] * RS;
    }
    double u[8][8], d[8], x[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      d[p] = ld(br[p] + C::OFF_RCP);
#pragma unroll
      for (int q = (p + 1) & ~1; q < 8; q += 2) {
        const double2 v = *reinterpret_cast<const double2*>(M + br[p] + (8 * K + q) * 8);
        u[p][q] = v.x;
        u[p][q + 1] = v.y;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[2 * q] = __shfl_sync(kFull, y[K].x, (lane & ~3) | q);
      x[2 * q + 1] = __shfl_sync(kFull, y[K].y, (lane & ~3) | q);
    }
#pragma unroll
    for (int q = 7; q >= 0; --q) {
      x[q] = x[q] * d[q];
#pragma unroll
      for (int p = q - 1; p >= 0; --p) x[p] = fma_(-u[p][q], x[q], x[p]);
    }
    // A fragments: right-hand side fr, positions 7 - fq and 3 - fq of the block
    const double a0 = (fq & 2) ? ((fq & 1) ? x[4] : x[5]) : ((fq & 1) ? x[6] : x[7]);
    const double a1 = (fq & 2) ? ((fq & 1) ? x[0] : x[1]) : ((fq & 1) ? x[2] : x[3]);
#pragma unroll
    for (int I = K - 1; I >= 0; --I) {
      dmma_m8n8k4(y[I], a0, -ld(row[I] + (8 * K + 7 - fq) * 8));
      dmma_m8n8k4(y[I], a1, -ld(row[I] + (8 * K + 3 - fq) * 8));
    }
    if (j.B && fr < j.nrhs) {
      double* out = j.B + (long long)(8 * K + 7 - fq) * j.ldb + j.b0 + fr;
      if (8 * K + 7 - fq < j.n) out[0] = a0;
      if (8 * K + 3 - fq < j.n) out[-4ll * j.ldb] = a1;
    }
  }
}

// The rows of the factor in pivot order, one chunk per lane and row (two where 8-byte
// chunks leave some over), four rows at a time: 9 instructions a row instead of 14.
template <int NP, int RS, int V>
__device__ __forceinline__ void tc_copy_rows(const unsigned char* M, char* g, int n, int lane, const int* ord) {
  using U = typename std::conditional<V == 16, uint4, uint2>::type;
  constexpr int S = (NP * 8 / V + 31) / 32;
  const int rowb = n * 8;
  const bool first = lane * V < rowb, second = S > 1 && (lane + 32) * V < rowb;
  M += first ? lane * V : 0;
  g += lane * V;
#pragma unroll 2
  for (int k = 0; k < n; k += 4) {
    const int4 o = *reinterpret_cast<const int4*>(ord + k);
    const int r[4] = {o.x, o.y, o.z, o.w};
    U a[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = *reinterpret_cast<const U*>(M + r[q] * RS);
      if (S > 1 && second) b[q] = *reinterpret_cast<const U*>(M + r[q] * RS + 32 * V);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q, g += rowb)
      if (k + q < n) {
        if (first) *reinterpret_cast<U*>(g) = a[q];
        if (S > 1 && second) *reinterpret_cast<U*>(g + 32 * V) = b[q];
      }
  }
}
template <int NP, int RS>
__device__ __forceinline__ void tc_copy_out(const unsigned char* M, double* A, int n, int lane, const int* ord) {
  if (vec_of<double>(A, n) == 16) tc_copy_rows<NP, RS, 16>(M, reinterpret_cast<char*>(A), n, lane, ord);
  else tc_copy_rows<NP, RS, 8>(M, reinterpret_cast<char*>(A), n, lane, ord);
}

// One matrix by a warp. A pivot step takes one reduction and one exchange: the lane that
// holds the largest key publishes {panel row, reciprocal, row} in one of two alternating
// records, and after the barrier every lane reads it. Latency bounds it, with the
// shared-memory pipe at 60% for 6 matrices of order 64 on an SM (order 64, 4 right-hand
// sides, 65,536 matrices 4137 -> 3928 us with its input copies; of a matrix alone, the
// solve and U12 21,000 -> 9,800 cycles, the pivot steps 30,000 -> 24,000). Two warps per
// matrix, a row per thread: a matrix alone 25 instead of 33 us, six 45 instead of 44 (the
// same order; 36 instead of 32 for eight of order 48), so one.
template <int NP, int NRHS>
__device__ __forceinline__ void lu_tc_matrix(unsigned char* M, const MatJob<double>& j, int lane) {
  using C = TcCfg<NP, NRHS>;
  using D = DivRange<double>;
  using T = double;
  constexpr int PB = C::PB, NC = C::NC, NCP = C::NCP, RS = C::RS, MR = C::MR, REC = C::REC;
  int* ord = reinterpret_cast<int*>(M + C::OFF_ORD);
  int* pmap = reinterpret_cast<int*>(M + C::OFF_MAP);
  auto at = [&](int r, int c) -> T& { return *reinterpret_cast<T*>(M + r * RS + c * 8); };
  auto vat = [&](int r, int c) -> double2& { return *reinterpret_cast<double2*>(M + r * RS + c * 8); };

  // ---- stage A and this lane's rows of right-hand sides; identity padding up to NP; the
  // columns that pad the right-hand sides to a whole tile take part in the MMAs and
  // start at zero
  const int n = j.n, rowb = n * 8;
  {
    const char* src = reinterpret_cast<const char*>(j.A);
    unsigned char* dst = M;
    // one chunk per lane and row, or two where 8-byte chunks leave some over
    auto rows = [&](auto vec, auto most) {
      constexpr int V = decltype(vec)::value, S = (decltype(most)::value + 31) / 32;
      src += lane * V;
      dst += lane * V;
      const bool first = lane * V < rowb, second = S > 1 && (lane + 32) * V < rowb;
#pragma unroll 8
      for (int r = 0; r < n; ++r, src += rowb, dst += RS) {
        if (first) cp_async<V>(dst, src);
        if (S > 1 && second) cp_async<V>(dst + 32 * V, src + 32 * V);
      }
    };
    if (vec_of<T>(j.A, n) == 16) rows(std::integral_constant<int, 16>(), std::integral_constant<int, NP / 2>());
    else rows(std::integral_constant<int, 8>(), std::integral_constant<int, NP>());
    cp_async_commit();
  }
  T rhs[MR][NRHS > 0 ? NRHS : 1];
#pragma unroll
  for (int s = 0; s < MR; ++s) {
    const int r = lane + 32 * s;
    const bool rowok = j.B && r < n;
    const T* brow = j.B + (rowok ? (long long)r * j.ldb + j.b0 : 0);
#pragma unroll
    for (int c = 0; c < NRHS; ++c) rhs[s][c] = (rowok && c < j.nrhs) ? brow[c] : T(0);
  }
  cp_async_wait<0>();
  __syncwarp();
  int row[MR];
  unsigned act[MR];  // key mask of this lane's rows, 0 once retired
#pragma unroll
  for (int s = 0; s < MR; ++s) {
    const int r = lane + 32 * s;
    row[s] = 32 * (s + 1) <= NP || r < NP ? r : NP - 1;
    act[s] = r < NP ? 0x7fffffffu : 0u;
    if (r >= NP) continue;
    for (int c = r >= n ? 0 : n; c < NP; ++c) at(r, c) = (r == c) ? T(1) : T(0);
#pragma unroll
    for (int c = 0; c < NRHS; ++c) at(r, NP + c) = rhs[s][c];
#pragma unroll
    for (int c = NC; c < NCP; ++c) at(r, c) = 0.0;
  }
  __syncwarp();
  int info = 0;

#pragma unroll 1
  for (int k0 = 0; k0 < NP; k0 += PB) {
    // ------------------------------------------------ 1. panel in registers
    T pan[MR][PB];
#pragma unroll
    for (int s = 0; s < MR; ++s)
#pragma unroll
      for (int i0 = 0; i0 < PB; i0 += 2) {
        const double2 v = vat(row[s], k0 + i0);
        pan[s][i0] = v.x;
        pan[s][i0 + 1] = v.y;
      }
    unsigned zb = 0;
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      const int k = k0 + i;
      unsigned char* rec = M + C::OFF_MAP + (i & 1) * REC;
      unsigned key[MR], m = 0, b = 0;
      T cand = T(1);
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        key[s] = hi_word(pan[s][i]) & act[s];
        cand = key[s] > m ? pan[s][i] : cand;
        m = max(m, key[s]);
      }
      m = __reduce_max_sync(kFull, m);
      const T rcand = rcp_in_range(cand);  // while the reduction runs
      auto publish = [&](unsigned char* to, int s, T rcp) {
#pragma unroll
        for (int jj = i & ~1; jj < PB; jj += 2) *reinterpret_cast<double2*>(to + jj * 8) = make_double2(pan[s][jj], pan[s][jj + 1]);
        *reinterpret_cast<uint4*>(to + 64) =
            make_uint4((unsigned)__double2loint(rcp), (unsigned)__double2hiint(rcp), (unsigned)row[s], 0u);
        *reinterpret_cast<T*>(M + row[s] * RS + C::OFF_RCP) = rcp;  // the last one stands: the step that retires the row
      };
      bool far = false;
      const unsigned lim = D::limit(m);
      unsigned tie = 0;
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        if (key[s] == m && act[s]) publish(rec, s, rcand);  // several on a tie: it is looked at again
        const unsigned x = __ballot_sync(kFull, key[s] == m);
        tie |= (x & (x - 1)) | (b ? x : 0u);
        b |= x;
        far |= D::outside(pan[s][i], lim);
      }
      far = __any_sync(kFull, far);
      __syncwarp();
      bool zero = false;
      // rare, by the whole warp: a tie (of high words), or a column whose largest entry is
      // tiny, huge, zero, infinite or NaN
      const bool wide = m - D::kLo > D::kHi - D::kLo;
      if ((tie != 0) | wide) {
        Candidates<T, MR> c;
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          c.v[s] = pan[s][i];
          c.act[s] = act[s];
        }
        const Choice q = exact_pivot<T, MR, 32>(c, ord, k, lane);
        zero = q.zero;
#pragma unroll
        for (int s = 0; s < MR; ++s)
          if (q.slot == s) publish(rec, s, rcp_(pan[s][i]));
        __syncwarp();
      }
      T uw[PB];
#pragma unroll
      for (int jj = i & ~1; jj < PB; jj += 2) {
        const double2 v = *reinterpret_cast<const double2*>(rec + jj * 8);
        uw[jj] = v.x;
        uw[jj + 1] = v.y;
      }
      const uint4 h = *reinterpret_cast<const uint4*>(rec + 64);
      const T ry = __hiloint2double((int)h.y, (int)h.x), vpk = uw[i];
      if (lane == 0) ord[k] = (int)h.z;
#pragma unroll
      for (int s = 0; s < MR; ++s) act[s] = (int)h.z == row[s] ? 0u : act[s];
      if (zero) {
        info = info == 0 ? k + 1 : info;
        zb |= 1u << i;
      } else {
        // l = a / pivot by the shared reciprocal with Markstein's correction; operands
        // outside its range take the IEEE division on a warp-uniform rare path
        T l[MR];
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          const T q = __dmul_rn(pan[s][i], ry);
          l[s] = __fma_rn(__fma_rn(-vpk, q, pan[s][i]), ry, q);
        }
        if (wide || far) {
#pragma unroll
          for (int s = 0; s < MR; ++s) l[s] = act[s] ? div_slow(pan[s][i], vpk) : T(0);
        }
#pragma unroll
        for (int s = 0; s < MR; ++s)
          if (act[s]) {  // a retired row keeps its U
            pan[s][i] = l[s];
#pragma unroll
            for (int jj = i + 1; jj < PB; ++jj) pan[s][jj] = fma_(-l[s], uw[jj], pan[s][jj]);
          }
      }
    }
    // the panel back to its rows, and the map of the rows still active
    unsigned ab[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      if (32 * (s + 1) <= NP || lane + 32 * s < NP) {
#pragma unroll
        for (int i0 = 0; i0 < PB; i0 += 2) vat(row[s], k0 + i0) = make_double2(pan[s][i0], pan[s][i0 + 1]);
      }
      ab[s] = __ballot_sync(kFull, act[s] != 0);
    }
    __syncwarp();
    const int j1 = k0 + PB;
    if (j1 >= NC) continue;
    int before = 0;
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      if (act[s]) pmap[j1 + before + __popc(ab[s] & ((1u << lane) - 1u))] = row[s];
      before += __popc(ab[s]);
    }
    // ------------------------------- 2. U12, a column per lane, and 3. the trailing
    // update (tensor cores); a panel without a zero pivot (the common case) takes the
    // forms without the zero-pivot selects
    if (zb == 0u) tc_u12<NP, NRHS, false>(M, ord, zb, k0, lane);
    else tc_u12<NP, NRHS, true>(M, ord, zb, k0, lane);
    __syncwarp();
    if (zb == 0u) tc_all_tiles<NP, NRHS, false>(M, ord, pmap, zb, k0, lane);
    else tc_all_tiles<NP, NRHS, true>(M, ord, pmap, zb, k0, lane);
    __syncwarp();
  }

  if constexpr (NRHS > 0) tc_backsolve<NP, NRHS>(M, ord, j, lane);
  if (lane == 0 && j.info) *j.info = info;
  if (j.piv)
    for (int k = lane; k < n; k += 32) j.piv[k] = position_of(ord, ord[k], k);
  if (j.Aout) tc_copy_out<NP, RS>(M, j.Aout, n, lane, ord);
  __syncwarp();
}

// Dense batch: a persistent CTA of at most WPC warps, one matrix per warp and round.
template <int NP, int NRHS, int WPC>
__global__ void __launch_bounds__(WPC * 32, 1) tc_kernel(SolveArgs<double> p) {
  extern __shared__ __align__(128) unsigned char smem[];
  using C = TcCfg<NP, NRHS>;
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), wpc = blockDim.x >> 5, lane = threadIdx.x & 31;
  unsigned char* M = smem + warp * C::WARPB;
  const long long nn = (long long)p.n * p.n, step = (long long)gridDim.x * wpc;
  for (long long m = (long long)blockIdx.x * wpc + warp; m < p.batch; m += step) {
    if (p.status && p.status[m] >= 0) continue;  // already solved: nothing to read or write
    // this warp's next matrix heads for L2 while this one is factored
    if (lane == 0 && m + step < p.batch) {
      prefetch_l2(p.A + (m + step) * nn, nn * 8);
      if (p.B) prefetch_l2(p.B + (m + step) * (long long)p.n * p.ldb, (long long)p.n * p.ldb * 8);
    }
    MatJob<double> j;
    j.live = true;
    j.A = p.A + m * nn;
    j.Aout = p.wf ? p.A + m * nn : nullptr;
    j.B = p.B ? p.B + m * (long long)p.n * p.ldb : nullptr;
    j.piv = (p.piv && p.wf) ? p.piv + m * p.n : nullptr;
    j.info = p.info ? p.info + m : nullptr;
    j.n = p.n;
    j.ldb = p.ldb;
    j.b0 = p.b0;
    j.nrhs = p.nrhs;
    lu_tc_matrix<NP, NRHS>(M, j, lane);
  }
}

}  // namespace dev
}  // namespace tsdx
