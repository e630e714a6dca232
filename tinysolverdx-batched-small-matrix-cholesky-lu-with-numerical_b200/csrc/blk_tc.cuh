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
//      order of the winners (position_of, rows.cuh);
//   2. U12: the panel's pivot rows on the trailing columns, one lane per column;
//   3. trailing update A22 -= L21 U12 on 8 x 8 tiles: tile (I, J) covers the active rows
//      8I .. 8I + 7 in physical order (gathered through a map of the rows still active)
//      and columns 8J .. 8J + 7, one m8n8k4 MMA per 4 columns of the panel (two per
//      tile).
// The back substitution runs in blocks of 8 rows on the same instruction: the block is
// solved by shuffles, then the rows above take it by tile products whose fragments count
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


// ---- 1-D bulk copies (TMA, this GPU's own memory, no multicast) on an mbarrier
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase of the given parity; false if it did not complete within
// kBulkWaitLimit polls (each poll may suspend the warp for a while).
constexpr int kBulkWaitLimit = 1 << 22;
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity) {
  for (int it = 0; it < kBulkWaitLimit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

template <int NP, int NRHS>
struct TcCfg {
  using B = BlkCfg<double, NP, NRHS, 32>;  // the one-warp row layout of blk.cuh
  static constexpr int RS = B::RS, MAT = B::MAT, MR = B::MR, NC = B::NC, NCP = B::NCP;
  static constexpr int PB = 8;
  static constexpr int NT = NP / 8 - 1;     // most row tiles below a panel
  // ord[NP] (physical row retired at each step), pmap[NP] (the active rows; before that,
  // the winners' records), then the mbarrier of the bulk loads
  static constexpr int OFF_BAR = (MAT + 2 * NP * 4 + 7) / 8 * 8;
  static constexpr int WARPB = (OFF_BAR + 8 + 15) / 16 * 16;
  static_assert(NP % 8 == 0 && NP >= 32 && NP <= 64, "one warp per matrix, two row slots at most");
  static_assert(NCP % 8 == 0, "columns in tiles of 8");
};

// Trailing update of one panel: NTI row tiles of 8 active rows (logical positions
// j1 .. NP - 1 through the position map) against the column tiles from j1 on, the
// right-hand-side tile included. A fragment (lane: tile row fr, k = fq): -l at panel
// columns k0 + fq and k0 + 4 + fq; B fragment (k = fq, column fr): the pivot rows of
// those steps (a zero-pivot step: a = -0, b = +0). NTI == 0: only the right-hand
// sides are left, and they have no active row.
template <int NP, int NRHS, int NTI, bool ZB>
__device__ __forceinline__ void tc_tiles(unsigned char* M, const int* ord, const int* pmap, unsigned zb, int k0,
                                         int lane) {
  if constexpr (NTI > 0) {
    using C = TcCfg<NP, NRHS>;
    constexpr int RS = C::RS, NCP = C::NCP;
    const int fr = lane >> 2, fq = lane & 3, j1 = k0 + 8;
    auto at = [&](int r, int c) -> double& { return *reinterpret_cast<double*>(M + r * RS + c * 8); };
    auto vat = [&](int r, int c) -> double2& { return *reinterpret_cast<double2*>(M + r * RS + c * 8); };
    const bool za = ZB && ((zb >> fq) & 1u), zc = ZB && ((zb >> (4 + fq)) & 1u);
    int prow[NTI];
    double a0[NTI], a1[NTI];
#pragma unroll
    for (int I = 0; I < NTI; ++I) {
      prow[I] = pmap[j1 + 8 * I + fr];
      a0[I] = za ? -0.0 : -at(prow[I], k0 + fq);
      a1[I] = zc ? -0.0 : -at(prow[I], k0 + 4 + fq);
    }
    const int ua = ord[k0 + fq], uc = ord[k0 + 4 + fq];
    for (int J = j1 / 8; J < NCP / 8; ++J) {
      const double b0 = za ? 0.0 : at(ua, 8 * J + fr);
      const double b1 = zc ? 0.0 : at(uc, 8 * J + fr);
      double2 c[NTI];
#pragma unroll
      for (int I = 0; I < NTI; ++I) c[I] = vat(prow[I], 8 * J + 2 * fq);
#pragma unroll
      for (int I = 0; I < NTI; ++I) {
        dmma_m8n8k4(c[I], a0[I], b0);
        dmma_m8n8k4(c[I], a1[I], b1);
      }
#pragma unroll
      for (int I = 0; I < NTI; ++I) vat(prow[I], 8 * J + 2 * fq) = c[I];
    }
  }
}

// U12 (the panel's pivot rows on the trailing columns, one lane per column) and the
// trailing update A22 -= L21 U12 on the tensor cores, for the panel at k0. ZB: the
// panel had a zero-pivot step, which enters both as fma(-(+0), +0, acc) == acc.
template <int NP, int NRHS, bool ZB>
__device__ __forceinline__ void tc_update(unsigned char* M, const int* ord, const int* pmap, unsigned zb, int k0,
                                          int lane) {
  using C = TcCfg<NP, NRHS>;
  using T = double;
  constexpr int PB = C::PB, NC = C::NC, RS = C::RS;
  const int j1 = k0 + PB;
  {
    int prs[PB];
#pragma unroll
    for (int i = 0; i < PB; ++i) prs[i] = ord[k0 + i] * RS;
    T l11[PB][PB];
#pragma unroll
    for (int i = 1; i < PB; ++i)
#pragma unroll
      for (int i2 = 0; i2 < i; ++i2)
        l11[i][i2] = (ZB && ((zb >> i2) & 1u)) ? 0.0 : *reinterpret_cast<const T*>(M + prs[i] + (k0 + i2) * 8);
    if (NC - j1 > 32) {
      // two columns per lane, interleaved: two independent chains
      const int jc0 = j1 + lane, jc1 = jc0 + 32;
      const bool two = jc1 < NC;
      T uz0[PB], uz1[PB];
#pragma unroll
      for (int i = 0; i < PB; ++i) {
        T* c0 = reinterpret_cast<T*>(M + prs[i] + jc0 * 8);
        T* c1 = reinterpret_cast<T*>(M + prs[i] + (two ? jc1 : jc0) * 8);
        T a0 = *c0, a1 = *c1;
#pragma unroll
        for (int i2 = 0; i2 < i; ++i2) {
          a0 = fma_(-l11[i][i2], uz0[i2], a0);
          a1 = fma_(-l11[i][i2], uz1[i2], a1);
        }
        uz0[i] = (ZB && ((zb >> i) & 1u)) ? 0.0 : a0;
        uz1[i] = (ZB && ((zb >> i) & 1u)) ? 0.0 : a1;
        if (i > 0) {
          *c0 = a0;
          if (two) *c1 = a1;
        }
      }
    } else {
      const int jc = j1 + lane;
      if (jc < NC) {
        T uz[PB];
#pragma unroll
        for (int i = 0; i < PB; ++i) {
          T* cell = reinterpret_cast<T*>(M + prs[i] + jc * 8);
          T acc = *cell;
#pragma unroll
          for (int i2 = 0; i2 < i; ++i2) acc = fma_(-l11[i][i2], uz[i2], acc);
          uz[i] = (ZB && ((zb >> i) & 1u)) ? 0.0 : acc;
          if (i > 0) *cell = acc;
        }
      }
    }
  }
  __syncwarp();
  switch ((NP - j1) / 8) {
    case 7: tc_tiles<NP, NRHS, 7, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 6: tc_tiles<NP, NRHS, 6, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 5: tc_tiles<NP, NRHS, 5, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 4: tc_tiles<NP, NRHS, 4, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 3: tc_tiles<NP, NRHS, 3, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 2: tc_tiles<NP, NRHS, 2, ZB>(M, ord, pmap, zb, k0, lane); break;
    case 1: tc_tiles<NP, NRHS, 1, ZB>(M, ord, pmap, zb, k0, lane); break;
    default: tc_tiles<NP, NRHS, 0, ZB>(M, ord, pmap, zb, k0, lane); break;
  }
  __syncwarp();
}

// Back substitution in blocks of 8 positions, from the last one down, on the right-hand
// sides that the factorization left in the augmented columns (one tile of 8 columns,
// zero past NRHS). Lane (fr, fq) holds columns 2 fq, 2 fq + 1 of position 8 I + fr of every
// block I. Step k of a block: the lanes of its row form x_k = y_k * RN(1/u_kk) and
// broadcast it, the rows above it in the block take y <- fma(-u, x_k, y); the blocks above
// take the 8 steps as two MMAs with the columns counted downwards, the same fused
// multiply-adds in the same order.
template <int NP, int NRHS>
__device__ __forceinline__ void tc_backsolve(const unsigned char* M, const int* ord, const MatJob<double>& j, int lane) {
  using C = TcCfg<NP, NRHS>;
  constexpr int RS = C::RS, NB = NP / 8;
  const int fr = lane >> 2, fq = lane & 3;
  const unsigned char* row[NB];
  double2 y[NB];
#pragma unroll
  for (int I = 0; I < NB; ++I) {
    row[I] = M + ord[8 * I + fr] * RS;
    y[I] = *reinterpret_cast<const double2*>(row[I] + (NP + 2 * fq) * 8);
  }
#pragma unroll
  for (int K = NB - 1; K >= 0; --K) {
    double u[8];
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
      const double2 v = *reinterpret_cast<const double2*>(row[K] + (8 * K + q) * 8);
      u[q] = v.x;
      u[q + 1] = v.y;
    }
    const double d = rcp_(*reinterpret_cast<const double*>(row[K] + (8 * K + fr) * 8));
#pragma unroll
    for (int q = 7; q >= 0; --q) {
      y[K].x = fr == q ? y[K].x * d : y[K].x;
      y[K].y = fr == q ? y[K].y * d : y[K].y;
      if (q == 0) continue;
      const double xx = __shfl_sync(kFull, y[K].x, 4 * q + fq), xy = __shfl_sync(kFull, y[K].y, 4 * q + fq);
      y[K].x = fr < q ? fma_(-u[q], xx, y[K].x) : y[K].x;
      y[K].y = fr < q ? fma_(-u[q], xy, y[K].y) : y[K].y;
    }
    if (K > 0) {
      // B fragments: x of rows 7 - fq and 3 - fq of the block, column fr
      const int s0 = 4 * (7 - fq) + (fr >> 1), s1 = 4 * (3 - fq) + (fr >> 1);
      const double p0 = __shfl_sync(kFull, y[K].x, s0), q0 = __shfl_sync(kFull, y[K].y, s0);
      const double p1 = __shfl_sync(kFull, y[K].x, s1), q1 = __shfl_sync(kFull, y[K].y, s1);
      const double b0 = (fr & 1) ? q0 : p0, b1 = (fr & 1) ? q1 : p1;
#pragma unroll
      for (int I = 0; I < K; ++I) {
        dmma_m8n8k4(y[I], -*reinterpret_cast<const double*>(row[I] + (8 * K + 7 - fq) * 8), b0);
        dmma_m8n8k4(y[I], -*reinterpret_cast<const double*>(row[I] + (8 * K + 3 - fq) * 8), b1);
      }
    }
  }
  if (j.live && j.B) {
#pragma unroll
    for (int I = 0; I < NB; ++I) {
      const int i = 8 * I + fr;
      if (i >= j.n) continue;
      double* brow = j.B + (long long)i * j.ldb + j.b0;
      if (2 * fq < j.nrhs) brow[2 * fq] = y[I].x;
      if (2 * fq + 1 < j.nrhs) brow[2 * fq + 1] = y[I].y;
    }
  }
}

// Returns false when the bulk load of the matrix did not complete (the matrix is then
// left unsolved with info = -1).
template <int NP, int NRHS>
__device__ __forceinline__ bool lu_tc_matrix(unsigned char* M, const MatJob<double>& j, int lane, unsigned& par) {
  using C = TcCfg<NP, NRHS>;
  using T = double;
  constexpr int MR = C::MR, PB = C::PB, NC = C::NC, NCP = C::NCP, RS = C::RS, NT = C::NT;
  int* ord = reinterpret_cast<int*>(M + C::MAT);
  int* pmap = ord + NP;
  auto at = [&](int r, int c) -> T& { return *reinterpret_cast<T*>(M + r * RS + c * 8); };
  auto vat = [&](int r, int c) -> double2& { return *reinterpret_cast<double2*>(M + r * RS + c * 8); };

  // ---- stage A and, while it lands, the right-hand sides in registers; identity
  // padding up to NP; the columns that pad the right-hand sides to a whole tile take
  // part in the MMAs and start at zero. Rows whose bytes and start are 16-byte
  // aligned arrive by one bulk copy each (TMA) on the warp's mbarrier, others by
  // per-lane cp.async: issuing 64 cp.async per lane for a 32 KB matrix stalls the
  // warp on the load/store unit for about 13k cycles on B200, the bulk copies take
  // two instructions per lane.
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(M + C::OFF_BAR);
  const int rowb = j.n * 8;
  const bool bulk = (rowb % 16 == 0) && ((reinterpret_cast<unsigned long long>(j.A) & 15) == 0);
  if (bulk) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier smem use before the async writes
    __syncwarp();
    if (lane == 0) mbar_expect_tx(bar, (unsigned)(rowb * j.n));
    __syncwarp();
    for (int r = lane; r < j.n; r += 32)
      bulk_g2s(M + r * RS, reinterpret_cast<const char*>(j.A) + (long long)r * rowb, (unsigned)rowb, bar);
  } else {
    seg_copy_in<T, 32, RS>(M, j.A, j.n, lane);
  }
  T rhs[MR][NRHS > 0 ? NRHS : 1];
#pragma unroll
  for (int s = 0; s < MR; ++s) {
    const int r = lane + 32 * s;
    const bool rowok = j.B && r < j.n;
    const T* brow = j.B + (rowok ? (long long)r * j.ldb + j.b0 : 0);
#pragma unroll
    for (int c = 0; c < NRHS; ++c) rhs[s][c] = (rowok && c < j.nrhs) ? brow[c] : T(0);
  }
  if (bulk) {
    const bool ok = mbar_wait_bounded(bar, par);
    if (!__all_sync(kFull, ok)) {
      // the load never completed: report the matrix, wait (bounded) for the copies
      // still in flight to this warp's shared memory, and stop
      if (lane == 0 && j.info) *j.info = -1;
      mbar_wait_bounded(bar, par);
      return false;
    }
    par ^= 1u;
  } else {
    cp_async_wait<0>();
  }
  __syncwarp();
#pragma unroll
  for (int s = 0; s < MR; ++s) {
    const int r = lane + 32 * s;
    if (r >= NP) continue;
    for (int c = r >= j.n ? 0 : j.n; c < NP; ++c) at(r, c) = (r == c) ? T(1) : T(0);
#pragma unroll
    for (int c = 0; c < NRHS; ++c) at(r, NP + c) = rhs[s][c];
#pragma unroll
    for (int c = NC; c < NCP; ++c) at(r, c) = 0.0;
  }
  __syncwarp();
  using D = DivRange<double>;
  unsigned act[MR];  // key mask of the lane's rows, 0 once retired
#pragma unroll
  for (int s = 0; s < MR; ++s) act[s] = lane + 32 * s < NP ? 0x7fffffffu : 0u;
  int info = 0;

  for (int k0 = 0; k0 < NP; k0 += PB) {
    // ------------------------------------------------ 1. panel in registers
    T pan[MR][PB];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s;
      const int rr = r < NP ? r : 0;
#pragma unroll
      for (int i0 = 0; i0 < PB; i0 += 2) {
        const double2 v = vat(rr, k0 + i0);
        pan[s][i0] = v.x;
        pan[s][i0 + 1] = v.y;
      }
    }
    unsigned zb = 0;
    // the winner's record (panel row, reciprocal) in the map's area, which is free until the
    // panel's map is written
    T* rec = reinterpret_cast<T*>(pmap);
    static_assert(NP * 4 >= 9 * 8, "the record fits the map");
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      const int k = k0 + i;
      unsigned key[MR], m = 0, b[MR];
      bool win[MR];
      T cand = T(1);
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        key[s] = hi_word(pan[s][i]) & act[s];
        cand = key[s] > m ? pan[s][i] : cand;
        m = max(m, key[s]);
      }
      m = __reduce_max_sync(kFull, m);
      T rcand = rcp_in_range(cand);  // of this lane's candidate, while the reduction runs
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        win[s] = key[s] == m;
        b[s] = __ballot_sync(kFull, win[s]);
      }
      Seg g;
      g.lane = lane;
      g.segbase = 0;
      int wr;
      const bool one = one_row<32, MR>(b, g, wr);
      bool zero = false;
      // rare, by the whole warp: a tie, or a column whose largest entry is zero, tiny,
      // huge, infinite or NaN
      const bool odd = !one || m - D::kLo > D::kHi - D::kLo;
      if (odd) {
        Candidates<T, MR> c;
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          c.v[s] = pan[s][i];
          c.act[s] = act[s];
        }
        const Choice w = exact_pivot<T, MR, 32>(c, ord, k, lane);
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          win[s] = w.slot == s;
          cand = win[s] ? pan[s][i] : cand;
        }
        wr = w.row;
        zero = w.zero;
        rcand = rcp_(cand);
      }
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        if (win[s]) {
#pragma unroll
          for (int jj = i & ~1; jj < PB; jj += 2)
            *reinterpret_cast<double2*>(rec + jj) = make_double2(pan[s][jj], pan[s][jj + 1]);
          rec[8] = rcand;
          ord[k] = wr;
          act[s] = 0u;
        }
      }
      __syncwarp();
      T uw[PB];
#pragma unroll
      for (int jj = i & ~1; jj < PB; jj += 2) {
        const double2 v = *reinterpret_cast<const double2*>(rec + jj);
        uw[jj] = v.x;
        uw[jj + 1] = v.y;
      }
      const T ry = rec[8];
      __syncwarp();  // all reads done before the next step's record
      if (zero) {
        info = info == 0 ? k + 1 : info;
        zb |= 1u << i;
      } else {
        // l = a / pivot by the shared reciprocal with Markstein's correction; operands
        // outside its range take the IEEE division on a warp-uniform rare path
        const T vpk = uw[i];
        T l[MR];
        bool slow = odd;
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          const T a = pan[s][i];
          const T q = __dmul_rn(a, ry);
          l[s] = __fma_rn(__fma_rn(-vpk, q, a), ry, q);
          slow = slow || D::outside(a, D::kLo);
        }
        if (__any_sync(kFull, slow)) {
#pragma unroll
          for (int s = 0; s < MR; ++s) l[s] = act[s] ? div_slow(pan[s][i], vpk) : T(0);
        }
        // a retired row keeps its U; the rows of this step's multipliers take the update
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          if (act[s]) {
            pan[s][i] = l[s];
#pragma unroll
            for (int jj = i + 1; jj < PB; ++jj) pan[s][jj] = fma_(-l[s], uw[jj], pan[s][jj]);
          }
        }
      }
    }
    // the panel back to its rows, and the map of the rows still active
    unsigned ab[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) ab[s] = __ballot_sync(kFull, act[s] != 0);
    int before = 0;
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s;
      if (r < NP) {
#pragma unroll
        for (int i0 = 0; i0 < PB; i0 += 2) vat(r, k0 + i0) = make_double2(pan[s][i0], pan[s][i0 + 1]);
        if (act[s]) pmap[k0 + PB + before + __popc(ab[s] & ((1u << lane) - 1u))] = r;
      }
      before += __popc(ab[s]);
    }
    __syncwarp();
    const int j1 = k0 + PB;
    if (j1 >= NC) continue;
    // ------------------------------- 2. U12 and 3. the trailing update (tensor
    // cores); a panel without a zero pivot (the common case) takes the forms without
    // the zero-pivot selects
    if (zb == 0u) tc_update<NP, NRHS, false>(M, ord, pmap, zb, k0, lane);
    else tc_update<NP, NRHS, true>(M, ord, pmap, zb, k0, lane);
  }

  if constexpr (NRHS > 0) tc_backsolve<NP, NRHS>(M, ord, j, lane);
  if (j.live) {
    if (j.piv) {
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int k = lane + 32 * s;
        if (k < j.n) j.piv[k] = position_of(ord, ord[k], k);
      }
    }
    if (lane == 0 && j.info) *j.info = info;
  }
  __syncwarp();
  if (j.live && j.Aout) seg_copy_out<T, 32, RS>(M, j.Aout, j.n, lane, ord);
  __syncwarp();
  return true;
}

// Dense batch: a persistent CTA of at most WPC warps, one matrix per warp per round.
template <int NP, int NRHS, int WPC>
__global__ void __launch_bounds__(WPC * 32, 1) tc_kernel(SolveArgs<double> p) {
  using C = TcCfg<NP, NRHS>;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31, wpc = blockDim.x >> 5;
  unsigned char* M = smem + warp * C::WARPB;
  const long long nn = (long long)p.n * p.n;
  const long long step = (long long)gridDim.x * wpc;
  if (lane == 0) mbar_init(reinterpret_cast<unsigned long long*>(M + C::OFF_BAR));
  __syncwarp();
  unsigned par = 0;  // parity of the mbarrier phase the next bulk load completes
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
    if (!lu_tc_matrix<NP, NRHS>(M, j, lane, par)) return;
  }
}

}  // namespace dev
}  // namespace tsdx
