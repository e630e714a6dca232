// Register-resident batched LU with partial pivoting and Cholesky: G lanes per
// matrix, each holding MR whole rows (right-hand sides appended as columns) in
// registers. Unblocked, right-looking, one column per step.
//
// LU step k (the winner is the physical row with the largest |a_ik|):
//   1. one reduction of the keys' high words over the segment, one ballot per row slot;
//      a single candidate wins, anything else (a tie, a zero, infinite or NaN column)
//      takes the exact comparison on a rare warp-uniform path;
//   2. the winner writes the rest of its row into the shared row that will hold the
//      result: the same store is the broadcast and the output;
//   3. every lane divides its own rows and updates them from broadcast 16-byte reads.
// Retired rows are never read again (their registers become zeros: the multiplier of a
// row over itself is 1), so nothing in the update is predicated. Multipliers go to
// shared memory once per 16 bytes of columns. Positions and pivots are not tracked in
// the loop: they follow from the order of the winners (position_of).
// Cholesky step k: the diagonal is broadcast by a shuffle; the lanes write column k of
// L into the unused upper part of shared row k, from where it is broadcast to every
// lane's update and, later, read as L^T by the back substitution.
//
// Each element receives the reference's chain of operations (see common.cuh), so
// factors, pivots and info are bit-identical to TinySolverDx's CPU backends.
#pragma once
#include <type_traits>

#include "blk.cuh"

namespace tsdx {
namespace dev {

// A row lives in registers as 64-bit units: two float32 or one float64, so that every
// unit is an aligned register pair, two of them are one 16-byte shared-memory access,
// and float32 arithmetic runs two elements to an instruction (fma.rn.f32x2; each half
// is rounded like the scalar operation).
template <class T> struct Unit;
template <> struct Unit<double> {
  using E = double;
  static constexpr int n = 1;
  __device__ static __forceinline__ double get(E v, int) { return v; }
  __device__ static __forceinline__ void set(E& v, int, double x) { v = x; }
  __device__ static __forceinline__ E dup(double x) { return x; }
  __device__ static __forceinline__ E fma(E m, E u, E c) { return __fma_rn(m, u, c); }
  __device__ static __forceinline__ E mul(E a, E b) { return __dmul_rn(a, b); }
  // c + RN(m * u): the product rounded before the addition
  __device__ static __forceinline__ E muladd(E m, E u, E c, E) { return __dadd_rn(c, __dmul_rn(m, u)); }
};
template <> struct Unit<float> {
  using E = unsigned long long;
  static constexpr int n = 2;
  __device__ static __forceinline__ E pack(float a, float b) {
    E r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
  }
  __device__ static __forceinline__ float get(E v, int i) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return i == 0 ? a : b;
  }
  __device__ static __forceinline__ void set(E& v, int i, float x) { v = i == 0 ? pack(x, get(v, 1)) : pack(get(v, 0), x); }
  __device__ static __forceinline__ E dup(float x) { return pack(x, x); }
  __device__ static __forceinline__ E fma(E m, E u, E c) {
    E d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(m), "l"(u), "l"(c));
    return d;
  }
  __device__ static __forceinline__ E mul(E a, E b) {
    E d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
  }
  __device__ static __forceinline__ E muladd(E m, E u, E c, E nz) {
    E d;
    // the product as m * u + (-0) with a -0 the compiler cannot see: mul.rn.f32x2 followed
    // by add.rn.f32x2 comes out as one fused operation (measured: results differ from
    // the separately rounded ones)
    asm("{\n .reg .b64 t;\n fma.rn.f32x2 t, %1, %2, %4;\n add.rn.f32x2 %0, %3, t;\n}"
        : "=l"(d)
        : "l"(m), "l"(u), "l"(c), "l"(nz));
    return d;
  }
};
// Shared constants of a rows kernel, at Seg::zrow: a row of zeros as long as the longest
// shared row (float64, order 64, 8 right-hand sides), then 16 bytes of float32 -0.
constexpr int kZeroRow = 592, kRowConst = kZeroRow + 16;
template <class E> struct __align__(16) Unit2 {
  E x, y;
};
// Shared-memory accesses at a 32-bit address plus a constant. Stores that not every lane
// makes stand in an ordinary branch: predicated store instructions came out several
// times as long (measured by code size: 30 more instructions in a step).
template <int OFF = 0> __device__ __forceinline__ Unit2<double> lds16(unsigned a, double) {
  Unit2<double> v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2+%3];" : "=d"(v.x), "=d"(v.y) : "r"(a), "n"(OFF) : "memory");
  return v;
}
template <int OFF = 0> __device__ __forceinline__ Unit2<unsigned long long> lds16(unsigned a, unsigned long long) {
  Unit2<unsigned long long> v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2+%3];" : "=l"(v.x), "=l"(v.y) : "r"(a), "n"(OFF) : "memory");
  return v;
}
template <int OFF = 0> __device__ __forceinline__ void sts16(unsigned a, double x, double y) {
  asm volatile("st.shared.f64 [%0+%3], %1;\n st.shared.f64 [%0+%4], %2;" ::"r"(a), "d"(x), "d"(y), "n"(OFF), "n"(OFF + 8) : "memory");
}
template <int OFF = 0> __device__ __forceinline__ void sts16(unsigned a, unsigned long long x, unsigned long long y) {
  asm volatile("st.shared.b64 [%0+%3], %1;\n st.shared.b64 [%0+%4], %2;" ::"r"(a), "l"(x), "l"(y), "n"(OFF), "n"(OFF + 8) : "memory");
}
__device__ __forceinline__ void sts(unsigned a, int x) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(x) : "memory"); }
__device__ __forceinline__ void sts(unsigned a, float x) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory"); }
__device__ __forceinline__ void sts(unsigned a, double x) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory"); }
// f(std::integral_constant<int, I>) for I = A, A + STEP, ... below B
template <int A, int B, int STEP, class F> __device__ __forceinline__ void unrolled(F&& f) {
  if constexpr (A < B) {
    f(std::integral_constant<int, A>());
    unrolled<A + STEP, B, STEP>(f);
  }
}

__device__ __forceinline__ unsigned hi_word(float v) { return __float_as_uint(v); }
__device__ __forceinline__ unsigned hi_word(double v) { return (unsigned)__double2hiint(v); }
__device__ __forceinline__ bool plain_zero(float v) { return __float_as_uint(v) == 0; }
__device__ __forceinline__ bool plain_zero(double v) { return __double_as_longlong(v) == 0; }
__device__ __forceinline__ unsigned abs_hi(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned abs_hi(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }

// RN(1/p) without a branch, for p in DivRange: from the hardware's approximation to
// within one ulp (float32 as it comes; float64 after a third-order Newton step), and
// Markstein's final step y + y (1 - p y), which rounds correctly from there unless p's
// significand is all ones (P. Markstein, IBM J. Res. Develop. 34(1), 1990). That last case
// needs the value before to be rounded up: 1/p then lies just above the middle of two
// neighbours, and the final step is right from the upper one. Checked against __frcp_rn for
// every float32 significand and against __drcp_rn for float64 ones at random and all ones,
// at exponents over the range, by tests/test_gpu_rare_paths.py::test_step_division_*.
__device__ __forceinline__ float rcp_in_range(float p) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(p));
  return __fmaf_rn(y, __fmaf_rn(-p, y, 1.0f), y);
}
__device__ __forceinline__ double rcp_in_range(double p) {
  const double a = fabs(p);
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = __fma_rn(-a, y, 1.0);
  y = __fma_ru(y, __fma_rn(e, e, e), y);
  return copysign(__fma_rn(y, __fma_rn(-a, y, 1.0), y), p);
}

// Where the shared-reciprocal division (div_by, common.cuh) of an x with |x| <= |p|
// needs no other check: no intermediate underflows and the remainder x - p q is exact,
// because ulp(p) ulp(q) >= ulp(x)^2 / 2 is still a representable number. float32: p in
// [2^-100, 2^100] and |x| >= max(2^-100, |p| 2^-120) (the quotient stays normal);
// float64: p in [2^-900, 2^900] and |x| >= max(2^-900, |p| 2^-900). A +0 numerator needs no
// check either; a -0 would lose its sign, so it counts as outside.
// Divisors are tested by the high word m of |p|, once per step. The tests are combined with
// & and |: && and || became branches (float64 LU on the tensor cores, a step of order 64
// alone on its SM 502 -> 373 cycles; float32 posv n = 45, 50,000 matrices 1056 -> 972 us, a
// mixed stream of 262,144 4323 -> 4147). Matrices scaled over 10^-250 .. 10^250 lie inside
// (float64 getrf, order 16, 34,179 of them 87 us, where p in [2^-600, 2^400] sent a third
// of them to the IEEE division and took 143; order 64, 4,096 203 and 559 us).
//
// kInf: from there on the high word belongs to an infinity or a NaN. A winner's high word
// in [1, kInf) that no other candidate shares decides the pivot, whatever the range. A tie
// needs the exact choice but no other division (integers of -1 .. 1, float32 LU of order 8:
// 26 % less time than with the IEEE division at every tie).
template <class T> struct DivRange;
template <> struct DivRange<float> {
  static constexpr unsigned kLo = (127u - 100u) << 23, kHi = (127u + 100u) << 23, kInf = 0x7f800000u;
  // the limit of |x| for a divisor m
  __device__ static __forceinline__ float limit(unsigned m) {
    return __int_as_float(__viaddmax_s32((int)m, -(120 << 23), (int)kLo));
  }
  __device__ static __forceinline__ bool outside(float x, float lim) { return (fabsf(x) < lim) & (__float_as_int(x) != 0); }
};
template <> struct DivRange<double> {
  static constexpr unsigned kLo = (1023u - 900u) << 20, kHi = (1023u + 900u) << 20, kInf = 0x7ff00000u;
  // the limit of |x|'s high word
  __device__ static __forceinline__ unsigned limit(unsigned m) {
    return (unsigned)__viaddmax_s32((int)m, -(900 << 20), (int)kLo);
  }
  __device__ static __forceinline__ bool outside(double x, unsigned lim) {
    return (((unsigned)__double2hiint(x) & 0x7fffffffu) < lim) & ((__double2hiint(x) | __double2loint(x)) != 0);
  }
};

// Maximum over the segment of G lanes, by every lane of the warp.
template <int G>
__device__ __forceinline__ unsigned seg_max(unsigned v, const Seg& g) {
  if constexpr (G == 32) {
    return __reduce_max_sync(kFull, v);
  } else if constexpr (G == 16) {
    // two full-warp reductions: a segment mask would serialise the segments
    const unsigned a = __reduce_max_sync(kFull, g.lane < 16 ? v : 0u);
    const unsigned b = __reduce_max_sync(kFull, g.lane < 16 ? 0u : v);
    return g.lane < 16 ? a : b;
  } else {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
    return v;
  }
}

template <class T, int NP, int NRHS, int GO>
struct RowCfg {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  static constexpr int UN = U::n, VN = 2 * UN;                 // elements per unit, per 16 bytes
  static constexpr int NCV = (C::NC + VN - 1) / VN * VN;       // LU columns, right-hand sides included
  // Columns held in registers at a time: the whole row up to order 16, else a panel of 8.
  // A later panel first catches up with the steps before it: the pivot rows and
  // multipliers are known, so this costs no search, and no more stores and updates than
  // updating it step by step. Whole rows above order 16 spill or leave too few warps, and
  // their fully unrolled steps do not fit the instruction cache (float32 LU, order 32, 4
  // right-hand sides, 262,144 matrices: whole rows 1576 us, unrolled panels of 8 1389).
  // Rolled panels of 8 against 16: Cholesky of order 48, 65,536 matrices, 4 right-hand sides
  // 972 and 1082 us in float32, 2122 and 2377 in float64; LU in float32 order 32, 131,072
  // 636 and 679, order 64 1877 and 1869 (without right-hand sides 1445 and 1273).
  static constexpr int PW = NP <= 16 ? NP : 8;
  static constexpr int LASTW = NCV - (NP - 1) / PW * PW;       // the last panel holds the right-hand sides
  static constexpr int RW = LASTW > PW ? LASTW : PW;
  static_assert(NP % VN == 0 && NP % PW == 0 && PW % VN == 0, "whole vectors of matrix columns, whole panels");
  static_assert(NCV * int(sizeof(T)) <= C::RS && C::RS <= kZeroRow, "the row of zeros stands in for any row");
  // A rolled loop over a panel's groups reads the vector at column k0 + Q in each of them,
  // past the panel's end in the later ones (values that are not used). in_row: for every
  // group, k0 = NP - VN included, that vector still lies in its row and its padding; else
  // the read has to be left out where it passes the panel's end.
  __host__ __device__ static constexpr bool in_row(int q) { return (NP + q) * int(sizeof(T)) <= C::RS; }
};

// The position, before step k, of a row still active: its own index, unless an earlier
// step j = index moved it to where that step's winner came from, and so on. With ord[j]
// the row retired at step j this is the first of r, ord[r], ord[ord[r]], ... at or above
// k. The pivot of step k (LAPACK's ipiv) is the position of ord[k]. A chain visits a row
// once, so it has at most k links.
__device__ __forceinline__ int position_of(const int* ord, int r, int k) {
#pragma unroll 1
  for (int t = 0; t < k && r < k; ++t) r = ord[r];
  return r;
}

// The exact pivot choice of the reference (common.cuh): the largest key wins, ties go
// to the smallest position, NaN wins only at position k. Every lane of the warp calls.
template <class T, int MR> struct Candidates {
  T v[MR];
  unsigned act[MR];
};
struct Choice {
  int slot, row, zero;  // the winner's slot on its lane (-1 elsewhere), its row, |pivot| == 0
};
template <class T, int MR, int G>
__device__ __noinline__ Choice exact_pivot(Candidates<T, MR> c, const int* ord, int k, int lsl) {
  using K = typename KeyT<T>::U;
  K bk = 0;
  int bp = 0x7fffffff, br = 0, slot = -1;
#pragma unroll
  for (int s = 0; s < MR; ++s) {
    if (!c.act[s]) continue;
    const int r = lsl + G * s, p = position_of(ord, r, k);
    const K key = isnan(c.v[s]) ? (p == k ? ~K(0) : K(0)) : key_bits(c.v[s]) + 1;
    if (key > bk || (key == bk && p < bp)) {
      bk = key;
      bp = p;
      br = r;
      slot = s;
    }
  }
  __syncwarp();
  const int mine = bp;
#pragma unroll 1
  for (int o = G / 2; o > 0; o >>= 1) {
    const K ok = __shfl_xor_sync(kFull, bk, o);
    const int op = __shfl_xor_sync(kFull, bp, o), orow = __shfl_xor_sync(kFull, br, o);
    if (ok > bk || (ok == bk && op < bp)) {
      bk = ok;
      bp = op;
      br = orow;
    }
  }
  return {mine == bp ? slot : -1, br, bk == K(1)};
}

// The rows (as a bit mask over lsl + G s) that hold the winning key; and the row of its
// lowest bit. One permute where the segment's rows are exactly 32.
template <int G, int MR>
__device__ __forceinline__ bool one_row(const unsigned (&b)[MR], const Seg& g, int& row) {
  if constexpr (G == 32 && MR == 2) {
    const unsigned x = b[0] | b[1];
    row = 31 - __clz(x) + (b[1] ? 32 : 0);
    return ((x & (x - 1)) | (b[0] ? b[1] : 0u)) == 0;
  } else if constexpr (G == 16 && MR == 2) {
    const unsigned x = __byte_perm(b[0], b[1], g.lane < 16 ? 0x5410 : 0x7632);
    row = 31 - __clz(x);
    return (x & (x - 1)) == 0;
  } else if constexpr (G * MR <= 32) {
    unsigned x = 0;
#pragma unroll
    for (int s = 0; s < MR; ++s) x |= ((b[s] >> g.segbase) & (G == 32 ? kFull : (1u << (G & 31)) - 1u)) << ((G * s) & 31);
    row = 31 - __clz(x);
    return (x & (x - 1)) == 0;
  } else {
    unsigned any = 0;
    int cnt = 0, ws = 0;
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const unsigned x = (b[s] >> g.segbase) & (G == 32 ? kFull : (1u << (G & 31)) - 1u);
      any |= x;
      cnt += __popc(x);
      if (s > 0) ws = x ? s : ws;
    }
    row = __ffs(any) - 1 + G * ws;
    return cnt == 1;
  }
}

// What a lane carries through the LU steps: per row slot act, the key mask (0 once the
// row is retired); per matrix info, the steps whose pivot was zero, and bad: a zero
// pivot over a column that does not hold plain zeros, left to the general kernel body.
template <int MR> struct RowState {
  unsigned act[MR];
  int info;
  bool bad;
  unsigned long long zmask;
};
template <class T, int NP, int NRHS, int GO>
using RowRegs = typename Unit<T>::E[BlkCfg<T, NP, NRHS, GO>::MR][RowCfg<T, NP, NRHS, GO>::RW / Unit<T>::n];

// VN steps of the LU on registers holding columns k0 .. k0 + W - 1 of each row; on
// return they hold columns k0 + VN .. k0 + W - 1 (moved down by the last step's update).
// Mu: shared address of the matrix; ord[k] <- the physical row retired at step k; cend:
// columns from there on are not this panel's.
template <class T, int NP, int NRHS, int GO, int W, bool ROLLED>
__device__ __forceinline__ void lu_rows_group(unsigned Mu, RowRegs<T, NP, NRHS, GO>& a,
                                              RowState<BlkCfg<T, NP, NRHS, GO>::MR>& st, int k0, int cend, int* ord,
                                              const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using R = RowCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  using E = typename U::E;
  using D = DivRange<T>;
  constexpr int G = C::G, MR = C::MR, RS = C::RS, VN = R::VN, UN = U::n, TS = int(sizeof(T));
  const unsigned own = Mu + g.lsl * RS + k0 * TS;  // this lane's row of slot 0 at column k0
  const unsigned ordu = Mu + C::MAT;               // ord as a shared address
#pragma unroll
  for (int i = 0; i < VN; ++i) {
    const int k = k0 + i;
    // ---- 1. the winner
    T x[MR];
    unsigned key[MR], m = 0, b[MR];
    bool win[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      x[s] = U::get(a[s][i / UN], i % UN);
      key[s] = hi_word(x[s]) & st.act[s];
      m = max(m, key[s]);
    }
    m = seg_max<G>(m, g);
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      win[s] = key[s] == m;
      b[s] = __ballot_sync(kFull, win[s]);
    }
    int wr;
    const bool one = one_row<G, MR>(b, g, wr);
    unsigned urow = Mu + wr * RS;
    // rare, by the whole warp: a tie (of high words), or a column whose largest entry is
    // zero, infinite or NaN
    bool zero = false;
    if (__any_sync(kFull, !one | (m - 1u >= D::kInf - 1u))) {
      Candidates<T, MR> c;
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        c.v[s] = x[s];
        c.act[s] = st.act[s];
      }
      const Choice w = exact_pivot<T, MR, G>(c, ord, k, g.lsl);
#pragma unroll
      for (int s = 0; s < MR; ++s) win[s] = w.slot == s;
      wr = w.row;
      urow = Mu + wr * RS;
      if (w.zero) {
        // the column stays as it is (plain zeros: a multiplier of +0), and a row of +0
        // leaves every element as it is: fma(-0, +0, c) == c
        zero = true;
        urow = g.zrow;
#pragma unroll
        for (int s = 0; s < MR; ++s) st.bad = st.bad || (st.act[s] && !plain_zero(x[s]));
        st.info = st.info == 0 ? k + 1 : st.info;
        st.zmask |= 1ull << k;
      }
    }
    // ---- 2. its row: output and broadcast
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      if (win[s]) {
        unrolled<0, W, VN>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          if (!ROLLED || q < W - R::PW + VN || k0 + q < cend) sts16<q * TS>(own + G * RS * s, a[s][q / UN], a[s][q / UN + 1]);
        });
        st.act[s] = 0u;
      }
    }
    if (g.lsl == 0) sts(ordu + 4 * k, wr);
    __syncwarp();
    urow += k0 * TS;
    const Unit2<E> u0 = lds16(urow, E());
    // ---- 3. multipliers
    const T piv = U::get(i / UN == 0 ? u0.x : u0.y, i % UN);
    const T ry = rcp_in_range(piv);
    const auto lim = D::limit(m);
    T l[MR];
    bool slow = m - D::kLo > D::kHi - D::kLo;
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const T q = x[s] * ry;
      l[s] = fma_(fma_(-piv, q, x[s]), ry, q);
      slow |= D::outside(x[s], lim);
    }
    if (__any_sync(kFull, slow)) {
#pragma unroll
      for (int s = 0; s < MR; ++s) l[s] = zero ? x[s] : st.act[s] ? div_slow(x[s], piv) : T(0);
    }
    // ---- 4. update
    E nl[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      nl[s] = U::dup(-l[s]);
      U::set(a[s][i / UN], i % UN, l[s]);
      if (UN == 2 && i % 2 == 0) U::set(a[s][i / UN], 1, fma_(-l[s], U::get(i / UN == 0 ? u0.x : u0.y, 1), U::get(a[s][i / UN], 1)));
      if (i < UN) a[s][1] = U::fma(nl[s], u0.y, a[s][1]);
      // the group's multipliers, before the registers move on
      if (i + 1 == VN && st.act[s]) sts16(own + G * RS * s, a[s][0], a[s][1]);
    }
    unrolled<VN, W, VN>([&](auto qc) {
      constexpr int q = decltype(qc)::value;
      if (ROLLED && !R::in_row(q) && k0 + q >= cend) return;
      const Unit2<E> u = lds16<q * TS>(urow, E());
      const int d = (i + 1 < VN ? q : q - VN) / UN;
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        a[s][d] = U::fma(nl[s], u.x, a[s][q / UN]);
        a[s][d + 1] = U::fma(nl[s], u.y, a[s][q / UN + 1]);
      }
    });
  }
}

// Brings a panel (registers holding W columns from c0 on) up to date with the steps
// 0 .. c0 - 1: the pivot row of each step is published (its final U), then every row
// takes the update with its own multiplier. Rows retired before a step update values
// that are never used.
template <class T, int NP, int NRHS, int GO, int W, bool ZEROS>
__device__ __forceinline__ void lu_rows_catch_up(unsigned Mu, RowRegs<T, NP, NRHS, GO>& a, unsigned long long zmask, int c0,
                                                 const int* ord, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using R = RowCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  using E = typename U::E;
  constexpr int G = C::G, MR = C::MR, RS = C::RS, VN = R::VN, UN = U::n, TS = int(sizeof(T));
#pragma unroll 1
  for (int k0 = 0; k0 < c0; k0 += VN) {
    Unit2<E> lv[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = g.lsl + G * s;
      lv[s] = lds16(Mu + (r < NP ? r : NP - 1) * RS + k0 * TS, E());
    }
#pragma unroll
    for (int i = 0; i < VN; ++i) {
      const int wr = ord[k0 + i];
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        if (wr == g.lsl + G * s) {
          unrolled<0, W, VN>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            sts16<q * TS>(Mu + (g.lsl + G * s) * RS + c0 * TS, a[s][q / UN], a[s][q / UN + 1]);
          });
        }
      }
      __syncwarp();
      const bool skip = ZEROS && ((zmask >> (k0 + i)) & 1);
      const unsigned urow = skip ? g.zrow : Mu + wr * RS + c0 * TS;
      E nl[MR];
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const T l = U::get(i / UN == 0 ? lv[s].x : lv[s].y, i % UN);
        nl[s] = U::dup(skip ? -T(0) : -l);
      }
#pragma unroll
      for (int q = 0; q < W; q += VN) {
        const Unit2<E> u = lds16(urow + q * TS, E());
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          a[s][q / UN] = U::fma(nl[s], u.x, a[s][q / UN]);
          a[s][q / UN + 1] = U::fma(nl[s], u.y, a[s][q / UN + 1]);
        }
      }
    }
  }
}

// VN steps of the Cholesky, same register contract (matrix columns only); b holds the
// right-hand sides. Shared row k receives L(j, k) at column j > k and y_k in the
// right-hand-side columns.
template <class T, int NP, int NRHS, int GO, int W>
__device__ __forceinline__ void chol_rows_group(unsigned Mu, RowRegs<T, NP, 0, GO>& a,
                                                T (&b)[BlkCfg<T, NP, NRHS, GO>::MR][NRHS > 0 ? NRHS : 1], int k0,
                                                int& info, typename Unit<T>::E nz, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using R = RowCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  using E = typename U::E;
  using D = DivRange<T>;
  constexpr int G = C::G, MR = C::MR, RS = C::RS, VN = R::VN, UN = U::n, TS = int(sizeof(T));
  constexpr bool FUSED = NP <= 16;  // n <= 16, as the reference's simd backend compiles it
#pragma unroll
  for (int i = 0; i < VN; ++i) {
    const int k = k0 + i;
    const int ds = k / G;
    T x[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) x[s] = U::get(a[s][i / UN], i % UN);
    T dv = x[0];
#pragma unroll
    for (int s = 1; s < MR; ++s) dv = ds == s ? x[s] : dv;
    const T d = __shfl_sync(kFull, dv, g.segbase + (k & (G - 1)));
    const bool bad = !(d > T(0));
    info = (bad && info == 0) ? k + 1 : info;
    const T lkk = sqrt_(bad ? T(1) : d);
    const T ry = rcp_in_range(lkk);
    const unsigned krow = Mu + k * RS;
    const unsigned m = abs_hi(lkk);
    const auto lim = D::limit(m);
    T l[MR];
    // an unscaled matrix may have |x| > lkk: the quotient is kept below 2^20 as well
    bool slow = m - D::kLo > D::kHi - D::kLo;
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const T q = x[s] * ry;
      l[s] = fma_(fma_(-lkk, q, x[s]), ry, q);
      slow |= (g.lsl + G * s > k) & (D::outside(x[s], lim) | !(fabs(q) <= T(0x1p+20)));
    }
    if (__any_sync(kFull, slow)) {
#pragma unroll
      for (int s = 0; s < MR; ++s) l[s] = g.lsl + G * s > k ? div_slow(x[s], lkk) : l[s];
    }
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = g.lsl + G * s;
      if (r > k && r < NP) sts(krow + r * TS, l[s]);
      if constexpr (NRHS > 0) {
        if (r == k) {
          // y_k = b_k / l_kk by the same reciprocal
          T y[NRHS];
          bool far = m - D::kLo > D::kHi - D::kLo;
#pragma unroll
          for (int c = 0; c < NRHS; ++c) {
            const T q = b[s][c] * ry;
            y[c] = fma_(fma_(-lkk, q, b[s][c]), ry, q);
            far |= D::outside(b[s][c], lim) | !(fabs(q) <= T(0x1p+20));
          }
          if (far) {
#pragma unroll
            for (int c = 0; c < NRHS; ++c) y[c] = div_slow(b[s][c], lkk);
          }
#pragma unroll
          for (int c = 0; c < NRHS; ++c) sts(krow + (NP + c) * TS, y[c]);
        }
      }
      U::set(a[s][i / UN], i % UN, r > k ? l[s] : (r == k ? lkk : x[s]));
    }
    __syncwarp();
    E nl[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) nl[s] = U::dup(-l[s]);
    if (i + 1 < VN) {
      const Unit2<E> u0 = lds16(krow + k0 * TS, E());
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int r = g.lsl + G * s;
#pragma unroll
        for (int e = i + 1; e < VN; ++e) {
          // row k keeps L(j, k) here: the group's store below writes it back unchanged
          const T ue = U::get(e / UN == 0 ? u0.x : u0.y, e % UN), ae = U::get(a[s][e / UN], e % UN);
          const T v = FUSED ? fma_(-l[s], ue, ae) : sub_mul(ae, l[s], ue);
          U::set(a[s][e / UN], e % UN, r > k ? v : (r == k ? ue : ae));
        }
      }
    } else {
      // the group's columns of L; from here on row k is read only past these columns
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int r = g.lsl + G * s;
        if (r >= k0 && r < NP) sts16(Mu + r * RS + k0 * TS, a[s][0], a[s][1]);
      }
    }
#pragma unroll
    for (int q = VN; q < W; q += VN) {
      if (R::PW < NP && !R::in_row(q) && k0 % R::PW + q >= R::PW) continue;
      const Unit2<E> u = lds16(krow + (k0 + q) * TS, E());
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int t = (i + 1 < VN ? q : q - VN) / UN;
        a[s][t] = FUSED ? U::fma(nl[s], u.x, a[s][q / UN]) : U::muladd(nl[s], u.x, a[s][q / UN], nz);
        a[s][t + 1] = FUSED ? U::fma(nl[s], u.y, a[s][q / UN + 1]) : U::muladd(nl[s], u.y, a[s][q / UN + 1], nz);
      }
    }
    if constexpr (NRHS > 0) {
#pragma unroll
      for (int c = 0; c < NRHS; ++c) {
        T y;
        if constexpr (sizeof(T) == 8) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(y) : "r"(krow + (NP + c) * TS) : "memory");
        else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(y) : "r"(krow + (NP + c) * TS) : "memory");
#pragma unroll
        for (int s = 0; s < MR; ++s) fma_if(b[s][c], g.lsl + G * s > k, l[s], y);
      }
    }
  }
}

// W staged columns from c0 on into registers.
template <class T, int G, int MR, int RS, int NP, int W, int NU>
__device__ __forceinline__ void rows_fetch(unsigned Mu, typename Unit<T>::E (&a)[MR][NU], int c0, const Seg& g) {
  using E = typename Unit<T>::E;
#pragma unroll
  for (int s = 0; s < MR; ++s) {
    const int r = g.lsl + G * s;
    const unsigned row = Mu + (r < NP ? r : NP - 1) * RS + c0 * int(sizeof(T));
#pragma unroll
    for (int q = 0; q < W / Unit<T>::n; q += 2) {
      const Unit2<E> v = lds16(row + q * 8, E());
      a[s][q] = v.x;
      a[s][q + 1] = v.y;
    }
  }
}

// All phases of an order whose whole rows are in registers, from column K0 on.
template <class T, int NP, int NRHS, int GO, int K0>
__device__ __forceinline__ void lu_rows_phases(unsigned Mu, RowRegs<T, NP, NRHS, GO>& a,
                                               RowState<BlkCfg<T, NP, NRHS, GO>::MR>& st, int* ord, const Seg& g) {
  using R = RowCfg<T, NP, NRHS, GO>;
  if constexpr (K0 < NP) {
    lu_rows_group<T, NP, NRHS, GO, R::NCV - K0, false>(Mu, a, st, K0, R::NCV, ord, g);
    lu_rows_phases<T, NP, NRHS, GO, K0 + R::VN>(Mu, a, st, ord, g);
  }
}
// The panel at c0, W columns of it (the last one's with the right-hand sides).
template <class T, int NP, int NRHS, int GO, int W>
__device__ __forceinline__ void lu_rows_panel(unsigned Mu, RowRegs<T, NP, NRHS, GO>& a,
                                              RowState<BlkCfg<T, NP, NRHS, GO>::MR>& st, int c0, int* ord, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using R = RowCfg<T, NP, NRHS, GO>;
  if (c0 > 0) {
    __syncwarp();
    rows_fetch<T, C::G, C::MR, C::RS, NP, W>(Mu, a, c0, g);
    if (__any_sync(kFull, st.zmask != 0)) lu_rows_catch_up<T, NP, NRHS, GO, W, true>(Mu, a, st.zmask, c0, ord, g);
    else lu_rows_catch_up<T, NP, NRHS, GO, W, false>(Mu, a, 0, c0, ord, g);
  }
#pragma unroll 1
  for (int k0 = c0; k0 < c0 + R::PW; k0 += R::VN) lu_rows_group<T, NP, NRHS, GO, W, true>(Mu, a, st, k0, c0 + W, ord, g);
}
// Panels in a rolled loop: a copy of the code per panel, with its column a constant, does
// not fit the instruction cache (order 64, 8 right-hand sides: Cholesky 13,900 instructions
// instead of 3,300, LU 10,700 instead of 5,600). float32 posv n = 45, 50,000 matrices, 3
// right-hand sides 1253 -> 1056 us, gesv n = 32, 262,144 1691 -> 1621, a mixed stream of
// 262,144 matrices 4946 -> 4323 (passes with their input copies).
template <class T, int NP, int NRHS, int GO>
__device__ __forceinline__ void lu_rows_panels(unsigned Mu, RowRegs<T, NP, NRHS, GO>& a,
                                               RowState<BlkCfg<T, NP, NRHS, GO>::MR>& st, int* ord, const Seg& g) {
  using R = RowCfg<T, NP, NRHS, GO>;
  if constexpr (R::PW == NP) {
    lu_rows_phases<T, NP, NRHS, GO, 0>(Mu, a, st, ord, g);
  } else {
    constexpr int LAST = R::LASTW == R::PW ? NP : NP - R::PW;  // from there on with right-hand sides
#pragma unroll 1
    for (int c0 = 0; c0 < LAST; c0 += R::PW) lu_rows_panel<T, NP, NRHS, GO, R::PW>(Mu, a, st, c0, ord, g);
    if constexpr (LAST < NP) lu_rows_panel<T, NP, NRHS, GO, R::LASTW>(Mu, a, st, LAST, ord, g);
  }
}
template <class T, int NP, int NRHS, int GO, int K0>
__device__ __forceinline__ void chol_rows_phases(unsigned Mu, RowRegs<T, NP, 0, GO>& a,
                                                 T (&b)[BlkCfg<T, NP, NRHS, GO>::MR][NRHS > 0 ? NRHS : 1], int& info,
                                                 typename Unit<T>::E nz, const Seg& g) {
  using R = RowCfg<T, NP, NRHS, GO>;
  if constexpr (K0 < NP) {
    chol_rows_group<T, NP, NRHS, GO, NP - K0>(Mu, a, b, K0, info, nz, g);
    chol_rows_phases<T, NP, NRHS, GO, K0 + R::VN>(Mu, a, b, info, nz, g);
  }
}
template <class T, int NP, int NRHS, int GO>
__device__ __forceinline__ void chol_rows_panels(unsigned Mu, RowRegs<T, NP, 0, GO>& a,
                                                 T (&b)[BlkCfg<T, NP, NRHS, GO>::MR][NRHS > 0 ? NRHS : 1], int& info,
                                                 typename Unit<T>::E nz, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using R = RowCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  using E = typename U::E;
  constexpr int G = C::G, MR = C::MR, RS = C::RS, VN = R::VN, UN = U::n, TS = int(sizeof(T)), W = R::PW;
  if constexpr (W == NP) {
    chol_rows_phases<T, NP, NRHS, GO, 0>(Mu, a, b, info, nz, g);
  } else {
#pragma unroll 1
    for (int c0 = 0; c0 < NP; c0 += W) {
      if (c0 > 0) {
        __syncwarp();
        // rows above the panel take their place in shared memory only: what their
        // registers hold is never used
        rows_fetch<T, G, MR, RS, NP, W>(Mu, a, c0, g);
#pragma unroll 1
        for (int k0 = 0; k0 < c0; k0 += VN) {
          Unit2<E> lv[MR];
#pragma unroll
          for (int s = 0; s < MR; ++s) {
            const int r = g.lsl + G * s;
            lv[s] = lds16(Mu + (r < NP ? r : NP - 1) * RS + k0 * TS, E());
          }
#pragma unroll
          for (int i = 0; i < VN; ++i) {
            E nl[MR];
#pragma unroll
            for (int s = 0; s < MR; ++s) nl[s] = U::dup(-U::get(i / UN == 0 ? lv[s].x : lv[s].y, i % UN));
#pragma unroll
            for (int q = 0; q < W; q += VN) {
              const Unit2<E> u = lds16(Mu + (k0 + i) * RS + (c0 + q) * TS, E());
#pragma unroll
              for (int s = 0; s < MR; ++s) {
                a[s][q / UN] = U::muladd(nl[s], u.x, a[s][q / UN], nz);
                a[s][q / UN + 1] = U::muladd(nl[s], u.y, a[s][q / UN + 1], nz);
              }
            }
          }
        }
      }
#pragma unroll 1
      for (int k0 = c0; k0 < c0 + W; k0 += VN) chol_rows_group<T, NP, NRHS, GO, W>(Mu, a, b, k0, info, nz, g);
    }
  }
}

// Column-oriented back substitution with reciprocal diagonals; lane lsl solves the
// positions lsl + G t. U(i, k) sits in shared row ord[i] (LU) or i (Cholesky: L^T), at
// column k. The operations of seg_backsolve (blk.cuh) in its order. The owner of x_k is
// known per slot, so there are no selects: one or two right-hand sides go by shuffle;
// more by shared memory, where x_k replaces y_k in its row and no update is predicated
// (a lane's own y is not needed any more).
template <class T, int NP, int NRHS, bool CHOL, int GO>
__device__ __forceinline__ void rows_backsolve(unsigned char* M, const int* ord, const MatJob<T>& j, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  using E = typename U::E;
  constexpr int G = C::G, MR = C::MR, RS = C::RS, UN = U::n, VN = 2 * UN, TS = int(sizeof(T));
  static_assert(G % VN == 0, "a vector of columns has its owners in one slot");
  constexpr bool SHARED = NRHS >= VN;
  constexpr int NU = SHARED ? NRHS / UN : NRHS;  // right-hand sides in registers: units, or elements
  const unsigned Mu = (unsigned)__cvta_generic_to_shared(M);
  T d[MR];
  unsigned rowp[MR];
  typename std::conditional<SHARED, E, T>::type y[MR][NU];
#pragma unroll
  for (int t = 0; t < MR; ++t) {
    const int i = g.lsl + G * t < NP ? g.lsl + G * t : NP - 1;
    const int r = CHOL ? i : ord[i];
    rowp[t] = Mu + r * RS;
    d[t] = rcp_(*reinterpret_cast<const T*>(M + r * RS + i * TS));
    if constexpr (SHARED) {
#pragma unroll
      for (int c = 0; c < NU; c += 2) {
        const Unit2<E> v = lds16(rowp[t] + NP * TS + c * 8, E());
        y[t][c] = v.x;
        y[t][c + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int c = 0; c < NU; ++c) y[t][c] = *reinterpret_cast<const T*>(M + r * RS + (NP + c) * TS);
    }
  }
#pragma unroll
  for (int t = MR - 1; t >= 0; --t) {  // the slot whose positions are being solved
    const int top = G * (t + 1) < NP ? G * (t + 1) : NP;
#pragma unroll 1
    for (int kb = top - VN; kb >= G * t; kb -= VN) {
      Unit2<E> u[MR];
#pragma unroll
      for (int s = 0; s <= t; ++s) u[s] = lds16(rowp[s] + kb * TS, E());
#pragma unroll
      for (int q = VN - 1; q >= 0; --q) {
        const int kl = kb + q - G * t;
        auto uq = [&](int s) { return U::get(q / UN == 0 ? u[s].x : u[s].y, q % UN); };
        if constexpr (SHARED) {
          const bool mine = g.lsl == kl;
          const E dd = U::dup(d[t]);
#pragma unroll
          for (int c = 0; c < NU; c += 2)
            if (mine) sts16(rowp[t] + NP * TS + c * 8, U::mul(y[t][c], dd), U::mul(y[t][c + 1], dd));
          __syncwarp();
          const unsigned xrow = Mu + (CHOL ? kb + q : ord[kb + q]) * RS + NP * TS;
          E nu[MR];
#pragma unroll
          for (int s = 0; s <= t; ++s) nu[s] = U::dup(-uq(s));
#pragma unroll
          for (int c = 0; c < NU; c += 2) {
            const Unit2<E> x = lds16(xrow + c * 8, E());
#pragma unroll
            for (int s = 0; s <= t; ++s) {
              y[s][c] = U::fma(nu[s], x.x, y[s][c]);
              y[s][c + 1] = U::fma(nu[s], x.y, y[s][c + 1]);
            }
          }
        } else {
          T x[NU];
#pragma unroll
          for (int c = 0; c < NU; ++c) x[c] = __shfl_sync(kFull, y[t][c] * d[t], g.segbase + kl);
#pragma unroll
          for (int s = 0; s < t; ++s)
#pragma unroll
            for (int c = 0; c < NU; ++c) y[s][c] = fma_(-uq(s), x[c], y[s][c]);
#pragma unroll
          for (int c = 0; c < NU; ++c) fma_if(y[t][c], g.lsl < kl, uq(t), x[c]);
        }
      }
    }
  }
  if (j.live && j.B) {
#pragma unroll
    for (int t = 0; t < MR; ++t) {
      const int i = g.lsl + G * t;
      if (i >= j.n) continue;
      T* brow = j.B + (long long)i * j.ldb + j.b0;
      if constexpr (SHARED) {
        const T* xr = reinterpret_cast<const T*>(M + (rowp[t] - Mu) + NP * TS);
#pragma unroll
        for (int c = 0; c < NRHS; ++c)
          if (c < j.nrhs) brow[c] = xr[c];
      } else {
#pragma unroll
        for (int c = 0; c < NU; ++c)
          if (c < j.nrhs) brow[c] = y[t][c] * d[t];
      }
    }
  }
}

// Calls f(row, chunk) for every chunk of VEC bytes of an n x n matrix, G lanes side by
// side. A matrix that fills its tile in 16-byte chunks is walked as one run of chunks
// with constant strides. Otherwise every row is taken by itself, its chunks dealt to the
// lanes: the addresses of a row are one multiply-add from the first's, where a run of
// chunks of any length costs about ten instructions a chunk to turn into rows (float32
// LU, 4 right-hand sides, rows going 4 bytes at a time: order 61, 32,768 matrices 1259 ->
// 1165 us; order 29, 131,072: 846 -> 759). UNROLL: 4 for plain copies; less where the body
// is longer, and then without the unrolled run, which spills there.
template <class T, int NP, int G, int VEC, int UNROLL = 4, class F>
__device__ __forceinline__ void walk_chunks(int n, int lsl, F&& f) {
  constexpr int RC = NP * int(sizeof(T)) / VEC;  // chunks of a row of the tile
  if constexpr (VEC == 16 && UNROLL == 4) {
    if (n == NP) {
#pragma unroll
      for (int i = 0; i < (NP * RC + G - 1) / G; ++i) {
        const int e = lsl + i * G;
        if (NP * RC % G == 0 || e < NP * RC) f(e / RC, e % RC);
      }
      return;
    }
  }
  const int rc = n * int(sizeof(T)) / VEC;
#pragma unroll UNROLL
  for (int r = 0; r < n; ++r) {
#pragma unroll
    for (int s = 0; s < (RC + G - 1) / G; ++s)
      if (lsl + G * s < rc) f(r, lsl + G * s);
  }
}

// Stages the job's matrix, identity-padded to NP, in shared memory (the copies are in
// flight while the right-hand sides are read).
template <class T, int NP, int NRHS, int GO>
__device__ __forceinline__ void rows_load(unsigned char* M, const MatJob<T>& j, const Seg& g, T (&rhs)[BlkCfg<T, NP, NRHS, GO>::MR][NRHS > 0 ? NRHS : 1]) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  constexpr int G = C::G, MR = C::MR, RS = C::RS, TS = int(sizeof(T));
  if (j.live) {
    const int vec = vec_of<T>(j.A, j.n), rowb = j.n * TS;
    const char* src = reinterpret_cast<const char*>(j.A);
    if (vec == 16) walk_chunks<T, NP, G, 16>(j.n, g.lsl, [&](int r, int c) { cp_async<16>(M + r * RS + c * 16, src + r * rowb + c * 16); });
    else if (vec == 8) walk_chunks<T, NP, G, 8>(j.n, g.lsl, [&](int r, int c) { cp_async<8>(M + r * RS + c * 8, src + r * rowb + c * 8); });
    else if constexpr (sizeof(T) == 4) walk_chunks<T, NP, G, 4>(j.n, g.lsl, [&](int r, int c) { cp_async<4>(M + r * RS + c * 4, src + r * rowb + c * 4); });
  }
  cp_async_commit();
#pragma unroll
  for (int s = 0; s < MR; ++s) {
    const int r = g.lsl + G * s;
    const bool rowok = j.live && j.B && r < j.n;
    const T* brow = rowok ? j.B + (long long)r * j.ldb + j.b0 : nullptr;
#pragma unroll
    for (int c = 0; c < NRHS; ++c) rhs[s][c] = (rowok && c < j.nrhs) ? brow[c] : T(0);
  }
  const int n = j.live ? j.n : 0;
  if (n < NP) {
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = g.lsl + G * s;
      T* row = reinterpret_cast<T*>(M + r * RS);
      if (r < n) {
        for (int c = n; c < NP; ++c) row[c] = T(0);
      } else if (r < NP) {
        for (int c = 0; c < NP * TS / 16; ++c) reinterpret_cast<uint4*>(row)[c] = make_uint4(0, 0, 0, 0);
        row[r] = T(1);
      }
    }
  }
  cp_async_wait<0>();
  __syncwarp();
}

// The LU of one matrix staged at shared address Mu (NP rows of RS bytes, NC columns, the
// right-hand sides included) for every input, one step at a time in shared memory: what
// lu_rows leaves to it is a zero pivot over a column that holds -0 or NaN. The reference's
// loop (kernels.hpp:91-119) with the rows behind a map; ord[k] <- the row at position k.
// Returns info. Out of line and sized at run time: few matrices need it.
template <class T>
__device__ __noinline__ int lu_plain(unsigned Mu, int RS, int NP, int NC, unsigned ordu, int lsl, int G) {
  using K = typename KeyT<T>::U;
  unsigned char* M = static_cast<unsigned char*>(__cvta_shared_to_generic(Mu));
  int* ord = static_cast<int*>(__cvta_shared_to_generic(ordu));
  auto row = [&](int p) { return reinterpret_cast<T*>(M + ord[p] * RS); };
  for (int p = lsl; p < NP; p += G) ord[p] = p;
  __syncwarp();
  int info = 0;
  for (int k = 0; k < NP; ++k) {
    K bk = 0;
    int bp = 0x7fffffff;
    for (int p = k + lsl; p < NP; p += G) {
      const T v = row(p)[k];
      const K key = isnan(v) ? (p == k ? ~K(0) : K(0)) : key_bits(v) + 1;
      if (key > bk || (key == bk && p < bp)) {
        bk = key;
        bp = p;
      }
    }
    for (int o = G / 2; o > 0; o >>= 1) {
      const K ok = __shfl_xor_sync(kFull, bk, o);
      const int op = __shfl_xor_sync(kFull, bp, o);
      if (ok > bk || (ok == bk && op < bp)) {
        bk = ok;
        bp = op;
      }
    }
    if (lsl == 0) {
      const int t = ord[k];
      ord[k] = ord[bp];
      ord[bp] = t;
    }
    __syncwarp();
    if (bk == K(1)) {
      info = info == 0 ? k + 1 : info;
    } else {
      const T* u = row(k);
      for (int p = k + 1 + lsl; p < NP; p += G) {
        T* x = row(p);
        const T l = div_(x[k], u[k]);
        x[k] = l;
        for (int c = k + 1; c < NC; ++c) x[c] = fma_(-l, u[c], x[c]);
      }
    }
    __syncwarp();
  }
  return info;
}

template <class T, int NP, int NRHS, int GO>
__device__ __forceinline__ void lu_rows(unsigned char* M, const MatJob<T>& j, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using R = RowCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  constexpr int G = C::G, MR = C::MR, RS = C::RS, UN = U::n;
  int* ord = reinterpret_cast<int*>(M + C::MAT);
  const unsigned Mu = (unsigned)__cvta_generic_to_shared(M);
  RowState<MR> st;
  {
    RowRegs<T, NP, NRHS, GO> a;
    T rhs[MR][NRHS > 0 ? NRHS : 1];
    rows_load<T, NP, NRHS, GO>(M, j, g, rhs);
    rows_fetch<T, G, MR, RS, NP, R::PW>(Mu, a, 0, g);
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = g.lsl + G * s;
#pragma unroll
      for (int c = NP; c < R::NCV; ++c) {
        const T v = c - NP < NRHS ? rhs[s][c - NP < NRHS ? c - NP : 0] : T(0);
        if (R::PW == NP) U::set(a[s][c / UN % (R::RW / UN)], c % UN, v);
        else if (r < NP) sts(Mu + r * RS + c * int(sizeof(T)), v);
      }
    }
    st.info = 0;
    st.bad = false;
    st.zmask = 0;
#pragma unroll
    for (int s = 0; s < MR; ++s) st.act[s] = g.lsl + G * s < NP ? 0x7fffffffu : 0u;
    lu_rows_panels<T, NP, NRHS, GO>(Mu, a, st, ord, g);
    __syncwarp();
  }
  if (__any_sync(kFull, st.bad)) {  // nothing has left shared memory yet: start over
    T rhs[MR][NRHS > 0 ? NRHS : 1];
    rows_load<T, NP, NRHS, GO>(M, j, g, rhs);
#pragma unroll
    for (int s = 0; s < MR; ++s)
#pragma unroll
      for (int c = 0; c < NRHS; ++c)
        if (g.lsl + G * s < NP) sts(Mu + (g.lsl + G * s) * RS + (NP + c) * int(sizeof(T)), rhs[s][c]);
    __syncwarp();
    st.info = lu_plain<T>(Mu, RS, NP, C::NC, Mu + C::MAT, g.lsl, G);
  }
  if constexpr (NRHS > 0) rows_backsolve<T, NP, NRHS, false, GO>(M, ord, j, g);
  if (j.live) {
    if (j.piv) {
#pragma unroll
      for (int t = 0; t < MR; ++t) {
        const int k = g.lsl + G * t;
        if (k < j.n) j.piv[k] = position_of(ord, ord[k], k);
      }
    }
    if (g.lsl == 0 && j.info) *j.info = st.info;
    if (j.Aout) {
      const int vec = vec_of<T>(j.Aout, j.n), rowb = j.n * int(sizeof(T));
      char* out = reinterpret_cast<char*>(j.Aout);
      if (vec == 16) walk_chunks<T, NP, G, 16>(j.n, g.lsl, [&](int r, int c) {
          *reinterpret_cast<uint4*>(out + r * rowb + c * 16) = *reinterpret_cast<const uint4*>(M + ord[r] * RS + c * 16); });
      else if (vec == 8) walk_chunks<T, NP, G, 8>(j.n, g.lsl, [&](int r, int c) {
          *reinterpret_cast<uint2*>(out + r * rowb + c * 8) = *reinterpret_cast<const uint2*>(M + ord[r] * RS + c * 8); });
      else if constexpr (sizeof(T) == 4) walk_chunks<T, NP, G, 4>(j.n, g.lsl, [&](int r, int c) {
          *reinterpret_cast<unsigned*>(out + r * rowb + c * 4) = *reinterpret_cast<const unsigned*>(M + ord[r] * RS + c * 4); });
    }
  }
  __syncwarp();
}

template <class T, int NP, int NRHS, int GO>
__device__ __forceinline__ void chol_rows(unsigned char* M, const MatJob<T>& j, const Seg& g) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  using U = Unit<T>;
  constexpr int G = C::G, MR = C::MR, RS = C::RS;
  const unsigned Mu = (unsigned)__cvta_generic_to_shared(M);
  RowRegs<T, NP, 0, GO> a;
  T b[MR][NRHS > 0 ? NRHS : 1];
  rows_load<T, NP, NRHS, GO>(M, j, g, b);
  rows_fetch<T, G, MR, RS, NP, RowCfg<T, NP, NRHS, GO>::PW>(Mu, a, 0, g);
  int info = 0;
  __syncwarp();  // every row is in registers before the first column overwrites its row
  chol_rows_panels<T, NP, NRHS, GO>(Mu, a, b, info, lds16(g.zrow + kZeroRow, typename U::E()).x, g);
  __syncwarp();
  if constexpr (NRHS > 0) rows_backsolve<T, NP, NRHS, true, GO>(M, nullptr, j, g);
  if (j.live) {
    if (g.lsl == 0 && j.info) *j.info = info;
    if (j.Aout) {
      // the lower triangle, zeros above it: of a chunk of vec bytes from element e0 on, the
      // words of the elements up to r
      constexpr int TW = int(sizeof(T)) / 4, UNR = 2;
      const int vec = vec_of<T>(j.Aout, j.n), rowb = j.n * int(sizeof(T));
      char* out = reinterpret_cast<char*>(j.Aout);
      if (vec == 16) walk_chunks<T, NP, G, 16, UNR>(j.n, g.lsl, [&](int r, int c) {
          uint4 v = *reinterpret_cast<const uint4*>(M + r * RS + c * 16);
          const int keep = (r + 1) * TW - 4 * c;
          v.x = keep > 0 ? v.x : 0u;
          v.y = keep > 1 ? v.y : 0u;
          v.z = keep > 2 ? v.z : 0u;
          v.w = keep > 3 ? v.w : 0u;
          *reinterpret_cast<uint4*>(out + r * rowb + c * 16) = v; });
      else if (vec == 8) walk_chunks<T, NP, G, 8, UNR>(j.n, g.lsl, [&](int r, int c) {
          uint2 v = *reinterpret_cast<const uint2*>(M + r * RS + c * 8);
          const int keep = (r + 1) * TW - 2 * c;
          v.x = keep > 0 ? v.x : 0u;
          v.y = keep > 1 ? v.y : 0u;
          *reinterpret_cast<uint2*>(out + r * rowb + c * 8) = v; });
      else if constexpr (sizeof(T) == 4) walk_chunks<T, NP, G, 4, UNR>(j.n, g.lsl, [&](int r, int c) {
          *reinterpret_cast<unsigned*>(out + r * rowb + c * 4) = c <= r ? *reinterpret_cast<const unsigned*>(M + r * RS + c * 4) : 0u; });
    }
  }
  __syncwarp();
}

// One matrix per segment: the body every dense and stream kernel runs.
template <class T, int NP, int NRHS, bool CHOL, int GO = 0>
__device__ __forceinline__ void blk_matrix(unsigned char* M, const MatJob<T>& j, const Seg& g) {
  if constexpr (CHOL) chol_rows<T, NP, NRHS, GO>(M, j, g);
  else lu_rows<T, NP, NRHS, GO>(M, j, g);
}

// The constants at Seg::zrow, once per CTA (kRowConst bytes of static shared memory).
__device__ __forceinline__ unsigned rows_constants(unsigned char* at) {
  for (int i = threadIdx.x; i < kRowConst / 4; i += blockDim.x) reinterpret_cast<int*>(at)[i] = i < kZeroRow / 4 ? 0 : (int)0x80000000;
  __syncthreads();
  return (unsigned)__cvta_generic_to_shared(at);
}

// Dense batch: one persistent CTA of at most WPC warps per SM; every round each segment
// takes the next matrix.
template <class T, int NP, int NRHS, int WPC, bool CHOL, int GO = 0>
__global__ void __launch_bounds__(WPC * 32, 1) blk_kernel(SolveArgs<T> p) {
  using C = BlkCfg<T, NP, NRHS, GO>;
  constexpr int G = C::G, S = C::S;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(16) unsigned char consts[kRowConst];
  // the warp index through a shuffle, so that the compiler knows it to be uniform: the
  // warp-wide operations below then need no divergence checks
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31, wpc = blockDim.x >> 5;
  Seg g;
  g.lane = lane;
  g.lsl = lane & (G - 1);
  g.segbase = (lane / G) * G;
  g.zrow = rows_constants(consts);
  unsigned char* M = smem + warp * C::WARPB + (lane / G) * C::SEGB;
  const long long nn = (long long)p.n * p.n;
  const long long per_round = (long long)gridDim.x * wpc * S;
  // warps own disjoint shared memory, so they run their rounds without a block barrier
  for (long long base = (long long)blockIdx.x * wpc * S; base < p.batch; base += per_round) {
    const long long m = base + (long long)warp * S + lane / G;
    {
      // this warp's next unit heads for L2 while this one is solved
      const long long nxt = base + per_round + (long long)warp * S;
      if (lane == 0 && nxt < p.batch) {
        const long long cnt = (p.batch - nxt) < S ? (p.batch - nxt) : S;
        prefetch_l2(p.A + nxt * nn, cnt * nn * (long long)sizeof(T));
        if (p.B) prefetch_l2(p.B + nxt * (long long)p.n * p.ldb, cnt * (long long)p.n * p.ldb * (long long)sizeof(T));
      }
    }
    MatJob<T> j;
    j.live = m < p.batch && !(p.status && p.status[m] >= 0);
    if (!__any_sync(kFull, j.live)) continue;
    const long long mm = j.live ? m : 0;
    j.A = p.A + mm * nn;
    j.Aout = p.wf ? p.A + mm * nn : nullptr;
    j.B = p.B ? p.B + mm * (long long)p.n * p.ldb : nullptr;
    j.piv = (p.piv && p.wf) ? p.piv + mm * p.n : nullptr;
    j.info = p.info ? p.info + mm : nullptr;
    j.n = p.n;
    j.ldb = p.ldb;
    j.b0 = p.b0;
    j.nrhs = p.nrhs;
    blk_matrix<T, NP, NRHS, CHOL, GO>(M, j, g);
  }
}

}  // namespace dev
}  // namespace tsdx
