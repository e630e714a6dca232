// Mixed-precision factorization + fp64 iterative refinement (gesv_ir / posv_ir).
//
// No reference counterpart: TinySolverDx only emulates fp16/bf16 on the CPU
// (precision.hpp:71-97). Per matrix (one warp, persistent CTA rounds):
//   1. A (fp64, global) is read once, coalesced, and written to shared memory as
//      an fp32 working matrix, scaled by powers of two (rows then columns, max
//      |a| -> 1, exact) so fp16 tensor-core operands stay in range.
//   2. The scaled matrix is factored in fp32 with partial pivoting (LU) or, for
//      symmetric positive definite input, without pivoting (A = L U with U = D L^T,
//      the Cholesky factor up to a diagonal: SPD matrices need no pivoting, and the
//      shared code keeps one fast path): 16-column panels in registers, a step's pivot
//      row published by the store that also writes it to the factor (as in rows.cuh), the
//      trailing update A22 -= L21 U12 either on the tensor cores (mma.sync m16n8k16,
//      fp16 or bf16 operands, fp32 accumulation) or on the fp32 CUDA cores, two columns
//      to an instruction, by tier.
//   3. x0 = A^{-1} b with the low-precision factors (fp32 triangular solves, a lane per
//      position, reciprocal pivots computed once after the factorization).
//   4. Refinement: r = b - A x in fp64 straight from A in global memory (rows
//      read coalesced, 32 row sums per lane folded by a transposing butterfly),
//      normwise backward error ||r|| / (||A||_F ||x|| + ||b||)
//      (runtime.cpp:230-242); stop when it is <= tol, else x += A^{-1} r with the
//      same factors.
// A matrix that does not converge within itmax steps (or meets a zero / non-
// positive pivot in low precision) is reported with status -1; the host then
// solves it with the plain fp64 kernel (the fallback is never silent).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "rows.cuh"

namespace tsdx {
namespace dev {

struct IrArgs {
  const double* A;            // (batch, n, n), not modified
  double* B;                  // (batch, n): right-hand side in, solution out
  int* info;                  // (batch) low-precision factorization info, or nullptr
  const signed char* tier;    // (batch) per-matrix tier, or nullptr -> default_tier
  int* status;                // (batch) refinement steps used, -1 = not converged
  double* bwd;                // (batch) final normwise backward error, or nullptr
  const int* idx;             // optional (batch) list of matrix indices to solve
  long long batch;
  int n, default_tier, itmax;
  double tol;
};

enum Tier { kTierF16 = 0, kTierBF16 = 1, kTierF32 = 2, kTierF64 = 3 };

__device__ __forceinline__ unsigned pack2(float lo, float hi, bool f16) {
  if (f16) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&h);
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&h);
}

// D = A(16x16) * B(16x8) + C, fp32 accumulation; A row-major, B column-major fragments.
__device__ __forceinline__ void mma16816(float* d, const unsigned* a, const unsigned* b, bool f16) {
  if (f16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int NP>
struct IrCfg {
  static constexpr int MR = (NP + 31) / 32;
  static constexpr int PB = 16;
  static constexpr int RSF = NP * 4 + 16;  // fp32 row: an odd number of 16-byte units
  static constexpr int F = NP * RSF;
  // ord (int), x (double), column scales, row scales (float; after the scaling, the
  // right-hand side on its way to the pivots' order)
  static constexpr int AUX = NP * 4 + NP * 8 + NP * 4 * 2 + 32;
  static constexpr int WARPB = (F + AUX + 127) / 128 * 128;
  // cooperative float4 passes: CG groups of 4 columns, RPI rows per pass
  static constexpr int CG = NP / 4;
  static constexpr int CGP = CG <= 4 ? 4 : CG <= 8 ? 8 : 16;
  static constexpr int RPI = 32 / CGP;
  static_assert(NP % 16 == 0, "tensor-core tiles need NP % 16 == 0");
};

template <int NP, bool SPD, int WPC>
__global__ void __launch_bounds__(WPC * 32, 1) ir_kernel(IrArgs p) {
  using C = IrCfg<NP>;
  constexpr int MR = C::MR, PB = C::PB, RSF = C::RSF, CG = C::CG, CGP = C::CGP, RPI = C::RPI;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31, wpc = blockDim.x >> 5;
  unsigned char* Fb = smem + warp * C::WARPB;
  int* ord = reinterpret_cast<int*>(Fb + C::F);
  double* xs = reinterpret_cast<double*>(Fb + C::F + NP * 4);
  float* csc = reinterpret_cast<float*>(Fb + C::F + NP * 12);
  float* rsd = csc + NP;
  const unsigned Fu = (unsigned)__cvta_generic_to_shared(Fb);
  using U2 = Unit<float>;
  auto F = [&](int r, int c) -> float& { return *reinterpret_cast<float*>(Fb + r * RSF + c * 4); };
  auto F4 = [&](int r, int c) -> float4& { return *reinterpret_cast<float4*>(Fb + r * RSF + c * 4); };
  const int n = p.n;
  const long long per_round = (long long)gridDim.x * wpc;
  const int q4 = lane % CGP, rho = lane / CGP;  // cooperative pass coordinates

  // A block barrier before every round keeps the warps on the same code. Without it they
  // drift apart over the rounds (a matrix takes two to four refinement steps) and their
  // instructions no longer fit the cache: general matrices, float32 tier, n = 17, 129,757 of
  // them 2796 us without and 1986 with it; n = 40, 156,250 6701 and 5069; n = 64, 61,035
  // 2967 and 2596. The code for SPD matrices of orders up to 16 fits, and is faster without
  // (n = 8, 600,000 matrices 3172 and 3537; the next one, n = 32, 244,140 3238 and 3237).
  constexpr bool LOCKSTEP = !(SPD && NP == 16);
  for (long long base = (long long)blockIdx.x * wpc; base < p.batch; base += per_round) {
    if constexpr (LOCKSTEP) __syncthreads();
    const long long t = base + warp;
    if (t >= p.batch) continue;
    const long long m = p.idx ? (long long)p.idx[t] : t;
    const int tier = p.tier ? (int)p.tier[m] : p.default_tier;
    if (tier >= kTierF64) {  // solved directly by the fp64 pass
      if (lane == 0 && p.status) p.status[m] = -1;
      continue;
    }
    const bool tc = tier == kTierF16 || tier == kTierBF16;
    const bool f16 = tier == kTierF16;
    const double* Ag = p.A + m * (long long)n * n;
    double* Bg = p.B + m * (long long)n;

    // ------------------------------------------ 1. load, scale, ||A||_F, b
    double afro = 0.0;
    float rsc[MR];
    {
      // coalesced row reads (lane c holds columns c, c + 32), unscaled fp32 copy
#pragma unroll 1
      for (int r0 = 0; r0 < n; r0 += 8) {
        double v[8][MR];
        load_rows<8, MR>(Ag, n, r0, lane, v);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int s = 0; s < MR; ++s) {
            const int r = r0 + j, c = lane + 32 * s;
            afro = fma(v[j][s], v[j][s], afro);
            if (r < n && c < n) F(r, c) = (float)v[j][s];
          }
      }
      if (n < NP) {  // identity padding
        for (int r = 0; r < NP; ++r)
#pragma unroll
          for (int s = 0; s < MR; ++s) {
            const int c = lane + 32 * s;
            if (c < NP && (r >= n || c >= n)) F(r, c) = (r == c) ? 1.f : 0.f;
          }
      }
      for (int o = 16; o > 0; o >>= 1) afro += __shfl_xor_sync(kFull, afro, o);
      __syncwarp();
      // row scales: each lane scans its own rows with 16-byte reads
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int r = lane + 32 * s;
        float mx = 0.f;
        if (r < n) {
#pragma unroll
          for (int c = 0; c < NP; c += 4) {
            const float4 v = F4(r, c);
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
          }
        }
        int e = 0;
        frexpf(mx, &e);
        rsc[s] = (r < n && mx > 0.f && isfinite(mx)) ? ldexpf(1.f, -e) : 1.f;
        if (r < NP) rsd[r] = rsc[s];
      }
      __syncwarp();
      // apply the row scales and take column maxima (lanes: 4 columns x RPI rows)
      float cm[4] = {0.f, 0.f, 0.f, 0.f};
      if (q4 < CG) {
        for (int r = rho; r < NP; r += RPI) {
          float4 v = F4(r, 4 * q4);
          const float sc = rsd[r];
          v.x *= sc; v.y *= sc; v.z *= sc; v.w *= sc;
          F4(r, 4 * q4) = v;
          cm[0] = fmaxf(cm[0], fabsf(v.x));
          cm[1] = fmaxf(cm[1], fabsf(v.y));
          cm[2] = fmaxf(cm[2], fabsf(v.z));
          cm[3] = fmaxf(cm[3], fabsf(v.w));
        }
      }
#pragma unroll
      for (int o = CGP; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) cm[i] = fmaxf(cm[i], __shfl_xor_sync(kFull, cm[i], o));
      if (rho == 0 && q4 < CG) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = 4 * q4 + i;
          int e = 0;
          frexpf(cm[i], &e);
          // SPD keeps symmetry: D A D with D the row scales
          const float cs = SPD ? rsd[c] : ((c < n && cm[i] > 0.f && isfinite(cm[i])) ? ldexpf(1.f, -e) : 1.f);
          csc[c] = cs;
        }
      }
      __syncwarp();
      if (q4 < CG) {
        const float4 cs = *reinterpret_cast<const float4*>(csc + 4 * q4);
        for (int r = rho; r < NP; r += RPI) {
          float4 v = F4(r, 4 * q4);
          v.x *= cs.x; v.y *= cs.y; v.z *= cs.z; v.w *= cs.w;
          F4(r, 4 * q4) = v;
        }
      }
      __syncwarp();
    }
    double bv[MR];
    double bnrm = 0.0;
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s;
      bv[s] = (r < n) ? Bg[r] : 0.0;
      bnrm = fma(bv[s], bv[s], bnrm);
    }
    for (int o = 16; o > 0; o >>= 1) bnrm += __shfl_xor_sync(kFull, bnrm, o);
    afro = sqrt(afro);
    bnrm = sqrt(bnrm);

    // ------------------------------------------------ 2. low-precision factor
    unsigned act[MR];  // key mask of the lane's rows, 0 once retired
#pragma unroll
    for (int s = 0; s < MR; ++s) act[s] = lane + 32 * s < NP ? 0x7fffffffu : 0u;
    int info = 0;
    for (int k0 = 0; k0 < NP; k0 += PB) {
      // a row's panel columns, two to a register pair
      U2::E pan[MR][PB / 2];
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int rr = (lane + 32 * s < NP) ? lane + 32 * s : 0;
#pragma unroll
        for (int i0 = 0; i0 < PB; i0 += 4) {
          const Unit2<U2::E> v = lds16(Fu + rr * RSF + (k0 + i0) * 4, U2::E());
          pan[s][i0 / 2] = v.x;
          pan[s][i0 / 2 + 1] = v.y;
        }
      }
#pragma unroll
      for (int i = 0; i < PB; ++i) {
        const int k = k0 + i;
        int wr = k;  // SPD: no pivoting (A = L U with U = D L^T)
        float x[MR];
        bool win[MR];
#pragma unroll
        for (int s = 0; s < MR; ++s) x[s] = U2::get(pan[s][i / 2], i % 2);
        if (!SPD) {
          // the largest |a_ik| by its bits (a NaN is larger than all), ties by position
          unsigned key[MR], m = 0, b[MR];
#pragma unroll
          for (int s = 0; s < MR; ++s) {
            key[s] = __float_as_uint(x[s]) & act[s];
            m = max(m, key[s]);
          }
          m = __reduce_max_sync(kFull, m);
#pragma unroll
          for (int s = 0; s < MR; ++s) {
            win[s] = key[s] == m;
            b[s] = __ballot_sync(kFull, win[s]);
          }
          Seg g;
          g.lane = lane;
          g.segbase = 0;
          if (!one_row<32, MR>(b, g, wr)) {
            int bp = 0x7fffffff;
            int q[MR];
#pragma unroll
            for (int s = 0; s < MR; ++s) {
              q[s] = (act[s] && key[s] == m) ? position_of(ord, lane + 32 * s, k) : 0x7fffffff;
              bp = min(bp, q[s]);
            }
            __syncwarp();
            bp = __reduce_min_sync(kFull, bp);
#pragma unroll
            for (int s = 0; s < MR; ++s) {
              win[s] = q[s] == bp;
              b[s] = __ballot_sync(kFull, win[s]);
            }
            one_row<32, MR>(b, g, wr);
          }
        } else {
#pragma unroll
          for (int s = 0; s < MR; ++s) win[s] = lane + 32 * s == k;
        }
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          if (win[s]) {
#pragma unroll
            for (int j = 0; j < PB; j += 4) sts16(Fu + (lane + 32 * s) * RSF + (k0 + j) * 4, pan[s][j / 2], pan[s][j / 2 + 1]);
            act[s] = 0u;
            ord[k] = lane + 32 * s;
          }
        }
        __syncwarp();
        U2::E u[PB / 2];
#pragma unroll
        for (int j = i & ~3; j < PB; j += 4) {
          const Unit2<U2::E> v = lds16(Fu + wr * RSF + (k0 + j) * 4, U2::E());
          u[j / 2] = v.x;
          u[j / 2 + 1] = v.y;
        }
        const float piv = U2::get(u[i / 2], i % 2);
        const bool zero = SPD ? (!(piv > 0.f) || !isfinite(piv)) : (!(piv != 0.f) || !isfinite(piv));
        if (zero && info == 0) info = k + 1;
        float ry = rcp_in_range(piv);
        const unsigned pb = abs_hi(piv);
        if (pb - DivRange<float>::kLo > DivRange<float>::kHi - DivRange<float>::kLo) ry = 1.f / piv;
        if (zero) ry = 0.f;
        // retired rows are in shared memory: what their registers hold is not used again
#pragma unroll
        for (int s = 0; s < MR; ++s) {
          const float l = x[s] * ry;
          U2::set(pan[s][i / 2], i % 2, l);
          if (i % 2 == 0) U2::set(pan[s][i / 2], 1, fmaf(-l, U2::get(u[i / 2], 1), U2::get(pan[s][i / 2], 1)));
          const U2::E nl = U2::dup(-l);
#pragma unroll
          for (int j = i / 2 + 1; j < PB / 2; ++j) pan[s][j] = U2::fma(nl, u[j], pan[s][j]);
        }
      }
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        if (!act[s]) continue;
#pragma unroll
        for (int i0 = 0; i0 < PB; i0 += 4) sts16(Fu + (lane + 32 * s) * RSF + (k0 + i0) * 4, pan[s][i0 / 2], pan[s][i0 / 2 + 1]);
      }
      __syncwarp();
      const int j1 = k0 + PB;
      if (j1 >= NP) continue;
      int ordp[PB];  // physical rows of the panel's pivots
#pragma unroll
      for (int i = 0; i < PB; ++i) ordp[i] = ord[k0 + i];
      {
        // U12: the panel's pivot rows on the trailing columns (unit-lower solve)
        for (int j = j1 + lane; j < NP; j += 32) {
          float u[PB];
#pragma unroll
          for (int i = 0; i < PB; ++i) {
            float acc = F(ordp[i], j);
#pragma unroll
            for (int i0 = 0; i0 < i; i0 += 4) {
              const float4 l = F4(ordp[i], k0 + i0);
              const float ll[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (i0 + e < i) acc = fmaf(-ll[e], u[i0 + e], acc);
            }
            u[i] = acc;
            if (i > 0) F(ordp[i], j) = acc;
          }
        }
        __syncwarp();
      }
      // trailing update of the rows still active
      if (tc) {
        const int g = lane >> 2, tq = lane & 3;
        unsigned ab[MR];
#pragma unroll
        for (int s = 0; s < MR; ++s) ab[s] = __ballot_sync(kFull, act[s] != 0);
#pragma unroll
        for (int rt = 0; rt < NP / 16; ++rt) {
          const int ra = rt * 16 + g, rb = ra + 8;
          // rows still being updated: those not yet retired
          const bool sa = (ab[ra >> 5] >> (ra & 31)) & 1u, sb = (ab[rb >> 5] >> (rb & 31)) & 1u;
          // L21 fragment (negated): rows ra/rb, panel columns k0 + [2tq, 2tq+1, 2tq+8, 2tq+9]
          unsigned af[4];
          af[0] = pack2(-F(ra, k0 + 2 * tq), -F(ra, k0 + 2 * tq + 1), f16);
          af[1] = pack2(-F(rb, k0 + 2 * tq), -F(rb, k0 + 2 * tq + 1), f16);
          af[2] = pack2(-F(ra, k0 + 2 * tq + 8), -F(ra, k0 + 2 * tq + 9), f16);
          af[3] = pack2(-F(rb, k0 + 2 * tq + 8), -F(rb, k0 + 2 * tq + 9), f16);
          for (int ct = j1 / 8; ct < NP / 8; ++ct) {
            const int c0 = ct * 8 + 2 * tq;
            // U12 fragment: B[k][n] = U(k0+k, col ct*8+g)
            unsigned bf[2];
            const int cg = ct * 8 + g;
            bf[0] = pack2(F(ord[k0 + 2 * tq], cg), F(ord[k0 + 2 * tq + 1], cg), f16);
            bf[1] = pack2(F(ord[k0 + 2 * tq + 8], cg), F(ord[k0 + 2 * tq + 9], cg), f16);
            float d[4] = {F(ra, c0), F(ra, c0 + 1), F(rb, c0), F(rb, c0 + 1)};
            mma16816(d, af, bf, f16);
            if (sa) { F(ra, c0) = d[0]; F(ra, c0 + 1) = d[1]; }
            if (sb) { F(rb, c0) = d[2]; F(rb, c0 + 1) = d[3]; }
          }
        }
      } else {
        // fp32 CUDA-core update, 8 columns at a time; each pivot-row segment is read
        // once for all of a lane's rows
        for (int jc = j1; jc < NP; jc += 8) {
          U2::E acc[MR][4];
#pragma unroll
          for (int s = 0; s < MR; ++s) {
            const int r = (lane + 32 * s < NP) ? lane + 32 * s : 0;
#pragma unroll
            for (int h = 0; h < 4; h += 2) {
              const Unit2<U2::E> v = lds16(Fu + r * RSF + (jc + 2 * h) * 4, U2::E());
              acc[s][h] = v.x;
              acc[s][h + 1] = v.y;
            }
          }
#pragma unroll
          for (int i = 0; i < PB; ++i) {
            const Unit2<U2::E> v0 = lds16(Fu + ordp[i] * RSF + jc * 4, U2::E());
            const Unit2<U2::E> v1 = lds16(Fu + ordp[i] * RSF + (jc + 4) * 4, U2::E());
#pragma unroll
            for (int s = 0; s < MR; ++s) {
              const U2::E nl = U2::dup(-U2::get(pan[s][i / 2], i % 2));
              acc[s][0] = U2::fma(nl, v0.x, acc[s][0]);
              acc[s][1] = U2::fma(nl, v0.y, acc[s][1]);
              acc[s][2] = U2::fma(nl, v1.x, acc[s][2]);
              acc[s][3] = U2::fma(nl, v1.y, acc[s][3]);
            }
          }
#pragma unroll
          for (int s = 0; s < MR; ++s) {
            if (!act[s]) continue;
            sts16(Fu + (lane + 32 * s) * RSF + jc * 4, acc[s][0], acc[s][1]);
            sts16(Fu + (lane + 32 * s) * RSF + (jc + 4) * 4, acc[s][2], acc[s][3]);
          }
        }
      }
      __syncwarp();
    }
    if (p.info && lane == 0) p.info[m] = info;
    // from here on lane l owns positions l and l + 32: their rows of the factor and
    // reciprocal pivots
    __syncwarp();
    unsigned rowp[MR];
    float rinv[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int k = lane + 32 * s < NP ? lane + 32 * s : NP - 1;
      rowp[s] = Fu + ord[k] * RSF;
      rinv[s] = 1.f / F(ord[k], k);
    }

    // ---------------------------------------- 3./4. solve and refine in fp64
    // lowsolve(v): v = D_r * rhs by physical row in; the scaled solution by position out
    auto lowsolve = [&](float* v) {
#pragma unroll
      for (int s = 0; s < MR; ++s)
        if (lane + 32 * s < NP) rsd[lane + 32 * s] = v[s];
      __syncwarp();
#pragma unroll
      for (int s = 0; s < MR; ++s) v[s] = lane + 32 * s < NP ? rsd[ord[lane + 32 * s]] : 0.f;
      // forward: y_k, then positions after k take -L(k', k) y_k
#pragma unroll
      for (int t2 = 0; t2 < MR; ++t2) {
        const int top = 32 * (t2 + 1) < NP ? 32 * (t2 + 1) : NP;
#pragma unroll 2
        for (int kb = 32 * t2; kb < top; kb += 4) {
          Unit2<U2::E> lv[MR];
#pragma unroll
          for (int s = t2; s < MR; ++s) lv[s] = lds16(rowp[s] + kb * 4, U2::E());
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int kl = kb + q - 32 * t2;
            const float y = __shfl_sync(kFull, v[t2], kl);
#pragma unroll
            for (int s = t2; s < MR; ++s) {
              const float w = fmaf(-U2::get(q / 2 ? lv[s].y : lv[s].x, q % 2), y, v[s]);
              v[s] = (s > t2 || lane > kl) ? w : v[s];
            }
          }
        }
      }
      // backward: x_k = y_k / U(k, k), then positions before k take -U(k', k) x_k
#pragma unroll
      for (int t2 = MR - 1; t2 >= 0; --t2) {
        const int top = 32 * (t2 + 1) < NP ? 32 * (t2 + 1) : NP;
#pragma unroll 2
        for (int kb = top - 4; kb >= 32 * t2; kb -= 4) {
          Unit2<U2::E> uv[MR];
#pragma unroll
          for (int s = 0; s <= t2; ++s) uv[s] = lds16(rowp[s] + kb * 4, U2::E());
#pragma unroll
          for (int q = 3; q >= 0; --q) {
            const int kl = kb + q - 32 * t2;
            const float x = __shfl_sync(kFull, v[t2] * rinv[t2], kl);
#pragma unroll
            for (int s = 0; s <= t2; ++s) {
              const float w = fmaf(-U2::get(q / 2 ? uv[s].y : uv[s].x, q % 2), x, v[s]);
              v[s] = (s < t2 || lane < kl) ? w : v[s];
            }
          }
        }
      }
#pragma unroll
      for (int s = 0; s < MR; ++s) v[s] = v[s] * rinv[s];
      __syncwarp();
    };
    // unscale the solution into xs
    auto gather = [&](const float* v, bool add) {
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int kk = lane + 32 * s;
        if (kk >= n) continue;
        const double xk = (double)v[s] * (double)csc[kk];
        xs[kk] = add ? xs[kk] + xk : xk;
      }
      __syncwarp();
    };
    // r = b - A x for the lane's rows lane + 32 s. Rows are read coalesced (lane c
    // multiplies columns c, c + 32) in chunks of 16; a transposing butterfly folds the
    // 16 partial sums of each lane so that lanes 2i and 2i + 1 both end with row
    // 16 ch + i, and one shuffle per chunk hands each row to its owning lane.
    auto residual = [&](double* rr) {
      constexpr int NCH = NP / 16;
      double xl[MR];
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int c = lane + 32 * s;
        xl[s] = (c < n) ? xs[c] : 0.0;
      }
      double cv[NCH];
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        double pp[16];
#pragma unroll
        for (int h = 0; h < 16; h += 8) {
          double v[8][MR];
          load_rows<8, MR>(Ag, n, 16 * ch + h, lane, v);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            double acc = 0.0;
#pragma unroll
            for (int s = 0; s < MR; ++s) acc = fma(v[j][s], xl[s], acc);
            pp[h + j] = acc;
          }
        }
#pragma unroll
        for (int o = 16, w = 8; w >= 1; o >>= 1, w >>= 1) {
          const bool up = (lane & o) != 0;
#pragma unroll
          for (int j = 0; j < w; ++j) {
            const double send = up ? pp[j] : pp[j + w];
            const double keep = up ? pp[j + w] : pp[j];
            pp[j] = keep + __shfl_xor_sync(kFull, send, o);
          }
        }
        cv[ch] = pp[0] + __shfl_xor_sync(kFull, pp[0], 1);
      }
      // row lane + 32 s is row (lane & 15) of chunk 2 s + (lane >> 4) (chunk 0 only for NP = 16)
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int r = lane + 32 * s;
        const double a = __shfl_sync(kFull, cv[(2 * s) < NCH ? 2 * s : NCH - 1], 2 * (lane & 15));
        const double b = __shfl_sync(kFull, cv[(2 * s + 1) < NCH ? 2 * s + 1 : NCH - 1], 2 * (lane & 15));
        const double sum = (lane >> 4) ? b : a;
        rr[s] = (r < n) ? bv[s] - sum : 0.0;
      }
    };
    float v[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s;
      v[s] = (r < n) ? (float)(bv[s] * (double)rsc[s]) : 0.f;
    }
    lowsolve(v);
    gather(v, false);
    int steps = 0;
    double be = 1.0, be_prev = 1e300;
    bool conv = false;
    for (int it = 0; it <= p.itmax + 1; ++it) {
      double rr[MR];
      residual(rr);
      double rn = 0.0, xn = 0.0;
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        rn = fma(rr[s], rr[s], rn);
        const int c = lane + 32 * s;
        if (c < n) xn = fma(xs[c], xs[c], xn);
      }
      for (int o = 16; o > 0; o >>= 1) {
        rn += __shfl_xor_sync(kFull, rn, o);
        xn += __shfl_xor_sync(kFull, xn, o);
      }
      be = sqrt(rn) / (afro * sqrt(xn) + bnrm);
      // converged once below tol AND at the fp64 floor: the last correction no longer
      // halved the backward error (or it is already below a quarter unit roundoff)
      if (be <= p.tol && (be > 0.5 * be_prev || be <= 0x1p-55)) { conv = true; break; }
      if (info != 0 || !(be < be_prev)) { conv = be <= p.tol; break; }
      if (steps == p.itmax + (be <= p.tol ? 1 : 0)) { conv = be <= p.tol; break; }
      be_prev = be;
      ++steps;
#pragma unroll
      for (int s = 0; s < MR; ++s) {
        const int r = lane + 32 * s;
        v[s] = (r < n) ? (float)(rr[s] * (double)rsc[s]) : 0.f;
      }
      lowsolve(v);
      gather(v, true);
    }
    if (lane == 0) {
      if (p.status) p.status[m] = (conv && info == 0) ? steps : -1;
      if (p.bwd) p.bwd[m] = be;
    }
    if (conv && info == 0)
      for (int c = lane; c < n; c += 32) Bg[c] = xs[c];
    __syncwarp();
  }
}

}  // namespace dev
}  // namespace tsdx
