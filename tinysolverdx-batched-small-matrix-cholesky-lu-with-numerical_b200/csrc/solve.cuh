// Triangular solves from an existing factor: potrs (L L^T x = b) and getrs
// (P L U x = b) — TinySolverDx kernels.hpp:184-227 driven by batched.hpp:248-268
// (which the reference always runs on the CPU; here they run on the GPU).
//
// Up to 16 right-hand sides at a time, one warp per matrix above order 12: the factor is
// staged to shared memory with cp.async, the right-hand sides live in registers. The forward
// substitution keeps the reference's chain (increasing k, fused multiply-add, and for
// Cholesky the division by l_ii); the backward substitution is column-oriented
// (decreasing k) and multiplies by the reciprocal of the diagonal, so X agrees with the
// reference to rounding.
//
//   float64: the right-hand sides are 8 x 8 accumulator tiles of the FP64 tensor cores.
//     Blocks of 8 rows are solved in registers by every lane of a right-hand side; the
//     rows below (above) take the block by one tile product per 8 rows, which
//     accumulates its four products in fragment order as fused multiply-adds (see
//     blk_tc.cuh); the backward pass numbers the fragments downwards. So every element
//     keeps its chain of operations.
//   float32: lane l owns rows l and l + 32; the solved row goes through shared memory
//     (which keeps it as the result) and every lane updates its rows, two columns to an
//     instruction.
//   Orders up to 12, both types: a lane per right-hand side, as many matrices in a warp as
//     that leaves room for.
#pragma once
#include "blk_tc.cuh"
#include "rows.cuh"

namespace tsdx {
namespace dev {

template <class T, int NP>
struct TrsCfg {
  static constexpr int RS = NP * int(sizeof(T)) + 16;  // an odd number of 16-byte units
  static constexpr int MAT = NP * RS;
  static constexpr int XB = 16 * int(sizeof(T));       // one solved row (float32)
  static constexpr int OFF_X = MAT, OFF_PERM = MAT + (sizeof(T) == 4 ? NP * XB : 0);
  static constexpr int WARPB = (OFF_PERM + 2 * NP * 4 + 127) / 128 * 128;
  static_assert(NP % 8 == 0, "row stride in an odd number of 16-byte units");
};

// Stages the factor, identity-padded to order np <= NP (a multiple of 4), and for LU the row that the pivots bring to
// each position: kernels.hpp:207-213 swaps rows j and piv[j] in increasing j, so a
// position's origin is found by following it backwards through the swaps. All positions
// are traced at once, one swap at a time; a pivot outside [0, n) is ignored.
template <class T, int NP, bool LU>
__device__ __forceinline__ void trs_stage(unsigned char* M, const T* A, const int* piv, int n, int np, int lane) {
  using C = TrsCfg<T, NP>;
  constexpr int RS = C::RS, TS = int(sizeof(T)), MR = (NP + 31) / 32;
  const int vec = vec_of<T>(A, n), rowb = n * TS;
  const char* src = reinterpret_cast<const char*>(A);
  if (vec == 16) walk_chunks<T, NP, 32, 16>(n, lane, [&](int r, int c) { cp_async<16>(M + r * RS + c * 16, src + r * rowb + c * 16); });
  else if (vec == 8) walk_chunks<T, NP, 32, 8>(n, lane, [&](int r, int c) { cp_async<8>(M + r * RS + c * 8, src + r * rowb + c * 8); });
  else if constexpr (sizeof(T) == 4) walk_chunks<T, NP, 32, 4>(n, lane, [&](int r, int c) { cp_async<4>(M + r * RS + c * 4, src + r * rowb + c * 4); });
  cp_async_commit();
  if (n < np) {
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s;
      T* row = reinterpret_cast<T*>(M + r * RS);
      if (r < n) {
        for (int c = n; c < np; ++c) row[c] = T(0);
      } else if (r < np) {
        for (int c = 0; c < np * TS / 16; ++c) reinterpret_cast<uint4*>(row)[c] = make_uint4(0, 0, 0, 0);
        row[r] = T(1);
      }
    }
  }
  if constexpr (LU) {
    int* pv = reinterpret_cast<int*>(M + C::OFF_PERM);
    int* perm = pv + NP;
    int q[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int k = lane + 32 * s;
      q[s] = k;
      if (k < n) {
        const int v = piv[k];
        if (v >= 0 && v < n) q[s] = v;
      }
      if (k < np) pv[k] = q[s];
      q[s] = k;
    }
    __syncwarp();
#pragma unroll 1
    for (int j0 = np - 4; j0 >= 0; j0 -= 4) {
      const int4 pj = *reinterpret_cast<const int4*>(pv + j0);
      const int pp[4] = {pj.x, pj.y, pj.z, pj.w};
#pragma unroll
      for (int j = 3; j >= 0; --j)
#pragma unroll
        for (int s = 0; s < MR; ++s) q[s] = q[s] == j0 + j ? pp[j] : (q[s] == pp[j] ? j0 + j : q[s]);
    }
#pragma unroll
    for (int s = 0; s < MR; ++s)
      if (lane + 32 * s < np) perm[lane + 32 * s] = q[s];
  }
}

// ---------------------------------------------------------------- float64
// NT tiles of 8 right-hand sides, transposed: lane (fr, fq) holds right-hand side fr of a
// tile at positions 8 I + 2 fq and 8 I + 2 fq + 1 of every block I. The four lanes of a
// right-hand side gather its 8 values of a block and each solves it in registers: one
// exchange per block, where the right-hand sides along the lanes took one per position
// (getrs n = 48, 12 right-hand sides, 32,768 matrices 387 -> 372 us). The reciprocals of
// the diagonal stand in the rows' padding. Orders run in the next multiple of 8 (one
// block): a block too many costs its loads, products and exchanges.
template <int NP, int NT, bool LU, int WPC>
__global__ void __launch_bounds__(WPC * 32, 1) trs_f64_kernel(SolveArgs<double> p) {
  using C = TrsCfg<double, NP>;
  constexpr int RS = C::RS, NB = NP / 8;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31, wpc = blockDim.x >> 5;
  const int fr = lane >> 2, fq = lane & 3;
  unsigned char* M = smem + warp * C::WARPB;
  const int* perm = reinterpret_cast<const int*>(M + C::OFF_PERM) + NP;
  auto at = [&](int r, int c) -> double { return *reinterpret_cast<const double*>(M + r * RS + c * 8); };
  const int n = p.n;
  const long long nn = (long long)n * n, step = (long long)gridDim.x * wpc;

  for (long long m = (long long)blockIdx.x * wpc + warp; m < p.batch; m += step) {
    if (lane == 0 && m + step < p.batch) {
      prefetch_l2(p.A + (m + step) * nn, nn * 8);
      prefetch_l2(p.B + (m + step) * (long long)n * p.ldb, (long long)n * p.ldb * 8);
    }
    trs_stage<double, NP, LU>(M, p.A + m * nn, LU ? p.piv + m * n : nullptr, n, NP, lane);
    if (LU) __syncwarp();
    double* Bm = p.B + m * (long long)n * p.ldb + p.b0;
    double2 c[NB][NT];
#pragma unroll
    for (int I = 0; I < NB; ++I) {
      const int r = 8 * I + 2 * fq;
      const int2 o = LU ? *reinterpret_cast<const int2*>(perm + r) : make_int2(r, r + 1);
      const double* row0 = Bm + (long long)o.x * p.ldb + fr;
      const double* row1 = Bm + (long long)o.y * p.ldb + fr;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        c[I][t].x = (r < n && 8 * t + fr < p.nrhs) ? row0[8 * t] : 0.0;
        c[I][t].y = (r + 1 < n && 8 * t + fr < p.nrhs) ? row1[8 * t] : 0.0;
      }
    }
    cp_async_wait<0>();
    __syncwarp();
#pragma unroll
    for (int s = 0; s < (NP + 31) / 32; ++s) {
      const int r = lane + 32 * s;
      if (r < NP) *reinterpret_cast<double*>(M + r * RS + NP * 8) = rcp_(at(r, r));
    }
    __syncwarp();

    auto rcpd = [&](int r) { return at(r, NP); };
    auto gather = [&](const double2& v, double (&x)[8]) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        x[2 * q] = __shfl_sync(kFull, v.x, (lane & ~3) | q);
        x[2 * q + 1] = __shfl_sync(kFull, v.y, (lane & ~3) | q);
      }
    };
    auto of4 = [&](double a, double b, double e, double f) { return (fq & 2) ? ((fq & 1) ? f : e) : ((fq & 1) ? b : a); };
    // the block's strict lower (upper) triangle, row by row
    auto lower = [&](int K, double (&l)[8][8]) {
#pragma unroll
      for (int i = 1; i < 8; ++i)
#pragma unroll
        for (int q = 0; q < i; q += 2) {
          const double2 v = *reinterpret_cast<const double2*>(M + (8 * K + i) * RS + (8 * K + q) * 8);
          l[i][q] = v.x;
          l[i][q + 1] = v.y;
        }
    };
    // forward: L y = P b
#pragma unroll
    for (int K = 0; K < NB; ++K) {
      double l[8][8], a0[NT], a1[NT];
      lower(K, l);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        double x[8];
        gather(c[K][t], x);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if constexpr (!LU) x[q] = div_by(x[q], at(8 * K + q, 8 * K + q), rcpd(8 * K + q));
#pragma unroll
          for (int i = q + 1; i < 8; ++i) x[i] = fma_(-l[i][q], x[q], x[i]);
        }
        a0[t] = of4(x[0], x[1], x[2], x[3]);
        a1[t] = of4(x[4], x[5], x[6], x[7]);
        c[K][t] = make_double2(of4(x[0], x[2], x[4], x[6]), of4(x[1], x[3], x[5], x[7]));
      }
#pragma unroll
      for (int I = K + 1; I < NB; ++I) {
        const double b0 = -at(8 * I + fr, 8 * K + fq), b1 = -at(8 * I + fr, 8 * K + 4 + fq);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          dmma_m8n8k4(c[I][t], a0[t], b0);
          dmma_m8n8k4(c[I][t], a1[t], b1);
        }
      }
    }
    // the padded positions have taken 0 * y, NaN where y is not finite: zero again, or the
    // backward pass, which starts with them, would carry it into every position
#pragma unroll
    for (int I = 0; I < NB; ++I) {
      const int r = 8 * I + 2 * fq;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        c[I][t].x = r < n ? c[I][t].x : 0.0;
        c[I][t].y = r + 1 < n ? c[I][t].y : 0.0;
      }
    }
    // backward: U x = y (LU) or L^T x = y (Cholesky), columns in decreasing order
#pragma unroll
    for (int K = NB - 1; K >= 0; --K) {
      double u[8][8], d[8], a0[NT], a1[NT];
      if constexpr (LU) {
#pragma unroll
        for (int i = 0; i < 7; ++i)
#pragma unroll
          for (int q = (i + 1) & ~1; q < 8; q += 2) {
            const double2 v = *reinterpret_cast<const double2*>(M + (8 * K + i) * RS + (8 * K + q) * 8);
            u[i][q] = v.x;
            u[i][q + 1] = v.y;
          }
      } else {
        lower(K, u);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) d[q] = rcpd(8 * K + q);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        double x[8];
        gather(c[K][t], x);
#pragma unroll
        for (int q = 7; q >= 0; --q) {
          x[q] = x[q] * d[q];
#pragma unroll
          for (int i = q - 1; i >= 0; --i) x[i] = fma_(-(LU ? u[i][q] : u[q][i]), x[q], x[i]);
        }
        a0[t] = of4(x[7], x[6], x[5], x[4]);
        a1[t] = of4(x[3], x[2], x[1], x[0]);
        if (8 * t + fr < p.nrhs) {
          double* out = Bm + (long long)(8 * K + 7 - fq) * p.ldb + 8 * t + fr;
          if (8 * K + 7 - fq < n) out[0] = a0[t];
          if (8 * K + 3 - fq < n) out[-4ll * p.ldb] = a1[t];
        }
      }
#pragma unroll
      for (int I = K - 1; I >= 0; --I) {
        const double b0 = LU ? -at(8 * I + fr, 8 * K + 7 - fq) : -at(8 * K + 7 - fq, 8 * I + fr);
        const double b1 = LU ? -at(8 * I + fr, 8 * K + 3 - fq) : -at(8 * K + 3 - fq, 8 * I + fr);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          dmma_m8n8k4(c[I][t], a0[t], b0);
          dmma_m8n8k4(c[I][t], a1[t], b1);
        }
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- float32
// NRHS columns in units of two (one: a single scalar column, exchanged by shuffle).
template <int NP, int NRHS, bool LU, int WPC>
__global__ void __launch_bounds__(WPC * 32, 1) trs_f32_kernel(SolveArgs<float> p) {
  using C = TrsCfg<float, NP>;
  using U = Unit<float>;
  using E = U::E;
  constexpr int RS = C::RS, XB = C::XB, MR = (NP + 31) / 32, NU = NRHS > 1 ? NRHS / 2 : 1;
  static_assert(NRHS == 1 || NRHS % 4 == 0, "whole 16-byte vectors");
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31, wpc = blockDim.x >> 5;
  unsigned char* M = smem + warp * C::WARPB;
  const unsigned Mu = (unsigned)__cvta_generic_to_shared(M), Xu = Mu + C::OFF_X;
  const int* perm = reinterpret_cast<const int*>(M + C::OFF_PERM) + NP;
  const int n = p.n, np = (n + 3) & ~3;  // the steps run to np
  const long long nn = (long long)n * n, step = (long long)gridDim.x * wpc;

  for (long long m = (long long)blockIdx.x * wpc + warp; m < p.batch; m += step) {
    if (lane == 0 && m + step < p.batch) {
      prefetch_l2(p.A + (m + step) * nn, nn * 4);
      prefetch_l2(p.B + (m + step) * (long long)n * p.ldb, (long long)n * p.ldb * 4);
    }
    trs_stage<float, NP, LU>(M, p.A + m * nn, LU ? p.piv + m * n : nullptr, n, np, lane);
    if (LU) __syncwarp();
    float* Bm = p.B + m * (long long)n * p.ldb + p.b0;
    E b[MR][NU];
    float b1[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s;
      const float* row = Bm + (long long)(LU && r < n ? perm[r] : r) * p.ldb;
      float v[NRHS > 1 ? NRHS : 2];
#pragma unroll
      for (int c = 0; c < NRHS; ++c) v[c] = (r < n && c < p.nrhs) ? row[c] : 0.f;
      b1[s] = v[0];
      if constexpr (NRHS > 1) {
#pragma unroll
        for (int c = 0; c < NU; ++c) b[s][c] = U::pack(v[2 * c], v[2 * c + 1]);
      }
    }
    cp_async_wait<0>();
    __syncwarp();
    float dg[MR], dinv[MR];
    unsigned own[MR], xown[MR];
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s < np ? lane + 32 * s : np - 1;
      own[s] = Mu + r * RS;
      xown[s] = Xu + r * XB;
      dg[s] = *reinterpret_cast<const float*>(M + r * RS + r * 4);
      dinv[s] = rcp_(dg[s]);
    }
    // forward: L y = P b; a row's y is final after its own step, where it is published
#pragma unroll
    for (int t = 0; t < MR; ++t) {
      const int top = min(32 * (t + 1), np);
#pragma unroll 1
      for (int k0 = 32 * t; k0 < top; k0 += 4) {
        Unit2<E> lv[MR];
#pragma unroll
        for (int s = t; s < MR; ++s) lv[s] = lds16(own[s] + k0 * 4, E());
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int kl = k0 + i - 32 * t;
          if constexpr (NRHS == 1) {
            const float y = __shfl_sync(kFull, LU ? b1[t] : div_by(b1[t], dg[t], dinv[t]), kl);
            if (!LU) b1[t] = lane == kl ? y : b1[t];
#pragma unroll
            for (int s = t; s < MR; ++s) {
              const float v = fma_(-U::get(i / 2 ? lv[s].y : lv[s].x, i % 2), y, b1[s]);
              b1[s] = (s > t || lane > kl) ? v : b1[s];
            }
          } else {
            if (lane == kl) {
#pragma unroll
              for (int c = 0; c < NU; c += 2) {
                E v0 = b[t][c], v1 = b[t][c + 1];
                if (!LU) {
                  v0 = U::pack(div_by(U::get(v0, 0), dg[t], dinv[t]), div_by(U::get(v0, 1), dg[t], dinv[t]));
                  v1 = U::pack(div_by(U::get(v1, 0), dg[t], dinv[t]), div_by(U::get(v1, 1), dg[t], dinv[t]));
                }
                sts16(xown[t] + c * 8, v0, v1);
              }
            }
            __syncwarp();
            E nl[MR];
#pragma unroll
            for (int s = t; s < MR; ++s) nl[s] = U::dup(-U::get(i / 2 ? lv[s].y : lv[s].x, i % 2));
#pragma unroll
            for (int c = 0; c < NU; c += 2) {
              const Unit2<E> y = lds16(Xu + (k0 + i) * XB + c * 8, E());
#pragma unroll
              for (int s = t; s < MR; ++s) {
                b[s][c] = U::fma(nl[s], y.x, b[s][c]);
                b[s][c + 1] = U::fma(nl[s], y.y, b[s][c + 1]);
              }
            }
          }
        }
      }
    }
    // (positions past n: zero, as in the float64 kernel)
    if constexpr (NRHS > 1) {
#pragma unroll
      for (int s = 0; s < MR; ++s)
#pragma unroll
        for (int c = 0; c < NU; c += 2) {
          const Unit2<E> y = lds16(xown[s] + c * 8, E());
          b[s][c] = lane + 32 * s < n ? y.x : E(0);
          b[s][c + 1] = lane + 32 * s < n ? y.y : E(0);
        }
      __syncwarp();
    } else {
#pragma unroll
      for (int s = 0; s < MR; ++s) b1[s] = lane + 32 * s < n ? b1[s] : 0.f;
    }
    // backward: U x = y (LU) or L^T x = y (Cholesky)
#pragma unroll
    for (int t = MR - 1; t >= 0; --t) {
      const int top = min(32 * (t + 1), np);
#pragma unroll 1
      for (int k0 = top - 4; k0 >= 32 * t; k0 -= 4) {
        float uv[MR][4];
#pragma unroll
        for (int s = 0; s <= t; ++s) {
          if constexpr (LU) {
            const float4 v = *reinterpret_cast<const float4*>(M + (own[s] - Mu) + k0 * 4);
            uv[s][0] = v.x; uv[s][1] = v.y; uv[s][2] = v.z; uv[s][3] = v.w;
          } else {
            const int r = lane + 32 * s < np ? lane + 32 * s : np - 1;
#pragma unroll
            for (int i = 0; i < 4; ++i) uv[s][i] = *reinterpret_cast<const float*>(M + (k0 + i) * RS + r * 4);
          }
        }
#pragma unroll
        for (int i = 3; i >= 0; --i) {
          const int kl = k0 + i - 32 * t;
          if constexpr (NRHS == 1) {
            const float x = __shfl_sync(kFull, b1[t] * dinv[t], kl);
#pragma unroll
            for (int s = 0; s <= t; ++s) {
              const float v = fma_(-uv[s][i], x, b1[s]);
              b1[s] = (s < t || lane < kl) ? v : b1[s];
            }
            b1[t] = lane == kl ? x : b1[t];
          } else {
            if (lane == kl) {
              const E dd = U::dup(dinv[t]);
#pragma unroll
              for (int c = 0; c < NU; c += 2) sts16(xown[t] + c * 8, U::mul(b[t][c], dd), U::mul(b[t][c + 1], dd));
            }
            __syncwarp();
            E nu[MR];
#pragma unroll
            for (int s = 0; s <= t; ++s) nu[s] = U::dup(-uv[s][i]);
#pragma unroll
            for (int c = 0; c < NU; c += 2) {
              const Unit2<E> x = lds16(Xu + (k0 + i) * XB + c * 8, E());
#pragma unroll
              for (int s = 0; s <= t; ++s) {
                b[s][c] = U::fma(nu[s], x.x, b[s][c]);
                b[s][c + 1] = U::fma(nu[s], x.y, b[s][c + 1]);
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int s = 0; s < MR; ++s) {
      const int r = lane + 32 * s;
      if (r >= n) continue;
      float* row = Bm + (long long)r * p.ldb;
      const float* x = reinterpret_cast<const float*>(M + C::OFF_X + r * XB);
#pragma unroll
      for (int c = 0; c < NRHS; ++c)
        if (c < p.nrhs) row[c] = NRHS == 1 ? b1[s] : x[c];
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- orders up to 12
// A lane per right-hand side and matrix: lg = log2 of the lanes per matrix (the right-hand
// sides rounded up to a power of two), 32 >> lg matrices per warp, all of a lane's column
// in registers, the factors of the unit as one run of elements in shared memory. No
// exchange between lanes and no padding; the operations and their order are those of the
// kernels above. With a warp per matrix and its padded tile, most lanes and most of the
// steps of these orders do nothing. Copies of the factors bound it, and for one right-hand
// side the shared memory of 32 matrices a warp. Against the warp per matrix and, before
// that one's padding, its unpadded form: float32 potrs, 400,000 matrices, 8 right-hand
// sides, n = 2 1486 and 318 us; n = 9, 12 right-hand sides 2007 and 1795, here 229; float64
// getrs, one right-hand side, n = 4, 400,000 matrices 488 and 253; n = 9, 231,481 matrices
// 304 and 262, here 52; n = 12, 130,208 matrices 178 and 182, here 57.
constexpr int kSmallWpc = 4;
__host__ __device__ constexpr int trs_small_stride(int n) { return (n * n) | 1; }  // elements: odd, for the banks
__host__ __device__ constexpr int trs_small_elems(int n, int lg) { return (32 >> lg) * trs_small_stride(n); }

template <class T, int NP, bool LU>
__global__ void __launch_bounds__(kSmallWpc * 32) trs_small_kernel(SolveArgs<T> p, int lg) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31, wpc = blockDim.x >> 5;
  const int n = p.n, nn = n * n, stride = trs_small_stride(n), S = 32 >> lg;
  T* F = reinterpret_cast<T*>(smem) + warp * trs_small_elems(n, lg);
  const T* own = F + (lane >> lg) * stride;
  const int col = lane & ((1 << lg) - 1);
  const int dm = 32 / nn, de = 32 - dm * nn;  // 32 elements on
  const int m_first = lane / nn, e_first = lane - m_first * nn;
  const long long step = (long long)gridDim.x * wpc * S;
  for (long long m0 = ((long long)blockIdx.x * wpc + warp) * S; m0 < p.batch; m0 += step) {
    const int cnt = (int)(p.batch - m0 < S ? p.batch - m0 : S);
    {
      const T* src = p.A + m0 * nn;
      int at = m_first * stride + e_first, e = e_first;
#pragma unroll 4
      for (int i = lane; i < cnt * nn; i += 32) {
        cp_async<int(sizeof(T))>(F + at, src + i);
        e += de;
        const bool wrap = e >= nn;
        e -= wrap ? nn : 0;
        at += dm * stride + de + (wrap ? stride - nn : 0);
      }
      cp_async_commit();
    }
    const long long m = m0 + (lane >> lg);
    const bool live = (lane >> lg) < cnt && col < p.nrhs;
    T* b = p.B + (live ? m * n * p.ldb + p.b0 + col : 0);
    T y[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) y[i] = (live && i < n) ? b[i * p.ldb] : T(0);
    if constexpr (LU) {
      // swaps in increasing k; a pivot outside [0, n) is ignored
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const int q = (live && k < n) ? p.piv[m * n + k] : k;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          if (j == k) continue;
          const bool s = q == j && j < n;
          const T t = y[k];
          y[k] = s ? y[j] : t;
          y[j] = s ? t : y[j];
        }
      }
    }
    cp_async_wait<0>();
    __syncwarp();
    if (live) {
      T d[NP];
#pragma unroll
      for (int k = 0; k < NP; ++k) d[k] = k < n ? rcp_(own[k * n + k]) : T(0);
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        if (k >= n) break;
        if constexpr (!LU) y[k] = div_by(y[k], own[k * n + k], d[k]);
#pragma unroll
        for (int i = k + 1; i < NP; ++i)
          if (i < n) y[i] = fma_(-own[i * n + k], y[k], y[i]);
      }
#pragma unroll
      for (int k = NP - 1; k >= 0; --k) {
        if (k >= n) continue;
        y[k] = y[k] * d[k];
#pragma unroll
        for (int i = k - 1; i >= 0; --i) y[i] = fma_(-(LU ? own[i * n + k] : own[k * n + i]), y[k], y[i]);
      }
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (i < n) b[i * p.ldb] = y[i];
    }
    __syncwarp();
  }
}

}  // namespace dev
}  // namespace tsdx
