// Learned precision-tier selector: per-matrix features and a 24-64-64-4 MLP with
// its own inference, training (forward + backward) and Adam kernels.
//
// No reference counterpart: TinySolverDx has no mixed-precision path on the GPU.
// The network predicts, per matrix, the cheapest tier {fp16, bf16, fp32, fp64}
// whose refinement (ir.cuh) converges; the refinement's own residual check and
// fp64 fallback make every prediction safe, a wrong one only costs time.
//
// Features (one warp per matrix, one coalesced fp64 pass over A). With
// d_i = |a_ii|, r_i = sum_j |a_ij| (row 1-norm), R_i = r_i - d_i, c_j = sum_i |a_ij|,
// L(x) = log10(max(x, 1e-300)), every feature clipped to [-30, 30]:
//   0 n/64             1 kind (0 SPD, 1 general)   2 L(max d) - L(min d)
//   3 L(max r) - L(min r)    4 L(max c) - L(min c)
//   5 L(max|a|) - L(max d)   6 L(max|a|) - L(min d)  (pivot-growth proxies)
//   7 fraction of rows with d_i > R_i
//   8 min_i (d_i - R_i) / r_i      9 mean_i (d_i - R_i) / r_i   (Gershgorin margins)
//  10 L(max_i (d_i + R_i)) - L(min_i (d_i - R_i))  (Gershgorin bound ratio)
//  11 1 if min_i (d_i - R_i) <= 0                  12 L(||A||_F) - L(max r)
//  13 L(max d) - L(mean d)   14 L(mean d) - L(min d)
//  15 std_i L(d_i)   16 std_i L(r_i)   17 std_j L(c_j)
//  18 max_i (L(r_i) - L(d_i))   19 mean_i (L(r_i) - L(d_i))
//  20 L(||strict lower||_F) - L(||strict upper||_F)
//  21 L(min d) - L(mean_{i != j} |a_ij|)     22 fraction of d_i < 1e-8 max d
//  23 max_j (L(c_j) - L(d_j))
//
// Network (float32): x' = (x - mu) * isd; h1 = relu(W1^T x' + b1) (24 -> 64);
// h2 = relu(W2^T h1 + b2) (64 -> 64); logits = W3^T h2 + b3 (64 -> 4).
// Parameter vector layout: W1[24][64], b1[64], W2[64][64], b2[64], W3[64][4], b3[4].
// Loss: class-weighted softmax cross entropy, sum_s w_{y_s} CE_s / batch.
#pragma once
#include <cuda_runtime.h>

#include "rows.cuh"

namespace tsdx {
namespace dev {

constexpr int kFeat = 24, kHid = 64, kTiers = 4;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kFeat * kHid, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
              kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kTiers, kParams = kOffB3 + kTiers;  // 6020
constexpr int kTrainBlock = 64;   // samples per training block
constexpr int kTrainThreads = 256;

// log10(max(x, 1e-300)) to about 1e-7 absolute: the binary exponent exactly plus a
// single-precision log2 of the mantissa (NaN maps to the clamp, like fmax does).
__device__ __forceinline__ double lg10(double x) {
  if (!(x >= 1e-300)) return -300.0;
  if (x > 1.7976931348623157e308) return 309.0;
  int e = 0;
  const double m = frexp(x, &e);  // x = m 2^e, m in [0.5, 1)
  return ((double)e + (double)__log2f((float)m)) * 0.30102999566398120;
}
__device__ __forceinline__ float clip30(double x) {
  if (!(x == x)) return 0.f;
  return (float)fmin(30.0, fmax(-30.0, x));
}
// Folds 16 values of every lane over the warp (op: sum or max); lanes 2 i and 2 i + 1 end
// with value i. The same additions as one xor butterfly per value, in 31 exchanges
// instead of 80.
template <class Op>
__device__ __forceinline__ double fold16(double (&v)[16], int lane, Op op) {
#pragma unroll
  for (int o = 16, w = 8; w >= 1; o >>= 1, w >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < w; ++j) {
      const double send = up ? v[j] : v[j + w];
      const double keep = up ? v[j + w] : v[j];
      v[j] = op(keep, __shfl_xor_sync(0xffffffffu, send, o));
    }
  }
  return op(v[0], __shfl_xor_sync(0xffffffffu, v[0], 1));
}

// One warp per matrix, one coalesced pass over A in registers: lane c accumulates
// columns c and c + 32 (SL column slots), row 1-norms come from per-lane partial sums of
// 16-row chunks (fold16), then each row's norm is handed to the lane that owns it (row r:
// lane r % 32, slot r / 32, the same lane that holds the diagonal a_rr as part of column
// r). The matrix's sums and extremes are folded 16 at a time, their logarithms and then
// the 24 features are computed by one lane each: on one lane, as before, they cost more
// than the pass over A (n = 32, 131,072 matrices).
template <int WPC, int SL>
__global__ void __launch_bounds__(WPC * 32, 2) features_kernel(const double* __restrict__ A, int n, long long batch,
                                                            const signed char* kind, int kind_all, float* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double INF = __longlong_as_double(0x7ff0000000000000LL);
  const long long nn = (long long)n * n;
  const double fn = (double)n;
  auto add = [](double p, double q) { return p + q; };
  auto mx = [](double p, double q) { return fmax(p, q); };
  // quantities: sums S0.. dsum fro lo up gsum sld sld2 slr slr2 rgsum offs slc slc2;
  // maxima X0.. dmax rmax amax gup rgmax cmax cgmax -dmin -rmin -gmin -cmin -gnmin.
  // Lane i's logarithm: of dmax dmin rmax rmin cmax cmin amax gup gmin dmean sqrt(fro)
  // sqrt(lo) sqrt(up) mean off-diagonal, and lane f's feature: a difference of two of
  // them, or of a sum or maximum.
  const int logx = lane == 0 ? 0 : lane == 1 ? 7 : lane == 2 ? 1 : lane == 3 ? 8 : lane == 4 ? 5 : lane == 5 ? 10
                 : lane == 6 ? 2 : lane == 7 ? 3 : 9;
  const int logs = lane == 9 ? 0 : lane == 10 ? 1 : lane == 11 ? 2 : lane == 12 ? 3 : 10;
  const int la = lane == 2 || lane == 13 ? 0 : lane == 3 ? 2 : lane == 4 ? 4 : lane == 5 || lane == 6 ? 6
               : lane == 10 ? 7 : lane == 12 ? 10 : lane == 14 ? 9 : lane == 20 ? 11 : 1;
  const int lb = lane == 2 || lane == 6 || lane == 14 ? 1 : lane == 3 ? 3 : lane == 4 ? 5 : lane == 5 ? 0
               : lane == 10 ? 8 : lane == 12 ? 2 : lane == 13 ? 9 : lane == 20 ? 12 : 13;
  const int fs = lane == 9 ? 4 : lane == 15 ? 5 : lane == 16 ? 7 : lane == 17 ? 11 : 9;
  const int fs2 = lane == 15 ? 6 : lane == 16 ? 8 : 12;
  const int fx = lane == 8 ? 11 : lane == 11 ? 9 : lane == 18 ? 4 : 6;
  for (long long m = (long long)blockIdx.x * WPC + warp; m < batch; m += (long long)gridDim.x * WPC) {
    const double* Ag = A + m * nn;
    double csum[SL] = {}, cdg[SL] = {}, cv[2 * SL] = {};
    double amax = 0, lo = 0, up = 0;
#pragma unroll
    for (int ch = 0; ch < 2 * SL; ++ch) {
      if (16 * ch < n) {
        double pp[16], v[16][SL];
        load_rows<16, SL>(Ag, n, 16 * ch, lane, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int r = 16 * ch + j;
          double acc = 0;
#pragma unroll
          for (int s = 0; s < SL; ++s) {
            const int c = lane + 32 * s;
            const double av = fabs(v[j][s]), v2 = v[j][s] * v[j][s];
            acc += av;
            csum[s] += av;
            amax = fmax(amax, av);
            if (c < r) lo += v2;
            else if (c > r) up += v2;
            else cdg[s] = av;
          }
          pp[j] = acc;
        }
        cv[ch] = fold16(pp, lane, add);
      }
    }
    double S[16] = {}, X[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) X[i] = -INF;
    X[0] = X[1] = X[3] = X[5] = 0;
    X[2] = amax;
    S[1] = lo + up;
    S[2] = lo;
    S[3] = up;
    int dom = 0;
    double dg[SL];
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      const double a0 = __shfl_sync(0xffffffffu, cv[2 * s], 2 * (lane & 15));
      const double a1 = __shfl_sync(0xffffffffu, cv[2 * s + 1], 2 * (lane & 15));
      const int r = lane + 32 * s;  // row r and column r
      const double ra = (lane >> 4) ? a1 : a0, d = cdg[s], R = ra - d, g = d - R, ca = csum[s];
      dg[s] = d;
      dom += __popc(__ballot_sync(0xffffffffu, r < n && d > R));
      if (r < n) {
        const double ld = lg10(d), lr = lg10(ra), lc = lg10(ca);
        S[0] += d;
        S[1] += d * d;
        S[4] += (ra > 0) ? g / ra : 0.0;
        S[5] += ld;
        S[6] += ld * ld;
        S[7] += lr;
        S[8] += lr * lr;
        S[9] += lr - ld;
        S[10] += R;
        S[11] += lc;
        S[12] += lc * lc;
        X[0] = fmax(X[0], d);
        X[1] = fmax(X[1], ra);
        X[3] = fmax(X[3], d + R);
        X[4] = fmax(X[4], lr - ld);
        X[5] = fmax(X[5], ca);
        X[6] = fmax(X[6], lc - ld);
        X[7] = fmax(X[7], -d);
        X[8] = fmax(X[8], -ra);
        X[9] = fmax(X[9], -g);
        X[10] = fmax(X[10], -ca);
        X[11] = fmax(X[11], (ra > 0) ? -(g / ra) : -0.0);  // the feature is its negative
      }
    }
    const double sum = fold16(S, lane, add), ext = fold16(X, lane, mx);  // lane i: value i / 2
    const double dmax = __shfl_sync(0xffffffffu, ext, 0);
    int tiny = 0;
#pragma unroll
    for (int s = 0; s < SL; ++s) tiny += __popc(__ballot_sync(0xffffffffu, lane + 32 * s < n && dg[s] < 1e-8 * dmax));
    // the logarithms, one per lane
    const double ex = __shfl_sync(0xffffffffu, ext, 2 * logx), su = __shfl_sync(0xffffffffu, sum, 2 * logs);
    double v = logx >= 7 ? -ex : ex;
    if (lane >= 9) v = lane == 9 ? su / fn : lane == 13 ? su / (fn * fn - fn) : sqrt(su);
    const double lg = lg10(v);
    // the features, one per lane
    const double diff = __shfl_sync(0xffffffffu, lg, la) - __shfl_sync(0xffffffffu, lg, lb);
    const double s1 = __shfl_sync(0xffffffffu, sum, 2 * fs), s2 = __shfl_sync(0xffffffffu, sum, 2 * fs2);
    const double x1 = __shfl_sync(0xffffffffu, ext, 2 * fx);
    double f = diff;
    if (lane == 0) f = fn / 64.0;
    else if (lane == 1) f = (kind ? (int)kind[m] : kind_all) ? 1.0 : 0.0;
    else if (lane == 7) f = (double)dom / fn;
    else if (lane == 22) f = (double)tiny / fn;
    else if (lane == 8) f = -x1;
    else if (lane == 11) f = -x1 <= 0 ? 1.0 : 0.0;
    else if (lane == 18 || lane == 23) f = x1;
    else if (lane == 9 || lane == 19) f = s1 / fn;
    else if (lane >= 15 && lane <= 17) f = sqrt(fmax(0.0, s2 / fn - (s1 / fn) * (s1 / fn)));
    else if (lane == 21 && n == 1) f = 0.0;
    if (lane < kFeat) out[m * kFeat + lane] = clip30(f);
  }
}

// Inference: one thread per sample, parameters broadcast from shared memory 16 bytes at
// a time, two hidden units to an instruction (each sum keeps its order). What bounds it:
// the float32 FMA rate and the registers of both hidden layers.
__global__ void __launch_bounds__(128) mlp_forward_kernel(const float* __restrict__ P, const float* __restrict__ norm,
                                                          const float* __restrict__ X, long long batch,
                                                          float* logits, signed char* tier) {
  using U = Unit<float>;
  __shared__ __align__(16) float w[kParams + 2 * kFeat];
  for (int i = threadIdx.x; i < kParams; i += blockDim.x) w[i] = P[i];
  for (int i = threadIdx.x; i < 2 * kFeat; i += blockDim.x) w[kParams + i] = norm[i];
  __syncthreads();
  const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= batch) return;
  const float* mu = w + kParams;
  const float* isd = mu + kFeat;
  auto pairs = [&](int off) { return *reinterpret_cast<const ulonglong2*>(w + off); };
  float x[kFeat];
#pragma unroll
  for (int k = 0; k < kFeat; ++k) x[k] = (X[s * kFeat + k] - mu[k]) * isd[k];
  U::E h1[kHid / 2];
#pragma unroll
  for (int j = 0; j < kHid / 2; j += 2) {
    const ulonglong2 b = pairs(kOffB1 + 2 * j);
    h1[j] = b.x;
    h1[j + 1] = b.y;
  }
#pragma unroll
  for (int k = 0; k < kFeat; ++k) {
    const U::E xk = U::dup(x[k]);
#pragma unroll
    for (int j = 0; j < kHid / 2; j += 2) {
      const ulonglong2 v = pairs(kOffW1 + k * kHid + 2 * j);
      h1[j] = U::fma(xk, v.x, h1[j]);
      h1[j + 1] = U::fma(xk, v.y, h1[j + 1]);
    }
  }
  U::E h2[kHid / 2];
#pragma unroll
  for (int j = 0; j < kHid / 2; j += 2) {
    const ulonglong2 b = pairs(kOffB2 + 2 * j);
    h2[j] = b.x;
    h2[j + 1] = b.y;
  }
#pragma unroll
  for (int k = 0; k < kHid; ++k) {
    const U::E hk = U::dup(fmaxf(U::get(h1[k / 2], k % 2), 0.f));
#pragma unroll
    for (int j = 0; j < kHid / 2; j += 2) {
      const ulonglong2 v = pairs(kOffW2 + k * kHid + 2 * j);
      h2[j] = U::fma(hk, v.x, h2[j]);
      h2[j + 1] = U::fma(hk, v.y, h2[j + 1]);
    }
  }
  ulonglong2 lp = pairs(kOffB3);
#pragma unroll
  for (int k = 0; k < kHid; ++k) {
    const U::E hk = U::dup(fmaxf(U::get(h2[k / 2], k % 2), 0.f));
    const ulonglong2 v = pairs(kOffW3 + k * kTiers);
    lp.x = U::fma(hk, v.x, lp.x);
    lp.y = U::fma(hk, v.y, lp.y);
  }
  const float lg[kTiers] = {U::get(lp.x, 0), U::get(lp.x, 1), U::get(lp.y, 0), U::get(lp.y, 1)};
  int best = 0;
#pragma unroll
  for (int c = 1; c < kTiers; ++c) best = lg[c] > lg[best] ? c : best;
  if (logits)
#pragma unroll
    for (int c = 0; c < kTiers; ++c) logits[s * kTiers + c] = lg[c];
  if (tier) tier[s] = (signed char)best;
}

// Training: a block of kTrainBlock samples runs forward and backward with its
// activations in shared memory and writes its partial gradient (kParams values) and
// partial loss to scratch; grad_reduce_kernel sums the partials. Activations are stored
// by unit, samples along the row (an odd number of 16-byte units), and every thread owns
// a 4 x 4 tile of each product, so that 16 multiply-adds take two 16-byte reads; one
// output per thread, as before, took two reads per multiply-add. Each sum runs in the
// order of its index.
constexpr int kRowS = kTrainBlock + 4;  // floats per unit row
struct TrainSmem {
  float w[kParams];
  float w2t[kHid][kRowS];  // W2 by its second index
  float x[kFeat][kRowS];
  float h1[kHid][kRowS];
  float h2[kHid][kRowS];
  float dh1[kHid][kRowS];
  float dh2[kHid][kRowS];
  float dl[kTiers][kRowS];
  float loss[kTrainBlock];
};
static_assert(kTrainBlock == 64 && kTrainThreads == 256 && kHid == 64, "4 x 4 tiles of 64 x 64 by 256 threads");

// acc[i][q] += sum_k a[k][4 ts + i] * b[k * bs + 4 tj + q], k < K in order
template <int K>
__device__ __forceinline__ void tile_product(float (&acc)[4][4], const float* a, const float* b, int bs, int ts, int tj) {
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    const float4 u = *reinterpret_cast<const float4*>(a + k * kRowS + 4 * ts);
    const float4 v = *reinterpret_cast<const float4*>(b + k * bs + 4 * tj);
    const float uu[4] = {u.x, u.y, u.z, u.w}, vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(uu[i], vv[q], acc[i][q]);
  }
}

__global__ void __launch_bounds__(kTrainThreads) mlp_train_kernel(const float* __restrict__ P,
                                                                   const float* __restrict__ norm,
                                                                   const float* __restrict__ X,
                                                                   const signed char* __restrict__ label,
                                                                   const float* __restrict__ cw, long long batch,
                                                                   float* partial) {
  extern __shared__ __align__(16) unsigned char tsm_raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(tsm_raw);
  const int t = threadIdx.x;
  for (int i = t; i < kParams; i += kTrainThreads) S.w[i] = P[i];
  for (int i = t; i < kHid * kHid; i += kTrainThreads) S.w2t[i % kHid][i / kHid] = P[kOffW2 + i];
  const long long s0 = (long long)blockIdx.x * kTrainBlock;
  const int live = (int)(batch - s0 < kTrainBlock ? batch - s0 : kTrainBlock);
  for (int i = t; i < kTrainBlock * kFeat; i += kTrainThreads) {
    const int s = i / kFeat, k = i % kFeat;
    S.x[k][s] = s < live ? (X[(s0 + s) * kFeat + k] - norm[k]) * norm[kFeat + k] : 0.f;
  }
  __syncthreads();
  const int ts = t >> 4, tj = t & 15;  // samples 4 ts .. + 3, units 4 tj .. + 3
  // forward
  auto layer = [&](const float (&in)[4][4], float (*h)[kRowS]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = 4 * ts + i < live ? fmaxf(in[i][q], 0.f) : 0.f;
      *reinterpret_cast<float4*>(&h[4 * tj + q][4 * ts]) = make_float4(v[0], v[1], v[2], v[3]);
    }
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = S.w[kOffB1 + 4 * tj + q];
  tile_product<kFeat>(acc, &S.x[0][0], S.w + kOffW1, kHid, ts, tj);
  layer(acc, S.h1);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = S.w[kOffB2 + 4 * tj + q];
  tile_product<kHid>(acc, &S.h1[0][0], S.w + kOffW2, kHid, ts, tj);
  layer(acc, S.h2);
  __syncthreads();
  {
    const int s = t & 63, q = t >> 6;
    float a = S.w[kOffB3 + q];
#pragma unroll 8
    for (int k = 0; k < kHid; ++k) a = fmaf(S.h2[k][s], S.w[kOffW3 + k * kTiers + q], a);
    S.dl[q][s] = a;  // logits for now
  }
  __syncthreads();
  if (t < kTrainBlock) {
    const int s = t;
    float lg[kTiers], mx = -3.0e38f;
#pragma unroll
    for (int c = 0; c < kTiers; ++c) {
      lg[c] = S.dl[c][s];
      mx = fmaxf(mx, lg[c]);
    }
    float z = 0.f;
#pragma unroll
    for (int c = 0; c < kTiers; ++c) z += expf(lg[c] - mx);
    const int y = s < live ? (int)label[s0 + s] : 0;
    const float wy = s < live ? (cw ? cw[y] : 1.f) : 0.f;
    const float scale = wy / (float)batch;
#pragma unroll
    for (int c = 0; c < kTiers; ++c) {
      const float pc = expf(lg[c] - mx) / z;
      S.dl[c][s] = scale * (pc - (c == y ? 1.f : 0.f));
    }
    float ly = lg[0];
#pragma unroll
    for (int c = 1; c < kTiers; ++c) ly = c == y ? lg[c] : ly;
    S.loss[s] = s < live ? scale * (logf(z) + mx - ly) : 0.f;
  }
  __syncthreads();
  // backward through the hidden layers
  auto masked = [&](const float (&in)[4][4], const float (*h)[kRowS], float (*d)[kRowS]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 hv = *reinterpret_cast<const float4*>(&h[4 * tj + q][4 * ts]);
      *reinterpret_cast<float4*>(&d[4 * tj + q][4 * ts]) =
          make_float4(hv.x > 0.f ? in[0][q] : 0.f, hv.y > 0.f ? in[1][q] : 0.f, hv.z > 0.f ? in[2][q] : 0.f,
                      hv.w > 0.f ? in[3][q] : 0.f);
    }
  };
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float a = 0.f;
#pragma unroll
      for (int c = 0; c < kTiers; ++c) a = fmaf(S.w[kOffW3 + (4 * tj + q) * kTiers + c], S.dl[c][4 * ts + i], a);
      acc[i][q] = a;
    }
  masked(acc, S.h2, S.dh2);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = 0.f;
  tile_product<kHid>(acc, &S.dh2[0][0], &S.w2t[0][0], kRowS, ts, tj);
  masked(acc, S.h1, S.dh1);
  __syncthreads();
  // parameter gradients over the block's samples: tiles of rows ra + 16 i (of the inputs)
  // and rb + 16 q (of the deltas), four samples at a time
  float* out = partial + (long long)blockIdx.x * (kParams + 1);
  auto grad_tile = [&](const float (*in)[kRowS], const float (*d)[kRowS], int rows, int off) {
    float g[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) g[i][q] = 0.f;
#pragma unroll 2
    for (int s = 0; s < kTrainBlock; s += 4) {
      float u[4][4], v[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(&in[ts + 16 * i < rows ? ts + 16 * i : 0][s]);
        const float4 b = *reinterpret_cast<const float4*>(&d[tj + 16 * i][s]);
        u[i][0] = a.x; u[i][1] = a.y; u[i][2] = a.z; u[i][3] = a.w;
        v[i][0] = b.x; v[i][1] = b.y; v[i][2] = b.z; v[i][3] = b.w;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int q = 0; q < 4; ++q) g[i][q] = fmaf(u[i][e], v[q][e], g[i][q]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (ts + 16 * i < rows)
#pragma unroll
        for (int q = 0; q < 4; ++q) out[off + (ts + 16 * i) * kHid + tj + 16 * q] = g[i][q];
  };
  grad_tile(S.h1, S.dh2, kHid, kOffW2);
  grad_tile(S.x, S.dh1, kFeat, kOffW1);
  {
    const int k = t >> 2, c = t & 3;
    float g = 0.f;
#pragma unroll 8
    for (int s = 0; s < kTrainBlock; ++s) g = fmaf(S.h2[k][s], S.dl[c][s], g);
    out[kOffW3 + t] = g;
  }
  if (t < 2 * kHid + kTiers + 1) {
    const float* row = t < kHid ? S.dh1[t] : t < 2 * kHid ? S.dh2[t - kHid] : t < 2 * kHid + kTiers ? S.dl[t - 2 * kHid] : S.loss;
    float g = 0.f;
#pragma unroll 8
    for (int s = 0; s < kTrainBlock; ++s) g += row[s];
    out[t < kHid ? kOffB1 + t : t < 2 * kHid ? kOffB2 + t - kHid : t < 2 * kHid + kTiers ? kOffB3 + t - 2 * kHid : kParams] = g;
  }
}

// grad[p] = sum over blocks of partial[b][p] (p = kParams is the loss), in a fixed order:
// a CTA takes 32 parameters, its 8 warps each an eighth of the blocks, then the eighths.
__global__ void __launch_bounds__(256) grad_reduce_kernel(const float* __restrict__ partial, int blocks, float* grad, float* loss) {
  __shared__ float part[8][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
  const int per = (blocks + 7) / 8, b0 = g * per, b1 = min(blocks, b0 + per);
  float v = 0.f;
  if (p <= kParams) {
#pragma unroll 8
    for (int b = b0; b < b1; ++b) v += partial[(long long)b * (kParams + 1) + p];
  }
  part[g][lane] = v;
  __syncthreads();
  if (g == 0 && p <= kParams) {
    for (int i = 1; i < 8; ++i) v += part[i][lane];
    if (p < kParams) grad[p] = v;
    else if (loss) *loss = v;
  }
}

// Adam (Kingma & Ba 2015) with bias correction.
__global__ void adam_kernel(float* P, const float* __restrict__ g, float* m, float* v, long long count, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  P[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace dev
}  // namespace tsdx
