// Host-side launchers: map a runtime (n, nrhs) onto a compiled (NP, NRHS) kernel
// and size a persistent grid from the occupancy of that kernel.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <string>

#include "blk3.cuh"
#include "rows.cuh"
#include "solve.cuh"
#include "blk_tc.cuh"

namespace tsdx {
namespace host {

using dev::SolveArgs;

// Errors of the CUDA runtime, per calling thread.
void set_cuda_error(cudaError_t e, const char* what);
std::atomic<long long>& launch_counter();

int device_sms(int dev);

// Per-device tables of the library (workspaces, streams, cached addresses) cover
// device ordinals [0, kMaxDevices); a higher ordinal is reported as TSDX_ERR_NODEV.
constexpr int kMaxDevices = 64;

// Compiled padded sizes; a matrix of order n runs in the smallest NP >= n
// (identity padding is exactly transparent to every result, see common.cuh).
inline int np_of(int n) {
  return n <= 4 ? 4 : n <= 8 ? 8 : n <= 16 ? 16 : n <= 24 ? 24 : n <= 32 ? 32 : n <= 40 ? 40 : n <= 48 ? 48 : n <= 56 ? 56 : 64;
}
// Right-hand sides are solved in passes of at most 8 columns.
inline int nrhs_bucket(int r) { return r == 0 ? 0 : r == 1 ? 1 : r <= 4 ? 4 : 8; }
template <class Kern>
int grid_for(Kern kern, int smem, long long ctas_needed, int threads = 128) {
  int devi = 0;
  cudaGetDevice(&devi);
  int occ = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem);
  if (e != cudaSuccess || occ < 1) occ = 1;
  const long long cap = (long long)device_sms(devi) * occ;
  return (int)(ctas_needed < cap ? (ctas_needed < 1 ? 1 : ctas_needed) : cap);
}

// Warps per CTA for this many work units of one warp each: the kernel's WPC, fewer when
// they would leave SMs without a CTA (float64 Cholesky of order 7, 5,959 matrices: 47 of
// 148 SMs with full CTAs).
inline int warps_for(long long units, int wpc) {
  int devi = 0;
  cudaGetDevice(&devi);
  const long long per_sm = (units + device_sms(devi) - 1) / device_sms(devi);
  return (int)(per_sm < 1 ? 1 : per_sm < wpc ? per_sm : wpc);
}

// Allows a kernel the smem bytes of dynamic shared memory that a call uses. most is the most
// that any of its calls uses, the same in every call: the limit belongs to the function on
// a device, so a call that set its own smaller need would lower it between another
// thread's prepare and launch.
constexpr int kMostSmem = 227 * 1024;  // of a block, less its static shared memory
template <class Kern>
int prepare(Kern kern, int smem, int most) {
  // (the 48 KB that need no leave hold a kernel's static shared memory as well)
  if (smem > 40 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) { set_cuda_error(e, "cudaFuncSetAttribute"); return -5; }
  }
  return 0;
}

// LU / Cholesky with rows in registers (rows.cuh): a persistent CTA per SM with as many
// warps as shared memory holds, at most 16. Between 12 and 16 it stays at 12: warps are
// dealt to four schedulers, so 13 to 15 cost the registers of 16 (128 a thread instead of
// 168) without its parallelism (float32, 4 right-hand sides: LU of order 24, 262,144
// matrices 869 us with 12, 978 with 15; order 56, 65,536 1686 and 1950 with 14; Cholesky of
// order 40 597 and 714 with 13; without right-hand sides within 2 %). A batch that 12 warps
// an SM do not quite hold pays a second round (float32 LU of order 52, 2,000 matrices 105
// us, 1,700 60).
template <class T, int NP, int NRHS, int GO = 0>
constexpr int blk_wpc() {
  constexpr int FIT = (227 * 1024 - dev::kRowConst) / dev::BlkCfg<T, NP, NRHS, GO>::WARPB;
  return FIT < 1 ? 1 : (FIT >= 16 ? 16 : FIT >= 12 ? 12 : FIT);
}

// Lanes per matrix (0: the layout's own choice; the matrices that share a warp run its
// steps together, so small orders spend fewer instructions each). Measured on B200 at
// 65,536 to 262,144 matrices against the next choice, factorizations alone (LU, Cholesky;
// us): order 8, 4 lanes float32 73 and 56, with 8 89 and 75, float64 101 and 75 against 116
// and 95; order 16, 8 lanes float32 232 and 148, with 16 259 and 232, float64 374 and 222
// against 376 and 329; order 24 float32, 8 lanes 586 and 384, with 16 640 and 556; order 32
// float32, 16 lanes 493 and 415, with 32 634 and 556; order 40 float32, 16 lanes 609 and
// 404, with 32 618 and 540. In float64 the next choice came out ahead there once panels
// ran in a rolled loop: order 24 with 8 lanes 1148 and 745 against 1172 and 845 with the 16
// taken here (with 4 right-hand sides 1316 and 1281 against 1685 and 1433), Cholesky of
// order 32 with 16 lanes 681 against 833 with 32, of order 40 837 against 943. Above that,
// one matrix per warp.
template <class T, int NP>
constexpr int blk_lanes() {
  constexpr bool F32 = sizeof(T) == 4;
  switch (NP) {
    case 8: return 4;
    case 16: return 8;
    case 24: return F32 ? 8 : 16;
    case 32: case 40: return F32 ? 16 : 32;
    default: return 0;
  }
}

// Two warps per matrix (blk2.cuh) for float64 LU of padded order 48..56: 1.10x (order 48)
// and 1.22x (56) the one-warp kernel on CUDA cores that rows.cuh replaced (65,536 to
// 131,072 matrices, 4 right-hand sides); slower at 40 and in float32.
template <class T, int NP, int NRHS>
int launch_blk2(const SolveArgs<T>& a, cudaStream_t st) {
  using C = dev::Blk2Cfg<T, NP, NRHS>;
  constexpr int FIT = (227 * 1024) / C::TEAMB;
  constexpr int TPC = FIT < 1 ? 1 : (FIT > 8 ? 8 : FIT);
  constexpr int SMEM = TPC * C::TEAMB;
  auto kern = dev::blk2_kernel<T, NP, NRHS, TPC>;
  if (int rc = prepare(kern, SMEM, SMEM)) return rc;
  const long long ctas = (a.batch + TPC - 1) / TPC;
  const int grid = grid_for(kern, SMEM, ctas, TPC * 64);
  kern<<<grid, TPC * 64, SMEM, st>>>(a);
  launch_counter().fetch_add(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e, "kernel launch"); return -5; }
  return 0;
}

// Two warps per matrix with look-ahead (blk3.cuh) for float64 LU of padded order 64:
// 1.10x the two-warp kernel (1.18x at n = 61) on B200, 65,536 matrices, 4 right-hand
// sides; slower than it at orders 40..56.
template <class T, int NP, int NRHS>
int launch_blk3(const SolveArgs<T>& a, cudaStream_t st) {
  using C = dev::Blk3Cfg<T, NP, NRHS>;
  constexpr int FIT = (227 * 1024) / C::TEAMB;
  constexpr int TPC = FIT < 1 ? 1 : (FIT > 8 ? 8 : FIT);
  constexpr int SMEM = TPC * C::TEAMB;
  // the panel warp also takes part of the trailing update (pivot steps counted as 3
  // chunk updates): +3.8 % at n = 64, -1.3 % at n = 61 on B200
  auto kern = dev::blk3_kernel<T, NP, NRHS, TPC, 3>;
  if (int rc = prepare(kern, SMEM, SMEM)) return rc;
  const long long ctas = (a.batch + TPC - 1) / TPC;
  const int grid = grid_for(kern, SMEM, ctas, TPC * 64);
  kern<<<grid, TPC * 64, SMEM, st>>>(a);
  launch_counter().fetch_add(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e, "kernel launch"); return -5; }
  return 0;
}

// LU kernel family: 0 = by order (the default), 1 = shared-memory blocked kernels
// with CUDA-core updates everywhere (rows.cuh / blk2.cuh / blk3.cuh), 3 = the float64
// tensor-core trailing update (blk_tc.cuh) at every padded order 32..64. Read once
// from TSDX_LU_KERNEL ("smem" or "tc"); all give bit-identical results.
int lu_kernel_family();

// float64 LU with the trailing update on the FP64 tensor cores (blk_tc.cuh): a
// persistent CTA per SM with as many one-matrix warps as shared memory holds.
template <int NP, int NRHS>
int launch_tc(const SolveArgs<double>& a, cudaStream_t st) {
  using C = dev::TcCfg<NP, NRHS>;
  constexpr int FIT = (227 * 1024) / C::WARPB;
  constexpr int WPC = FIT < 1 ? 1 : (FIT > 16 ? 16 : FIT);
  constexpr int SMEM = WPC * C::WARPB;
  auto kern = dev::tc_kernel<NP, NRHS, WPC>;
  if (int rc = prepare(kern, SMEM, SMEM)) return rc;
  const int wpc = warps_for(a.batch, WPC), smem = wpc * C::WARPB;
  const int grid = grid_for(kern, smem, (a.batch + wpc - 1) / wpc, wpc * 32);
  kern<<<grid, wpc * 32, smem, st>>>(a);
  launch_counter().fetch_add(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e, "kernel launch"); return -5; }
  return 0;
}

template <class T, int NP, int NRHS, bool CHOL>
int launch_blk(const SolveArgs<T>& a, cudaStream_t st) {
  // float64 LU from padded order 32 on: the tensor-core trailing update. Measured on B200
  // against the kernels on CUDA cores (4 right-hand sides, 131,072 matrices up to order 32,
  // 65,536 above, us): n=25 1080 and 1304, n=32 1084 and 1304, n=40 1066 and 1320, n=48 1574
  // and 2739, n=56 2332 and 3800, n=64 3229 and 4985. Odd orders above 48 run on
  // blk2/blk3: the line was drawn when rows came by bulk copies, which their 8-byte rows
  // did not allow. With the copies of today tc_kernel takes them too (TSDX_LU_KERNEL=tc) and
  // is the faster one, n=49 2307 and 3953, n=55 2421 and 4114, n=61 3389 and 5620.
  if constexpr (!CHOL && sizeof(T) == 8 && NP >= 32) {
    const int fam = lu_kernel_family();
    if (fam == 3 || (fam == 0 && (NP <= 48 || a.n % 2 == 0)))
      return launch_tc<NP, NRHS>(reinterpret_cast<const SolveArgs<double>&>(a), st);
  }
  if constexpr (!CHOL && sizeof(T) == 8 && NP == 64) return launch_blk3<T, NP, NRHS>(a, st);
  if constexpr (!CHOL && sizeof(T) == 8 && NP >= 48) return launch_blk2<T, NP, NRHS>(a, st);
  constexpr int GO = blk_lanes<T, NP>();
  using C = dev::BlkCfg<T, NP, NRHS, GO>;
  constexpr int WPC = blk_wpc<T, NP, NRHS, GO>();
  constexpr int SMEM = WPC * C::WARPB;
  auto kern = dev::blk_kernel<T, NP, NRHS, WPC, CHOL, GO>;
  if (int rc = prepare(kern, SMEM, SMEM)) return rc;
  const long long units = (a.batch + C::S - 1) / C::S;
  const int wpc = warps_for(units, WPC), smem = wpc * C::WARPB;
  const int grid = grid_for(kern, smem, (units + wpc - 1) / wpc, wpc * 32);
  kern<<<grid, wpc * 32, smem, st>>>(a);
  launch_counter().fetch_add(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e, "kernel launch"); return -5; }
  return 0;
}

// Triangular solves (solve.cuh): one warp per matrix, as many warps as shared memory and
// 128 registers a thread allow. W: tiles of 8 right-hand sides (float64) or columns
// (float32).
template <class T, int NP, int W, bool LU>
int launch_trs(const SolveArgs<T>& a, cudaStream_t st) {
  using C = dev::TrsCfg<T, NP>;
  constexpr int FIT = (227 * 1024) / C::WARPB;
  constexpr int WPC = FIT > 16 ? 16 : FIT;
  constexpr int SMEM = WPC * C::WARPB;
  auto kern = [] {
    if constexpr (sizeof(T) == 8) return dev::trs_f64_kernel<NP, W, LU, WPC>;
    else return dev::trs_f32_kernel<NP, W, LU, WPC>;
  }();
  if (int rc = prepare(kern, SMEM, SMEM)) return rc;
  const int wpc = warps_for(a.batch, WPC), smem = wpc * C::WARPB;
  const int grid = grid_for(kern, smem, (a.batch + wpc - 1) / wpc, wpc * 32);
  kern<<<grid, wpc * 32, smem, st>>>(a);
  launch_counter().fetch_add(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e, "kernel launch"); return -5; }
  return 0;
}

#define TSDX_NP_SWITCH(NPV, BODY)                 \
  switch (NPV) {                                  \
    case 4: { constexpr int NP_ = 4; BODY; }      \
    case 8: { constexpr int NP_ = 8; BODY; }      \
    case 16: { constexpr int NP_ = 16; BODY; }    \
    case 24: { constexpr int NP_ = 24; BODY; }    \
    case 32: { constexpr int NP_ = 32; BODY; }    \
    case 40: { constexpr int NP_ = 40; BODY; }    \
    case 48: { constexpr int NP_ = 48; BODY; }    \
    case 56: { constexpr int NP_ = 56; BODY; }    \
    default: { constexpr int NP_ = 64; BODY; }    \
  }
#define TSDX_RHS_SWITCH(RV, BODY)                 \
  switch (RV) {                                   \
    case 0: { constexpr int R_ = 0; BODY; }       \
    case 1: { constexpr int R_ = 1; BODY; }       \
    case 4: { constexpr int R_ = 4; BODY; }       \
    default: { constexpr int R_ = 8; BODY; }      \
  }

// One fused pass: factor A (and solve B columns [b0, b0 + nrhs), nrhs <= 8).
template <class T, bool CHOL>
int run_blk(const SolveArgs<T>& a, cudaStream_t st) {
  const int np = np_of(a.n), rb = nrhs_bucket(a.nrhs);
  TSDX_NP_SWITCH(np, TSDX_RHS_SWITCH(rb, return (launch_blk<T, NP_, R_, CHOL>(a, st))));
  return 0;
}

template <class T, int NP, bool LU>
int launch_trs_small(const SolveArgs<T>& a, cudaStream_t st) {
  auto kern = dev::trs_small_kernel<T, NP, LU>;
  constexpr int MOST = dev::kSmallWpc * dev::trs_small_elems(NP, 0) * int(sizeof(T));
  int lg = 0;
  while ((1 << lg) < a.nrhs) ++lg;
  const long long units = (a.batch + (32 >> lg) - 1) / (32 >> lg);
  const int wpc = warps_for(units, dev::kSmallWpc), smem = wpc * dev::trs_small_elems(a.n, lg) * int(sizeof(T));
  if (int rc = prepare(kern, smem, MOST)) return rc;
  const int grid = grid_for(kern, smem, (units + wpc - 1) / wpc, wpc * 32);
  kern<<<grid, wpc * 32, smem, st>>>(a, lg);
  launch_counter().fetch_add(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e, "kernel launch"); return -5; }
  return 0;
}

// One solve pass from a factor (nrhs <= kTrsRhs). Orders up to 12 take the kernel with a
// lane per right-hand side (measured up to there, beside it in solve.cuh: faster than the
// warp per matrix at every width). Above, orders run in the next multiple of 8 in float64
// (one block of the kernel; order 17, one right-hand side, 64,878 matrices getrs 184 us in
// 32, 135 in 24), of 16 in float32 (whose steps stop at the order anyway; the multiple
// only sets the shared memory).
constexpr int kTrsRhs = 16;
template <class T, bool LU, int W>
int run_trs_np(const SolveArgs<T>& a, cudaStream_t st) {
  if (a.n <= 4) return launch_trs_small<T, 4, LU>(a, st);
  if (a.n <= 8) return launch_trs_small<T, 8, LU>(a, st);
  if (a.n <= 12) return launch_trs_small<T, 12, LU>(a, st);
  if constexpr (sizeof(T) == 8) {
    switch ((a.n + 7) / 8) {
      case 3: return launch_trs<T, 24, W, LU>(a, st);
      case 5: return launch_trs<T, 40, W, LU>(a, st);
      case 7: return launch_trs<T, 56, W, LU>(a, st);
    }
  }
  switch ((a.n + 15) / 16) {
    case 1: return launch_trs<T, 16, W, LU>(a, st);
    case 2: return launch_trs<T, 32, W, LU>(a, st);
    case 3: return launch_trs<T, 48, W, LU>(a, st);
    default: return launch_trs<T, 64, W, LU>(a, st);
  }
}
template <class T, bool LU>
int run_trs(const SolveArgs<T>& a, cudaStream_t st) {
  if constexpr (sizeof(T) == 8) return a.nrhs > 8 ? run_trs_np<T, LU, 2>(a, st) : run_trs_np<T, LU, 1>(a, st);
  else
    return a.nrhs > 8 ? run_trs_np<T, LU, 16>(a, st) : a.nrhs > 4 ? run_trs_np<T, LU, 8>(a, st)
         : a.nrhs > 1 ? run_trs_np<T, LU, 4>(a, st) : run_trs_np<T, LU, 1>(a, st);
}

// Explicitly instantiated in the per-type translation units.
template <class T> int run_lu(const SolveArgs<T>& a, cudaStream_t st);
template <class T> int run_chol(const SolveArgs<T>& a, cudaStream_t st);
template <class T> int run_getrs(const SolveArgs<T>& a, cudaStream_t st);
template <class T> int run_potrs(const SolveArgs<T>& a, cudaStream_t st);

}  // namespace host
}  // namespace tsdx
