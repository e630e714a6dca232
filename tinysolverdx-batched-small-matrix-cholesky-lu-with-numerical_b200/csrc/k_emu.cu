// Launches of the emulated fp16 / bf16 kernels (emu.cuh) on device pointers, for the
// storage types float64, float32 and binary16 (as unsigned short).
#include <cuda_runtime.h>

#include <algorithm>

#include "emu.cuh"
#include "launch.cuh"

namespace tsdx {
namespace host {
namespace {

// one warp per matrix; at most 8 warps a CTA keep several CTAs of small orders per SM
template <class Kern, class... Args>
int launch(Kern kern, int warp_words, long long batch, cudaStream_t st, Args... args) {
  const int wpc = warps_for(batch, std::max(1, std::min(8, kMostSmem / (warp_words * 4)))), smem = wpc * warp_words * 4;
  if (int rc = prepare(kern, smem, kMostSmem)) return rc;
  const int grid = grid_for(kern, smem, (batch + wpc - 1) / wpc, wpc * 32);
  kern<<<grid, wpc * 32, smem, st>>>(args...);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e, "emulated format kernel"); return -5; }
  launch_counter().fetch_add(1);
  return 0;
}
template <class S> struct Storage { using type = S; };
template <> struct Storage<unsigned short> { using type = __half; };

template <int FMT, class S>
int factor(bool lu, S* A, int n, long long batch, int* piv, int* info, cudaStream_t st) {
  using G = typename Storage<S>::type;
  G* a = reinterpret_cast<G*>(A);
  const int words = dev::emu_factor_words(n);
  return lu ? launch(dev::emu_lu_kernel<FMT, G>, words, batch, st, a, n, batch, piv, info)
            : launch(dev::emu_cholesky_kernel<FMT, G>, words, batch, st, a, n, batch, info);
}
template <int FMT, class S>
int solve(bool lu, const S* F, const int* piv, int n, long long batch, S* B, int nrhs, cudaStream_t st) {
  using G = typename Storage<S>::type;
  const G* f = reinterpret_cast<const G*>(F);
  G* b = reinterpret_cast<G*>(B);
  const int words = dev::emu_factor_words(n) + 32 * n;
  return lu ? launch(dev::emu_solve_kernel<FMT, true, G>, words, batch, st, f, piv, n, batch, b, nrhs)
            : launch(dev::emu_solve_kernel<FMT, false, G>, words, batch, st, f, piv, n, batch, b, nrhs);
}
}  // namespace

template <class S>
int run_emu_factor(int fmt, bool lu, S* A, int n, long long batch, int* piv, int* info, cudaStream_t st) {
  return fmt == 0 ? factor<0, S>(lu, A, n, batch, piv, info, st) : factor<1, S>(lu, A, n, batch, piv, info, st);
}
template <class S>
int run_emu_solve(int fmt, bool lu, const S* F, const int* piv, int n, long long batch, S* B, int nrhs, cudaStream_t st) {
  return fmt == 0 ? solve<0, S>(lu, F, piv, n, batch, B, nrhs, st) : solve<1, S>(lu, F, piv, n, batch, B, nrhs, st);
}
#define TSDX_EMU(S)                                                                                              \
  template int run_emu_factor<S>(int, bool, S*, int, long long, int*, int*, cudaStream_t);                       \
  template int run_emu_solve<S>(int, bool, const S*, const int*, int, long long, S*, int, cudaStream_t);
TSDX_EMU(double)
TSDX_EMU(float)
TSDX_EMU(unsigned short)

}  // namespace host
}  // namespace tsdx
