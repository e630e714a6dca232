"""The shared-memory vectors that the register-row kernels read in their rolled loops,
from the layout constants of the kernels themselves: each lies in its own row, and the row
of zeros that a zero pivot reads is as long as any row."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = next(pathlib.Path(__file__).resolve().parents[1].glob("tinysolverdx*_b200")) / "csrc"
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = r"""
#include <cstdio>
#include "rows.cuh"
using namespace tsdx::dev;
template <class T, int NP, int NRHS, int G> int one() {
  using C = BlkCfg<T, NP, NRHS, G>;
  using R = RowCfg<T, NP, NRHS, G>;
  constexpr int TS = int(sizeof(T)), VN = R::VN;
  int bad = 0;
  if (R::PW == NP) return 0;
  for (int c0 = 0; c0 < NP; c0 += R::PW)
    for (int w : {R::PW, R::LASTW}) {
      if (w != R::PW && c0 + R::PW != NP) continue;  // the wide panel is the last one
      const int cend = c0 + w;
      for (int k0 = c0; k0 < c0 + R::PW; k0 += VN)
        for (int q = VN; q < w; q += VN) {
          if (!R::in_row(q) && k0 + q >= cend) continue;  // left out by the kernels
          const int end = (k0 + q + VN) * TS;
          bad += end > C::RS || end > kZeroRow;
        }
    }
  if (bad) std::printf("order %d, %d right-hand sides, %d bytes: %d reads\n", NP, NRHS, TS, bad);
  return bad;
}
template <class T, int NP, int G> int orders() {
  return one<T, NP, 0, G>() + one<T, NP, 1, G>() + one<T, NP, 2, G>() + one<T, NP, 4, G>() + one<T, NP, 8, G>();
}
template <class T> int types() {
  return orders<T, 8, 4>() + orders<T, 16, 8>() + orders<T, 24, 8>() + orders<T, 24, 16>() + orders<T, 24, 32>() +
         orders<T, 32, 16>() + orders<T, 32, 32>() + orders<T, 40, 16>() + orders<T, 40, 32>() + orders<T, 48, 32>() +
         orders<T, 56, 32>() + orders<T, 64, 32>();
}
int main() { return types<float>() + types<double>() ? 1 : 0; }
"""


@pytest.mark.skipif(not pathlib.Path(NVCC).exists(), reason="needs nvcc")
def test_rolled_reads_stay_in_their_row(tmp_path):
    src, exe = tmp_path / "layout.cu", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(CSRC), "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
