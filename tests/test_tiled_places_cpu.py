"""The one-pass kernel's collide warps write their cells in place.  For every tile
size: no two lanes share a word that one of them writes, every cell lies inside
its plane's slot, and a lane without a cell reads words that nobody writes."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "lbm_tiled.cuh"

template <int Q, int MODE>
int check() {
  using T = lbm::TileShape<Q>;
  constexpr uint32_t S = lbm::Sweep<Q>::SLOTS, N = 64 * T::NCW;
  const uint32_t words = lbm::tiled_smem_bytes<Q, MODE>() / 4;
  const uint32_t sync = words - sizeof(lbm::TileSync<Q>) / 4;
  const uint32_t ring = S * T::PLANE, stage = lbm::tiled_stage_bytes<Q, MODE>() / 4;
  for (uint32_t tyv = 1; tyv <= T::TY; ++tyv)
    for (uint32_t tzv = 1; tzv <= T::TZ; ++tzv)
      for (uint32_t s = 0; s < S; ++s) {
        std::vector<int> writer(words, -1);
        uint32_t cells = 0;
        for (uint32_t m = 0; m < N; ++m) {
          const auto p = lbm::collide_place<Q, MODE>(m, tyv, tzv);
          if (p.step == 0) continue;
          const uint32_t w = p.word + s * p.step;
          if (w < s * T::PLANE || w + Q > (s + 1) * T::PLANE) return 1;
          for (int q = 0; q < Q; ++q) {
            if (writer[w + q] >= 0) return 2;
            writer[w + q] = m;
          }
          ++cells;
        }
        if (cells != (tyv + 2 * T::HR) * (tzv + 2)) return 3;
        for (uint32_t m = 0; m < N; ++m) {
          const auto p = lbm::collide_place<Q, MODE>(m, tyv, tzv);
          if (p.step != 0) continue;
          const uint32_t w = p.word + s * p.step;
          if (w < ring + stage || w + Q > sync) return 4;
        }
      }
  return 0;
}
int main() {
  const int r[4] = {check<19, lbm::kOutAoS>(), check<19, lbm::kOutState>(),
                    check<9, lbm::kOutAoS>(), check<9, lbm::kOutState>()};
  std::printf("%d %d %d %d\n", r[0], r[1], r[2], r[3]);
  return 0;
}
"""


def test_collide_places_are_disjoint(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    src, exe = tmp_path / "places.cu", tmp_path / "places"
    src.write_text(SOURCE)
    csrc = os.path.join(ROOT, "maddening_b200", "csrc")
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", csrc, "-I",
                    os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0", "0"]
