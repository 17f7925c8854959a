"""Shared-memory layout of the strided FFT pass: a warp reads its twiddle tables behind a warp barrier
only, so no word of them may belong to another warp or to the tile, and 16-byte reads of a table must be
aligned. Checked for every instantiation (4 to 11 layers, 32- and 64-byte runs) from the kernel's own
layout functions, compiled for the host."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "proving_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "fft_layout.cuh"
using namespace cs;
template <int T, int EB>
int check() {
  constexpr int TA = T / 2, TB = T - TA;
  constexpr uint32_t warps = strided_warps<T, EB>();
  std::vector<int> owner(strided_smem_words<T, EB>(), -1);
  int bad = 0;
  for (uint32_t L = 0; L < (1u << (T + EB)); L++) {  // -2: the tile
    const uint32_t w = strided_pad<TA, EB>(L);
    if (w >= owner.size() || owner[w] != -1) { bad++; continue; }
    owner[w] = -2;
  }
  for (uint32_t warp = 0; warp < warps; warp++) {
    const uint32_t first[2] = {strided_high_table<T, EB>(warp), strided_low_table<T, EB>(warp)};
    const uint32_t words[2] = {1u << TB, (32u >> EB) << TB};
    for (int k = 0; k < 2; k++) {
      bad += first[k] % 4 != 0;
      for (uint32_t w = first[k]; w < first[k] + words[k]; w++) {
        if (w >= owner.size() || owner[w] != -1) { bad++; continue; }
        owner[w] = (int)warp;
      }
    }
  }
  if (bad) std::printf("T %d EB %d: %d words shared or out of range\n", T, EB, bad);
  return bad;
}
template <int T>
int check_both() {
  int bad = check<T, 3>();
  if constexpr (T <= 9) bad += check<T, 4>();
  return bad;
}
int main() {
  return check_both<4>() + check_both<5>() + check_both<6>() + check_both<7>() + check_both<8>() + check_both<9>() +
                 check_both<10>() + check_both<11>() ? 1 : 0;
}
"""


def test_every_warp_has_its_own_tables(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
