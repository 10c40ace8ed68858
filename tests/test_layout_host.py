"""Shared-memory layout of the generation-3 adjoint on grids of odd padded height (no GPU): every array
that the kernel reads in column pairs starts on an 8-byte boundary."""

from __future__ import annotations

import subprocess

from conftest import ROOT

SOURCE = r"""
#include <cstddef>
#include <initializer_list>
#define __host__
#define __device__
#define __forceinline__ inline
#include "LAYOUT"
int main() {
  for (int nx : {114, 144, 184})
    for (int nz = 60; nz <= 184; ++nz)
      for (int C : {1, 2, 3, 4, 6}) {
        const wg::A3Layout L = wg::a3_layout_rt(nx, 12, nz, 28, C, 71);
        for (int o : {L.off_vs, L.off_tx, L.off_u1x, L.off_tz, L.off_u1z, L.off_lpx, L.off_lzx, L.off_lpz, L.off_lzz, L.off_v2,
                      L.off_ga, L.off_prof, L.off_opb, L.off_src})
          if (o % 2) return 1;
      }
  return 0;
}
"""


def test_pair_arrays_are_eight_byte_aligned_for_odd_heights(tmp_path):
    csrc = ROOT / "wgnet_gb300" / "csrc"
    text = (csrc / "wave_kernels3_layout.h").read_text()
    device = (csrc / "wave_device.cuh").read_text()
    # the two row helpers of the device header, without its inline PTX
    rows = device[device.index("__host__ __device__ inline int split_row"):device.index("// Forward shared-memory layout")]
    text = text.replace('#include "wave_device.cuh"', "namespace wg {\nconstexpr int FD_PAD = 2;\n" + rows + "}\n")
    (tmp_path / "layout.h").write_text(text.replace("#pragma once", ""))
    (tmp_path / "t.cpp").write_text(SOURCE.replace("LAYOUT", "layout.h"))
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-o", str(exe), str(tmp_path / "t.cpp")], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
