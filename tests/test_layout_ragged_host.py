"""Shared-memory layouts of the generation-3 kernels (no GPU), for grids of any width and height: the arrays
that are read in column pairs and the mbarriers start on 8-byte boundaries, and no array runs into the next."""

from __future__ import annotations

import subprocess

from conftest import ROOT

SOURCE = r"""
#include <cstddef>
#include <initializer_list>
#define __host__
#define __device__
#define __forceinline__ inline
#include "layout.h"
int main() {
  for (bool rag : {false, true})
    for (int nx : {114, 116, 144, 184})
      for (int nz = 56; nz <= 184; ++nz)
        for (int C : {1, 2, 3, 4, 6})
          for (int nrec : {1, 70, 71, 139}) {
            const wg::F3Layout f = wg::f3_layout_rt(nx, 12, nz, 26, C, nrec, rag);
            for (int o : {f.off_u, f.off_apx, f.off_zx, f.off_apz, f.off_zz, f.off_v2, f.off_c2, f.off_bar})
              if (o % 2) return 1;
            if (f.off_src % 4) return 2;
            const int w = 2 * wg::g3_xsw(12, rag), zs = f.zs * nx;
            if (f.off_apx - f.off_u < 2 * f.lr * nx || f.off_zx - f.off_apx < 2 * f.maxrows * w || f.off_apz - f.off_zx < f.maxrows * w ||
                f.off_zz - f.off_apz < 2 * zs || f.off_v2 - f.off_zz < zs || f.off_rec - f.off_prof < 3 * (nx + nz) ||
                f.off_src - f.off_rec < 9 * nrec || f.off_bar - f.off_src < 8 + wg::G3_WAV_STEPS || f.total - f.off_bar < 4)
              return 3;
            const wg::A3Layout a = wg::a3_layout_rt(nx, 12, nz, 28, C, nrec, rag);
            for (int o : {a.off_vs, a.off_tx, a.off_u1x, a.off_tz, a.off_u1z, a.off_lpx, a.off_lzx, a.off_lpz, a.off_lzz, a.off_v2,
                          a.off_ga, a.off_prof, a.off_opb, a.off_src})
              if (o % 2) return 4;
            if (a.off_u1x - a.off_tx < a.maxrows * w || a.off_lzx - a.off_lpx < a.maxrows * w || a.off_opb - a.off_prof < 3 * (nx + nz))
              return 5;
          }
  return 0;
}
"""


def test_arrays_are_aligned_and_apart(tmp_path):
    csrc = ROOT / "wgnet_gb300" / "csrc"
    text = (csrc / "wave_kernels3_layout.h").read_text()
    device = (csrc / "wave_device.cuh").read_text()
    # the two row helpers of the device header, without its inline PTX
    rows = device[device.index("__host__ __device__ inline int split_row"):device.index("// Forward shared-memory layout")]
    text = text.replace('#include "wave_device.cuh"', "namespace wg {\nconstexpr int FD_PAD = 2;\n" + rows + "}\n")
    (tmp_path / "layout.h").write_text(text.replace("#pragma once", ""))
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-o", str(exe), str(tmp_path / "t.cpp")], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
