"""The assignment of a CTA's parts to its warps (no GPU): every part exactly once for any segment count, and
the schedulers' loads within two of the heaviest parts of each other where the warps divide evenly."""

from __future__ import annotations

import subprocess

from conftest import ROOT

SOURCE = r"""
#include "MAP"
int main() {
  const wg::WarpCosts costs[] = {{10, 5, 5, 0}, {10, 2, 2, 0}, {10, 30, 30, 4}, {10, 0, 0, 0}};
  for (const auto& c : costs)
    for (int C = 1; C <= 8; ++C)
      for (int NI = 1; NI <= 3; ++NI)
        for (int NSEG = 1; NSEG * (1 + NI) <= 32; ++NSEG)
          for (int S = 2; S <= 10; S += 4) {
            const int nz = C * S * NSEG + 3, W = 1 + NI, n = NSEG * W;  // the last CTA has rows beyond its segments
            int bounds[9];
            for (int r = 0; r <= C; ++r) bounds[r] = 2 + (nz - 4) * r / C;
            const wg::WarpMap m = wg::map_warps(bounds, C, S, NSEG, NI, nz, 24, c);
            for (int r = 0; r < C; ++r) {
              unsigned seen = 0;
              long load[4] = {}, most = 0;
              for (int w = 0; w < n; ++w) {
                const int v = m.id[r][w];
                if (v >= n || (seen >> v & 1)) return 1;
                seen |= 1u << v;
                long cost = 0;
                for (int z = bounds[r] + v / W * S; z < bounds[r] + (v / W + 1) * S && z < bounds[r + 1]; ++z)
                  cost += c.row + (v % W == 0 ? c.pml : 0) + (z < 24 || z >= nz - 24 ? c.strip : 0) +
                          ((r > 0 && z < bounds[r] + 2) || (r < C - 1 && z >= bounds[r + 1] - 2) ? c.halo : 0);
                load[w % 4] += cost;
                most = cost > most ? cost : most;
              }
              if (n % 4) continue;
              for (int a = 0; a < 4; ++a)
                for (int b = 0; b < 4; ++b)
                  if (load[a] - load[b] > 2 * most) return 2;
            }
          }
  return 0;
}
"""


def test_every_part_has_one_warp(tmp_path):
    src = ROOT / "wgnet_gb300" / "csrc" / "wave_warp_map.h"
    (tmp_path / "t.cpp").write_text(SOURCE.replace("MAP", str(src)))
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-o", str(exe), str(tmp_path / "t.cpp")], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
