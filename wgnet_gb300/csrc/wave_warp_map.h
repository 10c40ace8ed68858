// Which warp of a generation-3 CTA takes which part of its rows (plain C++: host and device).
#pragma once

namespace wg {

// Part of each warp, by CTA rank and warp: segment * (1 + interior warps) + role (role 0: the PML warp).
struct WarpMap {
  unsigned char id[8][32];
};

// Cost of a row per step, in tenths of an interior warp's row outside the strips, and what the PML warp,
// a row in a z strip and a row exchanged with a neighbouring CTA add to it.
struct WarpCosts {
  int row, pml, strip, halo;
};

// Shapes whose warps take the host's assignment. Measured (us; 64 models of 70 x 70, or 4 in
// clusters of three; 200 steps forward / adjoint), fixed roles -> map: {C 2, S 5} 4139 -> 4012 / 4800 ->
// 4880 (the adjoint takes {2, 4}), {2, 4} 4680 -> 4590 / 5240 -> 4660, {3, 4} 716 -> 692 / 771 -> 750.
// Elsewhere the map's registers or its order cost more than the balance gives: {3, 3} 696 -> 717, {4, 4}
// 590 -> 607, and with several interior warps per segment the adjoint spills (6.0 -> 6.6 ms on 100 x 100).
constexpr bool warps_mapped(int C, int S, int NI) { return NI == 1 && (C == 2 || (C == 3 && S == 4)); }

// Warp w issues from scheduler w % 4, and the parts of a CTA differ by up to a factor of four (PML warp or
// interior warp, z-strip rows or not): the heaviest part left goes to the scheduler with the least to
// issue so far that has a warp free. CTA r has the rows [bounds[r], bounds[r + 1]) of nz; segments of S
// rows, NSEG of them (at most 32 warps), NI interior warps each; rows z < region and z >= nz - region
// are strip rows.
inline WarpMap map_warps(const int* bounds, int C, int S, int NSEG, int NI, int nz, int region, const WarpCosts& c) {
  WarpMap m{};
  const int W = 1 + NI, n = NSEG * W;
  for (int rank = 0; rank < C && rank < 8; ++rank) {
    const int r0 = bounds[rank], r1 = bounds[rank + 1];
    int cost[32], order[32];
    for (int v = 0; v < n; ++v) {
      cost[v] = 0;
      for (int z = r0 + (v / W) * S; z < r0 + (v / W + 1) * S && z < r1; ++z) {
        cost[v] += c.row + (v % W == 0 ? c.pml : 0) + (z < region || z >= nz - region ? c.strip : 0);
        if ((rank > 0 && z < r0 + 2) || (rank < C - 1 && z >= r1 - 2)) cost[v] += c.halo;
      }
      int at = v;  // insertion by falling cost
      for (; at > 0 && cost[order[at - 1]] < cost[v]; --at) order[at] = order[at - 1];
      order[at] = v;
    }
    int load[4] = {}, used[4] = {};
    for (int k = 0; k < n; ++k) {
      int best = -1;
      for (int q = 0; q < 4; ++q)
        if (4 * used[q] + q < n && (best < 0 || load[q] < load[best])) best = q;
      const int last = (n - 1 - best) / 4;
      m.id[rank][4 * (last - used[best]) + best] = static_cast<unsigned char>(order[k]);
      load[best] += cost[order[k]];
      ++used[best];
    }
  }
  return m;
}

}  // namespace wg
