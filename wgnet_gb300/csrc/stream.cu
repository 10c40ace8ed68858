// Streamed path for grids too large for the resident kernels (for example 844 x 344 padded cells,
// 800 x 300 visible at 5 m): the wavefields of every (model, shot) unit live in HBM and each time
// step is one persistent launch over all units' tiles.
//
// A tile is 64 x 32 cells (x by z). A CTA walks the tiles of the step (unit-major, so neighbouring
// CTAs share halos in L2) with a two-stage TMA pipeline: while it updates one tile, the next tile's
// wavefield with its halo (72 x 36 floats; the x halo is rounded to 16 bytes) is already being
// copied into shared memory by cp.async.bulk.tensor, completion signalled on an mbarrier. Each
// thread owns a column pair over 2 (forward) or 4 rows; the vertical neighbours come from its column in shared
// memory, the horizontal ones from float2 loads beside it. Tiles that touch the C-PML read and
// write the packed PML strips (global memory, L1/L2 resident); interior tiles skip them entirely.
//
// Arithmetic follows the reference's operation order (splatForward.wgsl:48-121 and
// splatAdjoint.wgsl:58-131, restated in the resident kernels) with -fmad=false, so traces and
// gradients equal the f32 restatement bit for bit. The PML formulas are applied to every column
// pair that has a cell inside the adjoint's PML region; on cells outside a region the profiles are
// zero and the PML formula reduces exactly to the interior one.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "wave_launch.h"
#include "wave_packed.cuh"
#include "wgnet_gb300.h"

namespace wg {
namespace {

constexpr int TX_ = 64, TZ_ = 32;           // tile of cells per CTA iteration
constexpr int HX = 4, HZ = 2;               // halo loaded on each side (x rounded to 16 bytes)
constexpr int BX = TX_ + 2 * HX;            // 72 columns in shared memory
constexpr int BZ = TZ_ + 2 * HZ;            // 36 rows
constexpr int NTH = 256;                    // adjoint: 32 column pairs x 8 groups of 4 rows
constexpr int RPT = 4;                      // its rows per thread
constexpr unsigned kTileBytes = BX * BZ * 4;
constexpr long kWaitLimit = 1L << 22;       // mbarrier polls before giving up

struct SArgs {
  int nx, nz, units, shots;
  int tiles_x, tiles_z;
  int ssw;         // packed strip width per side (x strips: columns, z strips: rows)
  int region;      // PML region used for both axes (the adjoint's, pml + 3 FD_PAD)
  int nt, t, seg_t0;
  float rh, dt2, d2a, d2b;
  const float* prof;     // ax bx dbx (nx) | az bz dbz (nz)
  const float* wavelet;
  Stations st;
  const float* vel;      // [models][nz][nx] clamped padded velocity
  int rec_z0, rec_z1;    // rows holding receiver corners
  const int* tile_rec_start;  // [tiles + 1] receivers recorded by each tile (forward)
  const int* tile_rec;
  int* status;
  float* W;              // forward: wavefield ping-pong [2][units][nz][nx]; adjoint: lambda
  float* PX;             // forward a*psi_x ping-pong [2][units][nz][2 ssw]; adjoint psi_x ping-pong
  float* ZX;             // forward zeta_x [units][nz][2 ssw]; adjoint zeta_x ping-pong
  float* PZ;             // forward a*psi_z ping-pong [2][units][2 ssw][nx]; adjoint psi_z ping-pong
  float* ZZ;             // forward zeta_z [units][2 ssw][nx]; adjoint zeta_z ping-pong
  float* traces;         // [units][nt][nrec]
  float* stored;         // [units][seg][nz][nx], step t at t - seg_t0
  int seg;
  const float* residual; // [units][nt][nrec]
  float* gacc;           // [units][nz][nx]
  alignas(8) float nz2[2];  // -0, for packed products (wave_packed.cuh)
};

__device__ __forceinline__ float2 lds2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 ldg2(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }
__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }

__device__ __forceinline__ void put2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Bounded wait for the phase with parity `parity`; false when `limit` polls are reached.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, long limit = kWaitLimit) {
  const unsigned a = smem_u32(bar);
  for (long i = 0; i < limit; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// 3-D tiled TMA load of one tile box (x, z, buffer*units + unit) into shared memory.
__device__ __forceinline__ void tma_load(float* dst, const CUtensorMap* map, int x, int z, int u, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(z), "r"(u), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ int xstrip(int x, int nx, int ssw) { return x < ssw ? x : x - (nx - 2 * ssw); }

__device__ __forceinline__ void report(int* status) { atomicCAS(status, 0, ST_CUDA); }

// ------------------------------------------------------------------------------------------------
// Forward step t: u_next = v^2 dt^2 w + 2 u - u_prev over every unit, receivers read before the
// update, source after it (splatForward.wgsl:48-121).
// ------------------------------------------------------------------------------------------------
struct FwdMaps {
  CUtensorMap u;  // wavefield with halo: 72 x 36 boxes over [2 units][nz][nx]
  CUtensorMap p;  // wavefield without halo (the previous step): 64 x 32 boxes
  CUtensorMap v;  // velocity: 64 x 32 boxes over [models][nz][nx]
};
constexpr int FST = 2;                                        // forward pipeline stages
constexpr int FSTAGE_F = BZ * BX + 2 * TZ_ * TX_;             // floats per stage: U | P | V
constexpr size_t kFwdSmem = FST * FSTAGE_F * 4 + 128 + 16 * FST;

constexpr int FNTH = 512, FRPT = 2;    // forward: consumer threads, rows per thread
constexpr int FWD_THREADS = FNTH + 32;  // consumer warps + 1 producer warp

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One tile of a step's work, decoded once per CTA (by the thread that issues its copies) instead of by
// every thread: the divisions and the look-up of the shot's source were a third of an interior tile's
// instructions.
struct Job {
  int unit, tile, x0, z0;
  int shot, inner, src, model;  // inner: interior formulas only; src: the source's corners touch the tile
};

// Walks the jobs blockIdx.x, blockIdx.x + gridDim.x, ... of a step.
struct JobWalk {
  int unit, tile, du, dt;
  __device__ __forceinline__ explicit JobWalk(const SArgs& a) {
    const int tiles = a.tiles_x * a.tiles_z, first = blockIdx.x, step = gridDim.x;
    unit = first / tiles;
    tile = first - unit * tiles;
    du = step / tiles;
    dt = step - du * tiles;
  }
  __device__ __forceinline__ void advance(const SArgs& a) {
    const int tiles = a.tiles_x * a.tiles_z;
    unit += du;
    tile += dt;
    if (tile >= tiles) {
      tile -= tiles;
      ++unit;
    }
  }
  // A tile (with its halo) clear of the PML strips, the grid frame, the receivers' rows and this
  // unit's source corners is an inner one: every pair of every row takes the interior formulas.
  __device__ __forceinline__ Job decode(const SArgs& a) const {
    Job j;
    const int tz = tile / a.tiles_x;
    j.unit = unit;
    j.tile = tile;
    j.x0 = (tile - tz * a.tiles_x) * TX_;
    j.z0 = tz * TZ_;
    j.model = unit / a.shots;
    j.shot = unit - j.model * a.shots;
    const int c = __ldg(&a.st.src_cell[4 * j.shot]);  // the first of the 2 x 2 corner cells
    const int cz = c / a.nx, cx = c - cz * a.nx;
    j.src = cz + 1 >= j.z0 && cz < j.z0 + TZ_ && cx + 1 >= j.x0 && cx < j.x0 + TX_;
    const int m = a.ssw;
    j.inner = !j.src && j.x0 - HX >= m && j.x0 + TX_ + HX <= a.nx - m && j.z0 - HZ >= m && j.z0 + TZ_ + HZ <= a.nz - m &&
              !(j.z0 + TZ_ > a.rec_z0 && j.z0 <= a.rec_z1);
    return j;
  }
};

// Programmatic dependent launch: the next step's kernel may be scheduled as soon as this one's CTAs leave,
// and waits here, after its prologue, for this one's results.
__device__ __forceinline__ void wait_for_previous_step() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_step_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void prefetch_map(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// Bit 2 r + j: cell (zr + r, x + j) is a corner of the source.
template <int RPT>
__device__ __forceinline__ unsigned source_bits(const SArgs& a, int shot, int zr, int x) {
  unsigned m = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int d = __ldg(&a.st.src_cell[4 * shot + k]) - (zr * a.nx + x);
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const unsigned o = static_cast<unsigned>(d - r * a.nx);
      if (o < 2u) m |= 1u << (2 * r + o);
    }
  }
  return m;
}

// Issue the three copies of a job into stage buffer `st` with barrier `bar`.
__device__ __forceinline__ void issue_fwd(const SArgs& a, const FwdMaps& m, float* st, uint64_t* bar, const Job& j,
                                          int par) {
  mbar_expect_tx(bar, FSTAGE_F * 4);
  tma_load(st, &m.u, j.x0 - HX, j.z0 - HZ, par * a.units + j.unit, bar);
  tma_load(st + BZ * BX, &m.p, j.x0, j.z0, (1 - par) * a.units + j.unit, bar);
  tma_load(st + BZ * BX + TZ_ * TX_, &m.v, j.x0, j.z0, j.model, bar);
}

// Warp-specialised: the last warp (one lane) streams the jobs' tiles into FST stages (waiting on each
// stage's "empty" barrier before refilling it), the others update the tiles and release each stage
// with one arrival per warp. No CTA-wide barrier per tile: consumer warps run up to FST tiles
// apart. Every wait is bounded; a consumer that gives up records the error and leaves; the
// producer that gives up records it and waits (bounded) for the copies it issued.
// Latency bounds it: the C-PML tiles (43 % of those of the 844 x 344 grid) wait on their strips' values in
// L2. Decoding a job once per CTA, packed arithmetic (wave_packed.cuh) and the overlapped launch took a step
// of 16 shots of that grid from 38.5 to 31.5 us (storing terms) and from 36.2 to 30.9 (not); 16 warps of
// two rows a thread instead of 8 of four, with two stages, to 27.9 and 25.8, for all that they spill a
// little at 56 registers (three stages: 28.6 and 26.0; three CTAs of 8 warps: 29.0 and 26.8; four: 40.4
// and 37.4). Loading the strips ahead for four rows spilled and measured slower (44 us). The adjoint holds
// more and stays at 8 warps of four rows (16 of two: 55.8 against 51.5 us).
template <bool TRACES, bool STORE>
__global__ void __launch_bounds__(FWD_THREADS, 2) fwd_stream_kernel(const __grid_constant__ FwdMaps maps,
                                                                    const __grid_constant__ SArgs a) {
  extern __shared__ __align__(128) float fsm_raw[];
  float* stage = fsm_raw + ((128 - (smem_u32(fsm_raw) & 127)) & 127) / 4;  // [FST][U | P | V]
  uint64_t* full = reinterpret_cast<uint64_t*>(stage + FST * FSTAGE_F);
  uint64_t* empty = full + FST;
  __shared__ Job info[FST];
  const int tid = threadIdx.x;
  const int jobs = a.units * a.tiles_x * a.tiles_z;
  const int par = a.t & 1;
  const int nx = a.nx, nz = a.nz, ssw = a.ssw, region = a.region;
  const size_t cells = static_cast<size_t>(nx) * nz;
  const Pk pk{make_float2(a.nz2[0], a.nz2[1])};
  if (tid == 0) {
    for (int k = 0; k < FST; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], FNTH / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid == FNTH) {
    prefetch_map(&maps.u);
    prefetch_map(&maps.p);
    prefetch_map(&maps.v);
  }
  __syncthreads();
  wait_for_previous_step();
  let_next_step_launch();
  if (tid >= FNTH) {  // producer warp
    if (tid == FNTH) {
      int issued = 0;
      JobWalk walk(a);
      for (int job = blockIdx.x; job < jobs; job += gridDim.x, ++issued, walk.advance(a)) {
        const int s = issued % FST;
        if (issued >= FST && !mbar_wait(&empty[s], (issued / FST - 1) & 1)) {
          report(a.status);
          for (int k = 1; k <= FST && issued - k >= 0; ++k)  // the copies still landing
            mbar_wait(&full[(issued - k) % FST], ((issued - k) / FST) & 1);
          return;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        const Job j = walk.decode(a);
        info[s] = j;  // released to the consumers by the arrival on the full barrier
        issue_fwd(a, maps, stage + s * FSTAGE_F, &full[s], j, par);
      }
    }
    return;
  }
  const float f = __ldg(&a.wavelet[a.t]);
  const int pc = tid & 31, grp = tid >> 5;
  const size_t xs_unit = static_cast<size_t>(nz) * 2 * ssw;  // floats per unit of an x strip array
  const size_t zs_unit = static_cast<size_t>(2) * ssw * nx;
  const int sx = 2 * pc + HX, sz = FRPT * grp + HZ;
  int job = blockIdx.x;
  for (int i = 0; job < jobs; ++i, job += gridDim.x) {
    const int s = i % FST;
    if (!mbar_wait(&full[s], (i / FST) & 1)) {
      report(a.status);
      return;
    }
    const Job j = info[s];
    const int x = j.x0 + 2 * pc;
    const int zr = j.z0 + FRPT * grp;
    float* Wn = a.W + (static_cast<size_t>(1 - par) * a.units + j.unit) * cells;
    const float* T = stage + s * FSTAGE_F;
    const float* Pt = T + BZ * BX + FRPT * grp * TX_ + 2 * pc;
    const float* Vt = Pt + TZ_ * TX_;
    float* stp = STORE ? a.stored + (static_cast<size_t>(j.unit) * a.seg + (a.t - a.seg_t0)) * cells : nullptr;
    float2 col[FRPT + 4];
#pragma unroll
    for (int k = 0; k < FRPT + 4; ++k) col[k] = lds2(T + (sz - 2 + k) * BX + sx);

    if (j.inner) {
      // interior tile: no frame, PML, receivers or sources
#pragma unroll
      for (int r = 0; r < FRPT; ++r) {
        const int cell = (zr + r) * nx + x;
        const float2 A = lds2(T + (sz + r) * BX + sx - 2), B = lds2(T + (sz + r) * BX + sx + 2), u = col[r + 2];
        const float2 w = add2(pk.second(u, side_sum(A, u, B), add2(B, A), a.d2a, a.d2b),
                              pk.second(u, add2(col[r + 3], col[r + 1]), add2(col[r + 4], col[r]), a.d2a, a.d2b));
        const float2 v = lds2(Vt + r * TX_);
        const float2 n = sub2(add2(pk.mul(scale2(a.dt2, mul2(v, v)), w), add2(u, u)), lds2(Pt + r * TX_));
        if (STORE) __stcs(reinterpret_cast<float2*>(stp + cell), mul2(scale2(a.dt2, add2(v, v)), w));
        *reinterpret_cast<float2*>(Wn + cell) = n;
      }
      __syncwarp();
      if (pc == 0) mbar_arrive(&empty[s]);
      continue;
    }

    if (TRACES) {
      const int r0 = a.tile_rec_start[j.tile], r1 = a.tile_rec_start[j.tile + 1];
      for (int k = r0 + tid; k < r1; k += FNTH) {
        const int r = a.tile_rec[k];
        float acc = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int cell = a.st.rec_cell[4 * r + c];
          const int cz = cell / nx - (j.z0 - HZ), cx = cell % nx - (j.x0 - HX);
          acc = acc + a.st.rec_w[4 * r + c] * T[cz * BX + cx];
        }
        a.traces[(static_cast<size_t>(j.unit) * a.nt + a.t) * a.st.nrec + r] = acc;
      }
    }

    const bool xok = x >= FD_PAD && x + 1 < nx - FD_PAD;
    const bool xpml = x < region || x + 1 >= nx - region;
    const unsigned srcm = j.src ? source_bits<FRPT>(a, j.shot, zr, x) : 0u;
    float2 ax = make_float2(0.f, 0.f), bx = ax, dbx = ax;
    if (xok && xpml) {
      ax = ldg2(a.prof + x);
      bx = ldg2(a.prof + nx + x);
      dbx = ldg2(a.prof + 2 * nx + x);
    }
    const float2 opbx = make_float2(1.0f + bx.x, 1.0f + bx.y);
    const float* PXc = a.PX + (static_cast<size_t>(par) * a.units + j.unit) * xs_unit;
    float* PXn = a.PX + (static_cast<size_t>(1 - par) * a.units + j.unit) * xs_unit;
    float* ZXo = a.ZX + static_cast<size_t>(j.unit) * xs_unit;
    const float* PZc = a.PZ + (static_cast<size_t>(par) * a.units + j.unit) * zs_unit;
    float* PZn = a.PZ + (static_cast<size_t>(1 - par) * a.units + j.unit) * zs_unit;
    float* ZZo = a.ZZ + static_cast<size_t>(j.unit) * zs_unit;
    const int xc = xstrip(x, nx, ssw);
    // the rows' stores go to other cells than the strips' loads: through restrict-qualified pointers the
    // loads of a row may be issued ahead of the stores of the row before
    auto rows = [&](float* __restrict__ wn, float* __restrict__ pxn, float* __restrict__ zxo, float* __restrict__ pzn,
                    float* __restrict__ zzo, float* __restrict__ sto) {
#pragma unroll
      for (int r = 0; r < FRPT; ++r) {
        const int z = zr + r;
        if (!xok || z < FD_PAD || z >= nz - FD_PAD) continue;
        const int cell = z * nx + x;
        const float2 A = lds2(T + (sz + r) * BX + sx - 2), B = lds2(T + (sz + r) * BX + sx + 2), u = col[r + 2];
        float2 w = pk.second(u, side_sum(A, u, B), add2(B, A), a.d2a, a.d2b);
        if (xpml) {
          const float* row = PXc + z * 2 * ssw + xc;
          const float2 P0 = ld2(row - 2), P1 = ld2(row), P2 = ld2(row + 2);
          const float2 Z = ld2(zxo + z * 2 * ssw + xc);
          const float2 d1 = pk.first(side_diff(A, u, B), sub2(B, A), a.rh);
          const float2 da = pk.first(side_diff(P0, P1, P2), sub2(P2, P0), a.rh);
          const float2 tmp = add2(add2(pk.mul(opbx, w), pk.mul(dbx, d1)), da);
          const float2 az = pk.mul(ax, Z);
          w = add2(pk.mul(opbx, tmp), az);
          *reinterpret_cast<float2*>(zxo + z * 2 * ssw + xc) = add2(pk.mul(bx, tmp), az);
          *reinterpret_cast<float2*>(pxn + z * 2 * ssw + xc) = mul2(ax, add2(pk.mul(bx, d1), P1));
        }
        const float2 zm2 = col[r], zm1 = col[r + 1], zp1 = col[r + 3], zp2 = col[r + 4];
        const float2 d2z = pk.second(u, add2(zp1, zm1), add2(zp2, zm2), a.d2a, a.d2b);
        if (z < region || z >= nz - region) {
          const int zc = z < ssw ? z : z - (nz - 2 * ssw);
          const float az = __ldg(&a.prof[3 * nx + z]), bz = __ldg(&a.prof[3 * nx + nz + z]),
                      dbz = __ldg(&a.prof[3 * nx + 2 * nz + z]);
          const float opbz = 1.0f + bz;
          const float* q = PZc + zc * nx + x;
          const float2 Qm2 = ld2(q - 2 * nx), Qm1 = ld2(q - nx), Q0 = ld2(q), Qp1 = ld2(q + nx), Qp2 = ld2(q + 2 * nx);
          const float2 Z = ld2(zzo + zc * nx + x);
          const float2 d1 = pk.first(sub2(zp1, zm1), sub2(zp2, zm2), a.rh);
          const float2 da = pk.first(sub2(Qp1, Qm1), sub2(Qp2, Qm2), a.rh);
          const float2 tmp = add2(add2(pk.scale(opbz, d2z), pk.scale(dbz, d1)), da);
          const float2 aZ = pk.scale(az, Z);
          w = add2(w, add2(pk.scale(opbz, tmp), aZ));
          *reinterpret_cast<float2*>(zzo + zc * nx + x) = add2(pk.scale(bz, tmp), aZ);
          *reinterpret_cast<float2*>(pzn + zc * nx + x) = scale2(az, add2(pk.scale(bz, d1), Q0));
        } else {
          w = add2(w, d2z);
        }
        const float2 v = lds2(Vt + r * TX_);
        const float2 v2 = scale2(a.dt2, mul2(v, v));
        float2 n = sub2(add2(pk.mul(v2, w), add2(u, u)), lds2(Pt + r * TX_));
        if (STORE) __stcs(reinterpret_cast<float2*>(sto + cell), mul2(scale2(a.dt2, add2(v, v)), w));
        if (srcm & (3u << (2 * r))) {
          const int* sc = a.st.src_cell + 4 * j.shot;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (cell == sc[k]) n.x = n.x + (((-v2.x) * a.st.src_w[4 * j.shot + k]) * f);
            if (cell + 1 == sc[k]) n.y = n.y + (((-v2.y) * a.st.src_w[4 * j.shot + k]) * f);
          }
        }
        *reinterpret_cast<float2*>(wn + cell) = n;
      }
    };
    rows(Wn, PXn, ZXo, PZn, ZZo, stp);
    __syncwarp();
    if (pc == 0) mbar_arrive(&empty[s]);  // this warp is done with the stage
  }
}

// ------------------------------------------------------------------------------------------------
// Temporally blocked forward: TB_T steps per launch. Each job (unit, 64 x 32 tile) takes its tile
// with a halo of 2 TB_T cells per side (the stencil reaches 2 cells per step) into shared memory:
// u(t), u(t-1) and the velocity by TMA (double-buffered: the next job's boxes land while this one
// computes), and, on tiles that reach a C-PML strip, a*psi and zeta of the strip cells. It then
// advances the region TB_T steps in shared memory, the computed region shrinking by 2 cells per
// side per step, and writes back the tile: the halo cells are computed by every tile that holds
// them, with the same operations on the same values, so each cell's value is the per-step kernel's
// bit for bit (sources are injected into halo copies too; receivers are recorded by the tile that
// holds their first corner). Per step the wavefield crosses HBM once per TB_T steps instead of once
// per step. The state is read from one set and written to the other (sets alternate per launch),
// so no CTA overwrites cells a neighbouring CTA still has to read. Faster than one step per launch where a
// step is mostly latency (see blocked()); on large surveys the redundant halo updates (31 % of the
// work) make it slower (41 against 31 us a step for 16 shots of the 844 x 344 grid).
// ------------------------------------------------------------------------------------------------
constexpr int TB_T = 4;                      // time steps per launch
constexpr int TB_H = 2 * TB_T;               // halo per side
constexpr int TB_RX = TX_ + 2 * TB_H;        // 80 region columns (x offset 64 k - 8: 16-byte aligned)
constexpr int TB_RZ = TZ_ + 2 * TB_H;        // 48 region rows
constexpr int TB_N = TB_RX * TB_RZ;          // cells of a region
constexpr int TB_THREADS = 1024;
constexpr int TB_STAGE = 3 * TB_N;           // floats per stage: u(t) | u(t-1) | v
constexpr size_t kTbSmem = static_cast<size_t>(2 * TB_STAGE + 6 * TB_N) * 4 + 2 * 8 + 128;

struct TbArgs {
  SArgs a;         // geometry, stations, profiles, traces, stored terms, status; a.t = first step
  int nsub;        // steps of this launch, 1..TB_T
  int set_in;      // state set read (the other one is written)
  float* W;        // [2 sets][2 levels: u(t), u(t-1)][units][nz][nx]
  float* PX;       // a psi_x [2 sets][units][nz][2 ssw]
  float* ZX;       // zeta_x  [2 sets][units][nz][2 ssw]
  float* PZ;       // a psi_z [2 sets][units][2 ssw][nx]
  float* ZZ;       // zeta_z  [2 sets][units][2 ssw][nx]
};

template <bool TRACES, bool STORE>
__global__ void __launch_bounds__(TB_THREADS, 1) fwd_tb_kernel(const __grid_constant__ CUtensorMap umap,
                                                               const __grid_constant__ CUtensorMap vmap,
                                                               const __grid_constant__ TbArgs p) {
  extern __shared__ __align__(128) float tsm_raw[];
  float* sm = tsm_raw + ((128 - (smem_u32(tsm_raw) & 127)) & 127) / 4;
  float* stages = sm;             // [2][u(t) | u(t-1) | v]
  float* PXA = sm + 2 * TB_STAGE;  // a psi_x, two buffers (neighbours read x +- 2)
  float* PXB = PXA + TB_N;
  float* ZXr = PXB + TB_N;         // zeta_x (owner only, updated in place)
  float* PZA = ZXr + TB_N;         // a psi_z, two buffers
  float* PZB = PZA + TB_N;
  float* ZZr = PZB + TB_N;
  uint64_t* full = reinterpret_cast<uint64_t*>(ZZr + TB_N);
  const SArgs& a = p.a;
  const int tid = threadIdx.x;
  const int tiles = a.tiles_x * a.tiles_z;
  const int jobs = a.units * tiles;
  const int nx = a.nx, nz = a.nz, ssw = a.ssw, region = a.region;
  const size_t cells = static_cast<size_t>(nx) * nz;
  const size_t xs_unit = static_cast<size_t>(nz) * 2 * ssw, zs_unit = static_cast<size_t>(2) * ssw * nx;
  const int set_out = 1 - p.set_in;
  const Pk pk{make_float2(a.nz2[0], a.nz2[1])};
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_map(&umap);
    prefetch_map(&vmap);
  }
  __syncthreads();
  wait_for_previous_step();
  let_next_step_launch();
  auto issue = [&](int job, int s) {
    const int unit = job / tiles, tile = job % tiles;
    const int x = (tile % a.tiles_x) * TX_ - TB_H, z = (tile / a.tiles_x) * TZ_ - TB_H;
    float* st = stages + s * TB_STAGE;
    mbar_expect_tx(&full[s], TB_STAGE * 4);
    tma_load(st, &umap, x, z, (p.set_in * 2 + 0) * a.units + unit, &full[s]);
    tma_load(st + TB_N, &umap, x, z, (p.set_in * 2 + 1) * a.units + unit, &full[s]);
    tma_load(st + 2 * TB_N, &vmap, x, z, unit / a.shots, &full[s]);
  };
  if (tid == 0 && static_cast<int>(blockIdx.x) < jobs) issue(blockIdx.x, 0);
  int i = 0;
  for (int job = blockIdx.x; job < jobs; job += gridDim.x, ++i) {
    const int s = i & 1;
    const bool next = job + static_cast<int>(gridDim.x) < jobs;
    if (tid == 0 && next) {  // the other stage's last job ended with a CTA barrier
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(job + gridDim.x, 1 - s);
    }
    const bool ok = mbar_wait(&full[s], (i >> 1) & 1);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        report(a.status);
        if (next) mbar_wait(&full[1 - s], ((i + 1) >> 1) & 1);  // the copies still landing (bounded)
      }
      return;
    }
    const int unit = job / tiles, tile = job % tiles;
    const int x0 = (tile % a.tiles_x) * TX_, z0 = (tile / a.tiles_x) * TZ_;
    const int rx0 = x0 - TB_H, rz0 = z0 - TB_H;  // region origin in grid coordinates
    const int shot = unit % a.shots;
    float* U = stages + s * TB_STAGE;
    float* UP = U + TB_N;
    const float* V = UP + TB_N;
    const bool pml_tile = rx0 < ssw || rx0 + TB_RX > nx - ssw || rz0 < ssw || rz0 + TB_RZ > nz - ssw;
    if (pml_tile) {
      const float* PXi = p.PX + (static_cast<size_t>(p.set_in) * a.units + unit) * xs_unit;
      const float* ZXi = p.ZX + (static_cast<size_t>(p.set_in) * a.units + unit) * xs_unit;
      const float* PZi = p.PZ + (static_cast<size_t>(p.set_in) * a.units + unit) * zs_unit;
      const float* ZZi = p.ZZ + (static_cast<size_t>(p.set_in) * a.units + unit) * zs_unit;
      // pairs of columns (a pair lies in a strip or outside it: nx and ssw are even), loaded ahead of
      // their stores
      constexpr int PER = (TB_N / 2 + TB_THREADS - 1) / TB_THREADS;
      float2 px[PER], zx[PER], pz[PER], zz[PER];
#pragma unroll
      for (int it = 0; it < PER; ++it) {
        const int c = 2 * (tid + it * TB_THREADS);
        const int z = rz0 + c / TB_RX, x = rx0 + c % TB_RX;
        px[it] = zx[it] = pz[it] = zz[it] = make_float2(0.f, 0.f);
        if (c < TB_N && x >= 0 && x < nx && z >= 0 && z < nz) {
          if (x < ssw || x >= nx - ssw) {
            const int k = z * 2 * ssw + xstrip(x, nx, ssw);
            px[it] = ld2(PXi + k);
            zx[it] = ld2(ZXi + k);
          }
          if (z < ssw || z >= nz - ssw) {
            const int k = (z < ssw ? z : z - (nz - 2 * ssw)) * nx + x;
            pz[it] = ld2(PZi + k);
            zz[it] = ld2(ZZi + k);
          }
        }
      }
#pragma unroll
      for (int it = 0; it < PER; ++it) {
        const int c = 2 * (tid + it * TB_THREADS);
        if (c >= TB_N) break;
        // both buffers: a*psi of strip cells outside the C-PML region is never updated
        put2(PXA + c, px[it]);
        put2(PXB + c, px[it]);
        put2(ZXr + c, zx[it]);
        put2(PZA + c, pz[it]);
        put2(PZB + c, pz[it]);
        put2(ZZr + c, zz[it]);
      }
      __syncthreads();
    }
    const int* sc = a.st.src_cell + 4 * shot;
    const float* sw = a.st.src_w + 4 * shot;
    const int sc0 = __ldg(&sc[0]), sc1 = __ldg(&sc[1]), sc2 = __ldg(&sc[2]), sc3 = __ldg(&sc[3]);
    // the source's 2 x 2 corners against the region
    const int srz = sc0 / nx - rz0, srx = sc0 % nx - rx0;
    const bool src_near = srz >= -1 && srz < TB_RZ && srx >= -1 && srx < TB_RX;
    for (int k = 0; k < p.nsub; ++k) {
      const int t = a.t + k;
      const float f = __ldg(&a.wavelet[t]);
      const float* Uc = (k & 1) ? UP : U;  // u(t)
      float* Un = (k & 1) ? U : UP;        // u(t - 1), overwritten by u(t + 1)
      const float* Pc = (k & 1) ? PXB : PXA;
      float* Pn = (k & 1) ? PXA : PXB;
      const float* Qc = (k & 1) ? PZB : PZA;
      float* Qn = (k & 1) ? PZA : PZB;
      if (TRACES) {
        const int r0 = a.tile_rec_start[tile], r1 = a.tile_rec_start[tile + 1];
        for (int q = r0 + tid; q < r1; q += TB_THREADS) {
          const int r = a.tile_rec[q];
          float acc = 0.0f;
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            const int cell = a.st.rec_cell[4 * r + cc];
            acc = acc + a.st.rec_w[4 * r + cc] * Uc[(cell / nx - rz0) * TB_RX + (cell % nx - rx0)];
          }
          a.traces[(static_cast<size_t>(unit) * a.nt + t) * a.st.nrec + r] = acc;
        }
      }
      float* stp = STORE ? a.stored + (static_cast<size_t>(unit) * a.seg + (t - a.seg_t0)) * cells : nullptr;
      const int m = 2 * (k + 1);  // region of step k: 2 (k + 1) cells inside the loaded one
      const int pairs = (TB_RX - 2 * m) / 2, rows = TB_RZ - 2 * m;
      // idx / pairs for idx < pairs rows <= 1672 and 32 <= pairs <= 38: the reciprocal's error, under
      // pairs / 2^16 per unit, stays below one
      const int inv = (65536 + pairs - 1) / pairs;
      for (int idx = tid; idx < pairs * rows; idx += TB_THREADS) {
        const int qz = (idx * inv) >> 16;
        const int lz = m + qz, lx = m + 2 * (idx - qz * pairs);
        const int z = rz0 + lz, x = rx0 + lx;
        if (z < FD_PAD || z >= nz - FD_PAD || x < FD_PAD || x + 1 >= nx - FD_PAD) continue;
        const int c = lz * TB_RX + lx;
        const int cell = z * nx + x;
        const float2 u = lds2(Uc + c), A = lds2(Uc + c - 2), B = lds2(Uc + c + 2);
        float2 w = pk.second(u, side_sum(A, u, B), add2(B, A), a.d2a, a.d2b);
        if (pml_tile && (x < region || x + 1 >= nx - region)) {
          const float2 ax = ldg2(a.prof + x), bx = ldg2(a.prof + nx + x), dbx = ldg2(a.prof + 2 * nx + x);
          const float2 opbx = make_float2(1.0f + bx.x, 1.0f + bx.y);
          const float2 P0 = lds2(Pc + c - 2), P1 = lds2(Pc + c), P2 = lds2(Pc + c + 2);
          const float2 Z = lds2(ZXr + c);
          const float2 d1 = pk.first(side_diff(A, u, B), sub2(B, A), a.rh);
          const float2 da = pk.first(side_diff(P0, P1, P2), sub2(P2, P0), a.rh);
          const float2 tmp = add2(add2(pk.mul(opbx, w), pk.mul(dbx, d1)), da);
          const float2 az = pk.mul(ax, Z);
          w = add2(pk.mul(opbx, tmp), az);
          put2(ZXr + c, add2(pk.mul(bx, tmp), az));
          put2(Pn + c, mul2(ax, add2(pk.mul(bx, d1), P1)));
        }
        const float2 zm2 = lds2(Uc + c - 2 * TB_RX), zm1 = lds2(Uc + c - TB_RX), zp1 = lds2(Uc + c + TB_RX),
                     zp2 = lds2(Uc + c + 2 * TB_RX);
        const float2 d2z = pk.second(u, add2(zp1, zm1), add2(zp2, zm2), a.d2a, a.d2b);
        if (pml_tile && (z < region || z >= nz - region)) {
          const float az = __ldg(&a.prof[3 * nx + z]), bz = __ldg(&a.prof[3 * nx + nz + z]),
                      dbz = __ldg(&a.prof[3 * nx + 2 * nz + z]);
          const float opbz = 1.0f + bz;
          const float2 Qm2 = lds2(Qc + c - 2 * TB_RX), Qm1 = lds2(Qc + c - TB_RX), Q0 = lds2(Qc + c),
                       Qp1 = lds2(Qc + c + TB_RX), Qp2 = lds2(Qc + c + 2 * TB_RX);
          const float2 Z = lds2(ZZr + c);
          const float2 d1 = pk.first(sub2(zp1, zm1), sub2(zp2, zm2), a.rh);
          const float2 da = pk.first(sub2(Qp1, Qm1), sub2(Qp2, Qm2), a.rh);
          const float2 tmp = add2(add2(pk.scale(opbz, d2z), pk.scale(dbz, d1)), da);
          const float2 aZ = pk.scale(az, Z);
          w = add2(w, add2(pk.scale(opbz, tmp), aZ));
          put2(ZZr + c, add2(pk.scale(bz, tmp), aZ));
          put2(Qn + c, scale2(az, add2(pk.scale(bz, d1), Q0)));
        } else {
          w = add2(w, d2z);
        }
        const float2 v = lds2(V + c);
        const float2 v2 = scale2(a.dt2, mul2(v, v));
        float2 n = sub2(add2(pk.mul(v2, w), add2(u, u)), lds2(Un + c));
        if (STORE && lz >= TB_H && lz < TB_H + TZ_ && lx >= TB_H && lx < TB_H + TX_)
          __stcs(reinterpret_cast<float2*>(stp + cell), mul2(scale2(a.dt2, add2(v, v)), w));
        // sources: corners in the halo are injected too, so that halo copies match their owners
        if (src_near && (cell == sc0 || cell + 1 == sc0 || cell == sc1 || cell + 1 == sc1 || cell == sc2 ||
                         cell + 1 == sc2 || cell == sc3 || cell + 1 == sc3)) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int scq = q == 0 ? sc0 : q == 1 ? sc1 : q == 2 ? sc2 : sc3;
            if (cell == scq) n.x = n.x + (((-v2.x) * __ldg(&sw[q])) * f);
            if (cell + 1 == scq) n.y = n.y + (((-v2.y) * __ldg(&sw[q])) * f);
          }
        }
        put2(Un + c, n);
      }
      __syncthreads();
    }
    // write back the tile: u(t + nsub), u(t + nsub - 1), and the strip cells' C-PML state
    const int ns = p.nsub;
    const float* Ucur = (ns & 1) ? UP : U;
    const float* Uold = (ns & 1) ? U : UP;
    float* W0 = p.W + (static_cast<size_t>(set_out * 2 + 0) * a.units + unit) * cells;
    float* W1 = p.W + (static_cast<size_t>(set_out * 2 + 1) * a.units + unit) * cells;
    for (int idx = tid; idx < TZ_ * (TX_ / 4); idx += TB_THREADS) {
      const int lz = idx / (TX_ / 4), lx4 = 4 * (idx % (TX_ / 4));
      const int z = z0 + lz, x = x0 + lx4;
      if (z >= nz || x >= nx) continue;  // nx is a multiple of 4
      const int c = (lz + TB_H) * TB_RX + lx4 + TB_H;
      *reinterpret_cast<float4*>(W0 + z * nx + x) = *reinterpret_cast<const float4*>(Ucur + c);
      *reinterpret_cast<float4*>(W1 + z * nx + x) = *reinterpret_cast<const float4*>(Uold + c);
    }
    if (pml_tile) {
      const float* Pcur = (ns & 1) ? PXB : PXA;
      const float* Qcur = (ns & 1) ? PZB : PZA;
      float* PXo = p.PX + (static_cast<size_t>(set_out) * a.units + unit) * xs_unit;
      float* ZXo = p.ZX + (static_cast<size_t>(set_out) * a.units + unit) * xs_unit;
      float* PZo = p.PZ + (static_cast<size_t>(set_out) * a.units + unit) * zs_unit;
      float* ZZo = p.ZZ + (static_cast<size_t>(set_out) * a.units + unit) * zs_unit;
      for (int idx = tid; idx < TZ_ * TX_; idx += TB_THREADS) {
        const int lz = idx / TX_, lx = idx % TX_;
        const int z = z0 + lz, x = x0 + lx;
        if (z >= nz || x >= nx) continue;
        const int c = (lz + TB_H) * TB_RX + lx + TB_H;
        if (x < ssw || x >= nx - ssw) {
          const int k = z * 2 * ssw + xstrip(x, nx, ssw);
          PXo[k] = Pcur[c];
          ZXo[k] = ZXr[c];
        }
        if (z < ssw || z >= nz - ssw) {
          const int k = (z < ssw ? z : z - (nz - 2 * ssw)) * nx + x;
          PZo[k] = Qcur[c];
          ZZo[k] = ZZr[c];
        }
      }
    }
    __syncthreads();  // this stage and the C-PML arrays are free again
  }
}

// ------------------------------------------------------------------------------------------------
// Adjoint step t (reverse time): lambda_next = w + 2 lambda - lambda_prev + injected residuals,
// gradient += lambda * stored term (+ the source-term correction), splatAdjoint.wgsl:58-131.
// Derived terms v^2 dt^2 lambda (VS) and, in the PML strips, T = (1+b) VS + b zeta and
// U1 = db T + b psi are formed once per tile cell (halo included) in shared memory.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(NTH, 2) adj_stream_kernel(const __grid_constant__ CUtensorMap map,
                                                         const __grid_constant__ SArgs a) {
  extern __shared__ __align__(128) float dsm_raw[];
  // TMA destinations start on a 128-byte boundary
  float* dsm = dsm_raw + ((128 - (smem_u32(dsm_raw) & 127)) & 127) / 4;
  float* stage = dsm;                      // [2][BZ*BX] lambda tiles (TMA)
  float* VS = dsm + 2 * BZ * BX;           // [BZ*BX]
  float* TXs = VS + BZ * BX;
  float* U1Xs = TXs + BZ * BX;
  float* TZs = U1Xs + BZ * BX;
  float* U1Zs = TZs + BZ * BX;
  uint64_t* bar = reinterpret_cast<uint64_t*>(U1Zs + BZ * BX);
  const int tid = threadIdx.x;
  __shared__ Job info[2];
  const int jobs = a.units * a.tiles_x * a.tiles_z;
  const Pk pk{make_float2(a.nz2[0], a.nz2[1])};
  const int q = a.t & 1;  // lambda(t) in buffer q; lambda(t-1) is written into buffer 1 - q
  const int nx = a.nx, nz = a.nz, ssw = a.ssw, region = a.region;
  const size_t cells = static_cast<size_t>(nx) * nz;
  const size_t xs_unit = static_cast<size_t>(nz) * 2 * ssw;
  const size_t zs_unit = static_cast<size_t>(2) * ssw * nx;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_map(&map);
  }
  wait_for_previous_step();
  let_next_step_launch();
  // thread 0 decodes each job and issues its tile's copy, one job ahead
  JobWalk walk(a);
  auto issue = [&](int s) {
    const Job j = walk.decode(a);
    info[s] = j;
    mbar_expect_tx(&bar[s], kTileBytes);
    tma_load(stage + s * BZ * BX, &map, j.x0 - HX, j.z0 - HZ, q * a.units + j.unit, &bar[s]);
    walk.advance(a);
  };
  int job = blockIdx.x;
  if (tid == 0 && job < jobs) issue(0);
  __syncthreads();
  const float f = __ldg(&a.wavelet[a.t]);
  const float* sAX = a.prof;
  const float* sBX = a.prof + nx;
  const float* sDBX = a.prof + 2 * nx;
  const float* sAZ = a.prof + 3 * nx;
  const float* sBZ = sAZ + nz;
  const float* sDBZ = sBZ + nz;
  const int pc = tid & 31, grp = tid >> 5;
  // Halo pair of this thread (192 of the 256 threads): rows 0, 1, 34, 35 of the tile's 32 inner pairs, then
  // pairs 1 and 34 of its 32 inner rows. The stencils are axis-parallel: no corner is needed, and the
  // rows need the z strips' terms only, the columns the x strips' only.
  const bool hrow = tid < 4 * 32, hcol = !hrow && tid < 4 * 32 + 2 * TZ_;
  const int hk = hrow ? (tid / 32 < 2 ? tid / 32 : BZ - 4 + tid / 32) : HZ + (tid - 4 * 32) / 2;
  const int hj = hrow ? HX / 2 + tid % 32 : ((tid & 1) ? BX / 2 - 2 : 1);
  for (int i = 0; job < jobs; ++i, job += gridDim.x) {
    const int s = i & 1;
    const int nxt = job + gridDim.x;
    if (tid == 0 && nxt < jobs) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(s ^ 1);
    }
    const Job j = info[s];
    const int unit = j.unit, x0 = j.x0, z0 = j.z0, model = j.model, shot = j.shot;
    const float* vel = a.vel + static_cast<size_t>(model) * cells;
    const float* LPXc = a.PX + (static_cast<size_t>(q) * a.units + unit) * xs_unit;
    const float* LZXc = a.ZX + (static_cast<size_t>(q) * a.units + unit) * xs_unit;
    const float* LPZc = a.PZ + (static_cast<size_t>(q) * a.units + unit) * zs_unit;
    const float* LZZc = a.ZZ + (static_cast<size_t>(q) * a.units + unit) * zs_unit;
    const int x = x0 + 2 * pc;
    const int zr = z0 + RPT * grp;
    const bool xok = x >= FD_PAD && x + 1 < nx - FD_PAD;
    float* Ln = a.W + (static_cast<size_t>(1 - q) * a.units + unit) * cells;
    const float* st_t = a.stored + (static_cast<size_t>(unit) * a.seg + (a.t - a.seg_t0)) * cells;
    float* gacc = a.gacc + static_cast<size_t>(unit) * cells;
    const bool inner = j.inner;
    const int sx = 2 * pc + HX, sz = RPT * grp + HZ;

    // Everything that does not depend on the tile copy is requested before it is waited for: per own
    // cell the velocity, lambda_prev, the stored term, the gradient and the strips' psi and zeta, and
    // the halo pair's. (Read between the rows' stores, each strip value cost an L2 latency; with the
    // overlapped launch, packed arithmetic and one barrier less a step of 16 shots of the 844 x 344
    // grid went from 62 to 51.5 us, one of 10 shots of 344 x 194 from 18.3 to 14.4.)
    float2 vv[RPT], lpv[RPT], stv[RPT], gav[RPT], xP[RPT], xZ[RPT], zP[RPT], zZ[RPT];
    float2 hv = make_float2(0.f, 0.f), hP = hv, hZ = hv;
    const bool in_x = x < nx;                                     // own pair inside the grid (nx is even)
    const bool xs = !inner && in_x && (x < ssw || x >= nx - ssw);  // in an x strip
    const int xc = xstrip(x, nx, ssw);
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int z = zr + r;
      const bool ok = xok && z >= FD_PAD && z < nz - FD_PAD;
      const int cell = (ok ? z : FD_PAD) * nx + (ok ? x : FD_PAD);
      lpv[r] = ld2(Ln + cell);
      stv[r] = __ldcs(reinterpret_cast<const float2*>(st_t + cell));
      gav[r] = ld2(gacc + cell);
      vv[r] = in_x && z < nz ? ldg2(vel + static_cast<size_t>(z) * nx + x) : make_float2(0.f, 0.f);
      if (xs && z < nz) {
        xP[r] = ld2(LPXc + static_cast<size_t>(z) * 2 * ssw + xc);
        xZ[r] = ld2(LZXc + static_cast<size_t>(z) * 2 * ssw + xc);
      }
      if (!inner && in_x && z < nz && (z < ssw || z >= nz - ssw)) {
        const int zc = z < ssw ? z : z - (nz - 2 * ssw);
        zP[r] = ld2(LPZc + static_cast<size_t>(zc) * nx + x);
        zZ[r] = ld2(LZZc + static_cast<size_t>(zc) * nx + x);
      }
    }
    const int hz = z0 - HZ + hk, hx = x0 - HX + 2 * hj;
    const bool hin = (hrow || hcol) && hz >= 0 && hz < nz && hx >= 0 && hx < nx;
    const bool hxs = !inner && hcol && hin && (hx < ssw || hx >= nx - ssw);
    const bool hzs = !inner && hrow && hin && (hz < ssw || hz >= nz - ssw);
    if (hin) hv = ldg2(vel + static_cast<size_t>(hz) * nx + hx);
    if (hxs) {
      const size_t o = static_cast<size_t>(hz) * 2 * ssw + xstrip(hx, nx, ssw);
      hP = ld2(LPXc + o);
      hZ = ld2(LZXc + o);
    }
    if (hzs) {
      const size_t o = static_cast<size_t>(hz < ssw ? hz : hz - (nz - 2 * ssw)) * nx + hx;
      hP = ld2(LPZc + o);
      hZ = ld2(LZZc + o);
    }
    // a wait that runs out (the copy never completed) ends the kernel in every thread together, at
    // the barrier below
    const bool arrived = mbar_wait(&bar[s], (i >> 1) & 1);
    const float* L = stage + s * BZ * BX;

    // derived terms of the own cells and of the halo pair
    const float2 xb = xs ? ldg2(sBX + x) : make_float2(0.f, 0.f), xdb = xs ? ldg2(sDBX + x) : make_float2(0.f, 0.f);
    const float2 opxb = make_float2(1.0f + xb.x, 1.0f + xb.y);
    float2 vs[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int z = zr + r;
      const int o = (sz + r) * BX + sx;
      const float2 l = lds2(L + o);
      const bool in = in_x && z < nz;
      vs[r] = in ? mul2(scale2(a.dt2, mul2(vv[r], vv[r])), l) : make_float2(0.f, 0.f);
      put2(VS + o, vs[r]);
      if (xs && z < nz) {
        const float2 T = add2(pk.mul(opxb, vs[r]), pk.mul(xb, xZ[r]));
        put2(TXs + o, T);
        put2(U1Xs + o, add2(pk.mul(xdb, T), pk.mul(xb, xP[r])));
      }
      if (!inner && in && (z < ssw || z >= nz - ssw)) {
        const float bz = __ldg(&sBZ[z]), dbz = __ldg(&sDBZ[z]);
        const float2 T = add2(pk.scale(1.0f + bz, vs[r]), pk.scale(bz, zZ[r]));
        put2(TZs + o, T);
        put2(U1Zs + o, add2(pk.scale(dbz, T), pk.scale(bz, zP[r])));
      }
    }
    if (hrow || hcol) {
      const int o = hk * BX + 2 * hj;
      const float2 l = lds2(L + o);
      const float v0 = hin ? ((hv.x * hv.x) * a.dt2) * l.x : 0.0f, v1 = hin ? ((hv.y * hv.y) * a.dt2) * l.y : 0.0f;
      st2(VS + o, v0, v1);
      if (hxs) {
        const float2 b = ldg2(sBX + hx), db = ldg2(sDBX + hx);
        const float T0 = ((1.0f + b.x) * v0) + (b.x * hZ.x);
        const float T1 = ((1.0f + b.y) * v1) + (b.y * hZ.y);
        st2(TXs + o, T0, T1);
        st2(U1Xs + o, (db.x * T0) + (b.x * hP.x), (db.y * T1) + (b.y * hP.y));
      }
      if (hzs) {
        const float bz = __ldg(&sBZ[hz]), dbz = __ldg(&sDBZ[hz]);
        const float opbz = 1.0f + bz;
        const float T0 = (opbz * v0) + (bz * hZ.x);
        const float T1 = (opbz * v1) + (bz * hZ.y);
        st2(TZs + o, T0, T1);
        st2(U1Zs + o, (dbz * T0) + (bz * hP.x), (dbz * T1) + (bz * hP.y));
      }
    }
    if (__syncthreads_or(!arrived)) {
      if (tid == 0) {
        report(a.status);
        if (nxt < jobs) mbar_wait(&bar[s ^ 1], ((i + 1) >> 1) & 1);
      }
      return;
    }

    if (inner) {
      float* Lnf = a.W + (static_cast<size_t>(1 - q) * a.units + unit) * cells;
      float* gf = a.gacc + static_cast<size_t>(unit) * cells;
      // rows around the own four; the own ones are in registers
      const int so = sz * BX + sx;
      const float2 up2 = lds2(VS + so - 2 * BX), up1 = lds2(VS + so - BX), dn1 = lds2(VS + so + RPT * BX),
                   dn2 = lds2(VS + so + (RPT + 1) * BX);
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int cell = (zr + r) * nx + x;
        const float2 Vb = vs[r], Va = lds2(VS + so + r * BX - 2), Vc = lds2(VS + so + r * BX + 2);
        const float2 Vm2 = r >= 2 ? vs[r >= 2 ? r - 2 : 0] : (r == 1 ? up1 : up2);
        const float2 Vm1 = r >= 1 ? vs[r >= 1 ? r - 1 : 0] : up1;
        const float2 Vp1 = r + 1 < RPT ? vs[r + 1 < RPT ? r + 1 : r] : dn1;
        const float2 Vp2 = r + 2 < RPT ? vs[r + 2 < RPT ? r + 2 : r] : (r + 2 == RPT ? dn1 : dn2);
        const float2 w = add2(pk.second(Vb, side_sum(Va, Vb, Vc), add2(Vc, Va), a.rh, a.rh),
                              pk.second(Vb, add2(Vp1, Vm1), add2(Vp2, Vm2), a.rh, a.rh));
        const float2 lc = lds2(L + so + r * BX);
        // the shader starts the per-step gradient at +0; starting from the product itself differs
        // only in the sign of an exact zero
        put2(gf + cell, add2(gav[r], pk.mul(lc, stv[r])));
        put2(Lnf + cell, sub2(add2(w, add2(lc, lc)), lpv[r]));
      }
      __syncthreads();  // stage and VS are reused by the next tile
      continue;
    }

    const bool xpml = x < region || x + 1 >= nx - region;
    const int* sc = a.st.src_cell + 4 * shot;
    const float* res_t = a.residual + (static_cast<size_t>(unit) * a.nt + a.t) * a.st.nrec;
    const bool rec_rows = zr + RPT > a.rec_z0 && zr <= a.rec_z1;
    const unsigned srcm = j.src ? source_bits<RPT>(a, shot, zr, x) : 0u;
    float* LPXn = a.PX + (static_cast<size_t>(1 - q) * a.units + unit) * xs_unit;
    float* LZXn = a.ZX + (static_cast<size_t>(1 - q) * a.units + unit) * xs_unit;
    float* LPZn = a.PZ + (static_cast<size_t>(1 - q) * a.units + unit) * zs_unit;
    float* LZZn = a.ZZ + (static_cast<size_t>(1 - q) * a.units + unit) * zs_unit;
    float2 Ba = make_float2(0.f, 0.f), Bb = Ba, Bc = Ba, ax = Ba;
    if (xpml && xok) {
      Ba = ldg2(sBX + x - 2);
      Bb = ldg2(sBX + x);
      Bc = ldg2(sBX + x + 2);
      ax = ldg2(sAX + x);
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int z = zr + r;
      if (!xok || z < FD_PAD || z >= nz - FD_PAD) continue;
      const int cell = z * nx + x;
      const int so = (sz + r) * BX + sx;
      const float2 Vb = vs[r];
      float2 w;
      if (xpml) {
        const float2 Ta = lds2(TXs + so - 2), Tb = lds2(TXs + so), Tc = lds2(TXs + so + 2);
        const float2 Ua = lds2(U1Xs + so - 2), Ub = lds2(U1Xs + so), Uc = lds2(U1Xs + so + 2);
        const float2 qa = pk.mul(make_float2(1.0f + Ba.x, 1.0f + Ba.y), Ta), qb = pk.mul(make_float2(1.0f + Bb.x, 1.0f + Bb.y), Tb),
                     qc = pk.mul(make_float2(1.0f + Bc.x, 1.0f + Bc.y), Tc);
        const float2 du = pk.first(side_diff(Ua, Ub, Uc), sub2(Uc, Ua), a.rh);
        const float2 dd = pk.second(qb, side_sum(qa, qb, qc), add2(qc, qa), a.rh, a.rh);
        const float2 dt = pk.first(side_diff(Ta, Tb, Tc), sub2(Tc, Ta), a.rh);
        w = sub2(dd, du);
        const int xo = z * 2 * ssw + xc;
        put2(LPXn + xo, sub2(pk.mul(ax, xP[r]), pk.mul(ax, dt)));
        put2(LZXn + xo, add2(pk.mul(ax, Vb), pk.mul(ax, xZ[r])));
      } else {
        const float2 Va = lds2(VS + so - 2), Vc = lds2(VS + so + 2);
        w = pk.second(Vb, side_sum(Va, Vb, Vc), add2(Vc, Va), a.rh, a.rh);
      }
      if (z < region || z >= nz - region) {
        const float2 Tm2 = lds2(TZs + so - 2 * BX), Tm1 = lds2(TZs + so - BX), T0 = lds2(TZs + so),
                     Tp1 = lds2(TZs + so + BX), Tp2 = lds2(TZs + so + 2 * BX);
        const float2 Um2 = lds2(U1Zs + so - 2 * BX), Um1 = lds2(U1Zs + so - BX), Up1 = lds2(U1Zs + so + BX),
                     Up2 = lds2(U1Zs + so + 2 * BX);
        const float om2 = 1.0f + __ldg(&sBZ[z - 2]), om1 = 1.0f + __ldg(&sBZ[z - 1]), o0 = 1.0f + __ldg(&sBZ[z]),
                    op1 = 1.0f + __ldg(&sBZ[z + 1]), op2 = 1.0f + __ldg(&sBZ[z + 2]);
        const float2 du = pk.first(sub2(Up1, Um1), sub2(Up2, Um2), a.rh);
        const float2 dd = pk.second(scale2(o0, T0), add2(pk.scale(op1, Tp1), pk.scale(om1, Tm1)),
                                    add2(pk.scale(op2, Tp2), pk.scale(om2, Tm2)), a.rh, a.rh);
        const float2 dt = pk.first(sub2(Tp1, Tm1), sub2(Tp2, Tm2), a.rh);
        w = add2(w, sub2(dd, du));
        const int zo = (z < ssw ? z : z - (nz - 2 * ssw)) * nx + x;
        const float az = __ldg(&sAZ[z]);
        put2(LPZn + zo, sub2(pk.scale(az, zP[r]), pk.scale(az, dt)));
        put2(LZZn + zo, add2(pk.scale(az, Vb), pk.scale(az, zZ[r])));
      } else {
        const float2 Vm2 = lds2(VS + so - 2 * BX), Vm1 = lds2(VS + so - BX), Vp1 = lds2(VS + so + BX),
                     Vp2 = lds2(VS + so + 2 * BX);
        w = add2(w, pk.second(Vb, add2(Vp1, Vm1), add2(Vp2, Vm2), a.rh, a.rh));
      }
      const float2 lc = lds2(L + so);
      const float2 n = sub2(add2(w, add2(lc, lc)), lpv[r]);
      float n0 = n.x, n1 = n.y;
      float2 gr = pk.mul(lc, stv[r]);
      if (rec_rows) {
        const int e0 = a.st.csr[cell], e1 = a.st.csr[cell + 1], e2 = a.st.csr[cell + 2];
        for (int e = e0; e < e1; ++e) n0 = n0 + (a.st.ent_w[e] * res_t[a.st.ent_rec[e]]);
        for (int e = e1; e < e2; ++e) n1 = n1 + (a.st.ent_w[e] * res_t[a.st.ent_rec[e]]);
      }
      if (srcm & (3u << (2 * r))) {
        const float2 v = vv[r];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float wk = a.st.src_w[4 * shot + k];
          if (cell == sc[k]) gr.x = gr.x + lc.x * (((((-2.0f) * v.x) * a.dt2) * wk) * f);
          if (cell + 1 == sc[k]) gr.y = gr.y + lc.y * (((((-2.0f) * v.y) * a.dt2) * wk) * f);
        }
      }
      put2(gacc + cell, add2(gav[r], gr));
      st2(Ln + cell, n0, n1);
    }
    __syncthreads();  // stage and derived arrays are reused by the next tile
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------

struct Buf {
  void* p = nullptr;
  size_t bytes = 0;
  ~Buf() {
    if (p) cudaFree(p);
  }
  cudaError_t ensure(size_t need) {
    if (need <= bytes) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    cudaError_t e = cudaMalloc(&p, std::max<size_t>(need, 256));
    if (e != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
      return e;
    }
    bytes = need;
    return cudaSuccess;
  }
  float* f() const { return static_cast<float*>(p); }
};

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// Tensor map over [2 * units][nz][nx] floats with a 72 x 36 x 1 box; out-of-range elements read 0.
int make_map(CUtensorMap* m, const float* base, int nx, int nz, int depth, int box_x = BX, int box_z = BZ) {
  auto fn = encode_fn();
  if (!fn) return report_error(WG_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(nx), static_cast<cuuint64_t>(nz),
                              static_cast<cuuint64_t>(depth)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(nx) * 4, static_cast<cuuint64_t>(nx) * nz * 4};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(box_x), static_cast<cuuint32_t>(box_z), 1};
  const cuuint32_t es[3] = {1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return report_error(WG_ERR_CUDA, ("cuTensorMapEncodeTiled failed: " + std::to_string(r)).c_str());
  return WG_OK;
}

// Forward maps: the wavefield pair with and without halo, and the models' velocity.
int make_fwd_maps(FwdMaps* m, const float* W, const float* vel, int nx, int nz, int units, int models) {
  int rc = make_map(&m->u, W, nx, nz, 2 * units);
  if (rc == WG_OK) rc = make_map(&m->p, W, nx, nz, 2 * units, TX_, TZ_);
  if (rc == WG_OK) rc = make_map(&m->v, vel, nx, nz, models, TX_, TZ_);
  return rc;
}

constexpr size_t kAdjSmem = (7 * BZ * BX) * 4 + 16 + 128;

// Self-test of the time-out path: the kernels' bounded wait on an mbarrier that expects 16 bytes
// of a copy that is never issued. The wait gives up after `polls` polls, the CTA records ST_CUDA
// in `status` and the kernel returns (no copy is in flight, so there is nothing to drain).
__global__ void wait_timeout_probe_kernel(int* status, long polls) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_expect_tx(&bar, 16);  // the arrival; the 16 bytes never land
  __syncthreads();
  if (__syncthreads_or(mbar_wait(&bar, 0, polls) ? 0 : 1) && threadIdx.x == 0) report(status);
}

}  // namespace

int wait_timeout_selftest(int* d_status, long long polls, cudaStream_t st) {
  wait_timeout_probe_kernel<<<1, 64, 0, st>>>(d_status, static_cast<long>(polls));
  return cudaGetLastError() == cudaSuccess ? WG_OK : report_error(WG_ERR_CUDA, "wait self-test launch failed");
}

struct StreamWork {
  Buf vpad, mask, traces, energy, scale, part, stored, ckpt, gacc;
  Buf W, PX, ZX, PZ, ZZ;        // forward state
  Buf tb;                       // temporally blocked forward: two state sets
  bool tb_captured = false;     // a captured call reads them: the buffer stays where it is
  Buf L, LPX, LZX, LPZ, LZZ;    // adjoint state
  Buf tile_rec_start, tile_rec;
  int rec_tiles_nx = -1, rec_tiles_nz = -1, rec_z0 = 0, rec_z1 = -1;
  int fwd_blocks = 0, adj_blocks = 0, tb_blocks = 0, sms = 0;
};

StreamWork* stream_work_new() { return new StreamWork(); }
void stream_work_free(StreamWork* w) { delete w; }

namespace {

#define SW_CK(expr)                                                                                     \
  do {                                                                                                  \
    cudaError_t e_ = (expr);                                                                            \
    if (e_ != cudaSuccess) {                                                                            \
      cudaGetLastError();                                                                               \
      return report_error(e_ == cudaErrorMemoryAllocation ? WG_ERR_OOM : WG_ERR_CUDA,                   \
                          (std::string(#expr) + ": " + cudaGetErrorString(e_)).c_str());               \
    }                                                                                                   \
  } while (0)

int strip_width(const EngineView& v) { return ((v.grid.region_adj + 3) + 1) & ~1; }

// Receivers recorded by each tile: the tile that holds a receiver's first corner.
int setup_receivers(StreamWork* w, const EngineView& v, const int* h_rec_cell) {
  const int tx = (v.nx + TX_ - 1) / TX_, tz = (v.nz + TZ_ - 1) / TZ_;
  if (w->rec_tiles_nx == tx && w->rec_tiles_nz == tz) return WG_OK;
  std::vector<int> start(tx * tz + 1, 0), list(v.nrec);
  std::vector<int> tile_of(v.nrec);
  int z0 = v.nz, z1 = -1;
  for (int r = 0; r < v.nrec; ++r) {
    const int c = h_rec_cell[4 * r];
    const int cz = c / v.nx, cx = c % v.nx;
    tile_of[r] = (cz / TZ_) * tx + cx / TX_;
    ++start[tile_of[r] + 1];
    for (int k = 0; k < 4; ++k) {
      const int zz = h_rec_cell[4 * r + k] / v.nx;
      z0 = std::min(z0, zz);
      z1 = std::max(z1, zz);
    }
  }
  for (int t = 0; t < tx * tz; ++t) start[t + 1] += start[t];
  std::vector<int> fill(start.begin(), start.end() - 1);
  for (int r = 0; r < v.nrec; ++r) list[fill[tile_of[r]]++] = r;
  SW_CK(w->tile_rec_start.ensure(start.size() * 4));
  SW_CK(w->tile_rec.ensure(std::max<size_t>(list.size(), 1) * 4));
  SW_CK(cudaMemcpy(w->tile_rec_start.p, start.data(), start.size() * 4, cudaMemcpyHostToDevice));
  if (!list.empty()) SW_CK(cudaMemcpy(w->tile_rec.p, list.data(), list.size() * 4, cudaMemcpyHostToDevice));
  w->rec_tiles_nx = tx;
  w->rec_tiles_nz = tz;
  w->rec_z0 = z0;
  w->rec_z1 = z1;
  return WG_OK;
}

int occupancy(StreamWork* w) {
  if (w->sms) return WG_OK;
  int dev = 0, sms = 0, fb = 0, ab = 0;
  SW_CK(cudaGetDevice(&dev));
  SW_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  SW_CK(cudaFuncSetAttribute(adj_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kAdjSmem)));
  SW_CK(cudaFuncSetAttribute(fwd_stream_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kFwdSmem)));
  SW_CK(cudaFuncSetAttribute(fwd_stream_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kFwdSmem)));
  SW_CK(cudaFuncSetAttribute(fwd_stream_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kFwdSmem)));
  SW_CK(cudaFuncSetAttribute(fwd_tb_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kTbSmem)));
  SW_CK(cudaFuncSetAttribute(fwd_tb_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kTbSmem)));
  SW_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb, fwd_stream_kernel<true, true>, FWD_THREADS, kFwdSmem));
  SW_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ab, adj_stream_kernel, NTH, kAdjSmem));
  int tb = 0;
  SW_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&tb, fwd_tb_kernel<true, true>, TB_THREADS, kTbSmem));
  w->sms = sms;
  w->fwd_blocks = sms * std::max(fb, 1);
  w->adj_blocks = sms * std::max(ab, 1);
  w->tb_blocks = sms * std::max(tb, 1);
  return WG_OK;
}

SArgs base_args(StreamWork* w, const EngineView& v, int units) {
  SArgs a{};
  a.nx = v.nx;
  a.nz = v.nz;
  a.units = units;
  a.shots = v.shots;
  a.tiles_x = (v.nx + TX_ - 1) / TX_;
  a.tiles_z = (v.nz + TZ_ - 1) / TZ_;
  a.ssw = strip_width(v);
  a.region = v.grid.region_adj;
  a.nt = v.nt;
  a.rh = v.grid.rh;
  a.dt2 = v.grid.dt2;
  a.d2a = v.grid.d2a;
  a.d2b = v.grid.d2b;
  a.prof = v.grid.prof;
  a.wavelet = v.grid.wavelet;
  a.st = v.stations;
  a.rec_z0 = w->rec_z0;
  a.rec_z1 = w->rec_z1;
  a.tile_rec_start = static_cast<const int*>(w->tile_rec_start.p);
  a.tile_rec = static_cast<const int*>(w->tile_rec.p);
  a.status = v.d_status;
  a.nz2[0] = a.nz2[1] = -0.0f;
  return a;
}

size_t xs_floats(const EngineView& v) { return static_cast<size_t>(v.nz) * 2 * strip_width(v); }
size_t zs_floats(const EngineView& v) { return static_cast<size_t>(2) * strip_width(v) * v.nx; }

// Forward state buffers (zeroed) for `units` units.
int alloc_forward(StreamWork* w, const EngineView& v, int units, cudaStream_t st) {
  const size_t cells = static_cast<size_t>(v.nx) * v.nz;
  SW_CK(w->W.ensure(2 * units * cells * 4));
  SW_CK(w->PX.ensure(2 * units * xs_floats(v) * 4));
  SW_CK(w->ZX.ensure(units * xs_floats(v) * 4));
  SW_CK(w->PZ.ensure(2 * units * zs_floats(v) * 4));
  SW_CK(w->ZZ.ensure(units * zs_floats(v) * 4));
  SW_CK(cudaMemsetAsync(w->W.p, 0, 2 * units * cells * 4, st));
  SW_CK(cudaMemsetAsync(w->PX.p, 0, 2 * units * xs_floats(v) * 4, st));
  SW_CK(cudaMemsetAsync(w->ZX.p, 0, units * xs_floats(v) * 4, st));
  SW_CK(cudaMemsetAsync(w->PZ.p, 0, 2 * units * zs_floats(v) * 4, st));
  SW_CK(cudaMemsetAsync(w->ZZ.p, 0, units * zs_floats(v) * 4, st));
  return WG_OK;
}

// A step's launch, allowed to be scheduled while the step before it drains (see wait_for_previous_step).
template <class... P, class... A>
cudaError_t launch_step(void (*kernel)(P...), int blocks, int threads, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// One forward step over all units.
int fwd_step(StreamWork* w, const FwdMaps& map, SArgs a, int t, bool traces, bool store, cudaStream_t st) {
  a.t = t;
  const int jobs = a.units * a.tiles_x * a.tiles_z;
  const int blocks = std::min(jobs, w->fwd_blocks);
  note_launch();
  if (traces && store)
    SW_CK(launch_step(fwd_stream_kernel<true, true>, blocks, FWD_THREADS, kFwdSmem, st, map, a));
  else if (traces)
    SW_CK(launch_step(fwd_stream_kernel<true, false>, blocks, FWD_THREADS, kFwdSmem, st, map, a));
  else
    SW_CK(launch_step(fwd_stream_kernel<false, true>, blocks, FWD_THREADS, kFwdSmem, st, map, a));
  return WG_OK;
}

int adj_step(StreamWork* w, const CUtensorMap& map, SArgs a, int t, cudaStream_t st) {
  a.t = t;
  const int jobs = a.units * a.tiles_x * a.tiles_z;
  const int blocks = std::min(jobs, w->adj_blocks);
  note_launch();
  SW_CK(launch_step(adj_stream_kernel, blocks, NTH, kAdjSmem, st, map, a));
  return WG_OK;
}

// The blocked kernels' two state sets, in one allocation: a part that fails leaves nothing behind that
// the kernels of one step per launch, which then run, would miss.
struct TbLayout {
  size_t W, PX, ZX, PZ, ZZ, bytes;  // byte offsets, total
};

TbLayout tb_layout(const EngineView& v, int units) {
  const size_t nW = static_cast<size_t>(units) * v.nx * v.nz, nX = units * xs_floats(v), nZ = units * zs_floats(v);
  auto up = [](size_t floats) { return (floats * 4 + 255) & ~size_t(255); };
  TbLayout l{};
  l.PX = l.W + up(4 * nW);
  l.ZX = l.PX + up(2 * nX);
  l.PZ = l.ZX + up(2 * nX);
  l.ZZ = l.PZ + up(2 * nZ);
  l.bytes = l.ZZ + up(2 * nZ);
  return l;
}

// Temporally blocked forward over all units from the zero state, TB_T steps per launch: receivers
// into `traces` and, when `stored` is given, every step's gradient term (the store-all scheme).
int tb_forward(StreamWork* w, const EngineView& v, int units, int models, float* traces, float* stored,
               cudaStream_t st) {
  const TbLayout l = tb_layout(v, units);
  SW_CK(w->tb.ensure(l.bytes));
  SW_CK(cudaMemsetAsync(w->tb.p, 0, l.bytes, st));
  auto part = [&](size_t at) { return reinterpret_cast<float*>(static_cast<char*>(w->tb.p) + at); };
  CUtensorMap um, vm;
  int rc = make_map(&um, part(l.W), v.nx, v.nz, 4 * units, TB_RX, TB_RZ);
  if (rc == WG_OK) rc = make_map(&vm, w->vpad.f(), v.nx, v.nz, models, TB_RX, TB_RZ);
  if (rc != WG_OK) return rc;
  TbArgs p{};
  p.a = base_args(w, v, units);
  p.a.vel = w->vpad.f();
  p.a.traces = traces;
  p.a.stored = stored;
  p.a.seg = v.nt;
  p.a.seg_t0 = 0;
  p.W = part(l.W);
  p.PX = part(l.PX);
  p.ZX = part(l.ZX);
  p.PZ = part(l.PZ);
  p.ZZ = part(l.ZZ);
  const int jobs = units * p.a.tiles_x * p.a.tiles_z;
  const int blocks = std::min(jobs, w->tb_blocks);
  for (int t = 0, k = 0; t < v.nt; t += TB_T, ++k) {
    p.a.t = t;
    p.nsub = std::min(TB_T, v.nt - t);
    p.set_in = k & 1;
    note_launch();
    if (stored)
      SW_CK(launch_step(fwd_tb_kernel<true, true>, blocks, TB_THREADS, kTbSmem, st, um, vm, p));
    else
      SW_CK(launch_step(fwd_tb_kernel<true, false>, blocks, TB_THREADS, kTbSmem, st, um, vm, p));
  }
  return WG_OK;
}

// Whether a pass that starts from the zero state and writes no checkpoints runs temporally blocked: as
// the engine option says, or, where it was not set, when its tiles fit the chip in three waves (and there is
// memory for the second state set): a step is then
// mostly the latency of its launch and copies, which four steps share.
// us per step (recording traces), blocked against one step per launch, shots of 284 x 154 cells (25 tiles):
// 50 to 150 tiles 3.5 / 5.9, 200 5.8 / 6.7, 300 5.9 / 7.0, 325 (a third wave just begun) 8.8 / 9.0, 375 8.9 / 9.7,
// 450 8.8 / 10.3, 475 10.5 / 10.4, 525 11.2 / 10.6; shots of 464 x 224 cells (56 tiles): 280 6.0 / 6.7, 336 8.5 /
// 8.1, 392 8.5 / 9.1, 448 8.5 / 9.6, 504 11.1 / 9.7. A wave costs the same however full; the start of the third is
// the one place within the line where one step per launch can be as fast.
constexpr int kTbWaves = 3;
bool blocked(StreamWork* w, const EngineView& v, int units, cudaStream_t st) {
  if (v.tblock >= 0) return v.tblock != 0;
  const long jobs = static_cast<long>(units) * ((v.nx + TX_ - 1) / TX_) * ((v.nz + TZ_ - 1) / TZ_);
  if (jobs > static_cast<long>(kTbWaves) * w->tb_blocks) return false;
  // the choice is the library's: it does not allocate where the call is being captured into a graph, nor move
  // a buffer that a captured call reads
  const size_t need = tb_layout(v, units).bytes;
  const bool held = need <= w->tb.bytes, captured = being_captured(st);
  if (held && captured) w->tb_captured = true;
  if (held || captured || w->tb_captured) return held;
  return w->tb.ensure(need) == cudaSuccess;
}

// Checkpoint slot layout: [W(t) | W(t-1) | PX(t) | ZX | PZ(t) | ZZ] for all units.
size_t ckpt_slot_floats(const EngineView& v, int units) {
  const size_t cells = static_cast<size_t>(v.nx) * v.nz;
  return static_cast<size_t>(units) * (2 * cells + 2 * xs_floats(v) + 2 * zs_floats(v));
}

// Copy the forward state at the start of step t into (save) or out of (!save) a checkpoint slot.
int ckpt_copy(StreamWork* w, const EngineView& v, int units, int t, float* slot, bool save, cudaStream_t st) {
  const size_t cells = static_cast<size_t>(v.nx) * v.nz;
  const int par = t & 1;
  const size_t nW = units * cells, nX = units * xs_floats(v), nZ = units * zs_floats(v);
  float* parts[6] = {w->W.f() + par * nW, w->W.f() + (1 - par) * nW, w->PX.f() + par * nX, w->ZX.f(),
                     w->PZ.f() + par * nZ, w->ZZ.f()};
  const size_t sizes[6] = {nW, nW, nX, nX, nZ, nZ};
  size_t off = 0;
  for (int k = 0; k < 6; ++k) {
    float* dst = save ? slot + off : parts[k];
    const float* src = save ? parts[k] : slot + off;
    SW_CK(cudaMemcpyAsync(dst, src, sizes[k] * 4, cudaMemcpyDeviceToDevice, st));
    off += sizes[k];
  }
  return WG_OK;
}

}  // namespace

bool stream_supported(const EngineView& v, std::string* why) {
  if (v.nx % 4 != 0) {
    if (why) *why = "the streamed path needs a padded width divisible by 4 (nx_vis + 2 (pml + 2))";
    return false;
  }
  if (v.nx < 2 * strip_width(v) || v.nz < 2 * strip_width(v)) {
    if (why) *why = "grid too small for the streamed path's PML strips";
    return false;
  }
  return true;
}

int stream_simulate(StreamWork* w, const EngineView& v, const int* h_rec_cell, const float* d_vis, int models,
                    float* d_traces, cudaStream_t st, const StreamTimer& timer) {
  std::string why;
  if (!stream_supported(v, &why)) return report_error(WG_ERR_UNSUPPORTED, why.c_str());
  int rc = setup_receivers(w, v, h_rec_cell);
  if (rc != WG_OK) return rc;
  if ((rc = occupancy(w)) != WG_OK) return rc;
  const size_t cells = static_cast<size_t>(v.nx) * v.nz;
  const int units = models * v.shots;
  SW_CK(w->vpad.ensure(models * cells * 4));
  note_launch();
  SW_CK(launch_pad_velocity(d_vis, models, v.nx_vis, v.nz_vis, v.pad, v.vmin, v.vmax, w->vpad.f(), nullptr, st));
  if (blocked(w, v, units, st)) {
    timer.mark(0, true, st);
    if ((rc = tb_forward(w, v, units, models, d_traces, nullptr, st)) != WG_OK) return rc;
    timer.mark(0, false, st);
    return WG_OK;
  }
  if ((rc = alloc_forward(w, v, units, st)) != WG_OK) return rc;
  FwdMaps map;
  if ((rc = make_fwd_maps(&map, w->W.f(), w->vpad.f(), v.nx, v.nz, units, models)) != WG_OK) return rc;
  SArgs a = base_args(w, v, units);
  a.vel = w->vpad.f();
  a.W = w->W.f();
  a.PX = w->PX.f();
  a.ZX = w->ZX.f();
  a.PZ = w->PZ.f();
  a.ZZ = w->ZZ.f();
  a.traces = d_traces;
  timer.mark(0, true, st);
  for (int t = 0; t < v.nt; ++t)
    if ((rc = fwd_step(w, map, a, t, true, false, st)) != WG_OK) return rc;
  timer.mark(0, false, st);
  return WG_OK;
}

int stream_gradient(StreamWork* w, const EngineView& v, const int* h_rec_cell, const float* d_vis, const float* d_obs,
                    int models, double* d_loss, float* d_grad, cudaStream_t st, const StreamTimer& timer) {
  std::string why;
  if (!stream_supported(v, &why)) return report_error(WG_ERR_UNSUPPORTED, why.c_str());
  int rc = setup_receivers(w, v, h_rec_cell);
  if (rc != WG_OK) return rc;
  if ((rc = occupancy(w)) != WG_OK) return rc;
  const size_t cells = static_cast<size_t>(v.nx) * v.nz;
  const int units = models * v.shots;
  const size_t tr = static_cast<size_t>(v.nt) * v.nrec;
  SW_CK(w->vpad.ensure(models * cells * 4));
  SW_CK(w->mask.ensure(models * cells * 4));
  SW_CK(w->traces.ensure(units * tr * 4));
  SW_CK(w->energy.ensure(models * 8));
  SW_CK(w->scale.ensure(models * 4));
  SW_CK(w->part.ensure(static_cast<size_t>(models) * kRedParts * 8));
  SW_CK(w->gacc.ensure(units * cells * 4));
  note_launch();
  SW_CK(launch_pad_velocity(d_vis, models, v.nx_vis, v.nz_vis, v.pad, v.vmin, v.vmax, w->vpad.f(), w->mask.f(), st));
  note_launch();
  SW_CK(launch_energy(d_obs, models, v.shots * tr, static_cast<double*>(w->energy.p), w->scale.f(), v.d_status,
                      static_cast<double*>(w->part.p), st));
  if ((rc = alloc_forward(w, v, units, st)) != WG_OK) return rc;

  // Segment length: store every step's gradient terms when they fit in 70% of the free memory,
  // else checkpoints every k steps with k chosen (or given) so that one segment plus the
  // checkpoints fit.
  const size_t step_bytes = units * cells * 4;
  const size_t slot_bytes = ckpt_slot_floats(v, units) * 4;
  size_t free_b = 0, total_b = 0;
  SW_CK(cudaMemGetInfo(&free_b, &total_b));
  const size_t budget = free_b / 10 * 7 + w->stored.bytes + w->ckpt.bytes;
  int k = v.ck_every;
  if (k <= 0) {
    if (static_cast<size_t>(v.nt) * step_bytes <= budget) {
      k = v.nt;
    } else {
      k = 1;
      while (k < v.nt && (static_cast<size_t>(k) * step_bytes +
                          static_cast<size_t>((v.nt + k - 1) / k - 1) * slot_bytes) > budget) ++k;
      // prefer the smallest total memory among k that fit: sqrt balance
      int best = k;
      size_t best_mem = SIZE_MAX;
      for (int kk = k; kk <= std::min(v.nt, 4 * k + 64); ++kk) {
        const size_t mem = kk * step_bytes + static_cast<size_t>((v.nt + kk - 1) / kk - 1) * slot_bytes;
        if (mem <= budget && mem < best_mem) {
          best_mem = mem;
          best = kk;
        }
      }
      k = best;
    }
  }
  k = std::min(k, v.nt);
  const bool store_all = k >= v.nt;
  const int J = (v.nt + k - 1) / k;
  const int seg = store_all ? v.nt : k;
  SW_CK(w->stored.ensure(static_cast<size_t>(seg) * step_bytes));
  if (J > 1) SW_CK(w->ckpt.ensure(static_cast<size_t>(J - 1) * slot_bytes));

  // adjoint state (before the blocked forward's, which the pass can do without)
  const size_t xsf = xs_floats(v), zsf = zs_floats(v);
  SW_CK(w->L.ensure(2 * units * cells * 4));
  SW_CK(w->LPX.ensure(2 * units * xsf * 4));
  SW_CK(w->LZX.ensure(2 * units * xsf * 4));
  SW_CK(w->LPZ.ensure(2 * units * zsf * 4));
  SW_CK(w->LZZ.ensure(2 * units * zsf * 4));

  FwdMaps fmap;
  if ((rc = make_fwd_maps(&fmap, w->W.f(), w->vpad.f(), v.nx, v.nz, units, models)) != WG_OK) return rc;
  SArgs f = base_args(w, v, units);
  f.vel = w->vpad.f();
  f.W = w->W.f();
  f.PX = w->PX.f();
  f.ZX = w->ZX.f();
  f.PZ = w->PZ.f();
  f.ZZ = w->ZZ.f();
  f.traces = w->traces.f();
  f.stored = w->stored.f();
  f.seg = seg;
  f.seg_t0 = 0;
  timer.mark(0, true, st);
  if (store_all && blocked(w, v, units, st)) {
    if ((rc = tb_forward(w, v, units, models, w->traces.f(), w->stored.f(), st)) != WG_OK) return rc;
  } else {
    for (int t = 0; t < v.nt; ++t) {
      if (!store_all && t > 0 && t % k == 0)
        if ((rc = ckpt_copy(w, v, units, t, w->ckpt.f() + (t / k - 1) * (slot_bytes / 4), true, st)) != WG_OK)
          return rc;
      if ((rc = fwd_step(w, fmap, f, t, true, store_all, st)) != WG_OK) return rc;
    }
  }
  timer.mark(0, false, st);
  note_launch();
  SW_CK(launch_residual(w->traces.f(), d_obs, w->scale.f(), models, v.shots * tr, w->traces.f(), d_loss,
                        static_cast<double*>(w->part.p), st));

  SW_CK(cudaMemsetAsync(w->L.p, 0, 2 * units * cells * 4, st));
  SW_CK(cudaMemsetAsync(w->LPX.p, 0, 2 * units * xsf * 4, st));
  SW_CK(cudaMemsetAsync(w->LZX.p, 0, 2 * units * xsf * 4, st));
  SW_CK(cudaMemsetAsync(w->LPZ.p, 0, 2 * units * zsf * 4, st));
  SW_CK(cudaMemsetAsync(w->LZZ.p, 0, 2 * units * zsf * 4, st));
  SW_CK(cudaMemsetAsync(w->gacc.p, 0, units * cells * 4, st));
  CUtensorMap amap;
  if ((rc = make_map(&amap, w->L.f(), v.nx, v.nz, 2 * units)) != WG_OK) return rc;
  SArgs b = base_args(w, v, units);
  b.vel = w->vpad.f();
  b.W = w->L.f();
  b.PX = w->LPX.f();
  b.ZX = w->LZX.f();
  b.PZ = w->LPZ.f();
  b.ZZ = w->LZZ.f();
  b.residual = w->traces.f();
  b.stored = w->stored.f();
  b.seg = seg;
  b.gacc = w->gacc.f();
  for (int j = J - 1; j >= 0; --j) {
    const int t0 = store_all ? 0 : j * k, t1 = store_all ? v.nt : std::min(v.nt, t0 + k);
    if (!store_all) {
      timer.mark(1, true, st);
      if (j > 0) {
        if ((rc = ckpt_copy(w, v, units, t0, w->ckpt.f() + (j - 1) * (slot_bytes / 4), false, st)) != WG_OK) return rc;
      } else if ((rc = alloc_forward(w, v, units, st)) != WG_OK) {
        return rc;
      }
      f.seg_t0 = t0;
      for (int t = t0; t < t1; ++t)
        if ((rc = fwd_step(w, fmap, f, t, false, true, st)) != WG_OK) return rc;
      timer.mark(1, false, st);
    }
    b.seg_t0 = t0;
    timer.mark(2, true, st);
    for (int t = t1 - 1; t >= t0; --t)
      if ((rc = adj_step(w, amap, b, t, st)) != WG_OK) return rc;
    timer.mark(2, false, st);
  }
  note_launch();
  SW_CK(launch_fold(w->gacc.f(), w->mask.f(), models, v.shots, v.nx, v.nz, v.pad, v.nx_vis, v.nz_vis, d_grad, st));
  return WG_OK;
}

}  // namespace wg
