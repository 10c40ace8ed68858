// 3x3 convolutions of the update network on the 5th-generation tensor cores, with no im2col matrix:
// forward, data gradient and weight gradient read the activations' shifted pixels straight from
// [batch][h][w][64] bf16 by TMA (zero fill outside the image) and finish in the epilogue what separate
// passes did (ReLU, residual add, bf16 casts, ReLU masks, the sum over taps of the data gradient). The
// arithmetic is that of gemm_bf16_kernel on im2col columns followed by those passes, in the same
// order: every output is bit-identical to that route.
//
// What bounds them: a 64 -> 64 convolution of 32 x 70 x 70 pixels needs 11.6 GFLOP (6 us at the bf16
// rate) and reads or writes 20 to 120 MB of activations (3 to 18 us at the HBM rate); feeding every
// tap of every output tile from L2 is more than either (180 MB: 34 us with one TMA load per tap). So
// an output tile is 8 columns x 16 rows of an image and the three taps of a column come from one box
// of 16 + 2 dil rows (a row of 8 pixels is one swizzle atom, so a tap's operand starts dil atoms
// further): 3 to 6 loads' worth of bytes instead of 9. The weights (72 KB) stay in shared memory, one
// persistent CTA per SM keeps the next tile's boxes in flight, and the accumulators are double-buffered
// in tensor memory so that the epilogue of a tile overlaps the loads of the next.
#include <cuda_bf16.h>

#include <algorithm>

#include "tc_common.cuh"

namespace wg {
namespace {

// What the epilogue does with the FP32 accumulator y of a pixel and channel.
enum Epi : int {
  EPI_RELU16 = 0,    // out16 = bf16(max(y, 0))
  EPI_FIRST = 1,     // out16 = bf16(max(y, 0)); out32 = out16 > 0 ? y : 0
  EPI_RESID = 2,     // out32 = add32 + y; out16 = bf16(out32)
  EPI_OUT1 = 3,      // out32[pixel] = y of channel 0
  EPI_MASK16 = 4,    // data gradient: out16 = bf16(mask16 > 0 ? y : 0)
  EPI_ACC = 5,       // data gradient: out32 = add32 + y; out16 = bf16(out32)
  EPI_ACC_MASK = 6,  // data gradient: out16 = bf16(mask16 > 0 ? add32 + y : 0)
};

constexpr int CTW = 8, CTH = 16;                 // columns and rows of an output tile
constexpr int CBM = CTW * CTH;                   // pixels per tile
constexpr int CST = 8;                           // most boxes in flight
constexpr unsigned kTapBytes = CBM * 128;        // one tap of a tile: 128 pixels x 64 channels
constexpr unsigned kRing = 7 * kTapBytes;        // shared memory of the boxes in flight
constexpr int kMaxDil = 10;                      // three boxes of 16 + 2 dil rows fit the ring
constexpr int CEPI = 8;                          // epilogue warps
constexpr int CTHR = 64 + 32 * CEPI;             // producer warp, MMA warp, epilogue warps
constexpr int CLD = 68;                          // row stride (floats) of the epilogue's staging tile
constexpr int CKT = 9;                           // most k tiles (taps) of a tile

struct ConvArgs {
  int M, h, w, dil;
  int tiles, tiles_x, tiles_img; // output tiles: all, per row of tiles, per image
  int kt;                        // k tiles per output tile: 9 taps, or the 64-wide column blocks of a matrix
  int stages;                    // boxes in flight
  unsigned box;                  // bytes of a box
  const float* add32;            // [M][64]
  const __nv_bfloat16* mask16;   // [M][64]
  float* out32;
  __nv_bfloat16* out16;
  int* status;
  long polls;                    // limit of a wait
};

// Shared memory: weights [kt][N rows][128 B] | boxes in flight | staging tile | barriers.
constexpr size_t kConvSmem = CKT * 64 * 128 + kRing + CBM * CLD * 4 + 256 + 1024;

__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}

// Named barrier over the epilogue warps that ORs a predicate.
__device__ __forceinline__ bool epi_or(bool v) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
      "selp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(static_cast<int>(v)), "n"(32 * CEPI)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ void tmem_ld32(uint32_t addr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __halves2bfloat162(__float2bfloat16(a), __float2bfloat16(b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ bool bf16_positive(uint32_t pair, int hi) {
  const uint32_t bits = hi ? (pair & 0xffff0000u) : (pair << 16);
  return __uint_as_float(bits) > 0.0f;
}

// One tile is 128 pixels x N channels: 8 x 16 pixels of an image (in MATRIX mode 128 rows of the
// matrix). Warp 0 (one lane) loads the tile's boxes, warp 1 (one lane) issues the MMAs, warps 2-9 run the epilogue. The data gradient keeps
// one accumulator per tap (the reference route rounds each tap's product to FP32 before it sums the
// taps): the epilogue adds the nine in tap order. Every wait is bounded; a warp that gives up
// records the error and the others follow through their own waits; then the MMA lane waits (bounded) for
// every MMA it issued, those of an unfinished tile included, before the tensor memory is freed, and a
// thread for every copy before the CTA ends.
template <int MODE>
__global__ void __launch_bounds__(CTHR, 1) conv_kernel(const __grid_constant__ CUtensorMap mapA,
                                                       const __grid_constant__ CUtensorMap mapB,
                                                       const __grid_constant__ ConvArgs a) {
  constexpr bool DGRAD = MODE >= EPI_MASK16;
  constexpr bool MATRIX = MODE == EPI_FIRST;          // the A operand is a matrix [M][64 kt]
  constexpr int N = MODE == EPI_OUT1 ? 16 : 64;       // output channels of the MMA
  constexpr int NACC = DGRAD ? 4 : 2;                 // accumulators in tensor memory
  constexpr uint32_t TCOLS = NACC * N;                // columns of tensor memory
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
  unsigned char* sB = smem;
  unsigned char* sA = sB + CKT * 64 * 128;
  float* tile = reinterpret_cast<float*>(sA + kRing);
  uint64_t* full = reinterpret_cast<uint64_t*>(tile + CBM * CLD);
  uint64_t* empty = full + CST;
  uint64_t* acc_full = empty + CST;
  uint64_t* acc_empty = acc_full + NACC;
  uint64_t* wbar = acc_empty + NACC;
  uint64_t* drained = wbar + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  __shared__ int fail, boxes_issued;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kt = a.kt, tiles = a.tiles, stages = a.stages;
  const int boxes = MATRIX ? kt : 3;  // per tile
  if (tid == 0) {
    for (int s = 0; s < CST; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    for (int b = 0; b < NACC; ++b) {
      bar_init(&acc_full[b], 1);
      bar_init(&acc_empty[b], CEPI);
    }
    bar_init(wbar, 1);
    bar_init(drained, 1);
    fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)), "r"(TCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      bar_expect(wbar, static_cast<unsigned>(kt) * N * 128);
      for (int t = 0; t < kt; ++t) tma2d(sB + t * N * 128, &mapB, DGRAD ? 0 : 64 * t, DGRAD ? 64 * t : 0, wbar);
      int it = 0;
      bool ok = true;
      int s = 0, phase = 1;  // ring position; the parity of the phase before it, complete at first
      for (int tl = blockIdx.x; ok && tl < tiles; tl += gridDim.x) {
        const int n = tl / a.tiles_img, r = tl - n * a.tiles_img, ty = r / a.tiles_x, tx = r - ty * a.tiles_x;
        for (int t = 0; t < boxes; ++t, ++it) {
          if (it >= stages && !bar_wait(&empty[s], phase, a.polls)) {
            ok = false;
            break;
          }
          bar_expect(&full[s], a.box);
          if (MATRIX)
            tma2d(sA + s * a.box, &mapA, 64 * t, tl * CBM, &full[s]);
          else  // columns shifted by the tap's, rows from dil above the tile on
            tma_image(sA + s * a.box, &mapA, CTW * tx + (DGRAD ? 1 - t : t - 1) * a.dil, CTH * ty - a.dil, n, &full[s]);
          if (++s == stages) {
            s = 0;
            phase ^= 1;
          }
        }
      }
      boxes_issued = it;
      if (!ok) {
        fail = 1;
        atomicCAS(a.status, 0, ST_CUDA);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16(CBM, N);
      const uint32_t a0 = desc_lo(su32(sA)), b0 = desc_lo(su32(sB));
      const uint32_t box = a.box >> 4, row = a.dil * (CTW * 128 >> 4);  // a box, dil of its rows
      bool ok = bar_wait(wbar, 0, a.polls);
      int s = 0, phase = 0;                 // ring position of the next box and its parity
      int acc = 0, acc_phase = 1;           // next accumulator; the parity of the phase before it
      // one lane's loop over 36 MMAs per tile: descriptors and ring positions advance by additions
      auto take = [&](uint32_t& lo) {       // wait for the next box; its operand's descriptor
        if (!bar_wait(&full[s], phase, a.polls)) return false;
        lo = a0 + s * box;
        if (++s == stages) {
          s = 0;
          phase ^= 1;
        }
        return true;
      };
      auto mmas = [&](uint32_t at, uint32_t wt, bool first) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma_bf16_lo(tmem + acc * N, at + 2 * kk, wt + 2 * kk, idesc, !first || kk > 0);
      };
      auto open = [&]() {                   // wait until the next accumulator has been read
        if (!bar_wait(&acc_empty[acc], acc_phase, a.polls)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return true;
      };
      auto close = [&]() {
        mma_commit(&acc_full[acc]);
        if (++acc == NACC) {
          acc = 0;
          acc_phase ^= 1;
        }
      };
      for (int tl = blockIdx.x; ok && tl < tiles; tl += gridDim.x) {
        if constexpr (MATRIX) {
          if (!(ok = open())) break;
          for (int t = 0; ok && t < kt; ++t) {
            const int at = s;
            uint32_t lo;
            if (!(ok = take(lo))) break;
            mmas(lo, b0 + t * (N * 128 >> 4), t == 0);
            mma_commit(&empty[at]);
          }
          if (ok) close();
        } else {
          int at[3];
          uint32_t lo[3];
#pragma unroll
          for (int t = 0; t < 9; ++t) {
            if ((DGRAD || t == 0) && !(ok = open())) break;
            if (t < 3) {
              at[t] = s;
              if (!(ok = take(lo[t]))) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            mmas(lo[t % 3] + (DGRAD ? 2 - t / 3 : t / 3) * row, b0 + t * (N * 128 >> 4), DGRAD || t == 0);
            if (t >= 6) mma_commit(&empty[at[t - 6]]);
            if (DGRAD || t == 8) close();
          }
        }
      }
      if (!ok) {
        fail = 1;
        atomicCAS(a.status, 0, ST_CUDA);
      }
    }
    __syncwarp();
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;  // tensor memory lanes 32 quad.., columns 32 half..
    const int et = tid - 64;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    constexpr int PER = CBM * 16 / (32 * CEPI);  // float4 (4 channels) of the tile per thread
    bool ok = true;
    int r = 0;
    for (int tl = blockIdx.x; tl < tiles; tl += gridDim.x) {
      const int n = tl / a.tiles_img, rr = tl - n * a.tiles_img, ty = rr / a.tiles_x, tx = rr - ty * a.tiles_x;
      // linear pixel of a row of the tile; -1 outside the image
      auto pixel = [&](int i) -> long {
        if (MATRIX) return static_cast<long>(tl) * CBM + i < a.M ? static_cast<long>(tl) * CBM + i : -1;
        const int y = CTH * ty + i / CTW, x = CTW * tx + i % CTW;
        return y < a.h && x < a.w ? (static_cast<long>(n) * a.h + y) * a.w + x : -1;
      };
      if constexpr (MODE == EPI_OUT1) {
        const int b = r % NACC;
        ok = __all_sync(0xffffffffu, bar_wait(&acc_full[b], (r / NACC) & 1, a.polls));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (half == 0) {
          uint32_t v;
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(lane_addr + b * N));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const long m = pixel(row);
          if (m >= 0) a.out32[m] = __uint_as_float(v);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(&acc_empty[b]);
        ++r;
        continue;
      }
      // the other operands of the epilogue, requested before the accumulator is waited for
      float4 add[PER];
      uint2 msk[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int e = et + 32 * CEPI * k;
        const long m = pixel(e / 16);
        const long o = m * 64 + 4 * (e % 16);
        if (MODE == EPI_RESID || MODE == EPI_ACC || MODE == EPI_ACC_MASK)
          add[k] = m >= 0 ? *reinterpret_cast<const float4*>(a.add32 + o) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (MODE == EPI_MASK16 || MODE == EPI_ACC_MASK)
          msk[k] = m >= 0 ? *reinterpret_cast<const uint2*>(a.mask16 + o) : make_uint2(0, 0);
      }
      float v[32];
      if (DGRAD) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0.0f;
      }
      const int rounds = DGRAD ? kt : 1;
#pragma unroll 1
      for (int q = 0; q < rounds; ++q, ++r) {
        const int b = r % NACC;
        ok = ok && __all_sync(0xffffffffu, bar_wait(&acc_full[b], (r / NACC) & 1, a.polls));
        if (ok) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          float t[32];
          tmem_ld32(lane_addr + b * N + 32 * half, t);
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) bar_arrive(&acc_empty[b]);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = DGRAD ? v[i] + t[i] : t[i];
        }
      }
      // rows of the accumulator to whole rows of the output through the staging tile
#pragma unroll
      for (int i = 0; i < 32; i += 4)
        *reinterpret_cast<float4*>(tile + row * CLD + 32 * half + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      if (epi_or(!ok)) {
        ok = false;
        break;
      }
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int e = et + 32 * CEPI * k;
        const long m = pixel(e / 16);
        if (m < 0) continue;
        const int c = 4 * (e % 16);
        const long o = m * 64 + c;
        float4 y = *reinterpret_cast<const float4*>(tile + (e / 16) * CLD + c);
        if (MODE == EPI_RELU16 || MODE == EPI_FIRST) {
          const uint2 p = make_uint2(pack_bf16(fmaxf(y.x, 0.0f), fmaxf(y.y, 0.0f)), pack_bf16(fmaxf(y.z, 0.0f), fmaxf(y.w, 0.0f)));
          *reinterpret_cast<uint2*>(a.out16 + o) = p;
          if (MODE == EPI_FIRST)
            *reinterpret_cast<float4*>(a.out32 + o) =
                make_float4(bf16_positive(p.x, 0) ? y.x : 0.0f, bf16_positive(p.x, 1) ? y.y : 0.0f,
                            bf16_positive(p.y, 0) ? y.z : 0.0f, bf16_positive(p.y, 1) ? y.w : 0.0f);
        } else {
          if (MODE != EPI_MASK16) y = make_float4(add[k].x + y.x, add[k].y + y.y, add[k].z + y.z, add[k].w + y.w);
          if (MODE == EPI_RESID || MODE == EPI_ACC) *reinterpret_cast<float4*>(a.out32 + o) = y;
          if (MODE == EPI_MASK16 || MODE == EPI_ACC_MASK)
            y = make_float4(bf16_positive(msk[k].x, 0) ? y.x : 0.0f, bf16_positive(msk[k].x, 1) ? y.y : 0.0f,
                            bf16_positive(msk[k].y, 0) ? y.z : 0.0f, bf16_positive(msk[k].y, 1) ? y.w : 0.0f);
          *reinterpret_cast<uint2*>(a.out16 + o) = make_uint2(pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
        }
      }
      epi_or(false);  // the staging tile is free again
    }
    if (!ok) {
      fail = 1;
      if (lane == 0) atomicCAS(a.status, 0, ST_CUDA);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (fail && tid == 32) {  // the MMAs still running (a commit follows those of its own thread)
    mma_commit(drained);
    bar_wait(drained, 0);
  }
  __syncwarp();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
  if (fail && tid == 0) {  // the copies still landing
    bar_wait(wbar, 0);
    for (int k = 1; k <= stages && boxes_issued - k >= 0; ++k)
      bar_wait(&full[(boxes_issued - k) % stages], ((boxes_issued - k) / stages) & 1);
  }
}

// Weight gradient partials: part[z][k][n] = sum over the pixels of split z of x[pixel + tap(k)][c(k)]
// dy[pixel][n]. The reduction runs over pixels, which both operands hold as rows, so both are read as
// they lie (MN-major: 64 channels = 128 contiguous bytes per pixel). A CTA takes two taps (M = 128)
// of one split; its accumulator and the order of its k tiles are those of gemm_bf16_kernel on the
// transposed im2col columns (315 CTAs of 1 tile each for 64 splits, three to an SM).
constexpr int WST = 3;                              // pipeline stages
constexpr unsigned kWTile = 64 * 128;               // 64 pixels x 64 channels
constexpr unsigned kWStage = 3 * kWTile;            // two taps of x, dy
constexpr int WTHR = 128;
constexpr size_t kWgradSmem = WST * kWStage + 128 + 1024;

struct WgradArgs {
  int h, w, dil;
  int kdim;                // rows of a partial: 576, or the columns of a matrix
  int k_tiles, per_split;  // tiles of 64 pixels, and how many of them a split takes
  float* part;             // [splits][kdim][64]
  int* status;
};

template <bool MATRIX>  // x is a matrix [M][kdim] of columns instead of activations read per tap
__global__ void __launch_bounds__(WTHR, 3) wgrad_kernel(const __grid_constant__ CUtensorMap mapX,
                                                        const __grid_constant__ CUtensorMap mapY,
                                                        const __grid_constant__ WgradArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + WST * kWStage);
  uint64_t* empty = full + WST;
  uint64_t* done = empty + WST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  __shared__ int fail;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int blk = blockIdx.x;                                   // pair of taps (64-wide blocks of k)
  const bool two = 128 * blk + 64 < g.kdim;                     // the last pair may hold one
  const int kt0 = blockIdx.y * g.per_split;
  const int KT = min(g.per_split, g.k_tiles - kt0);
  if (tid == 0) {
    for (int s = 0; s < WST; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    bar_init(done, 1);
    fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)), "r"(64)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (tid == 0 && KT > 0) {
    Pixel pos(MATRIX ? 0 : kt0 * 64, g.h, g.w);  // of the next tile to load
    auto load = [&](int i) {
      const int s = i % WST, px = (kt0 + i) * 64;
      unsigned char* st = smem + s * kWStage;
      bar_expect(&full[s], (two ? 3 : 2) * kWTile);
      for (int j = 0; j < (two ? 2 : 1); ++j) {
        const int t = 2 * blk + j;
        if (MATRIX)
          tma2d(st + j * kWTile, &mapX, 64 * t, px, &full[s]);
        else
          tma_im2col(st + j * kWTile, &mapX, pos, g.dil, (t % 3) * g.dil, (t / 3) * g.dil, &full[s]);
      }
      tma2d(st + 2 * kWTile, &mapY, 0, px, &full[s]);
      if (!MATRIX) pos.advance(64, g.h, g.w);
    };
    for (int i = 0; i < KT && i < WST; ++i) load(i);
    constexpr uint32_t idesc = idesc_bf16(128, 64) | (1u << 15) | (1u << 16);  // both operands MN-major
    bool ok = true;
    int i = 0;
    for (; i < KT; ++i) {
      const int s = i % WST;
      if (!bar_wait(&full[s], (i / WST) & 1)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // MN-major operands: 64 channels (128 bytes) per pixel row, 8 pixel rows per 1024-byte atom, 64-channel
      // blocks kWTile apart
      const uint32_t lo = desc_lo(su32(smem + s * kWStage), kWTile);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)  // 16 pixels = two 8-row atoms further
        mma_bf16_lo(tmem, lo + (kk * 2048 >> 4), lo + ((2 * kWTile + kk * 2048) >> 4), idesc, i > 0 || kk > 0);
      mma_commit(&empty[s]);
      if (i >= 1 && i - 1 + WST < KT) {  // refill the stage of the tile before: its MMAs are mostly done
        const int p = i - 1;
        if (!bar_wait(&empty[p % WST], (p / WST) & 1)) {
          ok = false;
          break;
        }
        load(p + WST);
      }
    }
    if (ok) {
      mma_commit(done);
    } else {
      fail = 1;
      atomicCAS(g.status, 0, ST_CUDA);
      // drain (bounded): the last copies issued and the last commits of each stage
      const int loaded = min(KT, i + WST), committed = min(KT, i + 1);
      for (int k = 1; k <= WST && loaded - k >= 0; ++k) bar_wait(&full[(loaded - k) % WST], ((loaded - k) / WST) & 1);
      for (int k = 1; k <= WST && committed - k >= 0; ++k)
        bar_wait(&empty[(committed - k) % WST], ((committed - k) / WST) & 1);
    }
  }
  __syncthreads();
  bool have = !fail && KT > 0;
  have = __syncthreads_and(!have || bar_wait(done, 0)) && have;
  if (!have && !fail && KT > 0 && tid == 0) atomicCAS(g.status, 0, ST_CUDA);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  float* tile = reinterpret_cast<float*>(smem);  // the pipeline's buffers are idle now
  const int row = tid;
#pragma unroll
  for (int hlf = 0; hlf < 2; ++hlf) {
    float v[32];
    tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + 32 * hlf, v);
#pragma unroll
    for (int i = 0; i < 32; i += 4)
      *reinterpret_cast<float4*>(tile + row * CLD + 32 * hlf + i) =
          have ? make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  float* out = g.part + (static_cast<size_t>(blockIdx.y) * g.kdim + 128 * blk) * 64;
  for (int e = tid; e < (two ? 128 : 64) * 16; e += WTHR)
    *reinterpret_cast<float4*>(out + e * 4) = *reinterpret_cast<const float4*>(tile + (e / 16) * CLD + 4 * (e % 16));
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(64) : "memory");
}

// Data gradient of the one-channel output layer: dh[m][c] = sum over taps of bf16(dout[m - tap])
// w[tap][c] (products of two bf16 are exact in FP32; taps in order), with its bf16 copy, and dout as
// channel 0 of dout16 [M][64], whose other channels become zero. Writing these 8 bytes per value bounds
// it (80 MB for 32 images of 70 x 70). 16 threads take the channels of a run of ODG pixels of a row:
// their 36 weights stay in registers (24 us; 43 with the weights read from shared memory for every pixel,
// and 8 to clear dout16 beforehand).
constexpr int ODG = 10;
__global__ void __launch_bounds__(256) out_dgrad_kernel(const float* __restrict__ dout, const __nv_bfloat16* __restrict__ wt,
                                                        int runs, int h, int w, float* __restrict__ dh,
                                                        __nv_bfloat16* __restrict__ dh16,
                                                        __nv_bfloat16* __restrict__ dout16) {
  __shared__ __align__(16) float sw[9 * 64];
  for (int i = threadIdx.x; i < 9 * 64; i += blockDim.x) sw[i] = __bfloat162float(wt[static_cast<long>(i) * 64]);
  __syncthreads();
  const int c = 4 * (threadIdx.x % 16), across = (w + ODG - 1) / ODG;
  const int run = blockIdx.x * 16 + threadIdx.x / 16;
  if (run >= runs) return;
  float wv[9][4];
#pragma unroll
  for (int t = 0; t < 9; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) wv[t][j] = sw[t * 64 + c + j];
  const int row = run / across, x0 = (run - row * across) * ODG, y = row % h;
  const float* d0 = dout + static_cast<long>(row) * w;
  auto at = [&](int dy, int x) {  // bf16 of dout, zero outside the image
    return y - dy >= 0 && y - dy < h && x >= 0 && x < w ? __bfloat162float(__float2bfloat16(d0[x - static_cast<long>(dy) * w]))
                                                        : 0.0f;
  };
  float d[3][3];  // [row y + 1 .. y - 1][column x + 1 .. x - 1], the taps' order
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    d[r][0] = at(r - 1, x0);
    d[r][1] = at(r - 1, x0 - 1);
    d[r][2] = 0.0f;
  }
#pragma unroll 2
  for (int x = x0; x < min(x0 + ODG, w); ++x) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      d[r][2] = d[r][1];
      d[r][1] = d[r][0];
      d[r][0] = at(r - 1, x + 1);
    }
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      const int r = t / 3, q = t % 3;
      const bool in = y - (r - 1) >= 0 && y - (r - 1) < h && x - (q - 1) >= 0 && x - (q - 1) < w;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = in ? v[j] + d[r][q] * wv[t][j] : v[j];
    }
    const long o = (static_cast<long>(row) * w + x) * 64 + c;
    *reinterpret_cast<float4*>(dh + o) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<uint2*>(dh16 + o) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    *reinterpret_cast<uint2*>(dout16 + o) = make_uint2(c ? 0u : pack_bf16(d0[x], 0.0f), 0u);
  }
}

int sm_count() {
  static int n[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  return n[dev];
}

template <class K>
int allow_smem(K kernel, size_t bytes) {
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  return e == cudaSuccess ? WG_OK : report_error(WG_ERR_CUDA, cudaGetErrorString(e));
}

template <int MODE>
int conv_launch(const CUtensorMap& ma, const CUtensorMap& mb, const ConvArgs& a, cudaStream_t st) {
  const int sms = sm_count();
  if (sms < 1) return report_error(WG_ERR_CUDA, "no device");
  const int rc = allow_smem(conv_kernel<MODE>, kConvSmem);
  if (rc != WG_OK) return rc;
  note_launch();
  conv_kernel<MODE><<<a.tiles < sms ? a.tiles : sms, CTHR, kConvSmem, st>>>(ma, mb, a);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WG_OK : report_error(WG_ERR_CUDA, cudaGetErrorString(e));
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

bool bad_image(int batch, int h, int w, int dil) {
  return batch < 1 || h < 1 || w < 1 || dil < 1 || dil > kMaxDil || static_cast<long>(batch) * h * w > (1L << 30);
}

}  // namespace
}  // namespace wg

namespace wg {
namespace {

int conv(int mode, const void* d_act, int batch, int h, int w, int dil, const void* d_wgt, int kp, const float* d_add,
         const void* d_mask, float* d_out32, void* d_out16, int* d_status, void* stream, long polls) {
  const bool matrix = mode == EPI_FIRST, dgrad = mode >= EPI_MASK16;
  const bool needs_add = mode == EPI_RESID || mode == EPI_ACC || mode == EPI_ACC_MASK;
  const bool needs_mask = mode == EPI_MASK16 || mode == EPI_ACC_MASK;
  const bool needs32 = mode == EPI_FIRST || mode == EPI_RESID || mode == EPI_OUT1 || mode == EPI_ACC;
  if (mode < 0 || mode > EPI_ACC_MASK || !d_act || !d_wgt || !d_status || bad_image(batch, h, w, dil) || kp < 64 ||
      kp % 64 || kp > 64 * CKT || (!matrix && kp != 64 * CKT) || (needs_add && !d_add) || (needs_mask && !d_mask) ||
      (needs32 && !d_out32) || (mode != EPI_OUT1 && !d_out16))
    return report_error(WG_ERR_ARG, "conv: bad argument");
  if (!aligned16(d_act) || !aligned16(d_wgt) || !aligned16(d_add) || !aligned16(d_mask) || !aligned16(d_out32) ||
      !aligned16(d_out16))
    return report_error(WG_ERR_ARG, "conv: buffers must be 16-byte aligned");
  ConvArgs a{};
  a.M = batch * h * w;
  a.h = h;
  a.w = w;
  a.dil = dil;
  a.kt = kp / 64;
  a.add32 = d_add;
  a.mask16 = static_cast<const __nv_bfloat16*>(d_mask);
  a.out32 = d_out32;
  a.out16 = static_cast<__nv_bfloat16*>(d_out16);
  a.status = d_status;
  a.polls = polls;
  a.tiles_x = (w + CTW - 1) / CTW;
  a.tiles_img = a.tiles_x * ((h + CTH - 1) / CTH);
  a.tiles = matrix ? (a.M + CBM - 1) / CBM : batch * a.tiles_img;
  if (matrix) a.tiles_x = a.tiles_img = a.tiles;  // not an image: one row of tiles
  const int rows = CTH + 2 * dil;
  a.box = matrix ? kTapBytes : rows * CTW * 128;
  a.stages = std::min<int>(CST, kRing / a.box);
  CUtensorMap ma, mb;
  int rc = matrix ? map_bf16(&ma, d_act, a.M, kp, CBM) : map_image(&ma, d_act, batch, h, w, rows);
  if (rc != WG_OK) return rc;
  // weights: [n][kp] (boxes of 64 k x n rows), or for the data gradient [kp][64] (64 x 64 boxes)
  rc = dgrad ? map_bf16(&mb, d_wgt, kp, 64, 64) : map_bf16(&mb, d_wgt, 64, kp, mode == EPI_OUT1 ? 16 : 64);
  if (rc != WG_OK) return rc;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (mode) {
    case EPI_RELU16: return conv_launch<EPI_RELU16>(ma, mb, a, st);
    case EPI_FIRST: return conv_launch<EPI_FIRST>(ma, mb, a, st);
    case EPI_RESID: return conv_launch<EPI_RESID>(ma, mb, a, st);
    case EPI_OUT1: return conv_launch<EPI_OUT1>(ma, mb, a, st);
    case EPI_MASK16: return conv_launch<EPI_MASK16>(ma, mb, a, st);
    case EPI_ACC: return conv_launch<EPI_ACC>(ma, mb, a, st);
    default: return conv_launch<EPI_ACC_MASK>(ma, mb, a, st);
  }
}

}  // namespace
}  // namespace wg

extern "C" {

int wg_pc_conv(int mode, const void* d_act, int batch, int h, int w, int dil, const void* d_wgt, int kp,
               const float* d_add, const void* d_mask, float* d_out32, void* d_out16, int* d_status, void* stream) {
  return wg::conv(mode, d_act, batch, h, w, dil, d_wgt, kp, d_add, d_mask, d_out32, d_out16, d_status, stream,
                  wg::kTcWaitLimit);
}

int wg_selftest_conv_timeout(const void* d_act, int batch, int h, int w, const void* d_wgt, void* d_out16, int* d_status,
                             void* stream) {
  return wg::conv(wg::EPI_RELU16, d_act, batch, h, w, 1, d_wgt, 64 * wg::CKT, nullptr, nullptr, nullptr, d_out16, d_status,
                  stream, 0);
}

int wg_pc_wgrad_partials(int batch, int h, int w, int splits) {
  if (wg::bad_image(batch, h, w, 1) || splits < 1 || batch * h * w % 64) return 0;
  const int tiles = batch * h * w / 64, per_split = (tiles + splits - 1) / splits;
  return (tiles + per_split - 1) / per_split;
}

int wg_pc_conv_wgrad(const void* d_act, int columns, const void* d_dy, int batch, int h, int w, int dil, int splits,
                     float* d_partial, int* d_status, void* stream) {
  using namespace wg;
  if (!d_act || !d_dy || !d_partial || !d_status || bad_image(batch, h, w, dil) || splits < 1 || columns < 0 ||
      columns % 64 || columns > 64 * CKT)
    return report_error(WG_ERR_ARG, "conv_wgrad: bad argument");
  const int M = batch * h * w;
  if (M % 64) return report_error(WG_ERR_ARG, "conv_wgrad: batch * h * w must be a multiple of 64");
  if (!aligned16(d_act) || !aligned16(d_dy) || !aligned16(d_partial))
    return report_error(WG_ERR_ARG, "conv_wgrad: buffers must be 16-byte aligned");
  WgradArgs g{};
  g.h = h;
  g.w = w;
  g.dil = dil;
  g.kdim = columns ? columns : 64 * CKT;
  g.k_tiles = M / 64;
  g.per_split = (g.k_tiles + splits - 1) / splits;
  g.part = d_partial;
  g.status = d_status;
  CUtensorMap mx, my;
  int rc = columns ? map_bf16(&mx, d_act, M, columns, 64) : map_im2col(&mx, d_act, batch, h, w, dil, 64);
  if (rc != WG_OK) return rc;
  if ((rc = map_bf16(&my, d_dy, M, 64, 64)) != WG_OK) return rc;
  if ((rc = columns ? allow_smem(wgrad_kernel<true>, kWgradSmem) : allow_smem(wgrad_kernel<false>, kWgradSmem)) != WG_OK)
    return rc;
  const dim3 grid((g.kdim + 127) / 128, wg_pc_wgrad_partials(batch, h, w, splits));
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  note_launch();
  if (columns)
    wgrad_kernel<true><<<grid, WTHR, kWgradSmem, st>>>(mx, my, g);
  else
    wgrad_kernel<false><<<grid, WTHR, kWgradSmem, st>>>(mx, my, g);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WG_OK : report_error(WG_ERR_CUDA, cudaGetErrorString(e));
}

int wg_pc_out_dgrad(const float* d_dout, const void* d_wt, int batch, int h, int w, float* d_dh, void* d_dh16,
                    void* d_dout16, void* stream) {
  using namespace wg;
  if (!d_dout || !d_wt || !d_dh || !d_dh16 || !d_dout16 || bad_image(batch, h, w, 1))
    return report_error(WG_ERR_ARG, "out_dgrad: bad argument");
  if (!aligned16(d_dh) || !aligned16(d_dh16) || !aligned16(d_dout16)) return report_error(WG_ERR_ARG, "out_dgrad: buffers must be 16-byte aligned");
  note_launch();
  const long runs = static_cast<long>(batch) * h * ((w + ODG - 1) / ODG);
  out_dgrad_kernel<<<static_cast<unsigned>((runs + 15) / 16), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      d_dout, static_cast<const __nv_bfloat16*>(d_wt), static_cast<int>(runs), h, w, d_dh,
      static_cast<__nv_bfloat16*>(d_dh16), static_cast<__nv_bfloat16*>(d_dout16));
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WG_OK : report_error(WG_ERR_CUDA, cudaGetErrorString(e));
}

}  // extern "C"
