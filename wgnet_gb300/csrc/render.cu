// Additive anisotropic-Gaussian renderer (python/wgnet/render.py:34-109) and its vector-Jacobian
// product, for the 70 x 70 grid with 35 x 35 slots, each drawn in its 25 x 25 pixel window.
//
// Forward gathers: each pixel sums the slots whose window covers it, in increasing slot order (the
// order in which index_add_ accumulates on the CPU), from per-slot constants staged in shared
// memory; one thread computes a 2 x 2 pixel quad, so each slot's constants serve up to four pixels.
// Backward: one warp per slot reduces six moments over its window, from which its parameter gradients follow.
#include <cuda_runtime.h>

#include "wave_launch.h"
#include "wgnet_gb300.h"

namespace {

constexpr int GRID = 70;
constexpr int SIDE = 35;
constexpr int SLOTS = SIDE * SIDE;
constexpr int WIN = 12;
constexpr int NPAR = 6;

struct SlotC {
  float cx, cz, isx, isz, c, s, w;
};

__device__ __forceinline__ SlotC slot_consts(const float* p, int i) {
  const int iz = i / SIDE, ix = i % SIDE;
  SlotC k;
  k.cx = (2.0f * ix + 1.0f) + p[0];
  k.cz = (2.0f * iz + 1.0f) + p[1];
  k.isx = expf(-p[2]);
  k.isz = expf(-p[3]);
  sincosf(p[4], &k.s, &k.c);
  k.w = p[5];
  return k;
}

// One thread per 2 x 2 pixel quad (2n..2n+1, 2m..2m+1): row 2n is covered by the slots
// iz in [n-6, n+6], row 2n+1 by [n-5, n+6] (and the same for the columns), so each slot's
// constants, loaded once (two 128-bit loads), serve up to four pixels. Every pixel still sums its
// slots in increasing slot order. Blocks (QBLK threads, blockIdx.y) split a model's 1225 quads; each
// block stages all slot constants of its model (blockIdx.x). Small blocks spread a few models over the SMs and
// waste little in a last wave: 1 / 30 / 64 / 256 models take 39 / 40 / 54 / 157 us with 160 threads, 40 / 38 / 63 /
// 162 with 256, 47 / 45 / 71 / 173 with 416 (seven 32-bit loads per slot and 256 threads: 41 / 39 / 66 / 171).
// The arithmetic is the reference's, order and all: refinement takes decisions on misfits that a
// differently rounded field moves by 1e-4.
constexpr int QBLK = 160;
constexpr int QBLOCKS = (SLOTS + QBLK - 1) / QBLK;

__global__ void __launch_bounds__(QBLK) render_fwd_kernel(const float* __restrict__ params, float* __restrict__ field) {
  __shared__ float4 sh[2 * SLOTS];  // [cx cz isx isz] and [c s w 0] per slot
  const int b = blockIdx.x;
  const float* pb = params + static_cast<size_t>(b) * SLOTS * NPAR;
  for (int i = threadIdx.x; i < SLOTS; i += blockDim.x) {
    const SlotC k = slot_consts(pb + i * NPAR, i);
    sh[i] = make_float4(k.cx, k.cz, k.isx, k.isz);
    sh[SLOTS + i] = make_float4(k.c, k.s, k.w, 0.0f);
  }
  __syncthreads();
  const int q = blockIdx.y * QBLK + threadIdx.x;
  if (q >= SLOTS) return;
  const int n = q / SIDE, m = q % SIDE;
  const int iz0 = max(0, n - WIN / 2), iz1 = min(SIDE - 1, n + WIN / 2);
  const int ix0 = max(0, m - WIN / 2), ix1 = min(SIDE - 1, m + WIN / 2);
  const float fx0 = static_cast<float>(2 * m) + 0.5f, fx1 = static_cast<float>(2 * m + 1) + 0.5f;
  const float fz0 = static_cast<float>(2 * n) + 0.5f, fz1 = static_cast<float>(2 * n + 1) + 0.5f;
  float a00 = 0.0f, a01 = 0.0f, a10 = 0.0f, a11 = 0.0f;  // a[row][col]
  auto term = [](float fx, float fz, float cx, float cz, float c, float s, float isx, float isz, float w) {
    const float dx = fx - cx, dz = fz - cz;
    const float u = (dx * c + dz * s) * isx;
    const float v = (dz * c - dx * s) * isz;
    return w * expf(-0.5f * (u * u + v * v));
  };
  for (int iz = iz0; iz <= iz1; ++iz) {
    const bool row1 = iz >= n - WIN / 2 + 1;  // slot row iz also covers pixel row 2n + 1
    for (int ix = ix0; ix <= ix1; ++ix) {
      const bool col1 = ix >= m - WIN / 2 + 1;
      const float4 p = sh[iz * SIDE + ix], r = sh[SLOTS + iz * SIDE + ix];
      a00 += term(fx0, fz0, p.x, p.y, r.x, r.y, p.z, p.w, r.z);
      if (col1) a01 += term(fx1, fz0, p.x, p.y, r.x, r.y, p.z, p.w, r.z);
      if (row1) {
        a10 += term(fx0, fz1, p.x, p.y, r.x, r.y, p.z, p.w, r.z);
        if (col1) a11 += term(fx1, fz1, p.x, p.y, r.x, r.y, p.z, p.w, r.z);
      }
    }
  }
  float* f = field + static_cast<size_t>(b) * GRID * GRID + (2 * n) * GRID + 2 * m;
  *reinterpret_cast<float2*>(f) = make_float2(a00, a01);
  *reinterpret_cast<float2*>(f + GRID) = make_float2(a10, a11);
}

__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The gradient of a slot whose log scales lie far outside the activation's bounds (log 0.5 to log 6), where
// the moments below would overflow or lose their digits: every product formed per pixel, in unscaled
// distances, and reduced over the warp.
constexpr float kMomentScale = 4.0f;  // largest |log scale| that takes the moments
__device__ __noinline__ void render_bwd_direct(const SlotC k, const float* cb, int i, int lane, float* grad) {
  const int z0 = 2 * (i / SIDE) - WIN, x0 = 2 * (i % SIDE) - WIN;
  float g[NPAR] = {};
  for (int q = lane; q < (2 * WIN + 1) * (2 * WIN + 1); q += 32) {
    const int pz = z0 + q / (2 * WIN + 1), px = x0 + q % (2 * WIN + 1);
    if (pz < 0 || pz >= GRID || px < 0 || px >= GRID) continue;
    const float dx = (static_cast<float>(px) + 0.5f) - k.cx, dz = (static_cast<float>(pz) + 0.5f) - k.cz;
    const float ru = dx * k.c + dz * k.s, rv = dz * k.c - dx * k.s;
    const float u = ru * k.isx, v = rv * k.isz;
    const float e = expf(-0.5f * (u * u + v * v)), ct = cb[pz * GRID + px];
    const float ge = ct * k.w * e;  // cotangent times d/d(-0.5 (u^2 + v^2)) of the contribution
    // du/dcx = -c isx, dv/dcx = s isz; du/dcz = -s isx, dv/dcz = -c isz; dru/dangle = rv, drv/dangle = -ru
    g[0] += -ge * (u * (-k.c * k.isx) + v * (k.s * k.isz));
    g[1] += -ge * (u * (-k.s * k.isx) + v * (-k.c * k.isz));
    g[2] += ge * u * u;
    g[3] += ge * v * v;
    g[4] += -ge * (u * rv * k.isx - v * ru * k.isz);
    g[5] += ct * e;
  }
#pragma unroll
  for (int j = 0; j < NPAR; ++j) {
    for (int o = 16; o > 0; o >>= 1) g[j] += __shfl_down_sync(0xffffffffu, g[j], o);
    if (lane == 0) grad[j] = g[j];
  }
}

// One warp per slot: lane l takes window column l (25 of 32 lanes) and walks the window's rows inside
// the grid, so dx's products are loop constants and the pixel index needs no division. With
//   u = (dx c + dz s) / sx K,  v = (dz c - dx s) / sz K,  K = sqrt(log2(e) / 2)
// a slot's Gaussian is w 2^-(u^2 + v^2), one ex2. Six sums per slot, with E = cotangent x
// 2^-(u^2 + v^2): of E, E u, E v, E u^2, E v^2 and E u v; the parameter gradients are combinations
// of them (the amplitude and the coefficients are factored out). FP32
// issue bounds it, 13 operations and an ex2 per pixel. 256 models: 233 against 563 us with one
// pixel per lane of the flattened window and all six products formed per pixel.
__global__ void __launch_bounds__(256) render_bwd_kernel(const float* __restrict__ params, const float* __restrict__ cot,
                                                          int batch, float* __restrict__ grad) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= batch * SLOTS) return;
  const int b = warp / SLOTS, i = warp % SLOTS;
  const float* p = params + static_cast<size_t>(warp) * NPAR;
  constexpr float K = 0.84932180028801904f;
  const SlotC k = slot_consts(p, i);
  if (!(fabsf(p[2]) <= kMomentScale && fabsf(p[3]) <= kMomentScale)) {
    render_bwd_direct(k, cot + static_cast<size_t>(b) * GRID * GRID, i, lane, grad + static_cast<size_t>(warp) * NPAR);
    return;
  }
  const float uc = k.c * (k.isx * K), us = k.s * (k.isx * K), vc = k.c * (k.isz * K), vs = k.s * (k.isz * K);
  const int iz = i / SIDE, ix = i % SIDE;
  const int px = 2 * ix + lane - WIN;
  const int z0 = max(0, 2 * iz - WIN), z1 = min(GRID - 1, 2 * iz + WIN);
  float s = 0.f, su = 0.f, sv = 0.f, suu = 0.f, svv = 0.f, suv = 0.f;
  if (lane < 2 * WIN + 1 && px >= 0 && px < GRID) {
    const float* cb = cot + static_cast<size_t>(b) * GRID * GRID + px;
    const float dx = (static_cast<float>(px) + 0.5f) - k.cx;
    const float ux = dx * uc, vx = dx * vs;
#pragma unroll 5
    for (int pz = z0; pz <= z1; ++pz) {
      const float dz = (static_cast<float>(pz) + 0.5f) - k.cz;
      const float u = fmaf(dz, us, ux), v = fmaf(dz, vc, -vx);
      const float e = __ldg(cb + pz * GRID) * ex2(fmaf(-v, v, -(u * u)));
      const float eu = e * u, ev = e * v;
      s += e;
      su += eu;
      sv += ev;
      suu = fmaf(eu, u, suu);
      svv = fmaf(ev, v, svv);
      suv = fmaf(eu, v, suv);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    su += __shfl_down_sync(0xffffffffu, su, o);
    sv += __shfl_down_sync(0xffffffffu, sv, o);
    suu += __shfl_down_sync(0xffffffffu, suu, o);
    svv += __shfl_down_sync(0xffffffffu, svv, o);
    suv += __shfl_down_sync(0xffffffffu, suv, o);
  }
  if (lane == 0) {
    // the exponent is -(u^2 + v^2) ln 2 per natural unit: d/du 2^-(u^2 + v^2) = -2 ln2 u 2^-..., and
    // u^2 ln 2 = (unscaled u)^2 / 2. du/dcx = -uc, dv/dcx = vs; du/dcz = -us, dv/dcz = -vc;
    // du/dlog_sx = -u, dv/dlog_sz = -v; du/dangle = v sx^-1 / sz^-1, dv/dangle = -u sz^-1 / sx^-1
    const float g = 2.0f * 0.69314718055994531f * k.w;
    const float ratio = expf(p[3] - p[2]);  // sz / sx in log parameters: (1 / sx) / (1 / sz)
    float* o = grad + static_cast<size_t>(warp) * NPAR;
    o[0] = g * (uc * su - vs * sv);
    o[1] = g * (us * su + vc * sv);
    o[2] = g * suu;
    o[3] = g * svv;
    o[4] = -g * suv * (ratio - 1.0f / ratio);
    o[5] = s;
  }
}

}  // namespace

extern "C" int wg_render_fwd_dev(const float* d_params, int batch, float* d_field, void* stream) {
  if (batch < 0 || (batch > 0 && (!d_params || !d_field))) return wg::report_error(WG_ERR_ARG, "bad render arguments");
  if (batch == 0) return WG_OK;
  render_fwd_kernel<<<dim3(batch, QBLOCKS), QBLK, 0, static_cast<cudaStream_t>(stream)>>>(d_params, d_field);
  wg::note_launch();
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WG_OK : wg::report_error(WG_ERR_CUDA, cudaGetErrorString(e));
}

extern "C" int wg_render_bwd_dev(const float* d_params, const float* d_cot, int batch, float* d_grad, void* stream) {
  if (batch < 0 || (batch > 0 && (!d_params || !d_cot || !d_grad)))
    return wg::report_error(WG_ERR_ARG, "bad render arguments");
  if (batch == 0) return WG_OK;
  const int warps = batch * SLOTS;
  render_bwd_kernel<<<(warps + 7) / 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_params, d_cot, batch, d_grad);
  wg::note_launch();
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WG_OK : wg::report_error(WG_ERR_CUDA, cudaGetErrorString(e));
}
