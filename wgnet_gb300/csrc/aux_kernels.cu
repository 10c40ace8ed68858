// Small kernels around the time-stepping kernels: velocity padding, observed energy, residual and
// misfit, gradient shot-sum/mask/fold, causal band-limit FIR. All are HBM-bound elementwise or
// reduction passes; reductions use a fixed launch shape and a fixed tree so they are deterministic.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "wave_launch.h"

namespace wg {

namespace {

// Block-wide f64 sum with a fixed tree (deterministic for a fixed blockDim).
__device__ double block_sum(double v, double* sh) {
  const int tid = threadIdx.x;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((tid & 31) == 0) sh[tid >> 5] = v;
  __syncthreads();
  double r = 0.0;
  if (tid < 32) {
    r = (tid < static_cast<int>(blockDim.x >> 5)) ? sh[tid] : 0.0;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  return r;  // valid in thread 0
}

__global__ void pad_kernel(const float* __restrict__ vis, int nx_vis, int nz_vis, int pad, float vmin, float vmax,
                           float* __restrict__ padded, float* __restrict__ mask) {
  const int nx = nx_vis + 2 * pad, nz = nz_vis + 2 * pad;
  const int model = blockIdx.y;
  const size_t cells = static_cast<size_t>(nx) * nz;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<int>(cells); i += gridDim.x * blockDim.x) {
    const int z = i / nx, x = i % nx;
    const int vz = min(max(z - pad, 0), nz_vis - 1);
    const int vx = min(max(x - pad, 0), nx_vis - 1);
    const float v = vis[static_cast<size_t>(model) * nx_vis * nz_vis + vz * nx_vis + vx];
    if (mask) mask[model * cells + i] = (v > vmin && v < vmax) ? 1.0f : 0.0f;
    // Rust f32::clamp: NaN stays NaN.
    padded[model * cells + i] = v < vmin ? vmin : (v > vmax ? vmax : v);
  }
}

// The two f64 reductions over a model's traces. FP64 issues at 2 lanes per clock and SM, which bounds
// them, so a model's traces are split over up to kRedParts blocks (one block per model took 0.77 ms
// for 5 shots x 2001 x 70 and left the other SMs idle), and the square is one fused f64 operation
// (the product of two f32 is exact in f64, so nothing else rounds). A second launch adds a model's
// partial sums in a fixed order.
constexpr int kRedThreads = 256;
constexpr size_t kRedChunk = 8192;  // least values per block

inline int red_parts(size_t per_model) {
  return static_cast<int>(std::min<size_t>(kRedParts, (per_model + kRedChunk - 1) / kRedChunk));
}

__global__ void __launch_bounds__(kRedThreads) energy_kernel(const float* __restrict__ obs, size_t per_model,
                                                             double* __restrict__ part) {
  __shared__ double sh[32];
  const int model = blockIdx.y, parts = gridDim.x;
  const size_t chunk = (per_model + parts - 1) / parts;
  const size_t i0 = blockIdx.x * chunk, i1 = i0 + chunk < per_model ? i0 + chunk : per_model;
  const float* o = obs + static_cast<size_t>(model) * per_model;
  double acc = 0.0;
#pragma unroll 4
  for (size_t i = i0 + threadIdx.x; i < i1; i += kRedThreads) {
    const double d = static_cast<double>(o[i]);
    acc = __fma_rn(d, d, acc);
  }
  const double e = block_sum(acc, sh);
  if (threadIdx.x == 0) part[static_cast<size_t>(model) * kRedParts + blockIdx.x] = e;
}

__global__ void __launch_bounds__(kRedThreads) energy_final_kernel(const double* __restrict__ part, int parts,
                                                                   double* __restrict__ energy, float* __restrict__ scale,
                                                                   int* __restrict__ status) {
  __shared__ double sh[32];
  const int model = blockIdx.x;
  const double e = block_sum(threadIdx.x < parts ? part[static_cast<size_t>(model) * kRedParts + threadIdx.x] : 0.0, sh);
  if (threadIdx.x == 0) {
    energy[model] = e;
    scale[model] = static_cast<float>(1.0 / e);
    if (!(e > 0.0) && status) atomicExch(status, static_cast<int>(ST_ENERGY));
  }
}

// wave_wgpu.rs:13-54: d = p - obs; r = d * scale; e = 0.5 * d * d * scale (f32), summed in f64.
__global__ void __launch_bounds__(kRedThreads) residual_kernel(const float* pred, const float* __restrict__ obs,
                                                               const float* __restrict__ scale, size_t per_model, float* res,
                                                               double* __restrict__ part) {
  __shared__ double sh[32];
  const int model = blockIdx.y, parts = gridDim.x;
  const size_t chunk = (per_model + parts - 1) / parts;
  const size_t base = static_cast<size_t>(model) * per_model;
  const size_t i0 = base + blockIdx.x * chunk, end = base + per_model, i1 = i0 + chunk < end ? i0 + chunk : end;
  const float sc = scale[model];
  double acc = 0.0;
  // batches of four: pred and res may be one array, so the loads are issued ahead of the stores by hand
  for (size_t i = i0 + threadIdx.x; i < i1; i += 4 * kRedThreads) {
    float d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const size_t k = i + q * kRedThreads;
      d[q] = k < i1 ? pred[k] - obs[k] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const size_t k = i + q * kRedThreads;
      if (k < i1) {
        res[k] = d[q] * sc;
        acc += static_cast<double>(((0.5f * d[q]) * d[q]) * sc);
      }
    }
  }
  const double e = block_sum(acc, sh);
  if (threadIdx.x == 0) part[static_cast<size_t>(model) * kRedParts + blockIdx.x] = e;
}

__global__ void __launch_bounds__(kRedThreads) loss_final_kernel(const double* __restrict__ part, int parts,
                                                                 double* __restrict__ loss) {
  __shared__ double sh[32];
  const int model = blockIdx.x;
  const double e = block_sum(threadIdx.x < parts ? part[static_cast<size_t>(model) * kRedParts + threadIdx.x] : 0.0, sh);
  if (threadIdx.x == 0) loss[model] = e;
}

// wave_wgpu.rs:974-1005: the padded cells that fold onto a visible node, row-major (the reference's
// accumulation order), summed in f64. A node inside the grid has one cell and one thread; a node on
// the border has pad + 1 cells, a corner (pad + 1)^2, and gets a warp: the lanes load and shot-sum 32
// cells at a time, then the f64 sum runs over them in order. (A corner's 529 cells x 5 shots in one
// thread took 0.18 ms, all of it load latency.)
constexpr int kFoldThreads = 256;

__global__ void __launch_bounds__(kFoldThreads) fold_kernel(const float* __restrict__ gacc, const float* __restrict__ mask,
                                                            int shots, int nx, int nz, int pad, int nx_vis, int nz_vis,
                                                            int inner_blocks, float* __restrict__ grad) {
  const int model = blockIdx.y;
  const size_t cells = static_cast<size_t>(nx) * nz;
  const float* gm = gacc + static_cast<size_t>(model) * shots * cells;
  const float* mk = mask + static_cast<size_t>(model) * cells;
  float* out = grad + static_cast<size_t>(model) * nx_vis * nz_vis;
  auto cell_value = [&](size_t c) {
    float s = 0.0f;
    for (int k = 0; k < shots; ++k) s = s + gm[k * cells + c];
    return static_cast<double>(s * mk[c]);
  };
  if (static_cast<int>(blockIdx.x) < inner_blocks) {
    const int i = blockIdx.x * kFoldThreads + threadIdx.x;
    if (i >= nx_vis * nz_vis) return;
    const int vz = i / nx_vis, vx = i % nx_vis;
    if (vz == 0 || vz == nz_vis - 1 || vx == 0 || vx == nx_vis - 1) return;
    out[i] = static_cast<float>(0.0 + cell_value(static_cast<size_t>(vz + pad) * nx + vx + pad));
    return;
  }
  // border node b: the top row, the bottom row, then the two ends of each row in between
  const int lane = threadIdx.x & 31;
  const int b = (blockIdx.x - inner_blocks) * (kFoldThreads / 32) + (threadIdx.x >> 5);
  if (b >= 2 * nx_vis + 2 * (nz_vis - 2)) return;
  int vz, vx;
  if (b < 2 * nx_vis) {
    vz = b < nx_vis ? 0 : nz_vis - 1;
    vx = b % nx_vis;
  } else {
    vz = 1 + (b - 2 * nx_vis) / 2;
    vx = (b & 1) == 0 ? 0 : nx_vis - 1;
  }
  const int z_lo = (vz == 0) ? 0 : vz + pad, z_hi = (vz == nz_vis - 1) ? nz : vz + pad + 1;
  const int x_lo = (vx == 0) ? 0 : vx + pad, x_hi = (vx == nx_vis - 1) ? nx : vx + pad + 1;
  const int w = x_hi - x_lo, n = (z_hi - z_lo) * w;
  auto load = [&](int i) { return i < n ? cell_value(static_cast<size_t>(z_lo + i / w) * nx + x_lo + i % w) : 0.0; };
  double acc = 0.0, v = load(lane);
  for (int i0 = 0; i0 < n; i0 += 32) {
    const double next = load(i0 + 32 + lane);
    const int m = n - i0 < 32 ? n - i0 : 32;
    for (int l = 0; l < m; ++l) acc += __shfl_sync(0xffffffffu, v, l);
    v = next;
  }
  if (lane == 0) out[vz * nx_vis + vx] = static_cast<float>(acc);
}

// Causal FIR along time of [series][nt][nrec] traces: out[t] = sum over k, in order, of ker[k]
// x[t - (klen - 1) + k], times before 0 left out. One thread takes one trace (neighbouring threads
// neighbouring receivers, across series, so that no lane idles on 70 receivers) and R samples in
// a row: their inputs slide through registers, so a tap costs one load of x and one of ker for R
// products and sums, which FP32 issue then bounds (products and sums are not fused: each rounds as
// the one-sample-per-thread kernel's did, which two loads per product bounded). 16 models x 5 shots x
// 2001 x 70 at 377 taps: 0.35 against 3.2 ms; the FP32 bound is 0.21 ms (0.38 with the end of the record
// tested at every load and each load next to its use).
//
// R is 16, or 4 for small calls (few outputs, few taps that any of them has): those are one latency chain per
// thread, of R (R - 1) / 2 guarded taps and the window's loads, and want many short ones. Us for R = 4 / 16 (one
// sample per thread): 70 traces x 400 at 31 taps 3.9 / 6.8 (3.5), x 2001 at 31 4.0 / 6.9 (6.5); 1400 x 400 at
// 31 6.9 / 7.0 (17.4); 350 x 2001 at 101 19.9 / 12.1 (60.9); 70 x 400 at 377 28.3 / 18.6 (22.8). The line lies
// where the two meet.
constexpr int FIR_THREADS = 128;
constexpr long kFirFewProducts = 8L << 20;   // outputs times taps
constexpr int kFirFewTaps = 128;

// CHECK: fewer than R times, so a thread's samples may lie past the last; otherwise the last block of
// times starts at nt - R and stores only the samples that the one before it does not.
template <int FIR_R, bool CHECK>
__global__ void __launch_bounds__(FIR_THREADS) bandlimit_kernel(const float* __restrict__ in, const float* __restrict__ ker,
                                                                int klen, long traces, int nt, int nrec,
                                                                float* __restrict__ out) {
  const long c = blockIdx.x * static_cast<long>(FIR_THREADS) + threadIdx.x;
  if (c >= traces) return;
  const long base = (c / nrec) * nt * nrec + c % nrec;
  const float* x = in + base;
  const int first = blockIdx.y * FIR_R, t0 = CHECK ? first : min(first, nt - FIR_R);
  auto at = [&](int t) { return !CHECK || t < nt ? __ldg(x + static_cast<long>(t) * nrec) : 0.0f; };  // t >= 0
  float acc[FIR_R], win[FIR_R], next[FIR_R];
  // from tap k0 on, the taps of all FIR_R samples lie at times >= 0; before it sample j still has
  // the taps of times 0 .. j - 1
  const int k0 = max(0, klen - 1 - t0);
#pragma unroll
  for (int j = 0; j < FIR_R; ++j) {
    acc[j] = 0.0f;
    if (k0 > 0) {
#pragma unroll
      for (int ts = 0; ts < j; ++ts) {
        const int k = k0 - j + ts;
        if (k >= 0) acc[j] = acc[j] + __ldg(ker + k) * at(ts);
      }
    }
  }
  int ts = t0 - (klen - 1) + k0;  // time of tap k0 of sample 0
#pragma unroll
  for (int j = 0; j < FIR_R - 1; ++j) win[j] = at(ts + j);
  ts += FIR_R - 1;
  int k = k0;
  auto ahead = [&](int t) {  // the inputs of FIR_R taps, requested one round before their use
#pragma unroll
    for (int q = 0; q < FIR_R; ++q) next[q] = at(t + q);
  };
  if (k + FIR_R <= klen) ahead(ts);
  for (; k + FIR_R <= klen; k += FIR_R, ts += FIR_R) {
    // sample j reads time ts - (FIR_R - 1) + j + q at tap k + q: slot (j + q) % FIR_R
    float cur[FIR_R];
#pragma unroll
    for (int q = 0; q < FIR_R; ++q) cur[q] = next[q];
    if (k + 2 * FIR_R <= klen) ahead(ts + FIR_R);
#pragma unroll
    for (int q = 0; q < FIR_R; ++q) {
      win[(q + FIR_R - 1) % FIR_R] = cur[q];
      const float w = __ldg(ker + k + q);
#pragma unroll
      for (int j = 0; j < FIR_R; ++j) acc[j] = acc[j] + w * win[(j + q) % FIR_R];
    }
  }
#pragma unroll
  for (int q = 0; q < FIR_R - 1; ++q) {
    if (k + q < klen) {
      win[(q + FIR_R - 1) % FIR_R] = at(ts + q);
      const float w = __ldg(ker + k + q);
#pragma unroll
      for (int j = 0; j < FIR_R; ++j) acc[j] = acc[j] + w * win[(j + q) % FIR_R];
    }
  }
#pragma unroll
  for (int j = 0; j < FIR_R; ++j)
    if (t0 + j >= first && (!CHECK || t0 + j < nt)) out[base + static_cast<long>(t0 + j) * nrec] = acc[j];
}

// Zero-phase FIR low-pass and decimation to FP16: out[s][j][r] = sum_k ker[k] in[s][j*factor + k -
// center][r] (zero outside [0, nt)), for j < nt_out. One thread per output sample; the series' time
// window is read through L1.
__global__ void decimate_kernel(const float* __restrict__ in, const float* __restrict__ ker, int klen, int center,
                                int factor, int nt, int nrec, int nt_out, __half* __restrict__ out) {
  const int s = blockIdx.z;
  const int j = blockIdx.y;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrec) return;
  const float* x = in + static_cast<size_t>(s) * nt * nrec + r;
  const int t0 = j * factor - center;
  float acc = 0.0f;
  for (int k = 0; k < klen; ++k) {
    const int t = t0 + k;
    if (t >= 0 && t < nt) acc = acc + __ldg(&ker[k]) * __ldg(&x[static_cast<size_t>(t) * nrec]);
  }
  out[(static_cast<size_t>(s) * nt_out + j) * nrec + r] = __float2half_rn(acc);
}

__global__ void scale_kernel(const float* __restrict__ in, float alpha, size_t n, float* __restrict__ out) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = in[i] * alpha;
}

}  // namespace

cudaError_t launch_pad_velocity(const float* vis, int models, int nx_vis, int nz_vis, int pad, float vmin, float vmax,
                                float* padded, float* mask, cudaStream_t s) {
  const int cells = (nx_vis + 2 * pad) * (nz_vis + 2 * pad);
  dim3 grid((cells + 255) / 256, models);
  pad_kernel<<<grid, 256, 0, s>>>(vis, nx_vis, nz_vis, pad, vmin, vmax, padded, mask);
  return cudaGetLastError();
}

cudaError_t launch_energy(const float* observed, int models, size_t per_model, double* energy, float* scale,
                          int* status, double* scratch, cudaStream_t s) {
  const int parts = red_parts(per_model);
  energy_kernel<<<dim3(parts, models), kRedThreads, 0, s>>>(observed, per_model, scratch);
  energy_final_kernel<<<models, kRedThreads, 0, s>>>(scratch, parts, energy, scale, status);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_residual(const float* pred, const float* observed, const float* scale, int models,
                            size_t per_model, float* residual, double* loss, double* scratch, cudaStream_t s) {
  const int parts = red_parts(per_model);
  residual_kernel<<<dim3(parts, models), kRedThreads, 0, s>>>(pred, observed, scale, per_model, residual, scratch);
  loss_final_kernel<<<models, kRedThreads, 0, s>>>(scratch, parts, loss);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_fold(const float* gacc, const float* mask, int models, int shots, int nx, int nz, int pad,
                        int nx_vis, int nz_vis, float* grad, cudaStream_t s) {
  const int inner = (nx_vis * nz_vis + kFoldThreads - 1) / kFoldThreads;
  const int border = 2 * nx_vis + 2 * (nz_vis - 2), warps = kFoldThreads / 32;
  const dim3 grid(inner + (border + warps - 1) / warps, models);
  fold_kernel<<<grid, kFoldThreads, 0, s>>>(gacc, mask, shots, nx, nz, pad, nx_vis, nz_vis, inner, grad);
  return cudaGetLastError();
}

cudaError_t launch_bandlimit(const float* in, const float* ker, int klen, int series, int nt, int nrec, float* out,
                             cudaStream_t s) {
  const long traces = static_cast<long>(series) * nrec;
  const int taps = std::min(klen, nt);  // of an output, at most
  auto launch = [&](auto r) {
    constexpr int R = decltype(r)::value;
    const dim3 grid(static_cast<unsigned>((traces + FIR_THREADS - 1) / FIR_THREADS), (nt + R - 1) / R);
    if (nt < R)
      bandlimit_kernel<R, true><<<grid, FIR_THREADS, 0, s>>>(in, ker, klen, traces, nt, nrec, out);
    else
      bandlimit_kernel<R, false><<<grid, FIR_THREADS, 0, s>>>(in, ker, klen, traces, nt, nrec, out);
  };
  if (taps <= kFirFewTaps && traces * nt <= kFirFewProducts / taps)
    launch(std::integral_constant<int, 4>());
  else
    launch(std::integral_constant<int, 16>());
  return cudaGetLastError();
}

cudaError_t launch_decimate(const float* in, const float* ker, int klen, int center, int factor, int series, int nt,
                            int nrec, int nt_out, void* out_half, cudaStream_t s) {
  dim3 grid((nrec + 63) / 64, nt_out, series);
  decimate_kernel<<<grid, 64, 0, s>>>(in, ker, klen, center, factor, nt, nrec, nt_out, static_cast<__half*>(out_half));
  return cudaGetLastError();
}

cudaError_t launch_scale(const float* in, float alpha, size_t n, float* out, cudaStream_t s) {
  const int blocks = static_cast<int>(std::min<size_t>((n + 255) / 256, 152 * 16));
  scale_kernel<<<blocks > 0 ? blocks : 1, 256, 0, s>>>(in, alpha, n, out);
  return cudaGetLastError();
}

}  // namespace wg
