// Kernels of the learned update network (a dilated residual conv net on the 70x70 model grid):
// im2col of its 8-channel input, input features, the training loss and the Adam update. The convolutions
// themselves are tc_conv.cu's; col2im, the transposes, casts, sums and masks here are the separate passes
// that those fuse (with gemm_bf16_kernel the route that their results equal bit for bit).
// No reference counterpart: WGNet's refine() (python/wgnet/refine.py:41-169) has no learned part.
//
// Layouts: activations [B][H][W][C] (channels contiguous); im2col columns [M][Kp] with
// M = B H W, k = tap * C + c (tap = 3 ky + kx), zero for k >= 9 C; weights [N][Kp] (GEMM B operand)
// and their transpose [Kp][N] (the data-gradient GEMM's B operand). BF16 where a GEMM reads it,
// FP32 elsewhere.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "wave_launch.h"
#include "wgnet_gb300.h"

namespace {

// One block per image row and 32-bit arithmetic: writing the columns bounds it (40 MB for 32 images of
// 70 x 70 with 8 channels, 6 us at the HBM rate, now 12); with 64-bit
// divisions for each 16 bytes it took 21.
__global__ void im2col_kernel(const __nv_bfloat16* __restrict__ act, int H, int W, int C, int dil, int Kp,
                              __nv_bfloat16* __restrict__ col) {
  const long row = blockIdx.x;  // b H + y
  const int y = static_cast<int>(row % H);
  const unsigned kv = Kp / 8, n = W * kv;
  const __nv_bfloat16* in = act + row * W * C;
  uint4* out = reinterpret_cast<uint4*>(col + row * W * Kp);
  for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned x = i / kv, k8 = (i - x * kv) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (k8 < 9u * C) {
      const unsigned tap = k8 / C, c = k8 - tap * C, ty = tap / 3;
      const int dy = (static_cast<int>(ty) - 1) * dil, dx = (static_cast<int>(tap - 3 * ty) - 1) * dil;
      const int xs = static_cast<int>(x) + dx;
      if (y + dy >= 0 && y + dy < H && xs >= 0 && xs < W)
        v = *reinterpret_cast<const uint4*>(in + (static_cast<long>(dy) * W + xs) * C + c);
    }
    out[i] = v;
  }
}

// dact[m][c] (+)= sum over taps of dcol[m'][tap C + c], m' the pixel whose tap reads m.
__global__ void col2im_kernel(const float* __restrict__ dcol, int B, int H, int W, int C, int dil, int Kp,
                              float* __restrict__ dact, int accumulate) {
  const long M = static_cast<long>(B) * H * W;
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= M * C) return;
  const long m = i / C;
  const int c = static_cast<int>(i % C);
  const int x = static_cast<int>(m % W), y = static_cast<int>((m / W) % H);
  const long b = m / (static_cast<long>(W) * H);
  float acc = 0.0f;
#pragma unroll
  for (int tap = 0; tap < 9; ++tap) {
    const int ys = y - (tap / 3 - 1) * dil, xs = x - (tap % 3 - 1) * dil;
    if (ys >= 0 && ys < H && xs >= 0 && xs < W) acc += dcol[((b * H + ys) * W + xs) * Kp + tap * C + c];
  }
  dact[i] = accumulate ? dact[i] + acc : acc;
}

// out[c][r] = in[r][c] for a [R][Cc] bf16 matrix (32 x 32 tiles through shared memory).
__global__ void transpose_bf16_kernel(const __nv_bfloat16* __restrict__ in, long R, int Cc,
                                      __nv_bfloat16* __restrict__ out) {
  __shared__ __nv_bfloat16 t[32][33];
  const long r0 = static_cast<long>(blockIdx.x) * 32;
  const int c0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const long r = r0 + k;
    const int c = c0 + threadIdx.x;
    t[k][threadIdx.x] = (r < R && c < Cc) ? in[r * Cc + c] : __float2bfloat16(0.0f);
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int c = c0 + k;
    const long r = r0 + threadIdx.x;
    if (c < Cc && r < R) out[static_cast<long>(c) * R + r] = t[threadIdx.x][k];
  }
}

// out = bf16(relu ? max(x, 0) : x); column slice: rows of ld floats, first `cols` used, out [rows][cols]
__global__ void cast_bf16_kernel(const float* __restrict__ x, long rows, int ld, int cols, int relu,
                                 __nv_bfloat16* __restrict__ out) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= rows * cols) return;
  float v = x[(i / cols) * ld + i % cols];
  if (relu) v = fmaxf(v, 0.0f);
  out[i] = __float2bfloat16(v);
}

// out = a + b (fp32), and its bf16 copy when out_bf16 != null
__global__ void add_kernel(const float* __restrict__ a, const float* __restrict__ b, long n, float* __restrict__ out,
                           __nv_bfloat16* __restrict__ out_bf16) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const float v = a[i] + b[i];
  out[i] = v;
  if (out_bf16) out_bf16[i] = __float2bfloat16(v);
}

// out = d where mask > 0 else 0 (the ReLU derivative from the stored bf16 activation)
__global__ void relu_grad_kernel(const float* __restrict__ d, const __nv_bfloat16* __restrict__ mask, long n,
                                 float* __restrict__ out) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  out[i] = __bfloat162float(mask[i]) > 0.0f ? d[i] : 0.0f;
}

// Per-sample RMS of the gradient (f64 reduction, one block per sample: its chain of f64 additions
// bounds it, so 1024 threads take few terms each and the warps reduce in registers: 70 x 70 in 9.8 us, in
// 15.6 with 256 threads and a tree in shared memory).
constexpr int kRmsThreads = 1024;
__global__ void __launch_bounds__(kRmsThreads) rms_kernel(const float* __restrict__ g, int P, float* __restrict__ rms) {
  __shared__ double red[32];
  const float* x = g + static_cast<long>(blockIdx.x) * P;
  double s = 0.0;
  for (int i = threadIdx.x; i < P; i += kRmsThreads) s += static_cast<double>(x[i]) * x[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) rms[blockIdx.x] = static_cast<float>(sqrt(s / P));
  }
}

// Input features [B][H][W][8]: (v - 3) km/s, g / rms(g), one-hot band (4), depth z / H, 0.
__global__ void features_kernel(const float* __restrict__ vel_km, const float* __restrict__ grad,
                                const float* __restrict__ rms, const int* __restrict__ band, int B, int H, int W,
                                __nv_bfloat16* __restrict__ out) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  const long n = static_cast<long>(B) * H * W;
  if (i >= n) return;
  const int b = static_cast<int>(i / (static_cast<long>(H) * W));
  const int y = static_cast<int>((i / W) % H);
  const float r = rms[b];
  const int bd = band[b];
  float f[8];
  f[0] = vel_km[i] - 3.0f;
  f[1] = r > 0.0f ? grad[i] / r : 0.0f;
  for (int k = 0; k < 4; ++k) f[2 + k] = (bd == k) ? 1.0f : 0.0f;
  f[6] = static_cast<float>(y) / static_cast<float>(H);
  f[7] = 0.0f;
  __align__(16) __nv_bfloat16 o[8];
  for (int k = 0; k < 8; ++k) o[k] = __float2bfloat16(f[k]);
  *reinterpret_cast<uint4*>(out + i * 8) = *reinterpret_cast<const uint4*>(o);
}

// Mean squared error of scale * out[m][0] against target[m]; writes dL/d out[m][0] (other columns
// of the row untouched: they stay zero) and accumulates the loss (f64) per block into loss.
__global__ void mse_kernel(const float* __restrict__ out, int ld, const float* __restrict__ target, float scale,
                           long M, double* __restrict__ loss, float* __restrict__ dout) {
  __shared__ double red[256];
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  double l = 0.0;
  if (i < M) {
    const float e = scale * out[i * ld] - target[i];
    l = static_cast<double>(e) * e;
    dout[i * ld] = 2.0f * e * scale / static_cast<float>(M);
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, red[0] / static_cast<double>(M));
}

// Adam on FP32 master weights w32 [N][Kp]; the gradient is the sum, in split order, of the partials
// of the transposed weight gradient [S][Kp][N], kept in grad [N][Kp] if given. Writes the BF16 weights
// [N][Kp] and their transpose. All layers in one launch (blockIdx.y; one launch per layer left most SMs
// idle: 14 x 8.6 us). Reading the partials bounds it (110 MB for 63 splits of the network): a warp sums
// 32 neighbouring n of one k, 128-byte lines; a tile of 32 n x 8 k then turns over in shared memory so
// that every other access is whole 32-byte sectors too (from the summing layout each took 4 bytes of a
// sector: 94 us; now 23, 19 of them the partials at the HBM rate).
constexpr int kAdamLayers = 16;
struct AdamLayer {
  const float* partial;
  float *w32, *m1, *m2, *grad;
  __nv_bfloat16 *w, *wt;
  int S, N, Kp;
};
struct AdamArgs {
  AdamLayer layer[kAdamLayers];
  float lr, b1, b2, eps, c1, c2;
};

constexpr int ATN = 32, ATK = 8;  // tile of a block

__global__ void __launch_bounds__(ATN * ATK) adam_kernel(const __grid_constant__ AdamArgs a) {
  __shared__ float gs[ATN][ATK + 1];
  __shared__ __nv_bfloat16 qs[ATK][ATN + 2];
  const AdamLayer& L = a.layer[blockIdx.y];
  const int N = L.N, Kp = L.Kp, across = (N + ATN - 1) / ATN;
  const int n0 = static_cast<int>(blockIdx.x % across) * ATN;
  const long k0 = static_cast<long>(blockIdx.x / across) * ATK;
  if (k0 >= Kp) return;
  const int tn = threadIdx.x % ATN, tk = threadIdx.x / ATN;  // summing layout
  const bool in = n0 + tn < N && k0 + tk < Kp;
  const long t = (k0 + tk) * N + n0 + tn;
  if (L.partial) {
    float g = 0.0f;
    if (in) {
      const float* p = L.partial + t;
      const long step = static_cast<long>(Kp) * N;
      for (int s = 0; s < L.S; s += 16) {  // whole rounds of 16 loads in flight, also at the end
        float v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = s + u < L.S ? __ldcs(p + (s + u) * step) : 0.0f;
#pragma unroll
        for (int u = 0; u < 16; ++u) g = s + u < L.S ? g + v[u] : g;
      }
    }
    gs[tn][tk] = g;
    __syncthreads();
  }
  const int un = threadIdx.x / ATK, uk = threadIdx.x % ATK;  // updating layout
  if (n0 + un < N && k0 + uk < Kp) {
    const long i = static_cast<long>(n0 + un) * Kp + k0 + uk;
    float w = L.w32[i];
    if (L.partial) {
      const float g = gs[un][uk];
      const float m = a.b1 * L.m1[i] + (1.0f - a.b1) * g;
      const float v = a.b2 * L.m2[i] + (1.0f - a.b2) * g * g;
      L.m1[i] = m;
      L.m2[i] = v;
      w -= a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
      L.w32[i] = w;
      if (L.grad) L.grad[i] = g;
    }
    const __nv_bfloat16 q = __float2bfloat16(w);
    L.w[i] = q;
    qs[uk][un] = q;
  }
  __syncthreads();
  if (in) L.wt[t] = qs[tk][tn];
}

inline unsigned blocks(long n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

#define PC_LAUNCH(...)                                                         \
  do {                                                                         \
    wg::note_launch();                                                         \
    __VA_ARGS__;                                                               \
    cudaError_t e_ = cudaGetLastError();                                       \
    if (e_ != cudaSuccess) return wg::report_error(WG_ERR_CUDA, cudaGetErrorString(e_)); \
    return WG_OK;                                                              \
  } while (0)

}  // namespace

extern "C" {

int wg_pc_im2col(const void* act, int B, int H, int W, int C, int dil, int Kp, void* col, void* stream) {
  if (!act || !col || B < 1 || H < 1 || W < 1 || C < 8 || C % 8 || Kp % 64 || Kp < 9 * C || dil < 1)
    return wg::report_error(WG_ERR_ARG, "im2col: bad shape");
  PC_LAUNCH(im2col_kernel<<<static_cast<unsigned>(static_cast<long>(B) * H), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(act), H, W, C, dil, Kp, static_cast<__nv_bfloat16*>(col)));
}

int wg_pc_col2im(const float* dcol, int B, int H, int W, int C, int dil, int Kp, float* dact, int accumulate,
                 void* stream) {
  if (!dcol || !dact || B < 1 || C < 1 || Kp < 9 * C || dil < 1) return wg::report_error(WG_ERR_ARG, "col2im: bad shape");
  const long n = static_cast<long>(B) * H * W * C;
  PC_LAUNCH(col2im_kernel<<<blocks(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(dcol, B, H, W, C, dil, Kp,
                                                                                        dact, accumulate));
}

int wg_pc_transpose_bf16(const void* in, long R, int Cc, void* out, void* stream) {
  if (!in || !out || R < 1 || Cc < 1) return wg::report_error(WG_ERR_ARG, "transpose: bad shape");
  dim3 grid(static_cast<unsigned>((R + 31) / 32), static_cast<unsigned>((Cc + 31) / 32));
  PC_LAUNCH(transpose_bf16_kernel<<<grid, dim3(32, 8), 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(in), R, Cc, static_cast<__nv_bfloat16*>(out)));
}

int wg_pc_cast_bf16(const float* x, long rows, int ld, int cols, int relu, void* out, void* stream) {
  if (!x || !out || rows < 1 || cols < 1 || ld < cols) return wg::report_error(WG_ERR_ARG, "cast: bad shape");
  PC_LAUNCH(cast_bf16_kernel<<<blocks(rows * cols, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      x, rows, ld, cols, relu, static_cast<__nv_bfloat16*>(out)));
}

int wg_pc_add(const float* a, const float* b, long n, float* out, void* out_bf16, void* stream) {
  if (!a || !b || !out || n < 1) return wg::report_error(WG_ERR_ARG, "add: bad argument");
  PC_LAUNCH(add_kernel<<<blocks(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      a, b, n, out, static_cast<__nv_bfloat16*>(out_bf16)));
}

int wg_pc_relu_grad(const float* d, const void* mask, long n, float* out, void* stream) {
  if (!d || !mask || !out || n < 1) return wg::report_error(WG_ERR_ARG, "relu_grad: bad argument");
  PC_LAUNCH(relu_grad_kernel<<<blocks(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      d, static_cast<const __nv_bfloat16*>(mask), n, out));
}

int wg_pc_features(const float* vel_km, const float* grad, const int* band, int B, int H, int W, float* rms,
                   void* out, void* stream) {
  if (!vel_km || !grad || !band || !rms || !out || B < 1) return wg::report_error(WG_ERR_ARG, "features: bad argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  wg::note_launch();
  rms_kernel<<<B, kRmsThreads, 0, st>>>(grad, H * W, rms);
  const long n = static_cast<long>(B) * H * W;
  PC_LAUNCH(features_kernel<<<blocks(n, 256), 256, 0, st>>>(vel_km, grad, rms, band, B, H, W,
                                                            static_cast<__nv_bfloat16*>(out)));
}

int wg_pc_mse(const float* out, int ld, const float* target, float scale, long M, double* loss, float* dout,
              void* stream) {
  if (!out || !target || !loss || !dout || M < 1) return wg::report_error(WG_ERR_ARG, "mse: bad argument");
  PC_LAUNCH(mse_kernel<<<blocks(M, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(out, ld, target, scale, M, loss,
                                                                                     dout));
}

int wg_pc_adam_layers(int layers, const float* const* partial, const int* splits, const int* n, const int* kp,
                      float* const* w32, float* const* m1, float* const* m2, float* const* grad, void* const* w,
                      void* const* wt, float lr, float b1, float b2, float eps, int step, void* stream) {
  if (layers < 1 || layers > kAdamLayers || !n || !kp || !w32 || !m1 || !m2 || !w || !wt || (partial && !splits))
    return wg::report_error(WG_ERR_ARG, "adam: bad argument");
  AdamArgs a{};
  long most = 0;
  bool steps = false;
  for (int i = 0; i < layers; ++i) {
    const float* p = partial ? partial[i] : nullptr;
    if (!w32[i] || !m1[i] || !m2[i] || !w[i] || !wt[i] || n[i] < 1 || kp[i] < 1 || (p && (splits[i] < 1 || step < 1)))
      return wg::report_error(WG_ERR_ARG, "adam: bad argument");
    a.layer[i] = {p, w32[i], m1[i], m2[i], grad ? grad[i] : nullptr, static_cast<__nv_bfloat16*>(w[i]),
                  static_cast<__nv_bfloat16*>(wt[i]), p ? splits[i] : 0, n[i], kp[i]};
    const long tiles = static_cast<long>((n[i] + ATN - 1) / ATN) * ((kp[i] + ATK - 1) / ATK);
    most = tiles > most ? tiles : most;
    steps = steps || p;
  }
  a.lr = lr;
  a.b1 = b1;
  a.b2 = b2;
  a.eps = eps;
  a.c1 = steps ? 1.0f - powf(b1, static_cast<float>(step)) : 1.0f;
  a.c2 = steps ? 1.0f - powf(b2, static_cast<float>(step)) : 1.0f;
  PC_LAUNCH(adam_kernel<<<dim3(static_cast<unsigned>(most), layers), ATN * ATK, 0, static_cast<cudaStream_t>(stream)>>>(a));
}

int wg_pc_adam(const float* partial, int S, int N, int Kp, float* w32, float* m1, float* m2, float lr, float b1,
               float b2, float eps, int step, void* w, void* wt, void* stream) {
  return wg_pc_adam_layers(1, &partial, &S, &N, &Kp, &w32, &m1, &m2, nullptr, &w, &wt, lr, b1, b2, eps, step, stream);
}

}  // extern "C"
