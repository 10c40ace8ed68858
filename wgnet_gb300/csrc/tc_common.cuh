// Tensor-core building blocks shared by the update network's kernels (tc_gemm.cu, tc_conv.cu):
// bounded mbarrier waits, TMA loads, tcgen05 descriptors and instructions, tensor maps.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "wave_launch.h"
#include "wgnet_gb300.h"

namespace wg {
namespace {

constexpr long kTcWaitLimit = 1L << 22;  // mbarrier polls before giving up

__device__ __forceinline__ unsigned su32(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void bar_init(uint64_t* b, unsigned n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint64_t* b, unsigned parity, long limit = kTcWaitLimit) {
  const unsigned a = su32(b);
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

__device__ __forceinline__ void tma2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(su32(b))
      : "memory");
}

// Shared-memory matrix descriptor, K-major with the 128-byte swizzle: rows of 128 bytes, atoms of
// 8 rows (sbo = 1024 bytes between atoms along M/N; lbo unused for this layout, encoded as 1). The
// tile base is 1024-byte aligned, so the base-offset field stays 0.
__device__ __forceinline__ uint64_t sdesc_sw128(const void* p) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((su32(p) >> 4) & 0x3FFF);
  d |= static_cast<uint64_t>(1) << 16;              // leading byte offset (unused), 16 bytes
  d |= static_cast<uint64_t>(1024 >> 4) << 32;      // stride byte offset: 8 rows x 128 bytes
  d |= static_cast<uint64_t>(1) << 46;              // descriptor version for the 5th-generation tensor cores
  d |= static_cast<uint64_t>(2) << 61;              // layout: 128-byte swizzle
  return d;
}

// The same descriptor in halves: the upper one is constant, the lower one advances by (bytes >> 4), so that
// the lane that issues the MMAs spends two instructions on a pair of operands instead of some thirty
// (they, not the tensor core, set the pace of N = 64 tiles: 70 cycles per MMA).
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr, uint32_t lbo = 16) {
  return ((smem_addr >> 4) & 0x3FFF) | ((lbo >> 4) << 16);
}
__device__ __forceinline__ void mma_bf16_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 a, {%1, %5};\n\t"
      "mov.b64 b, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(static_cast<uint32_t>(acc)), "n"(kDescHi)
      : "memory");
}

// Instruction descriptor of kind::f16: BF16 A and B, FP32 D, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4)                                 // D format F32
         | (1u << 7)                               // A format BF16
         | (1u << 10)                              // B format BF16
         | (static_cast<uint32_t>(n >> 3) << 17)   // N / 8
         | (static_cast<uint32_t>(m >> 4) << 24);  // M / 16
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(b)) : "memory");
}

inline PFN_cuTensorMapEncodeTiled_v12000 encode() {
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

// 2-D map over a row-major [rows][K] bf16 matrix, boxes of 64 elements (128 bytes) x box_rows,
// written to shared memory with the 128-byte swizzle.
inline int map_bf16(CUtensorMap* m, const void* base, long rows, long K, int box_rows) {
  auto fn = encode();
  if (!fn) return report_error(WG_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
  const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t es[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return report_error(WG_ERR_CUDA, ("cuTensorMapEncodeTiled(bf16) failed: " + std::to_string(r)).c_str());
  return WG_OK;
}


// Activations [batch][h][w][64] bf16 as boxes of 8 columns x `rows` rows of one image, 128 bytes per
// pixel, 128-byte swizzle: a box row of 8 pixels is one 1024-byte swizzle atom. Pixels outside the
// image read zero.
inline int map_image(CUtensorMap* m, const void* base, int batch, int h, int w, int rows) {
  auto fn = encode();
  if (!fn) return report_error(WG_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[4] = {64, static_cast<cuuint64_t>(w), static_cast<cuuint64_t>(h), static_cast<cuuint64_t>(batch)};
  const cuuint64_t strides[3] = {128, static_cast<cuuint64_t>(w) * 128, static_cast<cuuint64_t>(w) * h * 128};
  const cuuint32_t box[4] = {64, 8, static_cast<cuuint32_t>(rows), 1};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return report_error(WG_ERR_CUDA, ("cuTensorMapEncodeTiled(image) failed: " + std::to_string(r)).c_str());
  return WG_OK;
}

__device__ __forceinline__ void tma_image(void* dst, const CUtensorMap* map, int x, int y, int n, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(x), "r"(y), "r"(n), "r"(su32(b))
      : "memory");
}

// Activations [batch][h][w][64] bf16 read pixel by pixel in their linear order, shifted by one tap of
// a same-padded 3x3 convolution of dilation `dil` (im2col mode: the base pixel runs over the image
// shifted by (-dil, -dil), the tap's offset (0..2) dil comes with the load; pixels outside the image
// or beyond the batch read zero). `pixels` x 128 bytes per load, 128-byte swizzle.
inline int map_im2col(CUtensorMap* m, const void* base, int batch, int h, int w, int dil, int pixels) {
  static PFN_cuTensorMapEncodeIm2col_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeIm2col", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeIm2col_v12000>(p);
  }();
  if (!fn) return report_error(WG_ERR_CUDA, "cuTensorMapEncodeIm2col is not available");
  const cuuint64_t dims[4] = {64, static_cast<cuuint64_t>(w), static_cast<cuuint64_t>(h), static_cast<cuuint64_t>(batch)};
  const cuuint64_t strides[3] = {128, static_cast<cuuint64_t>(w) * 128, static_cast<cuuint64_t>(w) * h * 128};
  const int corner[2] = {-dil, -dil};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, corner, corner, 64,
                        static_cast<cuuint32_t>(pixels), es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return report_error(WG_ERR_CUDA, ("cuTensorMapEncodeIm2col failed: " + std::to_string(r)).c_str());
  return WG_OK;
}

// Position of a linear pixel: the divisions are done once per tile, not once per tap (with one lane
// issuing the loads they bounded the convolutions).
struct Pixel {
  int n, y, x;
  __device__ __forceinline__ Pixel(int m, int h, int w) {
    n = m / (h * w);
    const int r = m - n * h * w;
    y = r / w;
    x = r - y * w;
  }
  __device__ __forceinline__ void advance(int pixels, int h, int w) {
    x += pixels;
    while (x >= w) {
      x -= w;
      if (++y == h) {
        y = 0;
        ++n;
      }
    }
  }
};

// Load of `pixels` (of the map) shifted pixels from p on, for the tap offset (ox, oy).
__device__ __forceinline__ void tma_im2col(void* dst, const CUtensorMap* map, const Pixel& p, int dil, int ox, int oy,
                                           uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6], {%7, %8};" ::"r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(p.x - dil), "r"(p.y - dil), "r"(p.n), "r"(su32(b)),
      "h"(static_cast<unsigned short>(ox)), "h"(static_cast<unsigned short>(oy))
      : "memory");
}

}  // namespace
}  // namespace wg
