// Explicit instantiation of the generation-3 kernels for grids of any width up to 144 (see wave_table.cu).
#include "wave_kernels3.cuh"

namespace wg {

template <>
cudaError_t fwd3r_dispatch<144, 12, 3, 6, 8, 2>(bool traces, bool store, const FwdArgs& a, size_t smem, cudaStream_t s) {
  return fwd3r_dispatch_impl<144, 12, 3, 6, 8, 2>(traces, store, a, smem, s);
}

template <>
cudaError_t adj3r_dispatch<144, 12, 3, 6, 8, 2>(const AdjArgs& a, size_t smem, cudaStream_t s) {
  return adj3r_dispatch_impl<144, 12, 3, 6, 8, 2>(a, smem, s);
}

}  // namespace wg
