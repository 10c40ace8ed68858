// Explicit instantiation of the generation-3 kernels for one launch shape (see wave_table.cu).
#include "wave_kernels3.cuh"

namespace wg {

template <>
cudaError_t fwd3_dispatch<144, 12, 4, 4, 9, 2>(bool traces, bool store, const FwdArgs& a, size_t smem, cudaStream_t s) {
  return fwd3_dispatch_impl<144, 12, 4, 4, 9, 2>(traces, store, a, smem, s);
}

template <>
cudaError_t adj3_dispatch<144, 12, 4, 4, 9, 2>(const AdjArgs& a, size_t smem, cudaStream_t s) {
  return adj3_dispatch_impl_pref<144, 12, 4, 4, 9, 2>(a, smem, s);
}

}  // namespace wg
