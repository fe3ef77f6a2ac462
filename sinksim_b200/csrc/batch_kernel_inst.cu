// The batch kernel for teams of SSB_INST_WARPS warps, for fleets when SSB_INST_FLEET is true, in both numerics.
#include "batch_kernel.cuh"

namespace ssb {

template <bool MIXED, int W, bool FLEET>
cudaError_t BatchKernel<MIXED, W, FLEET>::set_smem(std::size_t bytes) {
  return cudaFuncSetAttribute(run_batch<MIXED, W, FLEET>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

template <bool MIXED, int W, bool FLEET>
cudaError_t BatchKernel<MIXED, W, FLEET>::occupancy(int threads, std::size_t bytes, int* perSM) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(perSM, run_batch<MIXED, W, FLEET>, threads, bytes);
}

template <bool MIXED, int W, bool FLEET>
void BatchKernel<MIXED, W, FLEET>::launch(const DevModel& M, const DevBatch& B, const SlotLayout& L, int grid, int threads, std::size_t smem,
                                          cudaStream_t s) {
  run_batch<MIXED, W, FLEET><<<grid, threads, smem, s>>>(M, B, L);
}

template struct BatchKernel<false, SSB_INST_WARPS, SSB_INST_FLEET>;
template struct BatchKernel<true, SSB_INST_WARPS, SSB_INST_FLEET>;

}  // namespace ssb
