// Runtime-chain kernels, float.
#include "inst_runtime.cuh"

namespace mofft {
cudaError_t rt_launch_f32(const mofft_pass_args *p, cudaStream_t s) {
  return rt_launch<float>(p, s);
}
cudaError_t rt_prepare_f32(const mofft_pass_args *p) { return rt_prepare<float>(p); }
cudaError_t rt_prepare_columns_f32() { return rt_prepare_columns<float>(); }
}  // namespace mofft
