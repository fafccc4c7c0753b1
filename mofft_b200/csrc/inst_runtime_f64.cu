// Runtime-chain kernels, double.
#include "inst_runtime.cuh"

namespace mofft {
cudaError_t rt_launch_f64(const mofft_pass_args *p, cudaStream_t s) {
  return rt_launch<double>(p, s);
}
cudaError_t rt_prepare_f64(const mofft_pass_args *p) { return rt_prepare<double>(p); }
cudaError_t rt_prepare_columns_f64() { return rt_prepare_columns<double>(); }
}  // namespace mofft
