// Runtime-stage-list kernels of kernel bank 1 (like-terms codelets).
#include "fft_instances.cuh"

namespace mofft {
const Entry *entries_generic_lt(int *count) {
  static const Entry e[] = {
      GenericInst<float, false, 1>::entry("generic_float_lt"),
      GenericInst<double, false, 1>::entry("generic_double_lt"),
      GenericInst<float, true, 1>::entry("generic_float_wide_lt"),
      GenericInst<double, true, 1>::entry("generic_double_wide_lt"),
  };
  *count = (int)(sizeof(e) / sizeof(e[0]));
  return e;
}
}  // namespace mofft
