// Runtime-stage-list kernels of kernel bank 3 (vector-reuse codelets).
#include "fft_instances.cuh"

namespace mofft {
const Entry *entries_generic_vr(int *count) {
  static const Entry e[] = {
      GenericInst<float, false, 3>::entry("generic_float_vr"),
      GenericInst<double, false, 3>::entry("generic_double_vr"),
      GenericInst<float, true, 3>::entry("generic_float_wide_vr"),
      GenericInst<double, true, 3>::entry("generic_double_wide_vr"),
  };
  *count = (int)(sizeof(e) / sizeof(e[0]));
  return e;
}
}  // namespace mofft
