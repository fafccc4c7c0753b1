// Runtime-stage-list kernels of kernel bank 2 (even-odd codelets).
#include "fft_instances.cuh"

namespace mofft {
const Entry *entries_generic_eo(int *count) {
  static const Entry e[] = {
      GenericInst<float, false, 2>::entry("generic_float_eo"),
      GenericInst<double, false, 2>::entry("generic_double_eo"),
      GenericInst<float, true, 2>::entry("generic_float_wide_eo"),
      GenericInst<double, true, 2>::entry("generic_double_wide_eo"),
  };
  *count = (int)(sizeof(e) / sizeof(e[0]));
  return e;
}
}  // namespace mofft
