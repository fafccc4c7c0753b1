// Kernel registry and the launch shim behind the internal C-ABI of
// mofft_cuda.h.  Each registry entry is one compiled variant (precision, line
// length, threads per line, lines per CTA, in-CTA radix chain).  The host
// planner picks entries; the MEASURE planner times them.
#include <atomic>
#include <map>
#include <memory>
#include <tuple>
#include <vector>

#include "fft_instances.cuh"

using namespace mofft;

namespace {

const std::vector<Entry> &registry() {
  static const std::vector<Entry> all = [] {
    std::vector<Entry> v;
    const Entry *(*lists[])(int *) = {entries_generic, entries_generic_lt,
                                      entries_generic_eo, entries_generic_vr,
                                      entries_rows_f32,
                                      entries_rows_f64, entries_cols_f32,
                                      entries_cols_f64, entries_rows_mixed,
                                      entries_rows_even, entries_twin_f32,
                                      entries_cols_mixed, entries_tensor64,
                                      entries_tensor, entries_cluster};
    for (auto list : lists) {
      int n = 0;
      const Entry *e = list(&n);
      v.insert(v.end(), e, e + n);
    }
    return v;
  }();
  return all;
}

}  // namespace

extern "C" int mofft_cuda_kernel_count(void) { return (int)registry().size(); }

extern "C" const mofft_kernel_desc *mofft_cuda_kernel_get(int index) {
  const auto &r = registry();
  if (index < 0 || index >= (int)r.size()) return nullptr;
  return &r[index].desc;
}

extern "C" int mofft_cuda_kernels_of(int kind, int precision_bits, int length,
                                     const int **indices) {
  using Key = std::tuple<int, int, int>;
  static const std::map<Key, std::vector<int>> index = [] {
    std::map<Key, std::vector<int>> m;
    const auto &r = registry();
    for (int i = 0; i < (int)r.size(); ++i)
      m[Key(r[i].desc.kind, r[i].desc.precision_bits, r[i].desc.length)].push_back(i);
    return m;
  }();
  const auto it = index.find(Key(kind, precision_bits, length));
  if (it == index.end()) return 0;
  *indices = it->second.data();
  return (int)it->second.size();
}

extern "C" size_t mofft_cuda_generic_smem(int precision_bits, int length,
                                          int lines, int cols) {
  return precision_bits == 32 ? generic_smem<float>(length, lines, cols)
                              : generic_smem<double>(length, lines, cols);
}

// Opts one registry kernel into its shared memory on the current device.
static cudaError_t prepare_entry(int kernel) {
  const auto &r = registry();
  constexpr int kDevices = 64;
  int device = 0;
  const cudaError_t have = cudaGetDevice(&device);
  if (have != cudaSuccess) return have;
  if (device < 0 || device >= kDevices) return cudaErrorInvalidDevice;
  static const std::unique_ptr<std::atomic<bool>[]> done(
      new std::atomic<bool>[kDevices * r.size()]());
  std::atomic<bool> &mine = done[(size_t)device * r.size() + (size_t)kernel];
  if (mine.load(std::memory_order_acquire)) return cudaSuccess;
  const Entry &e = r[kernel];
  size_t smem = e.desc.smem_bytes;
  if (smem > 227 * 1024) smem = 227 * 1024;
  cudaError_t err =
      cudaFuncSetAttribute(e.func(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err == cudaSuccess && e.func_tail)
    err = cudaFuncSetAttribute(e.func_tail(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem);
  if (err == cudaSuccess) mine.store(true, std::memory_order_release);
  return err;
}

// Setting a kernel's attribute loads it, about 0.2 ms each, so a plan prepares the
// kernels that its passes launch and not the whole registry: the first plan of a
// process took 117 ms with all of them, 9 with its own.
extern "C" int mofft_cuda_prepare_pass(int kernel, const mofft_pass_args *args) {
  const auto &r = registry();
  if (kernel < 0 || kernel >= (int)r.size() || !args) return (int)cudaErrorInvalidValue;
  const mofft_kernel_desc &d = r[kernel].desc;
  if (d.kind == MOFFT_KERNEL_GENERIC && d.bank == 0 && d.radices[0] <= 16) {
    const cudaError_t err =
        d.precision_bits == 32 ? rt_prepare_f32(args) : rt_prepare_f64(args);
    if (err != cudaErrorNotSupported) return (int)err;
  }
  return (int)prepare_entry(kernel);
}

extern "C" int mofft_cuda_prepare_columns(int precision_bits) {
  for (int i = 0; i < (int)registry().size(); ++i) {
    const mofft_kernel_desc &d = registry()[i].desc;
    if (d.precision_bits != precision_bits || d.bank != 0 ||
        (d.kind != MOFFT_KERNEL_COLS && d.kind != MOFFT_KERNEL_GENERIC))
      continue;
    const cudaError_t err = prepare_entry(i);
    if (err != cudaSuccess) return (int)err;
  }
  return (int)(precision_bits == 32 ? rt_prepare_columns_f32() : rt_prepare_columns_f64());
}

extern "C" size_t mofft_cuda_kernel_aux_bytes(int kernel) {
  const auto &r = registry();
  if (kernel < 0 || kernel >= (int)r.size()) return 0;
  return r[kernel].fill_aux ? r[kernel].aux_bytes : 0;
}

extern "C" int mofft_cuda_kernel_fill_aux(int kernel, void *dst) {
  const auto &r = registry();
  if (kernel < 0 || kernel >= (int)r.size() || !r[kernel].fill_aux || !dst)
    return (int)cudaErrorInvalidValue;
  return r[kernel].fill_aux(dst);
}

extern "C" int mofft_cuda_launch_pass(int kernel, const mofft_pass_args *args,
                                      void *stream) {
  const auto &r = registry();
  if (kernel < 0 || kernel >= (int)r.size() || !args) return (int)cudaErrorInvalidValue;
  return (int)r[kernel].launch(args, static_cast<cudaStream_t>(stream));
}
