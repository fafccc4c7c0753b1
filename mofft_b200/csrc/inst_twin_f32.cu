// Twin one-pass FP32 kernels (two lines per thread, packed arithmetic).
#include "fft_instances.cuh"
#include "twin_fft.cuh"

namespace mofft {

template <int L, int TPL, int TP, int SH, int... Rs>
struct TwinInst {
  using G = TwinGeom<L, TPL, TP, SH>;
  static const void *func() {
    return reinterpret_cast<const void *>(&twin_kernel<L, TPL, TP, SH, Rs...>);
  }
  static cudaError_t launch(const mofft_pass_args *p, cudaStream_t s) {
    if (p->conj_in != p->conj_out) return cudaErrorInvalidValue;
    const long long grid = (p->batch + 2 * TP - 1) / (2 * TP);
    if (grid <= 0) return cudaSuccess;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    return launch_pass(func(), (unsigned)grid, G::THREADS, G::SMEM, rows_args<float>(p), p, s);
  }
  static Entry entry(const char *name) {
    Entry e{};
    e.desc.name = name;
    e.desc.precision_bits = 32;
    e.desc.kind = MOFFT_KERNEL_ROWS;
    e.desc.length = L;
    e.desc.lines = 2 * TP;
    e.desc.threads = G::THREADS;
    const int rs[] = {Rs...};
    e.desc.radix_count = (int)sizeof...(Rs);
    for (int i = 0; i < 8; ++i) e.desc.radices[i] = i < (int)sizeof...(Rs) ? rs[i] : 0;
    e.desc.smem_bytes = G::SMEM;
    e.launch = &launch;
    e.func = &func;
    return e;
  }
};

template <int L, int TPL, int C, int... Rs>
struct TwinColsInst {
  using G = TwinColsGeom<L, TPL, C>;
  static constexpr int kRadices[] = {Rs...};
  static constexpr size_t kSmemTail = G::super_smem(kRadices[0]);
  static_assert(kSmemTail <= 227 * 1024, "shared memory of one CTA");
  static const void *func() {
    return reinterpret_cast<const void *>(&twin_cols_kernel<L, TPL, C, true, Rs...>);
  }
  static const void *func_tail() {
    return reinterpret_cast<const void *>(&twin_cols_kernel<L, TPL, C, false, Rs...>);
  }
  static cudaError_t launch(const mofft_pass_args *p, cudaStream_t s) {
    if (p->total % L != 0 || (p->total / L) % C != 0) return cudaErrorInvalidValue;
    if (p->ns_outer != 1 && p->ns_outer % C != 0) return cudaErrorInvalidValue;
    const long long grid = (p->total / L) / C * p->batch;
    if (grid <= 0) return cudaSuccess;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const bool head = p->ns_outer == 1;
    return launch_pass(head ? func() : func_tail(), (unsigned)grid, G::THREADS,
                       head ? G::SMEM : kSmemTail, cols_args<float>(p), p, s);
  }
  static Entry entry(const char *name) {
    Entry e{};
    e.desc.name = name;
    e.desc.precision_bits = 32;
    e.desc.kind = MOFFT_KERNEL_COLS;
    e.desc.length = L;
    e.desc.lines = C;
    e.desc.threads = G::THREADS;
    e.desc.radix_count = (int)sizeof...(Rs);
    for (int i = 0; i < 8; ++i)
      e.desc.radices[i] = i < (int)sizeof...(Rs) ? kRadices[i] : 0;
    e.desc.smem_bytes = kSmemTail;
    e.launch = &launch;
    e.func = &func;
    e.func_tail = &func_tail;
    return e;
  }
};

#define TWINC(L, TPL, C, ...) \
  TwinColsInst<L, TPL, C, __VA_ARGS__>::entry("cols_float_" #L "_t" #TPL "_c" #C "_tw")
#define TWIN(L, TPL, TP, SH, ...) \
  TwinInst<L, TPL, TP, SH, __VA_ARGS__>::entry("rows_float_" #L "_t" #TPL "_p" #TP "_tw" #SH)

const Entry *entries_twin_f32(int *count) {
  static const Entry e[] = {
      TWIN(48, 8, 16, 4, 6, 8),
      TWIN(64, 8, 16, 4, 8, 8),
      TWIN(96, 12, 16, 4, 8, 12),
      TWIN(128, 8, 16, 4, 16, 8),
      TWIN(256, 16, 8, 4, 16, 16),
      TWIN(320, 64, 2, 4, 8, 5, 8),
      TWIN(384, 32, 4, 4, 16, 2, 12),
      TWIN(512, 32, 4, 4, 16, 16, 2),
      TWIN(1280, 128, 1, 4, 16, 5, 16),
      TWIN(1536, 128, 1, 4, 16, 6, 16),
      TWINC(512, 32, 16, 16, 16, 2),
      TWINC(384, 32, 16, 16, 12, 2),
      TWINC(320, 32, 16, 16, 10, 2),
  };
  *count = (int)(sizeof(e) / sizeof(e[0]));
  return e;
}
}  // namespace mofft
