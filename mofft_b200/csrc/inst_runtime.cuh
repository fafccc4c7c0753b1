// Launch of the runtime-chain kernels, instantiated per precision.
#pragma once
#include <string.h>

#include "fft_instances.cuh"
#include "runtime_fft.cuh"
#include "runtime_tile.h"

namespace mofft {

inline unsigned rt_magic(unsigned d) { return d <= 1 ? 0u : 0xffffffffu / d + 1u; }

template <typename T>
bool rt_pass_shape(const mofft_pass_args *p, RtShape *s) {
  if (p->in_table || p->out_table || p->batch <= 0) return false;
  const long long line_units = p->generic_cols ? p->total / p->length : 1;
  if (line_units < 1 || line_units > 0x7fffffffLL || p->ns_outer > 0x7fffffffLL) return false;
  return rt_shape(sizeof(T) == 4 ? 32 : 64, p->generic_cols != 0, p->length, p->radices,
                  p->radix_count, line_units * p->batch, line_units, s);
}

inline int rt_mode(const mofft_pass_args *p, const RtShape &s) {
  if (!p->generic_cols) return s.staged ? kRtStaged : kRtRows;
  return p->ns_outer == 1 ? kRtColsHead : kRtColsTail;
}

// Smallest register class that holds the chain's largest radix, or the
// several-butterfly kernels.
template <typename T, int MODE>
const void *rt_func(int max_radix, bool multi) {
  if constexpr (MODE != kRtStaged)   // one stage: one butterfly per thread
    if (multi) return reinterpret_cast<const void *>(&rt_kernel<T, MODE, 16, true>);
  if (max_radix <= 8) return reinterpret_cast<const void *>(&rt_kernel<T, MODE, 8, false>);
  if (max_radix <= 11) return reinterpret_cast<const void *>(&rt_kernel<T, MODE, 11, false>);
  return reinterpret_cast<const void *>(&rt_kernel<T, MODE, 16, false>);
}

template <typename T>
const void *rt_func(int mode, int max_radix, bool multi) {
  switch (mode) {
    case kRtRows: return rt_func<T, kRtRows>(max_radix, multi);
    case kRtStaged: return rt_func<T, kRtStaged>(max_radix, multi);
    case kRtColsHead: return rt_func<T, kRtColsHead>(max_radix, multi);
    default: return rt_func<T, kRtColsTail>(max_radix, multi);
  }
}

// cudaErrorNotSupported: the chain does not fit these kernels.
template <typename T>
cudaError_t rt_launch(const mofft_pass_args *p, cudaStream_t stream) {
  RtShape s;
  if (!rt_pass_shape<T>(p, &s)) return cudaErrorNotSupported;
  const bool cols = p->generic_cols != 0;
  RtArgs<T> a;
  memset(&a, 0, sizeof(a));
  a.in = static_cast<const cplx_t<T> *>(p->in);
  a.out = static_cast<cplx_t<T> *>(p->out);
  a.tw = static_cast<const cplx_t<T> *>(p->tw);
  a.tw_hi = static_cast<const cplx_t<T> *>(p->tw_hi);
  a.tw_lo = static_cast<const cplx_t<T> *>(p->tw_lo);
  a.batch = p->batch;
  a.in_dist = p->in_dist;
  a.out_dist = p->out_dist;
  a.ns_outer = cols ? p->ns_outer : 1;
  a.total_lines = cols ? (int)(p->total / p->length) : 1;
  a.split_shift = p->split_shift;
  a.length = p->length;
  a.lines = s.lines;
  while (cols && (1 << a.line_shift) < s.lines) ++a.line_shift;
  a.pitch = s.pitch;
  a.stage_count = p->radix_count;
  a.magic_len = rt_magic((unsigned)p->length);
  a.sign_in = p->conj_in ? T(-1) : T(1);
  a.sign_out = p->conj_out ? T(-1) : T(1);
  int ns = 1, twoff = 0, pad_in = 0;
  for (int i = 0; i < p->radix_count; ++i) {
    RtStage &st = a.st[i];
    const int R = p->radices[i];
    st.radix = R;
    st.ns = ns;
    st.bf = p->length / R;
    st.twoff = twoff;
    st.magic_bf = rt_magic((unsigned)st.bf);
    st.magic_ns = rt_magic((unsigned)ns);
    st.gpad = pad_in;
    st.gstep = st.bf + (st.bf / ns) * pad_in;
    st.sblk = ns * R + s.pad[i];
    pad_in = s.pad[i];
    twoff += stage_table_size(R, ns);
    ns *= R;
  }
  if (ns != p->length) return cudaErrorInvalidValue;
  const long long grid = cols ? ((long long)a.total_lines + s.lines - 1) / s.lines * p->batch
                              : (p->batch + s.lines - 1) / s.lines;
  if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  const void *func = rt_func<T>(rt_mode(p, s), s.max_radix, s.multi != 0);
  return launch_pass(func, (unsigned)grid, s.threads, s.smem, a, p, stream);
}

template <typename T>
cudaError_t rt_opt_in(int mode, int max_radix, bool multi) {
  return cudaFuncSetAttribute(rt_func<T>(mode, max_radix, multi),
                              cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}

// The kernels that a pass of this shape launches: both forms, since the tile
// depends on the launch's batch too (whether a tile fits does not).
template <typename T>
cudaError_t rt_prepare(const mofft_pass_args *p) {
  RtShape s;
  if (!rt_pass_shape<T>(p, &s)) return cudaErrorNotSupported;
  const int mode = rt_mode(p, s);
  const cudaError_t err = rt_opt_in<T>(mode, s.max_radix, false);
  return err != cudaSuccess || s.staged ? err : rt_opt_in<T>(mode, s.max_radix, true);
}

template <typename T>
cudaError_t rt_prepare_columns() {
  for (int mode : {kRtColsHead, kRtColsTail})
    for (int radix : {8, 11, 16})
      for (bool multi : {false, true}) {
        const cudaError_t err = rt_opt_in<T>(mode, radix, multi);
        if (err != cudaSuccess) return err;
      }
  return cudaSuccess;
}

}  // namespace mofft
