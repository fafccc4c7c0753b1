// Tile shapes of the runtime-chain kernels (runtime_fft.cuh): one rule, used
// by the planner (feasibility, reported lines and shared memory) and by the
// launch (which also knows the batch).
#pragma once

#include <stddef.h>

namespace mofft {

// Registers per thread of the kernels by register class (the chain's largest
// radix up to 8, 11, 16, or several butterflies): their cap when compiled, and
// the planner's occupancy.
constexpr int rt_registers(int precision_bits, bool cols, int max_radix, bool multi) {
  if (precision_bits == 32) {
    if (multi) return cols ? 80 : 64;
    return max_radix <= 8 ? (cols ? 48 : 40) : max_radix <= 11 ? (cols ? 64 : 48) : cols ? 80 : 56;
  }
  if (multi) return cols ? 128 : 112;
  return max_radix <= 8 ? (cols ? 72 : 64) : max_radix <= 11 ? (cols ? 88 : 80) : cols ? 128 : 104;
}

// Most threads of a CTA: what the register file holds of the class, in steps
// of the tile rule's timings.
constexpr int rt_max_threads(int precision_bits, bool cols, int max_radix, bool multi) {
  if (multi) return precision_bits == 32 ? (cols ? 768 : 1024) : 512;
  if (precision_bits == 32) return max_radix <= 11 || !cols ? 1024 : 768;
  if (max_radix <= 8) return cols ? 640 : 1024;
  if (max_radix <= 11) return cols ? 512 : 768;
  return 512;
}

// A CTA of the most threads fits the register file in every class.
constexpr bool rt_threads_fit() {
  for (int bits = 32; bits <= 64; bits += 32)
    for (int cols = 0; cols < 2; ++cols)
      for (int radix : {8, 11, 16})
        for (int multi = 0; multi < 2; ++multi)
          if (rt_registers(bits, cols != 0, radix, multi != 0) *
                  rt_max_threads(bits, cols != 0, radix, multi != 0) > 65536)
            return false;
  return true;
}
static_assert(rt_threads_fit(), "launch would exceed the register file");

struct RtShape {
  int lines;       // lines per CTA
  int threads;     // CTA threads: the most butterflies of any stage, whole warps
  int max_radix;   // largest radix of the chain
  int multi;       // several butterflies per thread (rt_per)
  int pitch;       // pairs per line (ROWS) / per element row (COLS)
  int staged;      // ROWS: global I/O goes through the tile
  int pad[16];     // pad pairs behind each block of the exchange after stage i
  size_t smem;
};

// Shape of the tile of `length` points with stage list `chain` (first stage
// first).  `units`: transforms of the launch (ROWS) or super-butterflies over
// all of them (COLS); `line_units`: super-butterflies of one transform (COLS).
// False when the chain does not fit the kernels.
bool rt_shape(int precision_bits, bool cols, int length, const int *chain, int count,
              long long units, long long line_units, RtShape *out);

}  // namespace mofft
