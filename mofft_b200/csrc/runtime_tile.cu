// Tile rule of the runtime-chain kernels.
#include "runtime_tile.h"

#include <string.h>

#include "fft_instances.cuh"
#include "runtime_fft.cuh"

namespace mofft {

static const size_t kSmemLimit = 227 * 1024;
static const int kSms = 148;   // of the B200, the only target

// Pad pairs behind each block of ns * radix points of an exchange.  First
// exchange: an even radix scatters at an even stride, one pad makes it odd.
// Later ones: the block pitch becomes congruent to the run length, so that the
// runs a row of lanes spans follow each other; long runs rarely meet.
static int exchange_pad(int ns, int radix, int row) {
  if (ns == 1) return radix % 2 == 0 ? 1 : 0;
  if (ns >= 4 * row) return 0;
  const int block = ns * radix;
  return ((ns - block) % row + row) % row;
}

// The tile of one kernel form (multi: several butterflies per thread).
static bool rt_form(int precision_bits, bool cols, bool multi, int length, const int *chain,
                    int count, long long units, long long line_units, RtShape *out) {
  const int row = precision_bits == 32 ? 16 : 8;
  const size_t cb = precision_bits == 32 ? 8 : 16;
  RtShape s;
  memset(&s, 0, sizeof(s));
  s.multi = multi;
  for (int i = 0; i < count; ++i)
    if (chain[i] > s.max_radix) s.max_radix = chain[i];
  // threads of a tile of n lines: every stage's butterflies in rt_per() rounds
  auto threads = [&](int n) {
    int most = 0;
    for (int i = 0; i < count; ++i) {
      const int per = multi ? rt_per(chain[i]) : 1;
      const int t = (n * (length / chain[i]) + per - 1) / per;
      if (t > most) most = t;
    }
    return most;
  };
  const int cap = rt_max_threads(precision_bits, cols, s.max_radix, multi);
  if (threads(1) > cap) return false;
  if (cols) {
    if (count < 2) return false;
    // adjacent lines per tile: runs of 128 bytes, narrower while the tile
    // exceeds the threads or half an SM's shared memory (runs of 64 bytes
    // still), or while the launch leaves SMs without a CTA
    int c = row;
    // tile rows of c + 1 pairs, and the first stage's table of line powers
    auto bytes = [&](int n) { return ((size_t)length * (n + 1) + (size_t)chain[0] * n) * cb; };
    const size_t half = kSmemLimit / 2;
    while (c > 1 && (threads(c) > cap || bytes(c) > kSmemLimit)) c /= 2;
    while (c > row / 2 && (threads(c) > 512 || bytes(c) > half)) c /= 2;
    while (c > row / 4 && (line_units + c - 1) / c * (units / line_units) < kSms) c /= 2;
    if (bytes(c) > kSmemLimit) return false;
    s.lines = c;
    s.pitch = c + 1;
    s.smem = bytes(c);
    s.threads = (threads(c) + 31) / 32 * 32;
    *out = s;
    return true;
  }
  int need = length, ns = 1;
  for (int i = 0; i + 1 < count; ++i) {
    s.pad[i] = exchange_pad(ns, chain[i], row);
    ns *= chain[i];
    const int words = length + (length / ns) * s.pad[i];
    if (words > need) need = words;
  }
  // lines per tile: about 256 threads, the count that fills whole warps best
  int lines = 1;
  if (threads(1) < 160) {
    const int most = 288 / threads(1);
    int best = -1;
    for (int n = (most + 1) / 2; n <= most; ++n) {
      const int t = threads(n), warps = (t + 31) / 32;
      const int fill = t * 64 / (warps * 32);   // of 64
      if (fill > best || (fill == best && t <= 256)) {
        best = fill;
        lines = n;
      }
    }
  }
  while (lines > 1 && (units + lines - 1) / lines < kSms) lines = (lines + 1) / 2;
  s.pitch = need;
  if (lines > 1) {
    const int want = (length / chain[0]) % row;
    while (s.pitch % row != want) ++s.pitch;
  }
  while (lines > 1 && (size_t)lines * s.pitch * cb > kSmemLimit / 2) --lines;
  s.lines = lines;
  s.smem = (size_t)lines * s.pitch * cb;
  if (s.smem > kSmemLimit) return false;
  s.threads = (threads(lines) + 31) / 32 * 32;
  // one stage: its only butterfly reads and writes whole short lines, so the
  // lines are copied through the tile.  More stages run direct however short
  // their runs (FP32 50 = 10 5 170 us through the tile, 111 direct; 25 157 and
  // 118; 144 174 and 90; FP64 26 = 13 2 298 and 120)
  s.staged = count < 2;
  *out = s;
  return true;
}

// Which form runs a chain.  One butterfly per thread wins while the stages
// need about the same threads (FP32 1000 = 10^3 120 against 131 us of 2^25
// points, 343 = 7^3 117 against 129, FP64 81 100 against 157); several win
// where the smallest radix asks for twice the threads of the largest, which
// then idle (FP32 4000 = 10 10 8 5 271 -> 186 us, 500 = 10 10 5 156 -> 120;
// FP64 2500 = 10 10 5 5 236 -> 158) or small radices for most of a CTA's
// (FP32 3125 = 5^5 236 -> 206; column passes of 625 points 656 -> 511).
static bool several_butterflies(int precision_bits, bool cols, int length, const int *chain,
                                int count, const RtShape &one) {
  int least = 64;
  for (int i = 0; i < count; ++i)
    if (chain[i] < least) least = chain[i];
  if (cols) return one.threads > 640;
  if (one.staged) return false;
  // short FP32 lines of unequal radices up to 8: a butterfly is too little work for a
  // thread of its own (20 = 5 4 195 -> 114, 28 = 7 4 209 -> 109)
  if (precision_bits == 32 && length < 64 && least <= 5 && one.max_radix > least &&
      one.max_radix <= 8)
    return true;
  return one.max_radix >= 2 * least || (least <= 5 && one.threads > 512);
}

bool rt_shape(int precision_bits, bool cols, int length, const int *chain, int count,
              long long units, long long line_units, RtShape *out) {
  if (count < 1 || count > kRtMaxStages || length < 2 || length > 16384) return false;
  for (int i = 0; i < count; ++i)
    if (chain[i] < 2 || chain[i] > 16) return false;
  RtShape several;
  const bool one = rt_form(precision_bits, cols, false, length, chain, count, units, line_units,
                           out);
  if (one && !several_butterflies(precision_bits, cols, length, chain, count, *out)) return true;
  if (!rt_form(precision_bits, cols, true, length, chain, count, units, line_units, &several))
    return one;
  *out = several;
  return true;
}

}  // namespace mofft

extern "C" int mofft_cuda_runtime_tile(int precision_bits, int cols, int length,
                                       const int *chain, int count, long long line_units,
                                       int *lines, int *threads, size_t *smem, int *ctas) {
  mofft::RtShape s;
  const long long many = 1LL << 24;
  if (line_units < 1 || line_units > 0x7fffffffLL) return 0;
  if (!mofft::rt_shape(precision_bits, cols != 0, length, chain, count,
                       cols ? many * line_units : many, line_units, &s))
    return 0;
  *lines = s.lines;
  *threads = s.threads;
  *smem = s.smem;
  const int regs = mofft::rt_registers(precision_bits, cols != 0, s.max_radix, s.multi != 0);
  int resident = 65536 / (regs * s.threads);
  if ((size_t)resident * (s.smem + 1024) > 228 * 1024)
    resident = (int)(228 * 1024 / (s.smem + 1024));
  if (resident * s.threads > 2048) resident = 2048 / s.threads;
  *ctas = resident < 1 ? 1 : resident;
  return 1;
}
