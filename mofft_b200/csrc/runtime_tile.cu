// Tile rule of the runtime-chain kernels.
#include "runtime_tile.h"

#include <string.h>

#include "fft_instances.cuh"
#include "runtime_fft.cuh"

namespace mofft {

static const size_t kSmemLimit = 227 * 1024;
static const int kSms = 148;


// Pad pairs behind each block of ns * radix points of an exchange.  First
// exchange: an even radix scatters at an even stride, one pad makes it odd.
// Later ones with runs shorter than a row of pairs: the block pitch becomes
// congruent to the run length.  Longer runs conflict at their ends only.
static int exchange_pad(int ns, int radix, int row) {
  if (ns == 1) return radix % 2 == 0 ? 1 : 0;
  if (ns >= row) return 0;
  const int block = ns * radix;
  return ((ns - block) % row + row) % row;
}

bool rt_shape(int precision_bits, bool cols, int length, const int *chain, int count,
              long long units, long long line_units, RtShape *out) {
  if (count < 1 || count > kRtMaxStages || length < 2 || length > 16384) return false;
  const int row = precision_bits == 32 ? 16 : 8;
  const size_t cb = precision_bits == 32 ? 8 : 16;
  RtShape s;
  memset(&s, 0, sizeof(s));
  int min_radix = 64;
  for (int i = 0; i < count; ++i) {
    if (chain[i] < 2 || chain[i] > 16) return false;
    if (chain[i] > s.max_radix) s.max_radix = chain[i];
    if (chain[i] < min_radix) min_radix = chain[i];
  }
  const int bf = length / min_radix;
  const int cap = rt_max_threads(precision_bits, cols, s.max_radix);
  if (bf > cap) return false;
  if (cols) {
    if (count < 2) return false;
    // adjacent lines per tile: runs of 128 bytes, narrower while the tile
    // exceeds the threads or half an SM's shared memory (runs of 64 bytes
    // still), or while the launch leaves SMs without a CTA
    int c = row;
    // tile rows of c + 1 pairs, and the first stage's table of line powers
    auto bytes = [&](int n) { return ((size_t)length * (n + 1) + (size_t)chain[0] * n) * cb; };
    const size_t half = kSmemLimit / 2;
    while (c > 1 && (c * bf > cap || bytes(c) > kSmemLimit)) c /= 2;
    while (c > row / 2 && (c * bf > 512 || bytes(c) > half)) c /= 2;
    while (c > row / 4 && (line_units + c - 1) / c * (units / line_units) < kSms) c /= 2;
    if (c < 1 || bytes(c) > kSmemLimit) return false;
    s.lines = c;
    s.pitch = c + 1;
    s.smem = bytes(c);
    s.threads = (c * bf + 31) / 32 * 32;
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
  if (bf < 160) {
    const int most = 288 / bf;
    int best = -1;
    for (int n = (most + 1) / 2; n <= most; ++n) {
      const int warps = (n * bf + 31) / 32;
      const int fill = n * bf * 64 / (warps * 32);   // of 64
      if (fill > best || (fill == best && n * bf <= 256)) {
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
  s.threads = (lines * bf + 31) / 32 * 32;
  // runs of the direct loads (L / first radix) and stores (L / last radix)
  // under 64 bytes: copy the lines through the tile instead (FP32 n = 144,
  // runs of 96 bytes: 174 us through the tile, 90 direct)
  const int in_run = length / chain[0], out_run = length / chain[count - 1];
  s.staged = count < 2 || in_run < row / 2 || out_run < row / 2;
  *out = s;
  return true;
}

}  // namespace mofft

extern "C" int mofft_cuda_runtime_tile(int precision_bits, int cols, int length,
                                       const int *chain, int count, long long line_units,
                                       int *lines, int *threads, size_t *smem) {
  mofft::RtShape s;
  const long long many = 1LL << 24;
  if (line_units < 1 || line_units > 0x7fffffffLL) return 0;
  if (!mofft::rt_shape(precision_bits, cols != 0, length, chain, count,
                       cols ? many * line_units : many, line_units, &s))
    return 0;
  *lines = s.lines;
  *threads = s.threads;
  *smem = s.smem;
  return 1;
}
