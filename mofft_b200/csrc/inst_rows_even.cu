// Single-pass kernels whose threads run the same number of butterflies in
// every stage, all on global memory directly.
//
// The 3*2^k and 5*2^k instances of inst_rows_mixed.cu start with the odd radix
// on L/16 threads, so a thread holds up to 24 points in that stage (its
// butterflies do not divide evenly) and as many registers.  Here the odd factor
// sits inside a radix of 10 or 12 (or a radix of its own with two to four
// butterflies a thread) behind a radix-16 or radix-8 stage: at most 16 points
// and 32 to 48 registers a thread in FP32 (64 to 70 before), up to 108 in FP64.
// A power of two first also makes the pad every 16 pairs free of bank conflicts
// (a bank simulation: 1.0-1.2 wavefronts per access against 1.35-1.9).  Lengths
// below 400 used to copy their lines through shared memory on both sides;
// reading and writing runs of L / radix points directly takes less, down to
// runs of 48 bytes.
//
// us per 2^25 FP32 / 2^24 FP64 points (copy floor 82), before -> now: FP32 64
// 93 -> 85, 80 122 -> 99, 160 130 -> 86, 192 115 -> 83, 320 133 -> 107, 384
// 134 -> 96, 640 103 -> 91, 1280 105 -> 95, 3072 101 -> 90; FP64 48 105 -> 81,
// 64 96 -> 82, 128 93 -> 81, 192 107 -> 84, 320 132 -> 90, 384 120 -> 87, 640
// 100 -> 89, 1280 119 -> 93, 2048 99 -> 88, 6144 168 -> 156.
// Tuned FP32 plans of 64, 320, 384, 1280 and 1536 points have moved on to the
// two-line kernels of twin_fft.cuh (80, 90, 85, 88 and 83 us).  FP64 128 looks
// its radix-16 twiddles up (ROWSTP), as the kernel that it replaced did: derived
// from four of them its rel-L2 error was 5 % larger (1.62e-16 -> 1.70e-16) for
// 80.6 instead of 81.7 us.
#include "fft_instances.cuh"

namespace mofft {
const Entry *entries_rows_even(int *count) {
  static const Entry e[] = {
      ROWSDP(float, 3072, 256, 1, 16, 12, 16),
      ROWSDP(float, 2560, 256, 1, 16, 10, 16),
      ROWSDP(float, 1536, 128, 2, 16, 6, 16),
      ROWSDP(float, 1280, 128, 2, 16, 5, 16),
      ROWSDP(float, 640, 64, 4, 16, 5, 8),
      ROWSDP(float, 384, 64, 4, 8, 6, 8),
      ROWSDP(float, 320, 64, 4, 8, 5, 8),
      ROWSDP(float, 192, 16, 16, 16, 12),
      ROWSDP(float, 160, 16, 16, 16, 10),
      ROWSDP(float, 128, 8, 32, 16, 8),
      ROWSDP(float, 96, 12, 16, 8, 12),
      ROWSDP(float, 80, 10, 16, 8, 10),
      ROWSDP(float, 64, 8, 32, 8, 8),
      ROWSDP(float, 48, 8, 32, 6, 8),
      ROWSDP(double, 6144, 768, 1, 8, 8, 8, 12),
      ROWSDP(double, 3072, 256, 1, 16, 12, 16),
      ROWSDP(double, 2048, 128, 1, 16, 16, 8),
      ROWSDP(double, 1280, 160, 1, 16, 10, 8),
      ROWSDP(double, 384, 64, 2, 8, 6, 8),
      ROWSDP(double, 320, 64, 2, 8, 5, 8),
      ROWSDP(double, 192, 16, 8, 16, 12),
      ROWSDP(double, 160, 16, 8, 16, 10),
      ROWSTP(double, 128, 16, 8, 8, 16),
      ROWSDP(double, 96, 12, 16, 8, 12),
      ROWSDP(double, 80, 10, 16, 8, 10),
      ROWSDP(double, 64, 8, 16, 8, 8),
      ROWSDP(double, 48, 8, 16, 6, 8),
      ROWSDP(double, 32, 4, 32, 8, 4),
      ROWSDP(double, 640, 80, 2, 8, 8, 10),
      ROWSDP(float, 768, 64, 2, 16, 12, 4),
  };
  *count = (int)(sizeof(e) / sizeof(e[0]));
  return e;
}
}  // namespace mofft
