// Runtime-chain kernels: one CTA tile of a line DFT whose radix chain is a
// launch argument, for the 13-smooth lengths without a compiled instance.
//
// A tile is `lines` lines of L points (ROWS: whole transforms; COLS: adjacent
// super-butterflies of a multi-pass transform).  A thread runs one butterfly
// per stage, or in the several-butterfly form as many as hold 16 points (eight
// of radix 2): it gathers R values each into registers, multiplies the stage
// twiddles, runs the straight-line radix-R codelet and, once every thread of
// the CTA has read, scatters into the same shared-memory tile.  So a tile needs
// one copy of its points (the ping-pong form this replaces kept four component
// arrays), and every value crosses shared memory as one {re, im} pair.
//
// Addresses.  With Ns the product of the radices applied so far, stage
// (R, Ns) scatters butterfly j to (j / Ns) Ns R + (j mod Ns) + k Ns and the
// next stage gathers j' + r L/R'.  The exchange between them inserts `pad`
// pairs behind each block of Ns R points.  Both sides stay linear in k and r
// (a block never divides L/R' unevenly), so an access costs one add, and the
// divisions by Ns and by the butterflies per line are multiplications by a
// precomputed reciprocal.  The pad makes the block pitch congruent to Ns
// modulo one 128-byte row of pairs, which spreads consecutive butterflies
// over distinct banks for every radix (without it the first stage's stride R
// conflicts gcd(R, 16) ways).
//
// Tile shape.  The chain decides the threads (the most butterflies of any
// stage), the register class its largest radix: variants for radices up to
// 8, 11 and 16 keep short codelets at the occupancy they can have.
//
// Bound by: issue slots and latency (0.71 instructions per scheduler and cycle
// at n = 343 before the stages were peeled), HBM for the short lengths that
// run direct.  Measured per 2^25 FP32 / 2^24 FP64 points (HBM floor 82 us),
// this against the ping-pong kernel: FP32 n = 100 801 -> 98 us, 343 1397 ->
// 117, 1000 1005 -> 122, 3375 976 -> 133, 10000 1441 -> 218, 50625 (two
// passes) 1849 -> 292; FP64 100 476 -> 86, 3375 672 -> 136, 50625 1233 -> 237.
// Every stage twiddle is looked up.  Deriving most of them as products of two
// others (6 loads instead of 15 at radix 16) took 0.4 % less time over 72
// lengths, 2 to 4 % less at these, but added 2 to 5 % to the rel-L2 error: FP32
// 343 1.062e-7 -> 1.092e-7, 3375 1.314e-7 -> 1.360e-7, FP64 343 1.937e-16 ->
// 1.977e-16.
#pragma once

#include "fft_device.cuh"
#include "runtime_tile.h"

namespace mofft {

constexpr int kRtMaxStages = 16;

struct RtStage {
  int radix;
  int ns;               // product of the earlier radices
  int bf;               // butterflies per line, L / radix
  int twoff;            // stage table offset in the pass's twiddle table
  unsigned magic_bf;    // ceil(2^32 / bf), 0 for bf == 1
  unsigned magic_ns;    // ceil(2^32 / ns), 0 for ns == 1
  int gpad;             // gather: pad pairs per block of ns points
  int gstep;            // gather: words between a butterfly's inputs
  int sblk;             // scatter: words between blocks of ns * radix points
};

template <typename T>
struct RtArgs {
  const cplx_t<T>* in;
  cplx_t<T>* out;
  const cplx_t<T>* tw;
  const cplx_t<T>* tw_hi;
  const cplx_t<T>* tw_lo;
  long long batch;
  long long in_dist;
  long long out_dist;
  long long ns_outer;       // COLS: product of the earlier passes' lengths
  int total_lines;          // COLS: lines of one transform, M / L
  int split_shift;
  int length;               // L
  int lines;                // lines of a full tile (COLS: a power of two)
  int line_shift;           // COLS: log2 lines
  int pitch;                // ROWS: pairs per line; COLS: pairs per element row
  int stage_count;
  unsigned magic_len;       // ceil(2^32 / L)
  T sign_in;
  T sign_out;
  RtStage st[kRtMaxStages];
};

// n / d for n d < 2^32 with m = ceil(2^32 / d); m == 0 stands for d == 1.
__device__ __forceinline__ int rt_div(int n, unsigned m) {
  return m ? (int)__umulhi((unsigned)n, m) : n;
}

// Stage twiddles v[r] *= w^r, every power from the table.
template <typename T, int R>
__device__ __forceinline__ void rt_twiddle(T (&vr)[R], T (&vi)[R],
                                           const cplx_t<T>* __restrict__ tw, int ns) {
#pragma unroll
  for (int r = 1; r < R; ++r) {
    const cplx_t<T> w = __ldg(tw + (r - 1) * ns);
    cmul<T>(vr[r], vi[r], w.x, w.y);
  }
}

// Kernel forms.  Stages are peeled (first / middle / last) so that each body
// computes only the addresses it uses.
enum RtMode {
  kRtRows = 0,      // whole transforms, first and last stage on global memory
  kRtStaged = 1,    // whole transforms of one stage, copied through the tile
  kRtColsHead = 2,  // first pass of a multi-pass transform (Ns = 1)
  kRtColsTail = 3   // later pass: super-stage twiddles, strided stores
};

// Where a butterfly of a stage lies.
template <typename T>
struct RtIo {
  bool act;
  int src, sstep, dst, dstep;     // tile addresses, in pairs
  const cplx_t<T>* gsrc;          // first stage on global memory
  cplx_t<T>* gdst;                // last stage on global memory
  long long gsstep, gdstep;
  const cplx_t<T>* tw;            // this butterfly's stage twiddles
  int j, line;
};

// A CTA's tile: which lines, and the place of each butterfly.
template <typename T, int MODE>
struct RtTile {
  static constexpr bool COLS = MODE >= kRtColsHead;
  const RtArgs<T>& a;
  const cplx_t<T>* in;
  long long b;                    // ROWS: first transform; COLS: the transform
  int j0, nl;                     // COLS: first line; lines inside the batch

  // butterfly w of stage s; only the fields the stage uses are computed
  template <bool FIRST, bool LAST>
  __device__ __forceinline__ RtIo<T> at(const RtStage& s, int w) const {
    RtIo<T> io;
    if (COLS) {
      io.line = w & (a.lines - 1);
      io.j = w >> a.line_shift;
      io.act = io.j < s.bf && io.line < nl;
    } else {
      io.line = rt_div(w, s.magic_bf);
      io.j = w - io.line * s.bf;
      io.act = io.line < nl;
    }
    const int j = io.j;
    const int step = COLS ? a.pitch : 1;   // pairs between a line's points
    const int base = COLS ? io.line : io.line * a.pitch;
    // first stage: Ns = 1 and the input is not padded; last: Ns R = L
    const int jq = FIRST ? j : LAST ? 0 : rt_div(j, s.magic_ns);
    const int jm = FIRST ? 0 : LAST ? j : j - jq * s.ns;
    io.src = base + (FIRST ? j : j + jq * s.gpad) * step;
    io.sstep = (FIRST ? s.bf : s.gstep) * step;
    io.dst = base + (jq * s.sblk + jm) * step;
    io.dstep = (FIRST ? 1 : s.ns) * step;
    io.tw = a.tw + s.twoff + jm;
    if (COLS) {
      const unsigned ns = (unsigned)a.ns_outer, jl = (unsigned)(j0 + io.line);
      const unsigned q = MODE == kRtColsTail ? jl / ns : 0u;
      io.gsrc = in + b * a.in_dist + jl + (long long)j * a.total_lines;
      io.gsstep = (long long)a.total_lines * s.bf;
      io.gdst = a.out + b * a.out_dist + (long long)q * ns * a.length + (jl - q * ns) +
                j * a.ns_outer;
      io.gdstep = a.ns_outer * s.ns;
    } else {
      io.gsrc = in + (b + io.line) * a.in_dist + j;
      io.gsstep = s.bf;
      io.gdst = a.out + (b + io.line) * a.out_dist + j;
      io.gdstep = s.ns;
    }
    return io;
  }
};

// Super-stage twiddle of a later column pass: v[r] *= b u^r with b =
// W^{jmod j} looked up by each thread and the powers u^r of the tile's lines
// in a table behind the tile (ColsLayout's scheme; here a line's jmod may wrap
// inside a tile).
template <typename T, int R>
__device__ __forceinline__ void rt_super_fill(const RtTile<T, kRtColsTail>& tile, int bf,
                                              cplx_t<T>* table) {
  const RtArgs<T>& a = tile.a;
  ColsLayout<T, 1, 1, true> lay;
  lay.tw_hi = a.tw_hi;
  lay.tw_lo = a.tw_lo;
  lay.split_shift = a.split_shift;
  for (int q = threadIdx.x; q < R << a.line_shift; q += blockDim.x) {
    lay.jmod = (unsigned)(tile.j0 + (q & (a.lines - 1))) % (unsigned)a.ns_outer;
    T wr, wi;
    lay.super_w((unsigned)((q >> a.line_shift) * bf), wr, wi);
    st_global<T>(table + q, wr, wi);
  }
}
template <typename T, int R>
__device__ __forceinline__ void rt_super_apply(const RtTile<T, kRtColsTail>& tile,
                                               const RtIo<T>& io, const cplx_t<T>* table,
                                               T (&vr)[R], T (&vi)[R]) {
  const RtArgs<T>& a = tile.a;
  ColsLayout<T, 1, 1, true> lay;
  lay.tw_hi = a.tw_hi;
  lay.tw_lo = a.tw_lo;
  lay.split_shift = a.split_shift;
  lay.jmod = (unsigned)(tile.j0 + io.line) % (unsigned)a.ns_outer;
  T br, bi;
  lay.super_w((unsigned)io.j, br, bi);
  cmul<T>(vr[0], vi[0], br, bi);
#pragma unroll
  for (int r = 1; r < R; ++r) {
    const cplx_t<T> u = table[(r << a.line_shift) + io.line];
    T xr = u.x, xi = u.y;
    cmul<T>(xr, xi, br, bi);
    cmul<T>(vr[r], vi[r], xr, xi);
  }
}

// One stage: PER butterflies per thread (w = thread + m * threads).
template <typename T, int MODE, int R, int PER, bool FIRST, bool LAST>
__device__ __forceinline__ void rt_stage(const RtTile<T, MODE>& tile, const RtStage& s,
                                         cplx_t<T>* sp) {
  constexpr Where SRC = FIRST && MODE != kRtStaged ? kGlobal : kShared;
  constexpr Where DST = LAST && (MODE == kRtRows || MODE == kRtColsTail) ? kGlobal : kShared;
  constexpr bool SUPER = FIRST && MODE == kRtColsTail;
  const RtArgs<T>& a = tile.a;
  T vr[PER][R], vi[PER][R];
#pragma unroll
  for (int m = 0; m < PER; ++m) {
    const RtIo<T> io = tile.template at<FIRST, LAST>(s, threadIdx.x + m * blockDim.x);
    if (io.act) {
      if constexpr (SRC == kGlobal) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const cplx_t<T> v = ld_global<T>(io.gsrc + r * io.gsstep);
          vr[m][r] = v.x;
          vi[m][r] = v.y * a.sign_in;
        }
      } else {
        const cplx_t<T>* p = sp + io.src;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const cplx_t<T> v = p[r * io.sstep];
          vr[m][r] = v.x;
          vi[m][r] = v.y;
        }
      }
      if constexpr (!SUPER) {
        if constexpr (!FIRST) rt_twiddle<T, R>(vr[m], vi[m], io.tw, s.ns);
        Dft<R>::fwd(vr[m], vi[m]);
      }
    } else {
      // defined on every path: a register that is only written under `act` and
      // read under it behind the barrier counts as live around the stage loop,
      // for every radix at once (the radix-8 class spilled 350 bytes a thread)
#pragma unroll
      for (int r = 0; r < R; ++r) vr[m][r] = vi[m][r] = T(0);
    }
  }
  if constexpr (SUPER) {
    cplx_t<T>* table = sp + a.length * a.pitch;
    rt_super_fill<T, R>(tile, s.bf, table);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const RtIo<T> io = tile.template at<FIRST, LAST>(s, threadIdx.x + m * blockDim.x);
      if (io.act) {
        rt_super_apply<T, R>(tile, io, table, vr[m], vi[m]);
        Dft<R>::fwd(vr[m], vi[m]);
      }
    }
  }
  if constexpr (SRC == kShared && DST == kShared) __syncthreads();
#pragma unroll
  for (int m = 0; m < PER; ++m) {
    const RtIo<T> io = tile.template at<FIRST, LAST>(s, threadIdx.x + m * blockDim.x);
    if (io.act) {
      if constexpr (DST == kGlobal) {
#pragma unroll
        for (int k = 0; k < R; ++k)
          st_global<T>(io.gdst + k * io.gdstep, vr[m][k], vi[m][k] * a.sign_out);
      } else {
        cplx_t<T>* p = sp + io.dst;
#pragma unroll
        for (int k = 0; k < R; ++k) st_global<T>(p + k * io.dstep, vr[m][k], vi[m][k]);
      }
    }
  }
  if constexpr (DST == kShared) __syncthreads();
}

// Butterflies a thread may run in a radix-R stage of the several-butterfly
// kernels (MULTI): as many as hold 16 points.
__host__ __device__ constexpr int rt_per(int radix) { return radix > 8 ? 1 : 16 / radix; }

template <typename T, int MODE, int MAXR, bool MULTI, bool FIRST, bool LAST>
__device__ __forceinline__ void rt_dispatch(const RtTile<T, MODE>& tile, const RtStage& s,
                                            cplx_t<T>* sp) {
#define MOFFT_RT_CASE(RR)                                                            \
  case RR:                                                                           \
    if constexpr (RR <= MAXR)                                                        \
      rt_stage<T, MODE, RR, MULTI ? rt_per(RR) : 1, FIRST, LAST>(tile, s, sp);       \
    break;
  switch (s.radix) {
    MOFFT_RT_CASE(2) MOFFT_RT_CASE(3) MOFFT_RT_CASE(4) MOFFT_RT_CASE(5)
    MOFFT_RT_CASE(6) MOFFT_RT_CASE(7) MOFFT_RT_CASE(8) MOFFT_RT_CASE(9)
    MOFFT_RT_CASE(10) MOFFT_RT_CASE(11) MOFFT_RT_CASE(12) MOFFT_RT_CASE(13)
    MOFFT_RT_CASE(14) MOFFT_RT_CASE(15) MOFFT_RT_CASE(16)
    default: break;
  }
#undef MOFFT_RT_CASE
}

// Registers are capped at the figures the planner's occupancy rests on
// (rt_registers), which every form meets without spills; uncapped, looking up all
// twiddles takes 56 to 64 where 48 and 56 do (FP32 1764 139 against 126 us of
// 2^25 points).
template <typename T, int MODE, int MAXR, bool MULTI>
__global__ void __maxnreg__((rt_registers(sizeof(T) == 4 ? 32 : 64, MODE >= kRtColsHead, MAXR,
                                          MULTI)))
rt_kernel(const __grid_constant__ RtArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx_t<T>* sp = reinterpret_cast<cplx_t<T>*>(smem_raw);
  constexpr bool COLS = MODE >= kRtColsHead;
  RtTile<T, MODE> tile{a, after_previous(a.in), 0, 0, 0};
  const int tid = threadIdx.x;
  const int L = a.length;
  const int last = a.stage_count - 1;
  if (COLS) {
    const unsigned groups = (unsigned)(a.total_lines + a.lines - 1) >> a.line_shift;
    const unsigned q = blockIdx.x / groups;
    tile.b = q;
    tile.j0 = (int)((blockIdx.x - q * groups) << a.line_shift);
    tile.nl = min(a.total_lines - tile.j0, a.lines);
  } else {
    tile.b = (long long)blockIdx.x * a.lines;
    tile.nl = (int)(a.batch - tile.b < a.lines ? a.batch - tile.b : a.lines);
  }
  const long long b = tile.b;
  const int points = tile.nl * L;
  if constexpr (MODE == kRtStaged) {
    // the tile's lines as they lie in global memory, kBatch loads in flight
    constexpr int kBatch = sizeof(T) == 4 ? 8 : 4;
    const cplx_t<T>* src = tile.in + b * a.in_dist;
    for (int q0 = tid; q0 < points; q0 += kBatch * blockDim.x) {
      cplx_t<T> v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const int q = q0 + k * (int)blockDim.x;
        const int ln = (int)__umulhi((unsigned)q, a.magic_len);
        if (q < points) v[k] = ld_global<T>(src + ln * a.in_dist + (q - ln * L));
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const int q = q0 + k * (int)blockDim.x;
        const int ln = (int)__umulhi((unsigned)q, a.magic_len);
        if (q < points) {
          v[k].y *= a.sign_in;
          sp[ln * a.pitch + (q - ln * L)] = v[k];
        }
      }
    }
    __syncthreads();
  }
  constexpr bool kStores = MODE == kRtRows || MODE == kRtColsTail;
  rt_dispatch<T, MODE, MAXR, MULTI, true, false>(tile, a.st[0], sp);
  const int middles = kStores ? last : last + 1;
  for (int i = 1; i < middles; ++i)
    rt_dispatch<T, MODE, MAXR, MULTI, false, false>(tile, a.st[i], sp);
  if constexpr (kStores) {
    rt_dispatch<T, MODE, MAXR, MULTI, false, true>(tile, a.st[last], sp);
  } else {
    // kRtColsHead: lines j0 .. j0+nl-1 are one contiguous block of the
    // output; kRtStaged: the tile's lines leave as they arrived
    cplx_t<T>* dst = a.out + b * a.out_dist + (COLS ? (long long)tile.j0 * L : 0);
    for (int q = tid; q < points; q += blockDim.x) {
      const int ln = (int)__umulhi((unsigned)q, a.magic_len);
      const int i = q - ln * L;
      const cplx_t<T> v = COLS ? sp[i * a.pitch + ln] : sp[ln * a.pitch + i];
      st_global<T>(COLS ? dst + q : dst + ln * a.out_dist + i, v.x, v.y * a.sign_out);
    }
  }
}

}  // namespace mofft
