// Twin one-pass kernels: every thread transforms two lines at once with packed
// FP32 arithmetic.
//
// The one-pass FP32 kernels issue 65 instructions a point (n = 4096, 71 % of
// the issue slots at full clock) and become issue-bound when the clock falls
// under load.  sm_100 executes add, sub, mul and fma on pairs of FP32 values
// (.f32x2) in one instruction.  Two transforms b, b+1 need the same operations
// on the same butterfly, so a thread keeps the real parts of both in one
// register pair and the imaginary parts in another: the codelets, twiddle
// products and exchanges, and all index arithmetic, are issued once for two
// lines.  A value pair crosses shared memory as one 16-byte access
// {reA, reB, imA, imB}, the layout of the FP64 pair tiles.
//
// Measured against the one-line instances (us, 2^26 points / 2^21 points in
// L2): 48 198 -> 187 / 7.3 -> 7.0, 64 163 -> 155 / 5.8 -> 5.5, 96 186 -> 177 / 7.4
// -> 7.9, 128 177 -> 161 / 6.0 -> 5.6, 256 158 -> 157 / 6.2 -> 5.7, 320 208 -> 176 /
// 7.9 -> 7.0, 384 184 -> 164 / 7.1 -> 6.7, 512 169 -> 156 / 7.4 -> 6.9, 1280 183 ->
// 174 / 7.5 -> 7.3, 1536 172 -> 163 / 7.1 -> 6.7.  Not built where one line
// already takes half an SM's tile or registers: a pair halves the resident CTAs,
// whose barriers then show (4096 170 -> 181, 8192 223 -> 291, 3072 171 -> 189,
// 2560 177 -> 205), nor where it loses in L2 (160, 192, 640, 768, 1024, 2048).
//
// Every stage twiddle is looked up.  Forming powers above w^3 as products took
// 1 % less time (5 % at 48 and 384: 95 -> 91, 85 -> 81 us of 2^25 points) and
// made the rel-L2 errors of 64, 128 and 256 points 5 % larger than the one-line
// kernels' (8.05e-8 -> 8.49e-8, 8.76e-8 -> 9.15e-8, 9.54e-8 -> 9.99e-8).  Looked
// up they are 8.05e-8, 8.75e-8 and 9.52e-8, and 320-1536 points are 7 to 10 %
// below the one-line kernels'.
#pragma once

#include "fft_device.cuh"

namespace mofft {

// Two FP32 values.  `neg` and `cst` are compile-time knowledge (every use is
// inlined and unrolled): a negation only flips `neg`, which the next add or sub
// absorbs, and a constant factor changes its sign for free.
struct TwinProd;
struct Twin {
  unsigned long long v;
  float c;         // value of a constant
  bool neg, cst;
  __device__ __forceinline__ Twin() : v(0), c(0.f), neg(false), cst(false) {}
  __device__ __forceinline__ explicit Twin(unsigned long long raw)
      : v(raw), c(0.f), neg(false), cst(false) {}
  __device__ __forceinline__ explicit Twin(double x)
      : v(0), c((float)x), neg(false), cst(true) {}
  __device__ __forceinline__ explicit Twin(int x)
      : v(0), c((float)x), neg(false), cst(true) {}
  __device__ __forceinline__ Twin(const TwinProd& p);
};

__device__ __forceinline__ unsigned long long twin_pack(float a, float b) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ void twin_unpack(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long twin_add(unsigned long long a,
                                                       unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long twin_sub(unsigned long long a,
                                                       unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long twin_mul(unsigned long long a,
                                                       unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long twin_fma(unsigned long long a,
                                                       unsigned long long b,
                                                       unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// The value itself: constants as a pair, a pending negation applied.
__device__ __forceinline__ unsigned long long twin_value(const Twin& a) {
  if (a.cst) return twin_pack(a.neg ? -a.c : a.c, a.neg ? -a.c : a.c);
  if (a.neg) return a.v ^ 0x8000000080000000ull;
  return a.v;
}
// Without its sign (for operations that take the sign elsewhere).
__device__ __forceinline__ unsigned long long twin_plain(const Twin& a) {
  return a.cst ? twin_pack(a.c, a.c) : a.v;
}
__device__ __forceinline__ Twin twin_signed(unsigned long long v, bool neg) {
  Twin r(v);
  r.neg = neg;
  return r;
}

// A product not yet added to anything.
struct TwinProd {
  Twin a, b;
};
__device__ __forceinline__ TwinProd operator*(const Twin& a, const Twin& b) {
  TwinProd p;
  p.a = a;
  p.b = b;
  return p;
}
__device__ __forceinline__ Twin twin_of(const TwinProd& p) {
  return twin_signed(twin_mul(twin_plain(p.a), twin_plain(p.b)), p.a.neg != p.b.neg);
}
__device__ __forceinline__ Twin operator-(const Twin& a) {
  Twin r = a;
  r.neg = !a.neg;
  return r;
}
__device__ __forceinline__ TwinProd operator-(const TwinProd& p) {
  TwinProd r = p;
  r.a.neg = !p.a.neg;
  return r;
}
__device__ __forceinline__ Twin operator+(const Twin& a) { return a; }
__device__ __forceinline__ Twin operator+(const Twin& a, const Twin& b) {
  if (a.neg == b.neg) return twin_signed(twin_add(twin_plain(a), twin_plain(b)), a.neg);
  if (b.neg) return twin_signed(twin_sub(twin_plain(a), twin_plain(b)), false);
  return twin_signed(twin_sub(twin_plain(b), twin_plain(a)), false);
}
__device__ __forceinline__ Twin operator-(const Twin& a, const Twin& b) { return a + (-b); }
__device__ __forceinline__ Twin::Twin(const TwinProd& p) { *this = twin_of(p); }
// a + p: the product's sign relative to a goes into a constant factor; two
// variable factors of the other sign multiply first.
__device__ __forceinline__ Twin operator+(const Twin& a, const TwinProd& p) {
  const bool flip = (p.a.neg != p.b.neg) != a.neg;
  if (!flip)
    return twin_signed(twin_fma(twin_plain(p.a), twin_plain(p.b), twin_plain(a)), a.neg);
  if (p.b.cst)
    return twin_signed(twin_fma(twin_plain(p.a), twin_pack(-p.b.c, -p.b.c), twin_plain(a)),
                       a.neg);
  if (p.a.cst)
    return twin_signed(twin_fma(twin_pack(-p.a.c, -p.a.c), twin_plain(p.b), twin_plain(a)),
                       a.neg);
  return a + twin_of(p);
}
__device__ __forceinline__ Twin operator+(const TwinProd& p, const Twin& a) { return a + p; }
__device__ __forceinline__ Twin operator-(const Twin& a, const TwinProd& p) { return a + (-p); }
__device__ __forceinline__ Twin operator-(const TwinProd& p, const Twin& a) { return (-a) + p; }
__device__ __forceinline__ Twin operator+(const TwinProd& p, const TwinProd& q) {
  return twin_of(p) + q;
}
__device__ __forceinline__ Twin operator-(const TwinProd& p, const TwinProd& q) {
  return twin_of(p) + (-q);
}

// Where a thread's two lines lie.
struct TwinLines {
  const float2* ga;
  const float2* gb;
  float2* oa;
  float2* ob;
  bool active, both;          // line A / both lines inside the batch
  ulonglong2* sp;             // the pair's shared tile
  unsigned long long sign;    // {1, 1} or {-1, -1}: conjugation on load and store
};

// x *= w with one scalar twiddle for both lines.
__device__ __forceinline__ void twin_rotate(Twin& xr, Twin& xi, float wr, float wi) {
  const Twin cr(twin_pack(wr, wr)), ci(twin_pack(wi, wi));
  const Twin r = xr * cr - xi * ci;
  const Twin i = xi * cr + xr * ci;
  xr = r;
  xi = i;
}

// Stage twiddles v[r] *= w^r, every power from the table: one load for both
// lines.
template <int R, int NS>
__device__ __forceinline__ void twin_twiddle(Twin (&vr)[R], Twin (&vi)[R],
                                             const float2* __restrict__ tw) {
#pragma unroll
  for (int r = 1; r < R; ++r) {
    const float2 w = __ldg(tw + (r - 1) * NS);
    twin_rotate(vr[r], vi[r], w.x, w.y);
  }
}

template <int L, int TPL, int SH, int NS, int TWOFF, int R, int... Rest>
struct TwinRunner {
  static constexpr int BF = L / R;
  static constexpr int PER = (BF + TPL - 1) / TPL;
  static constexpr bool EVEN = BF % TPL == 0;
  static constexpr bool FIRST = NS == 1;
  static constexpr bool LAST = sizeof...(Rest) == 0;
  __device__ __forceinline__ static int pad(int i) { return SH ? i + (i >> SH) : i; }
  __device__ __forceinline__ static void run(const TwinLines& t, int tid,
                                             const float2* __restrict__ tw) {
    Twin vr[PER][R], vi[PER][R];
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int j = tid + m * TPL;
      if (EVEN || j < BF) {
        if constexpr (FIRST) {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int i = j + r * BF;
            float2 a = make_float2(0.f, 0.f), b = a;
            if (t.active) a = ld_global<float>(t.ga + i);
            if (t.both) b = ld_global<float>(t.gb + i);
            vr[m][r] = Twin(twin_pack(a.x, b.x));
            vi[m][r] = Twin(twin_mul(twin_pack(a.y, b.y), t.sign));
          }
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const ulonglong2 v = t.sp[pad(j + r * BF)];
            vr[m][r] = Twin(v.x);
            vi[m][r] = Twin(v.y);
          }
          twin_twiddle<R, NS>(vr[m], vi[m], tw + TWOFF + j % NS);
        }
        Dft<R>::fwd(vr[m], vi[m]);
      }
    }
    if constexpr (!FIRST && !LAST) __syncthreads();
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int j = tid + m * TPL;
      if (EVEN || j < BF) {
        const int base = (j / NS) * NS * R + (j % NS);
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const int i = base + k * NS;
          if constexpr (LAST) {
            float ra, rb, ia, ib;
            twin_unpack(twin_value(vr[m][k]), ra, rb);
            twin_unpack(twin_mul(twin_value(vi[m][k]), t.sign), ia, ib);
            if (t.active) st_global<float>(t.oa + i, ra, ia);
            if (t.both) st_global<float>(t.ob + i, rb, ib);
          } else {
            t.sp[pad(i)] = make_ulonglong2(twin_value(vr[m][k]), twin_value(vi[m][k]));
          }
        }
      }
    }
    if constexpr (!LAST) {
      __syncthreads();
      TwinRunner<L, TPL, SH, NS * R, TWOFF + stage_table_size(R, NS), Rest...>::run(t, tid, tw);
    }
  }
};

// TP line pairs per CTA, TPL threads per pair.
template <int L, int TPL, int TP, int SH>
struct TwinGeom {
  static constexpr int THREADS = TPL * TP;
  static constexpr int PITCH = pair_pitch<double>(L, TPL, TP, SH);
  static constexpr size_t SMEM = (size_t)TP * PITCH * 16;
  // 128 registers: 16 points of two lines take 64
  static constexpr int MIN_RAW = 65536 / (128 * ((THREADS + 31) / 32 * 32));
  static constexpr int MIN_CTAS = MIN_RAW < 1 ? 1 : MIN_RAW;
};

template <int L, int TPL, int TP, int SH, int... Rs>
__global__ void __launch_bounds__(TPL * TP, (TwinGeom<L, TPL, TP, SH>::MIN_CTAS))
twin_kernel(const RowsArgs<float> args) {
  static_assert(StageProduct<L, Rs...>::value == L, "radices must multiply to L");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RowsArgs<float> a = args;
  a.in = after_previous(args.in);
  const int pair = threadIdx.x / TPL;
  const long long b = 2 * ((long long)blockIdx.x * TP + pair);
  TwinLines t;
  t.active = b < a.batch;
  t.both = b + 1 < a.batch;
  t.ga = t.active ? batch_in<float>(a.in, a.in_dist, a.in_table, b) : a.in;
  t.gb = t.both ? batch_in<float>(a.in, a.in_dist, a.in_table, b + 1) : t.ga;
  t.oa = t.active ? batch_out<float>(a.out, a.out_dist, a.out_table, b) : a.out;
  t.ob = t.both ? batch_out<float>(a.out, a.out_dist, a.out_table, b + 1) : t.oa;
  t.sp = reinterpret_cast<ulonglong2*>(smem_raw) + pair * TwinGeom<L, TPL, TP, SH>::PITCH;
  t.sign = twin_pack(a.sign, a.sign);
  TwinRunner<L, TPL, SH, 1, 0, Rs...>::run(t, threadIdx.x % TPL, a.tw);
}

// ---------------------------------------------------------------------------
// Twin column passes: a thread runs the same butterfly of two adjacent lines
// (2 pr, 2 pr + 1) of the tile.  Their elements are adjacent in global memory,
// so one 16-byte access moves both where the transform starts on a 16-byte
// boundary (8-byte accesses where it does not), and in the tile one 16-byte
// word {reA, reB, imA, imB}.  Stage twiddles are the same for both lines; the
// line powers of a later pass (ColsLayout::super_fill) are kept as packed pairs.
//
// Lines of 320-512 points are bound by their tiles: 8 lines on 256 threads move
// 64-byte runs, and 16 lines of the one-line form take 512 threads at 64
// registers.  Two lines a thread give 16 lines, 128-byte runs, on 256 threads
// at 116 registers with two CTAs per SM.  us per 2^25 points, 8 lines -> 16
// lines one a thread -> 16 lines two a thread: 512 x 160 224 -> 211 -> 199, 512
// x 192 220 -> 206 -> 194, 256 x 512 209 -> 209 -> 199, 512 x 1024 261 -> 248
// -> 237; 512 x 512 239 -> 218 (256 x 1024 takes 220); as the narrow side of
// 327680 and 393216, 320 and 384 points take
// 279 -> 254 and 260 -> 249.  In L2 (2^21 points) 131072 16.1 -> 14.1; one
// transform alone, with half the CTAs, 8.4 -> 7.9.  Not built for 64-256 points, whose one-line
// tiles already move 128-byte runs (256 x 256 184 -> 187, 64 x 64 170 -> 168),
// nor for 640-2048 points, whose 16-line tiles leave one CTA per SM (512 x
// 1024 237 -> 245).
// ---------------------------------------------------------------------------
template <int L, int TPL, int C>
struct TwinColsGeom {
  static constexpr int P = C / 2;                 // line pairs
  static constexpr int THREADS = TPL * P;
  static constexpr int PITCH = P + 1;             // 16-byte words per element row
  static constexpr size_t SMEM = (size_t)L * PITCH * 16;
  static constexpr size_t super_smem(int first_radix) {
    return SMEM + (size_t)first_radix * P * 16;
  }
  static constexpr int MIN_RAW = 65536 / (128 * ((THREADS + 31) / 32 * 32));
  static constexpr int MIN_CTAS = MIN_RAW < 1 ? 1 : MIN_RAW;
};

template <int L, int TPL, int C, bool HEAD>
struct TwinCols {
  using G = TwinColsGeom<L, TPL, C>;
  const ColsArgs<float>& a;
  const float2* gin;          // element 0 of line 2 pr
  float2* gout;
  long long in_stride, out_stride;
  bool in16, out16;           // 16-byte aligned pairs
  ulonglong2* sp;             // the tile
  ulonglong2* sw;             // line powers (later passes)
  unsigned jmod;              // of line 2 pr
  int pr;
  unsigned long long sign_in, sign_out;

  // W^{jm i} of one line from the two-level table
  __device__ __forceinline__ float2 power(unsigned jm, unsigned i) const {
    ColsLayout<float, 1, 1, true> lay;
    lay.tw_hi = a.tw_hi;
    lay.tw_lo = a.tw_lo;
    lay.split_shift = a.split_shift;
    lay.jmod = jm;
    float2 w;
    lay.super_w(i, w.x, w.y);
    return w;
  }

  template <int NS, int TWOFF, int R, int... Rest>
  __device__ __forceinline__ void run(int t, const float2* __restrict__ tw) const {
    constexpr int BF = L / R;
    constexpr int PER = (BF + TPL - 1) / TPL;
    constexpr bool EVEN = BF % TPL == 0;
    constexpr bool FIRST = NS == 1;
    constexpr bool LAST = sizeof...(Rest) == 0;
    constexpr bool STORE = LAST && !HEAD;
    Twin vr[PER][R], vi[PER][R];
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int j = t + m * TPL;
      if (EVEN || j < BF) {
        if constexpr (FIRST) {
          const float2* p = gin + (long long)j * in_stride;
          const long long step = (long long)BF * in_stride;
          if (in16) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
              vr[m][r] = Twin(twin_pack(v.x, v.z));
              vi[m][r] = Twin(twin_mul(twin_pack(v.y, v.w), sign_in));
              p += step;
            }
          } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const float2 x = ld_global<float>(p), y = ld_global<float>(p + 1);
              vr[m][r] = Twin(twin_pack(x.x, y.x));
              vi[m][r] = Twin(twin_mul(twin_pack(x.y, y.y), sign_in));
              p += step;
            }
          }
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const ulonglong2 v = sp[(j + r * BF) * G::PITCH + pr];
            vr[m][r] = Twin(v.x);
            vi[m][r] = Twin(v.y);
          }
        }
      }
    }
    if constexpr (FIRST && !HEAD) {
      // the tile's line powers u^r, filled while the loads are in flight
      for (int q = threadIdx.x; q < R * G::P; q += G::THREADS) {
        const unsigned jm = jmod - 2u * (unsigned)pr + 2u * (unsigned)(q % G::P);
        const unsigned i = (unsigned)(q / G::P * BF);
        const float2 x = power(jm, i), y = power(jm + 1, i);
        sw[q] = make_ulonglong2(twin_pack(x.x, y.x), twin_pack(x.y, y.y));
      }
      __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int j = t + m * TPL;
      if (EVEN || j < BF) {
        if constexpr (FIRST && !HEAD) {
          const float2 x = power(jmod, (unsigned)j), y = power(jmod + 1, (unsigned)j);
          const Twin br(twin_pack(x.x, y.x)), bi(twin_pack(x.y, y.y));
#pragma unroll
          for (int r = 0; r < R; ++r) {
            Twin wr = br, wi = bi;
            if (r > 0) {
              const ulonglong2 u = sw[r * G::P + pr];
              const Twin ur(u.x), ui(u.y);
              wr = ur * br - ui * bi;
              wi = ui * br + ur * bi;
            }
            const Twin xr = vr[m][r] * wr - vi[m][r] * wi;
            const Twin xi = vi[m][r] * wr + vr[m][r] * wi;
            vr[m][r] = xr;
            vi[m][r] = xi;
          }
        }
        if constexpr (!FIRST) twin_twiddle<R, NS>(vr[m], vi[m], tw + TWOFF + j % NS);
        Dft<R>::fwd(vr[m], vi[m]);
      }
    }
    if constexpr (!FIRST && !STORE) __syncthreads();
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int j = t + m * TPL;
      if (EVEN || j < BF) {
        const int base = (j / NS) * NS * R + (j % NS);
        if constexpr (STORE) {
          float2* p = gout + (long long)base * out_stride;
          const long long step = (long long)NS * out_stride;
#pragma unroll
          for (int k = 0; k < R; ++k) {
            float ra, rb, ia, ib;
            twin_unpack(twin_value(vr[m][k]), ra, rb);
            twin_unpack(twin_mul(twin_value(vi[m][k]), sign_out), ia, ib);
            if (out16) {
              *reinterpret_cast<float4*>(p) = make_float4(ra, ia, rb, ib);
            } else {
              st_global<float>(p, ra, ia);
              st_global<float>(p + 1, rb, ib);
            }
            p += step;
          }
        } else {
#pragma unroll
          for (int k = 0; k < R; ++k)
            sp[(base + k * NS) * G::PITCH + pr] =
                make_ulonglong2(twin_value(vr[m][k]), twin_value(vi[m][k]));
        }
      }
    }
    if constexpr (!STORE) __syncthreads();
    if constexpr (!LAST) run<NS * R, TWOFF + stage_table_size(R, NS), Rest...>(t, tw);
  }
};

template <int L, int TPL, int C, bool HEAD, int... Rs>
__global__ void __launch_bounds__(TPL * C / 2, (TwinColsGeom<L, TPL, C>::MIN_CTAS))
twin_cols_kernel(const ColsArgs<float> args) {
  static_assert(StageProduct<L, Rs...>::value == L, "radices must multiply to L");
  static_assert(C % 2 == 0, "lines in pairs");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using G = TwinColsGeom<L, TPL, C>;
  ColsArgs<float> a = args;
  a.in = after_previous(args.in);
  long long b, j0;
  cols_tile<L, C>(a, b, j0);
  const int pr = threadIdx.x % G::P;
  const unsigned ns = (unsigned)a.ns_outer;             // a multiple of C, or 1
  const unsigned j = (unsigned)j0 + 2u * (unsigned)pr;
  const unsigned jq = HEAD ? 0u : j / ns, jm = j - jq * ns;
  const float2* in_b = batch_in<float>(a.in, a.in_dist, a.in_table, b);
  float2* out_b = batch_out<float>(a.out, a.out_dist, a.out_table, b);
  const long long stride = a.total / L;                 // a multiple of C
  TwinCols<L, TPL, C, HEAD> tc{a,
                               in_b + j,
                               out_b + (long long)jq * ns * L + jm,
                               stride,
                               (long long)ns,
                               (reinterpret_cast<uintptr_t>(in_b) & 15) == 0,
                               (reinterpret_cast<uintptr_t>(out_b) & 15) == 0,
                               reinterpret_cast<ulonglong2*>(smem_raw),
                               reinterpret_cast<ulonglong2*>(smem_raw + G::SMEM),
                               jm,
                               pr,
                               twin_pack(a.sign_in, a.sign_in),
                               twin_pack(a.sign_out, a.sign_out)};
  tc.template run<1, 0, Rs...>(threadIdx.x / G::P, a.tw);
  if constexpr (HEAD) {
    // lines j0 .. j0+C-1 are one contiguous block of the output
    float2* dst = out_b + j0 * L;
    for (int q = threadIdx.x; q < G::P * L; q += G::THREADS) {
      const int p = q / L, k = q - p * L;
      const ulonglong2 v = tc.sp[k * G::PITCH + p];
      float ra, rb, ia, ib;
      twin_unpack(v.x, ra, rb);
      twin_unpack(twin_mul(v.y, tc.sign_out), ia, ib);
      st_global<float>(dst + (2 * p) * L + k, ra, ia);
      st_global<float>(dst + (2 * p + 1) * L + k, rb, ib);
    }
  }
}

}  // namespace mofft
