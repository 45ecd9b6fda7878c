// The FP64 block FFT in 64-bit block fixed point (BlockFFT<double, ...>).
//
// GB300 issues 2 FP64 lanes per SM and clock and about 128 of 32-bit integer
// adds, 30 of 32 x 32 -> 64-bit multiply-adds: an FP64 butterfly add costs
// what 27 64-bit integer adds cost, an FP64 complex product (2.26 SM clocks)
// what 4.4 integer ones of 62-bit operands cost (0.52).  A transform needs
// one common scale only, so it runs on integers: the vector is scaled by a
// power of two so that no stage can overflow, transformed with 64-bit adds
// and 62-bit twiddles, and converted back.
//
// Scale and error.  Every value's magnitude after stage s is at most
// min(R_s max|x|, sum|x|) 4^-(s-1): R_s the product of the radices so far,
// and each twiddle product divides by 4 (the twiddles are scaled by 2^62 and
// the product keeps the upper 64 bits), which about keeps pace with the
// growth of a radix-8 stage (sqrt 8 for noise).  It is also at most
// sqrt(R_1 sum|x|^2), R_1 the first radix (Cauchy and Schwarz over the R_s
// values that it sums: sqrt(R_s) 4^-(s-1) falls from stage to stage).  The
// smaller of the last and the largest over the stages of the first two is
// scaled to just under 2^62 (the products and the sqrt(1/2) rotations need one
// more bit).  The rounding noise is about 2.5 units per output.  Flat vectors
// take the first bound, single values the second, a few peaks on noise (the
// brackets of an intermittent field) the third.
//   Relative L2 error over that of the same transform in FP64 arithmetic, the
// worst of noise, its powers, peaks of 5 to 640 on it, power laws and single
// modes, n = 512 .. 8192: 0.74, 0.64, 0.82, 0.98, 0.89; without the third bound
// 0.74, 1.18, 1.71, 2.7, 3.3.  A 1024^2 2-D transform against long double (white
// noise / k^-3 / one mode): 1.1e-16 / 6.7e-17 / 5.9e-17, with FP64 arithmetic
// 3.1e-16 / 2.6e-16 / 3.3e-16.  2048^2 there and back: 548 -> 156 us.
#pragma once

#include <vector>

#include "r2d3c_fft.cuh"

namespace r2d3c {

struct fx {
  long long x, y;
};

__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
// limbs of a = a1 2^32 + a0 with both signed
__device__ __forceinline__ int limb0(long long a) { return (int)a; }
__device__ __forceinline__ int limb1(long long a) { return (int)(a >> 32) + (int)((unsigned)a >> 31); }

// a w / 4 for w = (c + i s) 2^62 in signed limbs (c0, c1, s0, s1): the upper
// 64 bits of the two sums of products, their middle terms rounded, the
// product of the low limbs (below half a unit, of either sign) left out.
// |a| <= 2^62 keeps every sum inside 63 bits.
__device__ __forceinline__ fx fx_twmul(fx a, int4 w) {
  const int x0 = limb0(a.x), x1 = limb1(a.x), y0 = limb0(a.y), y1 = limb1(a.y);
  const int n0 = -w.z, n1 = -w.w;
  fx r;
  long long m = mad_wide(x1, w.x, 0x80000000ll);
  m = mad_wide(x0, w.y, m);
  m = mad_wide(y1, n0, m);
  m = mad_wide(y0, n1, m);
  r.x = mad_wide(x1, w.y, mad_wide(y1, n1, (long long)(int)(m >> 32)));
  m = mad_wide(x1, w.z, 0x80000000ll);
  m = mad_wide(x0, w.w, m);
  m = mad_wide(y1, w.x, m);
  m = mad_wide(y0, w.y, m);
  r.y = mad_wide(x1, w.w, mad_wide(y1, w.y, (long long)(int)(m >> 32)));
  return r;
}
// a / 4 rounded to nearest, ties to even: ties one way would add up over the
// elements of a transform, and over the transforms of a plane, in the lowest
// modes
__device__ __forceinline__ fx fx_quarter(fx a) {
  a.x = (a.x + (1 + (int)(((unsigned)a.x >> 2) & 1u))) >> 2;
  a.y = (a.y + (1 + (int)(((unsigned)a.y >> 2) & 1u))) >> 2;
  return a;
}
// a K / 2^64 for a constant |K| < 2^63 (a may use all 63 bits)
template <long long K>
__device__ __forceinline__ long long fx_mulk(long long a) {
  constexpr int k0 = (int)K, k1 = (int)((K - (long long)k0) >> 32);
  const int a0 = limb0(a), a1 = limb1(a);
  long long m = mad_wide(a1, k0, 0x80000000ll);
  m = mad_wide(a0, k1, m);
  return mad_wide(a1, k1, (long long)(int)(m >> 32));
}
// Fractions of 2^64: 1 - cos(pi/4), 1 - cos(pi/8), sin(pi/8)
constexpr long long kFx1mR2 = 0x4AFB0CCC06219B7Cll;
constexpr long long kFx1mC8 = 0x137CA1866B95CEBBll;
constexpr long long kFxS8 = 0x61F78A9ABAA58B47ll;

// a exp(-2 pi i I16 / 16)
template <int I16>
__device__ __forceinline__ fx fx_rot(fx a) {
  if constexpr (I16 == 0) {
    return a;
  } else if constexpr (I16 == 4) {
    return fx{a.y, -a.x};
  } else if constexpr (I16 == 2) {
    const long long p = a.x + a.y, q = a.y - a.x;
    return fx{p - fx_mulk<kFx1mR2>(p), q - fx_mulk<kFx1mR2>(q)};
  } else if constexpr (I16 == 6) {
    const long long p = a.y - a.x, q = -a.x - a.y;
    return fx{p - fx_mulk<kFx1mR2>(p), q - fx_mulk<kFx1mR2>(q)};
  } else {
    // (C - i S) with C = cos(pi/8) = 1 - k, S = sin(pi/8), and its turns
    if constexpr (I16 == 1) {
      return fx{a.x - fx_mulk<kFx1mC8>(a.x) + fx_mulk<kFxS8>(a.y), a.y - fx_mulk<kFx1mC8>(a.y) - fx_mulk<kFxS8>(a.x)};
    } else if constexpr (I16 == 3) {
      return fx{fx_mulk<kFxS8>(a.x) + a.y - fx_mulk<kFx1mC8>(a.y), fx_mulk<kFxS8>(a.y) - a.x + fx_mulk<kFx1mC8>(a.x)};
    } else if constexpr (I16 == 5) {
      return fx{a.y - fx_mulk<kFx1mC8>(a.y) - fx_mulk<kFxS8>(a.x), fx_mulk<kFx1mC8>(a.x) - a.x - fx_mulk<kFxS8>(a.y)};
    } else {
      return fx{fx_mulk<kFx1mC8>(a.x) - a.x + fx_mulk<kFxS8>(a.y), fx_mulk<kFx1mC8>(a.y) - a.y - fx_mulk<kFxS8>(a.x)};
    }
  }
}

// In-register forward DFT of R points (radix-2 decimation in time)
template <int R> struct FxDFT {
  template <int K>
  static __device__ __forceinline__ void bfly(fx* u, const fx* e, const fx* o) {
    if constexpr (K < R / 2) {
      const fx t = fx_rot<(K * 16) / R>(o[K]);
      u[K] = fx{e[K].x + t.x, e[K].y + t.y};
      u[K + R / 2] = fx{e[K].x - t.x, e[K].y - t.y};
      bfly<K + 1>(u, e, o);
    }
  }
  static __device__ __forceinline__ void run(fx* u) {
    fx e[R / 2], o[R / 2];
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
      e[i] = u[2 * i];
      o[i] = u[2 * i + 1];
    }
    FxDFT<R / 2>::run(e);
    FxDFT<R / 2>::run(o);
    bfly<0>(u, e, o);
  }
};
template <> struct FxDFT<1> {
  static __device__ __forceinline__ void run(fx*) {}
};

// x 2^s for c = e + 62 - s, e the biased exponent of the vector's largest
// value: rounded to nearest.  (Truncation towards zero would leave an error
// that has the sign of x, which a field of one sign or a skewed one carries
// into its lowest modes.)  fx_round: (h, l) >> r with one guard bit, the sign
// s (0 or -1) by complement, ((t ^ s) + 1) >> 1: halves away from zero.
__device__ __forceinline__ long long fx_round(unsigned h, unsigned l, int r, int s) {
  if (r & 32) {
    l = h;
    h = 0;
  }
  l = __funnelshift_r(l, h, r) ^ (unsigned)s;
  h = (h >> (r & 31)) ^ (unsigned)s;
  return ((long long)(((unsigned long long)h << 32) | l) + 1) >> 1;
}
// SUB: the vector may hold subnormals (fx_sub); otherwise a zero exponent
// means a value far below the last place, whatever its mantissa
__device__ __forceinline__ bool fx_sub(int e) { return e < 128; }
template <bool SUB = false>
__device__ __forceinline__ long long fx_from(double x, int c) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  int e = (hi >> 20) & 0x7ff;
  unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  if constexpr (SUB) {
    if (e == 0) {
      e = 1;
      mh &= 0xfffffu;
    }
  }
  // the mantissa's top bit at 62, so that a shift by 63 leaves nothing
  return fx_round(__funnelshift_l(lo, mh, 10), lo << 10, min(c - 1 - e, 63), hi >> 31);
}
// |K x| with sign flip sg (0 or -1): as fx_from with the mantissa times the
// normalised factor F = |K| << clz(|K|) (32 bits) and c less 32 - clz(|K|)
template <bool SUB = false>
__device__ __forceinline__ long long fx_from_mul(double x, unsigned F, int sg, int c) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  int e = (hi >> 20) & 0x7ff;
  unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  if constexpr (SUB) {
    if (e == 0) {
      e = 1;
      mh &= 0xfffffu;
    }
  }
  const unsigned long long t = (unsigned long long)(lo << 11) * F;
  const unsigned long long m = (unsigned long long)__funnelshift_l(lo, mh, 11) * F + (unsigned)(t >> 32);
  const int r = c - e;
  return r < 64 ? fx_round((unsigned)(m >> 32), (unsigned)m, r, sg ^ (hi >> 31)) : 0;
}
__device__ __forceinline__ unsigned fx_upper(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// The largest upper word of the thread's values, at least 1 where any is not
// zero (subnormals below 2^-1042 have none): mh with the values' lower words
// joined in lo
__device__ __forceinline__ unsigned fx_any(unsigned mh, unsigned lo) { return max(mh, lo ? 1u : 0u); }
// |x| 2^(1023 - ew) in FP32 from x's upper word (the mantissa's upper 20 bits;
// below 2^-126: 0)
__device__ __forceinline__ float fx_mag(unsigned up, int ew) {
  return __int_as_float(max((int)up - ((ew - 127) << 20), 0) << 3);
}

// The FP64 value of a 2^k by integer operations (the FP64 pipe's own
// conversion takes half an SM clock a value), rounded to nearest (halves away
// from zero); kb = k + 1023 + 63, for results in the normal range
__device__ __forceinline__ double fx_to(long long a, int kb) {
  const int sg = (int)(a >> 63);
  const unsigned long long m = (unsigned long long)(a < 0 ? -a : a);
  unsigned h = (unsigned)(m >> 32), l = (unsigned)m;
  if (h == 0) {
    h = l;
    l = 0;
    kb -= 32;
  }
  const int z = __clz(h);
  const unsigned g = __funnelshift_l(l, h, z);
  l <<= (z & 31);
  // the mantissa with its top bit at 63, shifted to 52; the implicit bit adds
  // one to the exponent field, a carry out of the rounding another
  const unsigned ql = __funnelshift_r(l, g, 11), qh = (g >> 11) + ((unsigned)(kb - z - 1) << 20);
  const unsigned long long q = (((unsigned long long)qh << 32) | ql) + ((l >> 10) & 1u);
  const int hi = h ? (int)(q >> 32) | (sg & (int)0x80000000) : 0;
  return __hiloint2double(hi, (int)(unsigned)q);
}

// the same for any k, and NaN where the vector's largest exponent e says so
static __device__ __noinline__ double fx_to_far(long long a, int e, int k) {
  return e == 0x7ff ? __hiloint2double(0x7ff80000, 0) : scalbn(fx_to(a, 1086), k);
}
// the values a 2^k of one vector: by integers, or by the FP64 pipe in kernels
// that leave it idle
struct FxOut {
  int e, k;
  bool plain;  // no value leaves the normal range
  __device__ __forceinline__ FxOut(int e_, int k_) : e(e_), k(k_), plain(k_ > -1000 && k_ < 900 && e_ != 0x7ff) {}
  __device__ __forceinline__ double operator()(long long a) const {
    return plain ? fx_to(a, k + 1086) : fx_to_far(a, e, k);
  }
  __device__ __forceinline__ double pipe(long long a) const {
    if (!plain) return fx_to_far(a, e, k);
    const double d = __ll2double_rn(a);
    const int hi = __double2hiint(d);
    return __hiloint2double(hi ? hi + (k << 20) : 0, __double2loint(d));
  }
};

// One length-N FP64 transform by TPF = N/E threads: the interface of the
// general BlockFFT (thread `lane` holds x[lane + q*TPF], then X[lane + q*TPF]),
// the arithmetic in block fixed point (above).  An inverse transform is the
// forward one with real and imaginary parts exchanged.  A vector with an
// infinity or a NaN gives NaN throughout.
template <int N, int E, bool ILV_OK>
struct BlockFFT<double, N, E, 1, ILV_OK> {
  using T = double;
  static_assert((N & (N - 1)) == 0 && N >= E && E >= 2, "N, E powers of two");
  static constexpr int TPF = N / E;
  static constexpr int LOGN = ilog2(N);
  static constexpr int LOGE = ilog2(E);
  static constexpr int NST = (LOGN + LOGE - 1) / LOGE;
  static constexpr int LAST_R = 1 << (LOGN - LOGE * (NST - 1));
  static constexpr int PADSH = 3;  // one 16-byte element every 128 bytes
  static constexpr int WARPS = TPF > 32 ? TPF / 32 : 0;
  static_assert(WARPS <= 32, "one lane per warp in the scale's reduction");
  static constexpr int RED = N + (N >> PADSH);  // the warps' partial maxima and sums
  static constexpr int SMEM_ELEMS = RED + WARPS;
  static constexpr size_t SMEM_BYTES = (size_t)SMEM_ELEMS * sizeof(double2);

  static __device__ __forceinline__ int pad(int i) { return i + (i >> PADSH); }
  // pad(base + r step): one address and constant offsets where the carry into
  // the padding is known (base a multiple of R for step 1)
  static __device__ __forceinline__ int pad_add(int base, int r, int step, int R) {
    if (step % 8 == 0) return pad(base) + r * (step + step / 8);
    if (step == 1 && R == 8) return pad(base) + r;
    return pad(base + r * step);
  }
  static __host__ __device__ constexpr int radix(int s) { return s == NST - 1 ? LAST_R : E; }
  static __host__ __device__ constexpr int ns_of(int s) {
    int ns = 1;
    for (int i = 0; i < s; ++i) ns *= radix(i);
    return ns;
  }
  static __host__ __device__ constexpr int tw_off(int s) {
    int off = 0;
    for (int i = 1; i < s; ++i) off += ns_of(i) * (radix(i) - 1);
    return off;
  }
  static constexpr int TW_ELEMS = tw_off(NST) > 0 ? tw_off(NST) : 1;

  // The scale of a vector in two steps.  warp_base: from the thread's largest
  // upper word (sign cleared) the biased exponent of the warp's (or the
  // group's, below 32 threads) largest component; every magnitude is then
  // taken relative to it in FP32 (fx_mag), which loses no exponent range; mh
  // becomes the warp's largest word (0: all zero, whatever fx_mag says).
  // combine: from the thread's largest magnitude mx of a component, the sum l1
  // of its values' larger components and the sum l2 of their squares the group's
  // biased exponent e and the scale s, such that x 2^(s - (e - 1023)) is the
  // fixed-point value.
  static constexpr int SUB = TPF < 32 ? TPF : 32;
  static __device__ __forceinline__ int warp_base(unsigned& mh) {
    if constexpr (TPF >= 32) {
      mh = __reduce_max_sync(0xffffffffu, mh);
    } else {
#pragma unroll
      for (int o = SUB / 2; o > 0; o >>= 1) mh = max(mh, __shfl_xor_sync(0xffffffffu, mh, o));
    }
    return max((int)(mh >> 20), 1);
  }
  static __device__ __forceinline__ float sub_max(float m) {  // m >= 0: ordered as its bits
    if constexpr (TPF >= 32) {
      return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    } else {
#pragma unroll
      for (int o = SUB / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      return m;
    }
  }
  // The bound by the squares (l2) is taken from four stages on (n >= 1024); with
  // three the other two leave the error below 0.75 times FP64's.
  static constexpr bool L2 = NST >= 4;
  static_assert(!L2 || (TPF >= 64 && E <= 16 && WARPS <= 16), "the ranges of lanes_sum");
  static __device__ __forceinline__ float shfl_sum(float v, int o0) {
#pragma unroll
    for (int o = o0; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  // 2^LG times the sum of v over the warp, every v to half a unit of 2^-LG (v <=
  // 2^(23 - LG)): one integer reduction instead of five shuffles and additions.
  template <int LG>
  static __device__ __forceinline__ float lanes_sum(float v) {
    const unsigned u = __reduce_add_sync(0xffffffffu, __float_as_uint(fmaf(v, (float)(1 << LG), 8388608.f)));
    return (float)(u - 32u * 0x4b000000u);
  }
  // 2^-k and 2^k for the exponent k of mx >= 1 (or mx = 0)
  static __device__ __forceinline__ void unit_of(float mx, float& down, float& up) {
    up = __int_as_float(__float_as_int(fmaxf(mx, 1.f)) & 0x7f800000);
    down = __int_as_float((254 << 23) - __float_as_int(up));
  }
  static __device__ __forceinline__ void combine(int ew, float mx, float l1, float l2, int lane, int4* red, int& e,
                                                 int& s) {
    mx = sub_max(mx);
    e = ew;
    if constexpr (L2) {
      // per thread below 2 E and 4 E in units of mx
      float down, up;
      unit_of(mx, down, up);
      l1 = lanes_sum<17>(l1 * down) * (up * 0x1p-17f);
      l2 = lanes_sum<16>(l2 * down * down) * (up * up * 0x1p-16f);
    } else {
      l1 = shfl_sum(l1, SUB / 2);
    }
    if constexpr (TPF > 32) {
      if ((lane & 31) == 0)
        red[lane >> 5] = make_int4(ew, __float_as_int(mx), __float_as_int(l1), __float_as_int(l2));
      __syncthreads();
      const int4 w = red[lane & (WARPS - 1)];
      e = __reduce_max_sync(0xffffffffu, w.x);
      const float f = __int_as_float(max(127 + w.x - e, 0) << 23);
      mx = sub_max(__int_as_float(w.y) * f);
      l1 = __int_as_float(w.z) * f;
      if constexpr (L2) {  // (every warp's entry is read by 32 / WARPS lanes)
        constexpr float r = (float)WARPS / 32.f;
        float down, up;
        unit_of(mx, down, up);
        l1 = lanes_sum<12>(l1 * down) * (up * 0x1p-12f * r);
        l2 = lanes_sum<11>(__int_as_float(w.w) * f * f * down * down) * (up * up * 0x1p-11f * r);
      } else {
        l1 = shfl_sum(l1, WARPS / 2);
      }
    }
    s = scale_of(mx, l1, l2) - (e == 1 ? 2 : 0);  // (subnormals: taken up to twice too small or large)
    if (l1 == 0.f) {  // all zero
      e = 1023;
      s = 0;
    }
  }
  // s for magnitudes relative to the vector's exponent
  static __device__ __forceinline__ int scale_of(float mx, float l1, float l2) {
    // upper bounds: |z| <= sqrt(2) max(|re|, |im|), the truncated lower words,
    // the FP32 sums (lanes_sum: 2^-12 and 2^-9 of mx, 2^-11 and 2^-8 of mx^2)
    mx *= 1.41423f;
    l1 *= L2 ? 1.41425f * 1.0025f : 1.41425f;
    float b = 0.f, g = 1.f;
#pragma unroll
    for (int st = 0; st < NST; ++st) {
      b = fmaxf(b, fminf(mx * (float)ns_of(st + 1), l1) * g);
      g *= 0.25f;
    }
    int x = (__float_as_int(b) >> 23) - 127;  // b < 2^(x + 1)
    // sqrt(R_s) 4^-(s-1) is largest at the first stage (R <= 16); half the
    // exponent is the root's
    if constexpr (L2) x = min(x, ((__float_as_int(l2 * (2.0001f * 1.0046f * (float)E)) >> 23) - 127) >> 1);
    return min(61 - x, 61);
  }
  // The scale of a vector whose real and imaginary parts are scaled apart, so
  // that the smaller one keeps its own precision: each part relative to its
  // own largest exponent e1, e2 (equal to the other's where it is all zero).
  // Values 0 or normal; ew, l1 and l2 of each part as for combine (p: part 1,
  // q: part 2).  Takes two elements of red a warp.
  static __device__ __forceinline__ void combine2(int ewp, int ewq, float p1, float q1, float p2, float q2, int lane,
                                                  int4* red, int& e1, int& e2, int& s) {
    e1 = ewp;
    e2 = ewq;
    float l1, l2 = 0.f;
    if constexpr (TPF > 32) {
      if constexpr (L2) {
        p1 = lanes_sum<17>(p1);
        q1 = lanes_sum<17>(q1);
        p2 = lanes_sum<16>(p2);
        q2 = lanes_sum<16>(q2);
      } else {
        p1 = shfl_sum(p1, 16);
        q1 = shfl_sum(q1, 16);
      }
      if ((lane & 31) == 0) {
        red[lane >> 5] = make_int4(ewp, ewq, __float_as_int(p1), __float_as_int(q1));
        if constexpr (L2) red[WARPS + (lane >> 5)] = make_int4(__float_as_int(p2), __float_as_int(q2), 0, 0);
      }
      __syncthreads();
      const int4 w = red[lane & (WARPS - 1)];
      e1 = __reduce_max_sync(0xffffffffu, w.x);
      e2 = __reduce_max_sync(0xffffffffu, w.y);
      const float f1 = __int_as_float(max(127 + w.x - e1, 0) << 23), f2 = __int_as_float(max(127 + w.y - e2, 0) << 23);
      l1 = __int_as_float(w.z) * f1 + __int_as_float(w.w) * f2;
      if constexpr (L2) {
        const int4 v = red[WARPS + (lane & (WARPS - 1))];
        constexpr float r = (float)WARPS / 32.f;
        l1 = lanes_sum<12>(l1 * 0x1p-17f) * (0x1p-12f * r);
        l2 = lanes_sum<11>((__int_as_float(v.x) * f1 * f1 + __int_as_float(v.y) * f2 * f2) * 0x1p-16f) * (0x1p-11f * r);
      } else {
        l1 = shfl_sum(l1, WARPS / 2);
      }
    } else {
      l1 = shfl_sum(p1 + q1, SUB / 2);
    }
    s = scale_of(2.f, 0.70711f * l1, 0.50001f * l2);  // (the sums are of |z| and |z|^2 themselves)
    if (e1 == 1) e1 = e2 == 1 ? 1023 : e2;
    if (e2 == 1) e2 = e1;
  }

  // both steps for the values v
  static __device__ __forceinline__ void scale(const double2 (&v)[E], int lane, int4* red, int& e, int& s) {
    unsigned mh = 0, lo = 0;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      mh = max(mh, max(fx_upper(v[q].x), fx_upper(v[q].y)));
      lo |= __double2loint(v[q].x) | __double2loint(v[q].y);
    }
    mh = fx_any(mh, lo);
    const int ew = warp_base(mh);
    float mx = 0.f, l1 = 0.f, l2 = 0.f;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const float a = fx_mag(max(fx_upper(v[q].x), fx_upper(v[q].y)), ew);
      mx = fmaxf(mx, a);
      l1 += a;
      l2 = fmaf(a, a, l2);
    }
    combine(ew, mh ? mx : 0.f, mh ? l1 : 0.f, mh ? l2 : 0.f, lane, red, e, s);
  }

  // Position of value i of one component in a buffer of N 8-byte values
  // (HALF: real parts, then imaginary parts go through it; half the shared
  // memory, twice the barriers): every access of the stages is free of bank
  // conflicts.
  static __device__ __forceinline__ int pos8(int i) { return i ^ ((i >> LOGE) & 15); }
  // of value lane + q TPF
  static __device__ __forceinline__ int pos8(int lane, int q) {
    if constexpr (TPF % (16 << LOGE) == 0) return pos8(lane) + q * TPF;
    else return pos8(lane + q * TPF);
  }

  template <int S, int NS, bool HALF>
  static __device__ __forceinline__ void stage(fx (&v)[E], int lane, longlong2* sm, const int4* __restrict__ tw) {
    constexpr int R = radix(S);
    constexpr int B = E / R;
    constexpr int LOGNS = ilog2(NS);
#pragma unroll
    for (int m = 0; m < B; ++m) {
      if constexpr (NS > 1) {
        const int jm = (lane + m * TPF) & (NS - 1);
        const int4* tb = tw + tw_off(S) + jm;
        v[m] = fx_quarter(v[m]);
#pragma unroll
        for (int r = 1; r < R; ++r) v[m + r * B] = fx_twmul(v[m + r * B], __ldg(&tb[(r - 1) * NS]));
      }
      fx u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = v[m + r * B];
      FxDFT<R>::run(u);
#pragma unroll
      for (int r = 0; r < R; ++r) v[m + r * B] = u[r];
    }
    if constexpr (S < NST - 1 && HALF) {
      long long* s8 = reinterpret_cast<long long*>(sm);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int m = 0; m < B; ++m) {
          const int j = lane + m * TPF;
          const int base = ((j >> LOGNS) << (LOGNS + ilog2(R))) + (j & (NS - 1));
#pragma unroll
          for (int r = 0; r < R; ++r) s8[pos8(base + r * NS)] = h ? v[m + r * B].y : v[m + r * B].x;
        }
        fft_sync<TPF>();
#pragma unroll
        for (int q = 0; q < E; ++q) (h ? v[q].y : v[q].x) = s8[pos8(lane, q)];
        fft_sync<TPF>();
      }
      stage<S + 1, NS * R, HALF>(v, lane, sm, tw);
    } else if constexpr (S < NST - 1) {
#pragma unroll
      for (int m = 0; m < B; ++m) {
        const int j = lane + m * TPF;
        const int base = ((j >> LOGNS) << (LOGNS + ilog2(R))) + (j & (NS - 1));
#pragma unroll
        for (int r = 0; r < R; ++r)
          sm[pad_add(base, r, NS, R)] = make_longlong2(v[m + r * B].x, v[m + r * B].y);
      }
      fft_sync<TPF>();
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const longlong2 w = sm[pad_add(lane, q, TPF, 1)];
        v[q] = fx{w.x, w.y};
      }
      fft_sync<TPF>();
      stage<S + 1, NS * R, HALF>(v, lane, sm, tw);
    }
  }

  // forward transform of fixed-point values in place, divided by 4 at every
  // stage but the first: the results are u 2^out_exp(e, s)
  template <bool HALF = false>
  static __device__ __forceinline__ void run_fx(fx (&u)[E], int lane, void* sm, const int4* __restrict__ tw) {
    stage<0, 1, HALF>(u, lane, reinterpret_cast<longlong2*>(sm), tw);
  }
  static __device__ __forceinline__ int out_exp(int e, int s) { return e - 1023 - s + 2 * (NST - 1); }

  // X[k] = sum_x x[x] exp(DIR*2*pi*i*x*k/N), unnormalised
  template <int DIR>
  static __device__ __forceinline__ void run(double2 (&v)[1][E], int lane, double2* sm,
                                             const int4* __restrict__ tw) {
    int e, s;
    scale(v[0], lane, reinterpret_cast<int4*>(sm + RED), e, s);
    fx u[E];
    const int c = e + 62 - s;
    from<(DIR > 0)>(v[0], e, c, u);
    run_fx(u, lane, sm, tw);
    const FxOut out(e, out_exp(e, s));
#pragma unroll
    for (int q = 0; q < E; ++q) v[0][q] = mkc<T>(out(DIR < 0 ? u[q].x : u[q].y), out(DIR < 0 ? u[q].y : u[q].x));
  }
  // the values in fixed point (SWAP: real and imaginary parts exchanged)
  template <bool SWAP>
  static __device__ __forceinline__ void from(const double2 (&v)[E], int e, int c, fx (&u)[E]) {
    if (!fx_sub(e)) {
#pragma unroll
      for (int q = 0; q < E; ++q) u[q] = fx{fx_from(SWAP ? v[q].y : v[q].x, c), fx_from(SWAP ? v[q].x : v[q].y, c)};
    } else {
#pragma unroll
      for (int q = 0; q < E; ++q)
        u[q] = fx{fx_from<true>(SWAP ? v[q].y : v[q].x, c), fx_from<true>(SWAP ? v[q].x : v[q].y, c)};
    }
  }

  // Natural-order result to shared memory (Hermitian split of packed pairs)
  static __device__ __forceinline__ void to_smem(const double2 (&v)[1][E], int lane, double2* sm) {
#pragma unroll
    for (int q = 0; q < E; ++q) sm[pad(lane + q * TPF)] = v[0][q];
  }
  static __device__ __forceinline__ double2 from_smem(int, int k, const double2* sm) { return sm[pad(k)]; }
};

// ---------------------------------------------------------------------------
// Host: the twiddles in fixed point.  cos and sin of 2 pi k / n in
// double-double (Taylor series of the first octant, exact symmetries beyond),
// rounded to 2^-62.
// ---------------------------------------------------------------------------
struct dd {
  double h, l;
};
inline dd dd_norm(double h, double l) {
  const double s = h + l;
  return dd{s, l - (s - h)};
}
inline dd dd_mul(dd a, dd b) {
  const double p = a.h * b.h;
  return dd_norm(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
inline dd dd_add(dd a, dd b) {
  const double s = a.h + b.h, t = s - a.h;
  return dd_norm(s, ((a.h - (s - t)) + (b.h - t)) + (a.l + b.l));
}
inline dd dd_div(dd a, double b) {
  const double q = a.h / b;
  return dd_norm(q, (std::fma(-q, b, a.h) + a.l) / b);
}
inline long long dd_fix62(dd a) {  // round(a 2^62), |a| <= 1
  const double s = 4611686018427387904.0;  // 2^62: both products are exact
  const double h = a.h * s, ih = std::nearbyint(h);
  return (long long)ih + (long long)std::nearbyint((h - ih) + a.l * s);
}
inline void fx_unit_roots(int n, std::vector<long long>& c, std::vector<long long>& s) {
  c.resize(n);
  s.resize(n);
  const dd twopi{6.283185307179586477, 2.449293598294706414e-16};
  for (int k = 0; k <= n / 8; ++k) {
    const dd a = dd_div(dd_mul(twopi, dd{(double)k, 0.0}), (double)n);  // n is a power of two: exact
    const dd a2 = dd_mul(a, a);
    dd tc{1.0, 0.0}, ts = a, sc = tc, ss = ts;
    for (int i = 1; i <= 11; ++i) {  // (pi/4)^24 / 24! < 2^-87
      tc = dd_div(dd_mul(tc, a2), -(double)((2 * i - 1) * (2 * i)));
      ts = dd_div(dd_mul(ts, a2), -(double)((2 * i) * (2 * i + 1)));
      sc = dd_add(sc, tc);
      ss = dd_add(ss, ts);
    }
    c[k] = dd_fix62(sc);
    s[k] = dd_fix62(ss);
  }
  for (int k = n / 8 + 1; k <= n / 4; ++k) {
    c[k] = s[n / 4 - k];
    s[k] = c[n / 4 - k];
  }
  for (int k = n / 4 + 1; k <= n / 2; ++k) {
    c[k] = -c[n / 2 - k];
    s[k] = s[n / 2 - k];
  }
  for (int k = n / 2 + 1; k < n; ++k) {
    c[k] = c[n - k];
    s[k] = -s[n - k];
  }
}
inline void fx_limbs(long long a, int& a0, int& a1) {
  a0 = (int)(unsigned)(unsigned long long)a;
  if (a0 == (-2147483647 - 1)) {  // its negative has no limb: one unit (2^-62) off instead
    a += 1;
    a0 += 1;
  }
  a1 = (int)((a - (long long)a0) >> 32);
}
// the stage-major table of BlockFFT<double, N, E>: exp(-2 pi i k / N) 2^62
template <int N, int E>
void build_fx_twiddles(int4* out, const std::vector<long long>& c, const std::vector<long long>& s) {
  using F = BlockFFT<double, N, E, 1>;
  for (int st = 1; st < F::NST; ++st) {
    const int ns = F::ns_of(st), r = F::radix(st), stride = N / (ns * r);
    for (int jm = 0; jm < ns; ++jm)
      for (int q = 1; q < r; ++q) {
        const int k = q * jm * stride;
        int4& w = out[F::tw_off(st) + (q - 1) * ns + jm];
        fx_limbs(c[k], w.x, w.y);
        fx_limbs(-s[k], w.z, w.w);
      }
  }
}

// table of the transform of type T (the FP32 one from the FP64 roots)
template <typename T, int N, int E>
void build_twiddle_table(tw_t<T>* out) {
  if constexpr (sizeof(T) == 8) {
    std::vector<long long> c, s;
    fx_unit_roots(N, c, s);
    build_fx_twiddles<N, E>(out, c, s);
  } else {
    std::vector<double> c(N), s(N);
    host_unit_roots(N, c.data(), s.data());
    build_stage_twiddles<T, N, E>(out, c.data(), s.data());
  }
}

}  // namespace r2d3c
