// The three passes of the FP64 path (see r2d3c_kernels.cuh): one kx column or
// row per transform group, the transforms in block fixed point
// (r2d3c_fx.cuh), everything around them kept off the FP64 pipe (2 lanes per
// SM and clock) where integers can do it.
//
// Per launch at 4096^2 (us; FP64 arithmetic, the transforms alone in fixed
// point, these kernels): A 2556, 841, 381; B 5227, 1697, 942; C 1179, 594,
// 270.  What bounds them now (ncu): A and B the issue of integer instructions
// (52-57% of the slots, ALU pipe 55-56%), C the FP64 pipe of the update (70%)
// and the latency of its loads; DRAM 11-33% of peak.
#pragma once

#include "r2d3c_kernels.cuh"

namespace r2d3c {

// 64 registers a thread: two 512-thread CTAs (four of 256) share an SM, so
// that one's integer stages run beside the other's loads and FP64 operations
// (n = 8192 holds 16 elements a thread: one CTA).  The mixed planes are
// pair-tiled (mix_idx<N, 2>): a column writes and a row reads whole 32-byte
// sectors.
template <int N>
struct P64 {
  using C = Cfg<double, N, 1>;
  using F = typename C::FFT;
  static constexpr int E = C::E, TPF = C::TPF;
  static constexpr int MINB = E == 8 ? 1024 / C::THREADS : 1;
  // no position lane + q TPF of element q is retained (|k| <= N/3)
  static __host__ __device__ constexpr bool dead(int q) { return q * TPF > N / 3 && (q + 1) * TPF <= N - N / 3; }
};

// --------------------------------------------------------------------------
// pass A: the derivative multipliers k and -k (kx^2 + ky^2) are whole numbers
// below 2^32 (n <= 4096), so they join the conversion to fixed point as an
// integer factor of the mantissa (exact but for the last of 62 bits).  The
// results are converted by the FP64 pipe, which is idle otherwise: 364 ->
// 285 instructions a point, 488 -> 440 us at 4096^2.
// --------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(P64<N>::C::THREADS, P64<N>::MINB)
k_passA64(const double2* __restrict__ ps, const double2* __restrict__ vz, double2* __restrict__ tf, DevGrid gd,
          const int4* __restrict__ tw, Batch bs) {
  using P = P64<N>;
  using F = typename P::F;
  using T = double;
  constexpr int E = P::E, TPF = P::TPF;
  ps += blockIdx.y * bs.spec;
  vz += blockIdx.y * bs.spec;
  tf += blockIdx.y * bs.tf;
  R2D3C_SMEM_DECL
  const int g = threadIdx.x / TPF, lane = threadIdx.x % TPF;
  double2* sm = smbase_ + (size_t)g * F::SMEM_ELEMS;
  // groups per CTA and field chunks are launch-time choices, as in k_passA
  const int kx = blockIdx.x * (blockDim.x / TPF) + g;
  const int fpc = 6 / gridDim.z, f0 = blockIdx.z * fpc;
  const size_t plane = (size_t)gd.M * N;
#pragma unroll 1
  for (int f = f0; f < f0 + fpc; ++f) {
    // psi for fields 0-3, vz for fields 4-5; the column is re-read for every
    // field, from L2
    const double2* sp = (f < 4 ? ps : vz) + (size_t)kx * N;
    const bool lap = f == 2 || f == 3;
    // the multiplier of element q, (0,k)*(x,y) = (-k*y, k*x): derivk2 dir 1 (k
    // = kx) / dir 2 (k = ky); laplak2: -ka2*a
    auto mult = [&](int q) -> int {
      const int ky = ky_of(lane + q * TPF, N);
      return (f & 1) ? ky : kx;
    };
    auto absmult = [&](int q) -> unsigned {
      const int ky = ky_of(lane + q * TPF, N), k = mult(q);
      const unsigned a = (unsigned)(k < 0 ? -k : k);
      return (N < 8192 && lap) ? a * (unsigned)(kx * kx + ky * ky) : a;
    };
    double2 x[E];
    unsigned mh = 0, lo = 0;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      if (P::dead(q)) continue;
      const int ky = ky_of(lane + q * TPF, N), k2 = kx * kx + ky * ky;
      const bool in = kx < gd.M && (ky <= gd.L && -ky <= gd.L) && k2 <= gd.kmaxi;
      x[q] = in ? __ldcg(sp + lane + q * TPF) : czero<T>();
      if (mult(q) == 0) {  // 0 times a finite value: no part in the vector's scale
        if (fx_upper(x[q].x) < 0x7ff00000u) x[q].x = 0.0;
        if (fx_upper(x[q].y) < 0x7ff00000u) x[q].y = 0.0;
      }
      if constexpr (N >= 8192) {  // k (kx^2 + ky^2) may exceed 32 bits: the Laplacian first
        if (lap) x[q] = mkc<T>(x[q].x * (double)k2, x[q].y * (double)k2);
      }
      mh = max(mh, max(fx_upper(x[q].x), fx_upper(x[q].y)));
      lo |= __double2loint(x[q].x) | __double2loint(x[q].y);
    }
    mh = fx_any(mh, lo);
    const int ew = F::warp_base(mh);
    float mx = 0.f, l1 = 0.f, l2 = 0.f;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      if (P::dead(q)) continue;
      // (outside the retained disc x = 0: the factor's wrap-around is harmless)
      const float a = fx_mag(max(fx_upper(x[q].x), fx_upper(x[q].y)), ew) * __uint2float_ru(absmult(q));
      mx = fmaxf(mx, a);
      l1 += a;
      l2 = fmaf(a, a, l2);
    }
    int e, s;
    F::combine(ew, mh ? mx : 0.f, mh ? l1 : 0.f, mh ? l2 : 0.f, lane, reinterpret_cast<int4*>(sm + F::RED), e, s);
    const int c = e + 62 - s;
    const bool sub = fx_sub(e);
    fx u[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
      if (P::dead(q)) {
        u[q] = fx{0, 0};
        continue;
      }
      const unsigned k = absmult(q);
      const int z = __clz(k);
      const unsigned kn = k << (z & 31);
      const int sg = (mult(q) >> 31) ^ (lap ? -1 : 0), cz = c - 32 + z;
      // the inverse transform takes (re, im) = (-K y, K x) exchanged
      u[q] = sub ? fx{fx_from_mul<true>(x[q].x, kn, sg, cz), fx_from_mul<true>(x[q].y, kn, ~sg, cz)}
                 : fx{fx_from_mul(x[q].x, kn, sg, cz), fx_from_mul(x[q].y, kn, ~sg, cz)};
    }
    F::run_fx(u, lane, sm, tw);
    const FxOut out(e, F::out_exp(e, s));
    if (kx < gd.M) {
      double2* dst = tf + (size_t)f * plane + mix_idx<N, 2>(kx, lane, gd.M);
#pragma unroll
      for (int q = 0; q < E; ++q) dst[(size_t)q * TPF * gd.M] = mkc<T>(out.pipe(u[q].y), out.pipe(u[q].x));
    }
  }
}

// --------------------------------------------------------------------------
// pass B.  A row's three packed spectra, brackets and forward transform by
// one group.
//   - The packed spectrum Z = A + i B of two planes is formed in fixed point:
//     a thread converts A and B once for each of its retained kx and adds
//     them to Z[kx] and to Z[N - kx], which goes to its owner through shared
//     memory.
//   - The physical values stay in fixed point (their scales known per
//     transform); only the products are FP64.
//   - The exchanges go through a buffer of N 8-byte values, one component at
//     a time, and the first bracket waits in global memory: with z1 held in
//     shared memory a 4096-point row takes 97 KB, so that two CTAs share an SM
//     (one CTA of 128 registers a thread: 1640 us).
//   - The Hermitian split of the result adds in fixed point and converts only
//     the retained kx.
// --------------------------------------------------------------------------
template <int N>
struct PassB64 {
  using P = P64<N>;
  using F = typename P::F;
  static constexpr int E = P::E, TPF = P::TPF;
  static constexpr int KQ = (N / 3 + TPF) / TPF;  // elements q that hold retained kx = lane + q TPF <= N/3
  // per group: the exchange buffer (mirror slots: re of kx at kx, im at N/2 +
  // 1 + kx), the scale's reduction, z1
  static constexpr size_t XB = (size_t)(N + 8) * 8;
  static constexpr size_t RED = (size_t)(F::WARPS > 0 ? F::WARPS : 1) * (F::L2 ? 32 : 16);  // (combine2's)
  static constexpr size_t GROUP = XB + RED + (size_t)N * 16;
  static constexpr int MIRROR = N / 2 + 1;

  // One packed inverse transform: u is the physical row pair in fixed point,
  // exchanged (u.y + i u.x) 2^k; e = 0x7ff where a value is not finite.
  static __device__ __forceinline__ void inverse(const double2* pa, const double2* pb, int y,
                                                 int M, int lane, unsigned char* sm, const int4* __restrict__ tw,
                                                 fx (&u)[E], int& e, int& k) {
    double2 a[KQ], b[KQ];
    unsigned mh = 0, lo = 0;
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      const int kx = lane + q * TPF;
      const size_t i = mix_idx<N, 2>(kx < M ? kx : 0, y, M);
      a[q] = kx < M ? __ldcg(pa + i) : make_double2(0.0, 0.0);
      b[q] = kx < M ? __ldcg(pb + i) : make_double2(0.0, 0.0);
      if (kx == 0) a[q].y = b[q].y = 0.0;  // Im of the kx = 0 column is ignored
      mh = max(mh, max(max(fx_upper(a[q].x), fx_upper(a[q].y)), max(fx_upper(b[q].x), fx_upper(b[q].y))));
      lo |= __double2loint(a[q].x) | __double2loint(a[q].y) | __double2loint(b[q].x) | __double2loint(b[q].y);
    }
    mh = fx_any(mh, lo);
    const int ew = F::warp_base(mh);
    float mx = 0.f, l1 = 0.f, l2 = 0.f;
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      // |Z| <= |A| + |B|; |Z[kx]|^2 + |Z[N - kx]|^2 = 2 (|A|^2 + |B|^2)
      const float ma = fx_mag(max(fx_upper(a[q].x), fx_upper(a[q].y)), ew);
      const float mb = fx_mag(max(fx_upper(b[q].x), fx_upper(b[q].y)), ew);
      const float p = ma + mb, w = lane + q * TPF == 0 ? 1.f : 2.f;  // Z[kx] and Z[N - kx]
      mx = fmaxf(mx, p);
      l1 = fmaf(w, p, l1);
      l2 = fmaf(w, fmaf(ma, ma, mb * mb), l2);
    }
    int s;
    F::combine(ew, mh ? mx : 0.f, mh ? l1 : 0.f, mh ? l2 : 0.f, lane, reinterpret_cast<int4*>(sm + XB), e, s);
    k = F::out_exp(e, s);
    const int c = e + 62 - s;
    const bool sub = fx_sub(e);
    long long* mir = reinterpret_cast<long long*>(sm);
#pragma unroll
    for (int q = 0; q < E; ++q) u[q] = fx{0, 0};
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      const int kx = lane + q * TPF;
      long long ax, ay, bx, by;
      if (!sub) {
        ax = fx_from(a[q].x, c), ay = fx_from(a[q].y, c);
        bx = fx_from(b[q].x, c), by = fx_from(b[q].y, c);
      } else {
        ax = fx_from<true>(a[q].x, c), ay = fx_from<true>(a[q].y, c);
        bx = fx_from<true>(b[q].x, c), by = fx_from<true>(b[q].y, c);
      }
      u[q] = fx{ay + bx, ax - by};
      if (kx >= 1 && kx < M) {
        mir[kx] = bx - ay;
        mir[MIRROR + kx] = ax + by;
      }
    }
    fft_sync<TPF>();
#pragma unroll
    for (int q = 0; q < E; ++q) {
      if ((q + 1) * TPF <= N - N / 3) continue;  // no mirrored position
      const int kx = N - (lane + q * TPF);
      if (kx < M) u[q] = fx{mir[kx], mir[MIRROR + kx]};
    }
    fft_sync<TPF>();
    F::template run_fx<true>(u, lane, sm, tw);
  }

  // The brackets' row (p1 2^k1 and p2 2^k2 of this thread's positions, NaN
  // where not finite) to mixed space: the forward transform of p1 + i p2,
  // split, times inv_n4 = 2^-4 log2 N, for kx < kxo (FULL: up to N/2).
  template <bool FULL>
  static __device__ __forceinline__ void forward(const double (&p1)[E], const double (&p2)[E], int k1, int k2, int y,
                                                 int kxo, int nh, int lane, unsigned char* sm,
                                                 const int4* __restrict__ tw, double2* __restrict__ o1,
                                                 double2* __restrict__ o2, bool store) {
    // the two brackets scaled apart: with one scale the smaller one's kx = 0
    // modes, which the split does not mix, took the larger one's rounding.
    // (A product of fixed-point values is 0 or at least 1: no subnormals.)
    unsigned m1 = 0, m2 = 0;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      m1 = max(m1, fx_upper(p1[q]));
      m2 = max(m2, fx_upper(p2[q]));
    }
    const int w1 = F::warp_base(m1), w2 = F::warp_base(m2);
    float s1 = 0.f, s2 = 0.f, t1 = 0.f, t2 = 0.f;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const float a = fx_mag(fx_upper(p1[q]), w1), b = fx_mag(fx_upper(p2[q]), w2);
      s1 += a;
      s2 += b;
      t1 = fmaf(a, a, t1);
      t2 = fmaf(b, b, t2);
    }
    int e1, e2, s;
    F::combine2(w1, w2, m1 ? s1 : 0.f, m2 ? s2 : 0.f, m1 ? t1 : 0.f, m2 ? t2 : 0.f, lane,
                reinterpret_cast<int4*>(sm + XB), e1, e2, s);
    const int c1 = e1 + 62 - s, c2 = e2 + 62 - s;
    fx u[E];
#pragma unroll
    for (int q = 0; q < E; ++q) u[q] = fx{fx_from(p1[q], c1), fx_from(p2[q], c2)};
    F::template run_fx<true>(u, lane, sm, tw);
    // mirrored values to the owner of kx (W[N - kx]; kx = 0: its own)
    long long* mir = reinterpret_cast<long long*>(sm);
    constexpr int top = FULL ? N / 2 : N / 3;  // largest kx stored
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int kx = N - (lane + q * TPF);
      if ((q + 1) * TPF <= N - top) continue;
      if (kx <= top) {
        mir[kx] = u[q].x;
        mir[MIRROR + kx] = u[q].y;
      }
    }
    fft_sync<TPF>();
    // (-1: the halves of the split)
    const bool bad = e1 == 0x7ff || e2 == 0x7ff;
    const FxOut out1(bad ? 0x7ff : e1, F::out_exp(e1, s) + k1 - 4 * F::LOGN - 1);
    const FxOut out2(bad ? 0x7ff : e2, F::out_exp(e2, s) + k2 - 4 * F::LOGN - 1);
#pragma unroll
    for (int q = 0; q < E; ++q) {
      if (q * TPF > top) continue;
      const int kx = lane + q * TPF;
      if (store && kx < kxo) {
        const fx w = u[q];
        const fx m = kx == 0 ? w : fx{mir[kx], mir[MIRROR + kx]};
        const size_t i = mix_idx<N, 2>(kx, y, nh);
        o1[i] = make_double2(out1(w.x + m.x), out1(w.y - m.y));
        o2[i] = make_double2(out2(w.y + m.y), out2(m.x - w.x));
      }
    }
    fft_sync<TPF>();  // the buffer is free for the next row
  }

  // CFL maximum of |grad psi|^2 over z1 = u 2^k (CFL_condition,
  // pseudospec2D_Rot2D3C.f90:867-874), folded into the run's encoded maximum
  static __device__ __forceinline__ void cfl_max(const fx (&u)[E], int e, int k, bool on, unsigned long long* enc) {
    double m = 0.0;
    if (on) {
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const double x = __ll2double_rn(u[q].x), y = __ll2double_rn(u[q].y);
        m = fmax(m, x * x + y * y);
      }
      m = e == 0x7ff ? 0.0 : scalbn(m, 2 * k);
    }
    m = group_max<TPF>(m);
    if (on && group_first<TPF>()) atomicMax(enc, enc_ordered(m));
  }
  // a transform's value (held exchanged) in FP64, without its 2^k
  static __device__ __forceinline__ double2 value(fx u) {
    return make_double2(__ll2double_rn(u.y), __ll2double_rn(u.x));
  }
  // z1.re z.im - z1.im z.re
  static __device__ __forceinline__ double bracket(double2 a, fx u, bool finite) {
    const double2 z = value(u);
    const double p = fma(a.x, z.y, -(a.y * z.x));
    return finite ? p : __hiloint2double(0x7ff80000, 0);
  }
};

// One row per group.  The first bracket overwrites the row's second plane pair,
// which only this row reads and which is in fixed point by then (4 M doubles,
// N <= 3 M).  (A loop over rows by persistent CTAs spilled 400 bytes a thread.)
template <int N, bool CFL, bool FULL>
__global__ void __launch_bounds__(P64<N>::C::THREADS, P64<N>::MINB)
k_passB64(double2* tf, double2* __restrict__ pb, int kxo, DevGrid gd, const int4* __restrict__ tw,
          unsigned long long* __restrict__ cfl_enc, Batch bs) {
  using B = PassB64<N>;
  constexpr int E = B::E, TPF = B::TPF;
  extern __shared__ __align__(16) unsigned char smraw_[];
  const int g = threadIdx.x / TPF, lane0 = threadIdx.x % TPF;
  unsigned char* sm = smraw_ + (size_t)g * B::GROUP;
  double2* hold = reinterpret_cast<double2*>(sm + B::XB + B::RED);
  tf += blockIdx.y * bs.tf;
  pb += blockIdx.y * bs.pb;
  cfl_enc += blockIdx.y * kScalStride;
  const size_t plane = (size_t)gd.M * N, oplane = (size_t)gd.nh * N;
  int y = blockIdx.x * (blockDim.x / TPF) + g;
  const bool ok = y < N;
  if (!ok) y = 0;  // surplus groups compute row 0 and store nothing
  // slots of the first bracket: values q, q + 1 of this thread
  auto slot = [&](int lane, int q) -> double2* {
    const int j = lane + (q >> 1) * TPF;
    return tf + (size_t)(j < gd.M ? 2 : 3) * plane + mix_idx<N, 2>(j < gd.M ? j : j - gd.M, y, gd.M);
  };
  int e1 = 0, k1 = 0, kb1 = 0, kb2 = 0;
  // the later planes' rows (both of the pair's) into L2 while the first
  // transform runs
  if (lane0 < 4 && !(y & 1)) prefetch_l2(tf + (size_t)(2 + lane0) * plane + (size_t)(y >> 1) * gd.M * 2, (size_t)2 * gd.M);
#pragma unroll 1
  for (int f = 0; f < 3; ++f) {
    // the transform's addresses are derived from an opaque lane index every
    // time, not hoisted out of the loop into registers that spill
    const int lane = opaque(lane0);
    fx u[E];
    int e, k;
    B::inverse(tf + (size_t)(2 * f) * plane, tf + (size_t)(2 * f + 1) * plane, y, gd.M, lane, sm, tw, u, e, k);
    if (f == 0) {
      if constexpr (CFL) B::cfl_max(u, e, k, ok, cfl_enc);
      e1 = e;
      k1 = k;
#pragma unroll
      for (int q = 0; q < E; ++q) hold[lane + q * TPF] = B::value(u[q]);
    } else {
      const bool fin = e1 != 0x7ff && e != 0x7ff;
      if (f == 1) {
        kb1 = k1 + k;
#pragma unroll
        for (int q = 0; q < E; q += 2) {
          const double2 p = make_double2(B::bracket(hold[lane + q * TPF], u[q], fin),
                                         B::bracket(hold[lane + (q + 1) * TPF], u[q + 1], fin));
          if (ok) *slot(lane, q) = p;
        }
      } else {  // z1 is done with: its place takes the second bracket
        kb2 = k1 + k;
#pragma unroll
        for (int q = 0; q < E; ++q) {
          double2* h = &hold[lane + q * TPF];
          h->x = B::bracket(*h, u[q], fin);
        }
      }
    }
  }
  const int lane = opaque(lane0);
  double p1[E], p2[E];
#pragma unroll
  for (int q = 0; q < E; q += 2) {
    const double2 p = __ldcg(slot(lane, q));
    p1[q] = p.x;
    p1[q + 1] = p.y;
  }
#pragma unroll
  for (int q = 0; q < E; ++q) p2[q] = hold[lane + q * TPF].x;
  B::template forward<FULL>(p1, p2, kb1, kb2, y, kxo, gd.nh, lane, sm, tw, pb, pb + oplane, ok);
}

// small grids: the three inverse transforms of a row side by side in three
// groups of one CTA (k_passB_split); the same values, so the same bits
template <int N>
struct SplitB64 {
  using B = PassB64<N>;
  static constexpr int THREADS = 3 * B::TPF;
  static constexpr bool OK = THREADS <= 384;
  // per group: exchange buffer and reduction; the three rows; their exponents
  static constexpr size_t SMEM = 3 * (B::XB + B::RED) + (size_t)3 * N * 16 + 3 * 16;
};
template <int N, bool CFL>
__global__ void __launch_bounds__(SplitB64<N>::THREADS)
k_passB64_split(const double2* __restrict__ tf, double2* __restrict__ pb, int kxo, DevGrid gd,
                const int4* __restrict__ tw, unsigned long long* __restrict__ cfl_enc, Batch bs) {
  using B = PassB64<N>;
  constexpr int E = B::E, TPF = B::TPF;
  extern __shared__ __align__(16) unsigned char smraw_[];
  const int j = threadIdx.x / TPF, lane = threadIdx.x % TPF;
  unsigned char* sm = smraw_ + (size_t)j * (B::XB + B::RED);
  fx* res = reinterpret_cast<fx*>(smraw_ + 3 * (B::XB + B::RED));  // [pair j][x]
  int2* ek = reinterpret_cast<int2*>(res + 3 * N);
  tf += blockIdx.y * bs.tf;
  pb += blockIdx.y * bs.pb;
  cfl_enc += blockIdx.y * kScalStride;
  const size_t plane = (size_t)gd.M * N;
  fx u[E];
  int e, k;
  B::inverse(tf + (size_t)(2 * j) * plane, tf + (size_t)(2 * j + 1) * plane, blockIdx.x, gd.M, lane, sm, tw, u, e, k);
  if constexpr (CFL) B::cfl_max(u, e, k, j == 0, cfl_enc);
#pragma unroll
  for (int q = 0; q < E; ++q) res[(size_t)j * N + lane + q * TPF] = u[q];
  if (lane == 0) ek[j] = make_int2(e, k);
  __syncthreads();
  const int2 s1 = ek[0], s2 = ek[1], s3 = ek[2];
  const bool f2 = s1.x != 0x7ff && s2.x != 0x7ff, f3 = s1.x != 0x7ff && s3.x != 0x7ff;
  double p1[E], p2[E];
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const int x = lane + q * TPF;
    const double2 z1 = B::value(res[x]);
    p1[q] = B::bracket(z1, res[N + x], f2);
    p2[q] = B::bracket(z1, res[2 * N + x], f3);
  }
  // every group runs the forward transform (their barriers are uniform), the first stores
  B::template forward<false>(p1, p2, s1.y + s2.y, s1.y + s3.y, blockIdx.x, kxo, gd.nh, lane, sm, tw, pb,
                             pb + (size_t)gd.nh * N, j == 0);
}

// --------------------------------------------------------------------------
// pass C: the coefficients of the update that depend only on the wavenumber,
// laid out once per parameter set (k_rk_table): per retained (kx, |ky|), row
// stride L + 1, the dissipation rates nu k^2nn + hnu k^-2mm of both fields
// and 1/k^2 (and 2 Omega |ky| per |ky|).  In the update itself they took
// some 20 of its 36 FP64 operations per element and field.
// --------------------------------------------------------------------------
struct RkTab {
  const double *d1, *d2;  // [run][M][L+1]
  const double* ik2;      // [M][L+1]
  const double* wk;       // [run][L+1]
  size_t run;             // M (L+1)
};

static __global__ void k_rk_table(double* d1, double* d2, double* ik2, double* wk, DevGrid gd,
                                  const StepCoef* __restrict__ scs) {
  const StepCoef sc = scs[blockIdx.y];
  const size_t w = (size_t)gd.L + 1, total = (size_t)gd.M * w;
  d1 += blockIdx.y * total;
  d2 += blockIdx.y * total;
  wk += blockIdx.y * w;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int kx = (int)(i / w), ky = (int)(i % w);
    const double ka2 = (double)(kx * kx + ky * ky);
    const double inv = 1.0 / ka2;
    d1[i] = sc.nu * powi(ka2, sc.nn) + sc.hnu * powi(inv, sc.mm);
    d2[i] = sc.nuv * powi(ka2, sc.nnv) + sc.hnuv * powi(inv, sc.mmv);
    if (blockIdx.y == 0) ik2[i] = inv;
    if (i < w) wk[i] = sc.w2 * (double)ky;
  }
}

// Each CTA transforms one bracket of its columns (blockIdx.z: 0 [psi, -k^2
// psi], 1 [psi, vz]) and updates the field it drives: C1 needs the first
// bracket and C2's input, C2 the second and C1's input (see k_passC).
template <int N>
constexpr size_t kPassC64Group = P64<N>::F::SMEM_BYTES + 16;  // per group: transform, dt/o
template <int N>
__global__ void __launch_bounds__(P64<N>::C::THREADS, P64<N>::MINB)
k_passC64(const double2* __restrict__ pb, const double2* c1in, const double2* c2in, const double2* ps,
          const double2* vz, const double2* __restrict__ fp, const double2* __restrict__ fz, double2* c1out,
          double2* c2out, DevGrid gd, RkTab tab, const double* __restrict__ scal, int o, const int4* __restrict__ tw,
          Batch bs, const double2* __restrict__ tau5, const double2* __restrict__ tau6) {
  using P = P64<N>;
  using F = typename P::F;
  using T = double;
  constexpr int E = P::E, TPF = P::TPF;
  const bool second = blockIdx.z != 0;
  const size_t rs = blockIdx.y * bs.spec;
  R2D3C_SMEM_DECL
  const int g = threadIdx.x / TPF, lane = threadIdx.x % TPF;
  double2* sm = smbase_ + (size_t)g * (kPassC64Group<N> / 16);
  const int kx = blockIdx.x * (blockDim.x / TPF) + g;  // groups per CTA: a launch-time choice
  const bool ok = kx < gd.M;
  const size_t col = (size_t)(ok ? kx : 0) * N;
  const double2* other = (second ? c1in : c2in) + rs + col;  // the Coriolis term's field
  const double2* base = (second ? vz : ps) + rs + col;
  const double2* force = (second ? fz : fp) + rs + col;
  const double2* tau = second ? tau6 : tau5;
  double2* out = (second ? c2out : c1out) + rs + col;
  // dt/o (:581), divided by one thread
  double* tsh = reinterpret_cast<double*>(sm + F::SMEM_ELEMS);
  if (lane == 0) *tsh = scal[blockIdx.y * kScalStride] / (double)o;
  // the update's inputs into L2 while the transform runs
  if (lane < 4 && ok) {
    const double2* src = lane == 0 ? other : lane == 1 ? base : lane == 2 ? force : (tau ? tau + col : nullptr);
    if (src) prefetch_columns_l2<double>(src, 1, N, gd.L);
  }
  {
    double2 v[E];
    const double2* src = pb + blockIdx.y * bs.pb + (second ? (size_t)gd.nh * N : 0) + mix_idx<N, 2>(ok ? kx : 0, lane, gd.nh);
#pragma unroll
    for (int q = 0; q < E; ++q) v[q] = __ldcg(src + (size_t)q * TPF * gd.nh);
    int e, s;
    F::scale(v, lane, reinterpret_cast<int4*>(sm + F::RED), e, s);
    fx u[E];
    F::template from<false>(v, e, e + 62 - s, u);
    F::run_fx(u, lane, sm, tw);
    // through shared memory (every thread reads only what it wrote): the
    // registers are the update's
    const FxOut val(e, F::out_exp(e, s));
#pragma unroll
    for (int q = 0; q < E; ++q)
      if (!P::dead(q)) sm[lane + q * TPF] = mkc<T>(val(u[q].x), val(u[q].y));
  }
  if (!ok) return;
  const double t = *tsh;  // (written before the transform's barriers)
  const size_t tr = (size_t)kx * (gd.L + 1);
  const double* dt = (second ? tab.d2 : tab.d1) + blockIdx.y * tab.run + tr;
  const double* ik2t = tab.ik2 + tr;
  const double* wk = tab.wk + blockIdx.y * (size_t)(gd.L + 1);
  // the elements with retained rows, two at a time with their loads in flight
  // together
  constexpr int RB = 2, LO = PassB64<N>::KQ, LIVE = 2 * LO;
  static_assert(LIVE <= E && LIVE % RB == 0, "retained rows at both ends");
#pragma unroll 1
  for (int i0 = 0; i0 < LIVE; i0 += RB) {
    double2 a[RB], p[RB], f[RB];
    double d[RB], i2[RB], w[RB];
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int q = i0 + b < LO ? i0 + b : i0 + b + E - LIVE;
      const int j = lane + q * TPF, ky = ky_of(j, N), k2 = kx * kx + ky * ky, ay = ky < 0 ? -ky : ky;
      if (ay <= gd.L && k2 <= gd.kmaxi && k2 >= 1) {
        a[b] = __ldcg(other + j);
        p[b] = __ldcg(base + j);
        f[b] = __ldcg(force + j);
        d[b] = dt[ay];
        w[b] = wk[ay];
        if (!second) i2[b] = ik2t[ay];
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int q = i0 + b < LO ? i0 + b : i0 + b + E - LIVE;
      const int j = lane + q * TPF, ky = ky_of(j, N), k2 = kx * kx + ky * ky, ay = ky < 0 ? -ky : ky;
      if (ay > gd.L) continue;
      double2 r = czero<T>();
      if (k2 <= gd.kmaxi && k2 >= 1) {  // ka2 <= kmax .and. ka2 > tiny (:580)
        double2 c = sm[j];
        if (tau) {  // learned subgrid tendency of the bracket
          const double2 u = tau[col + j];
          c = mkc<T>(c.x + u.x, c.y + u.y);
        }
        const double wy = ky < 0 ? -w[b] : w[b];  // 2 Omega ky
        const double r3 = recip(fma(d[b], t, 1.0));
        double ux, uy;  // (:583-592)
        if (second) {
          ux = fma(-wy, a[b].y, c.x) + f[b].x;
          uy = fma(wy, a[b].x, c.y) + f[b].y;
        } else {
          ux = fma(fma(-wy, a[b].y, -c.x), i2[b], f[b].x);
          uy = fma(fma(wy, a[b].x, -c.y), i2[b], f[b].y);
        }
        r = mkc<T>(fma(ux, t, p[b].x) * r3, fma(uy, t, p[b].y) * r3);
      }
      out[j] = r;
    }
  }
}

}  // namespace r2d3c
