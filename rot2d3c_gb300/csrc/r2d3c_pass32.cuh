// Passes B and C of the FP32 path for large grids.
//
// Per launch (us), at n = 2048 / 4096 / 8192, before (one CTA per SM with
// everything held in shared memory, or staged by cp.async; at 8192 one row per
// CTA) and now: B 60 / 247 / 2660 -> 57 / 234 / 1216, C 36 / 137 / 394 -> 29 /
// 102 / 490 (the 8192^2 C pays for the pair-tiled layout that its B takes).
// B waits on its loads (planes and twiddles: 61 KB of (hi, lo) pairs a
// 4096-point transform, of which L1 keeps a fifth) and issues in 51% of the
// slots; C on its update's loads, DRAM 41% of peak.
//   Tried for B: radix 8 with 64 registers and 32 warps an SM (262 us), most of
// z1 in global memory so that L1 holds the twiddles (268).  For C: the shared
// memory carve-out at its maximum, which left L1 28 KB (134).
#pragma once

#include "r2d3c_kernels.cuh"

namespace r2d3c {

// Pass C: radix 8 (16 at n = 8192), 64 registers a thread (128), so that two
// CTAs of 512 threads share an SM.  From n = 1024 on: 12.9 us there against
// 13.2 for the best launch shape of k_passC, 101 against 135 at 4096.
template <int N>
struct LeanC32 {
  static constexpr bool OK = N >= 1024;
  using C = Cfg<float, N, 2>;
  using F = typename C::FFT;
  static constexpr int E = C::E, TPF = C::TPF;
  static constexpr int MINB = E == 8 ? 1024 / (TPF < 64 ? 64 : TPF) : 1;
  static constexpr size_t SMEM = (size_t)2 * F::SMEM_ELEMS * 8;
};
// Pass B: radix 16, 128 registers a thread, two CTAs of 256 threads (n = 4096)
// per SM.  From n = 2048 on (at 1024 radix 16 took 20.9 us, k_passB_pipe 18.9).
template <int N>
struct LeanB32 {
  static constexpr bool OK = N >= 2048;
  static constexpr int E = 16, TPF = N / E;
  using F = BlockFFT<float, N, E, 2>;
  static constexpr int MINB = 512 / (TPF < 32 ? 32 : TPF);
  static constexpr int KQ = (N / 3 + TPF) / TPF;          // elements q that hold retained kx = lane + q TPF <= N/3
  static constexpr size_t XB = (size_t)N * 8 + 16;        // exchange buffer (N float2; mirror slots 0 .. N/2)
  static constexpr size_t SMEM = XB + (size_t)2 * N * 8;  // and z1 of both rows
};
template <typename T, int N>
constexpr bool kLeanB = sizeof(T) == 4 && LeanB32<N>::OK;
template <typename T, int N>
constexpr bool kLeanC = sizeof(T) == 4 && LeanC32<N>::OK;

// One row pair: the packed spectra are formed once per retained kx, their
// mirrored halves reaching the owners of N - kx through shared memory; the
// exchanges move one component of both rows at a time through a buffer of N
// float2, and the first bracket overwrites the row pair's second plane pair,
// which only this CTA reads and which is used up by then: 96 KB a CTA at n =
// 4096.
template <int N, bool CFL, bool FULL>
__device__ __forceinline__ void passB_lean_pair(int rp, float2* tf, float2* __restrict__ pb, int kxo, const DevGrid& gd,
                                                float inv_n4, const float4* __restrict__ tw,
                                                unsigned long long* __restrict__ cfl_enc, unsigned char* smraw) {
  using T = float;
  using L = LeanB32<N>;
  using F = typename L::F;
  constexpr int E = L::E, TPF = L::TPF, KQ = L::KQ;
  float2* sm = reinterpret_cast<float2*>(smraw);
  float4* hold = reinterpret_cast<float4*>(smraw + L::XB);  // z1: (row 0, row 1)
  const int lane0 = threadIdx.x;
  const int M = gd.M;
  const size_t pl4 = (size_t)M * (N / 2);  // a plane, in float4 (two rows of one column)
  float4* P = reinterpret_cast<float4*>(tf) + (size_t)rp * M;
  // slots of the first bracket: both rows at positions q, q + 1 of this thread
  auto slot = [&](int lane, int q) -> float4* {
    const int j = lane + (q >> 1) * TPF;
    return P + (j < M ? 2 * pl4 + j : 3 * pl4 + (j - M));
  };
  // the later planes' rows into L2 while the first transforms run
  if (lane0 < 4) prefetch_l2(P + (2 + lane0) * pl4, (size_t)M);
  cpx<T> v[2][E];
#pragma unroll 1
  for (int f = 0; f < 4; ++f) {
    // addresses derived from an opaque lane index: not hoisted out of the loop
    // into registers that spill
    const int lane = opaque(lane0);
    if (f < 3) {
      const float4* pa = P + 2 * f * pl4;
      const float4* pc = pa + pl4;
      float4* mir = reinterpret_cast<float4*>(sm);  // Z[N - kx] of both rows at kx
#pragma unroll
      for (int q = 0; q < E; ++q) v[0][q] = v[1][q] = czero<T>();
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        const int k = lane + q * TPF;
        if (k < M) {
          const float4 a = __ldcg(pa + k), b = __ldcg(pc + k);
          if (k == 0) {  // Im of the kx = 0 column is ignored
            v[0][q] = mkc<T>(a.x, b.x);
            v[1][q] = mkc<T>(a.z, b.z);
          } else {
            v[0][q] = mkc<T>(a.x - b.y, a.y + b.x);
            v[1][q] = mkc<T>(a.z - b.w, a.w + b.z);
            mir[k] = make_float4(a.x + b.y, b.x - a.y, a.z + b.w, b.z - a.w);
          }
        }
      }
      fft_sync<TPF>();
#pragma unroll
      for (int q = 0; q < E; ++q) {
        if ((q + 1) * TPF <= N - N / 3) continue;  // no mirrored position
        const int k = N - (lane + q * TPF);
        if (k < M) {
          const float4 w = mir[k];
          v[0][q] = mkc<T>(w.x, w.y);
          v[1][q] = mkc<T>(w.z, w.w);
        }
      }
      fft_sync<TPF>();
    } else {
      // the forward transform is the inverse one of the conjugate, conjugated
#pragma unroll
      for (int q = 0; q < E; q += 2) {
        const float4 p = __ldcg(slot(lane, q));
        const float4 b0 = hold[lane + q * TPF], b1 = hold[lane + (q + 1) * TPF];
        v[0][q] = mkc<T>(p.x, -b0.x);
        v[1][q] = mkc<T>(p.y, -b0.y);
        v[0][q + 1] = mkc<T>(p.z, -b1.x);
        v[1][q + 1] = mkc<T>(p.w, -b1.y);
      }
    }
    F::template run<+1, true>(v, lane, sm, tw);
    if (f == 0) {
      if constexpr (CFL) cfl_max_sq<T, 2, E, TPF>(v, cfl_enc);
#pragma unroll
      for (int q = 0; q < E; ++q) hold[lane + q * TPF] = make_float4(v[0][q].x, v[0][q].y, v[1][q].x, v[1][q].y);
    } else if (f == 1) {
#pragma unroll
      for (int q = 0; q < E; q += 2) {
        const float4 a = hold[lane + q * TPF], b = hold[lane + (q + 1) * TPF];
        *slot(lane, q) = make_float4((a.x * v[0][q].y - a.y * v[0][q].x) * inv_n4,
                                                      (a.z * v[1][q].y - a.w * v[1][q].x) * inv_n4,
                                                      (b.x * v[0][q + 1].y - b.y * v[0][q + 1].x) * inv_n4,
                                                      (b.z * v[1][q + 1].y - b.w * v[1][q + 1].x) * inv_n4);
      }
    } else if (f == 2) {  // z1 is done with: its place takes the second bracket
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const float4 a = hold[lane + q * TPF];
        *reinterpret_cast<float2*>(&hold[lane + q * TPF]) =
            make_float2((a.x * v[0][q].y - a.y * v[0][q].x) * inv_n4, (a.z * v[1][q].y - a.w * v[1][q].x) * inv_n4);
      }
    }
  }
  // v holds the conjugate of W; W[N - k] goes to the owner of k
  const int lane = opaque(lane0);
  float4* mir = reinterpret_cast<float4*>(sm);
  constexpr int top = FULL ? N / 2 : N / 3;  // largest kx stored
  const size_t oplane = (size_t)gd.nh * N;
  const T h = (T)0.5;
#pragma unroll
  for (int q = 0; q < E; ++q) {
    if ((q + 1) * TPF <= N - top) continue;
    const int k = N - (lane + q * TPF);
    if (k <= top) mir[k] = make_float4(v[0][q].x, v[0][q].y, v[1][q].x, v[1][q].y);
  }
  fft_sync<TPF>();
#pragma unroll
  for (int q = 0; q < E; ++q) {
    if (q * TPF > top) continue;
    const int k = lane + q * TPF;
    if (k < kxo) {
      cpx<T> o1[2], o2[2];
      const float4 m = k == 0 ? make_float4(v[0][q].x, v[0][q].y, v[1][q].x, v[1][q].y) : mir[k];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const cpx<T> w = mkc<T>(v[t][q].x, -v[t][q].y);
        const cpx<T> u = t ? mkc<T>(m.z, -m.w) : mkc<T>(m.x, -m.y);
        o1[t] = mkc<T>((w.x + u.x) * h, (w.y - u.y) * h);
        o2[t] = mkc<T>((w.y + u.y) * h, (u.x - w.x) * h);
      }
      const size_t off = mix_idx<N, 2>(k, 2 * rp, gd.nh);
      store_rows(pb, off, o1);
      store_rows(pb + oplane, off, o2);
    }
  }
}

// LOOP: persistent CTAs, row pairs blockIdx.x, blockIdx.x + gridDim.x, ...
template <int N, bool CFL, bool FULL, bool LOOP>
__global__ void __launch_bounds__(LeanB32<N>::TPF, LeanB32<N>::MINB)
k_passB_lean(float2* tf, float2* __restrict__ pb, int kxo, DevGrid gd, float inv_n4, const float4* __restrict__ tw,
             unsigned long long* __restrict__ cfl_enc, Batch bs) {
  tf += blockIdx.y * bs.tf;
  pb += blockIdx.y * bs.pb;
  cfl_enc += blockIdx.y * kScalStride;
  extern __shared__ __align__(16) unsigned char smraw_[];
  if constexpr (LOOP) {
#pragma unroll 1
    for (int rp = blockIdx.x; rp < N / 2; rp += gridDim.x) {
      passB_lean_pair<N, CFL, FULL>(rp, tf, pb, kxo, gd, inv_n4, tw, cfl_enc, smraw_);
      fft_sync<LeanB32<N>::TPF>();  // the mirror slots are read
    }
  } else {
    passB_lean_pair<N, CFL, FULL>(blockIdx.x, tf, pb, kxo, gd, inv_n4, tw, cfl_enc, smraw_);
  }
}

// Pass C, one bracket of a column pair per CTA (blockIdx.z: 0 [psi, -k^2 psi]
// and the update of C1, 1 [psi, vz] and C2): nothing is held, so a CTA takes
// the transform's buffer only.
template <int N>
__global__ void __launch_bounds__(LeanC32<N>::TPF, LeanC32<N>::MINB)
k_passC_lean(const float2* __restrict__ pb, const float2* c1in, const float2* c2in, const float2* ps,
             const float2* vz, const float2* __restrict__ fp, const float2* __restrict__ fz, float2* c1out,
             float2* c2out, DevGrid gd, const StepCoef* __restrict__ scs, const double* __restrict__ scal, int o,
             const float4* __restrict__ tw, Batch bs, const float2* __restrict__ tau5,
             const float2* __restrict__ tau6) {
  using T = float;
  using L = LeanC32<N>;
  using F = typename L::F;
  constexpr int E = L::E, TPF = L::TPF;
  const size_t rs = blockIdx.y * bs.spec;
  const int chunk = blockIdx.z, kx0 = 2 * blockIdx.x, lane = threadIdx.x;
  R2D3C_SMEM_DECL
  cpx<T>* sm = smbase_;
  if (lane < 4) {  // the update's inputs into L2 while the transform runs
    const cpx<T>* tau = chunk ? tau6 : tau5;
    const cpx<T>* src = lane == 0 ? (chunk ? c1in : c2in) + rs : lane == 1 ? (chunk ? vz : ps) + rs
                      : lane == 2 ? (chunk ? fz : fp) + rs : tau;
    const int ncol = min(2, gd.M - kx0);
    if (src) prefetch_columns_l2<T>(src + (size_t)kx0 * N, ncol, N, gd.L);
  }
  cpx<T> v[2][E];
  {
    // lane pair (2p, 2p+1): the even lane loads column kx0's rows (2p, 2p+1),
    // the odd lane column kx0+1's; one swap gives each its own row of both
    const cpx<T>* src = pb + blockIdx.y * bs.pb + (size_t)chunk * gd.nh * N;
    const bool odd = lane & 1;
    const int kx = kx0 + (odd ? 1 : 0);
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int y = (lane + q * TPF) & ~1;
      const float4 w = __ldcg(reinterpret_cast<const float4*>(src + mix_idx<N, 2>(kx, y, gd.nh)));
      const float rx = __shfl_xor_sync(0xffffffffu, odd ? w.x : w.z, 1);
      const float ry = __shfl_xor_sync(0xffffffffu, odd ? w.y : w.w, 1);
      v[0][q] = odd ? mkc<T>(rx, ry) : mkc<T>(w.x, w.y);
      v[1][q] = odd ? mkc<T>(w.z, w.w) : mkc<T>(rx, ry);
    }
  }
  F::template run<-1>(v, lane, sm, tw);
  const StepCoef sc = scs[blockIdx.y];
  const T tmp1 = (T)(scal[blockIdx.y * kScalStride] / (double)o);  // :581
  if (chunk == 0) {  // the update reads the first bracket's columns from sm
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int q = 0; q < E; ++q) sm[t * N + lane + q * TPF] = v[t][q];
    passC_update_pairs<T, N, 2, E, TPF, 0>(sm, sm, v, lane, kx0, c1in + rs, c2in + rs, ps + rs, vz + rs, fp + rs,
                                           fz + rs, c1out + rs, c2out + rs, gd, sc, tmp1, tau5, tau6, 0);
  } else {
    passC_update_pairs<T, N, 2, E, TPF, 1>(sm, sm, v, lane, kx0, c1in + rs, c2in + rs, ps + rs, vz + rs, fp + rs,
                                           fz + rs, c1out + rs, c2out + rs, gd, sc, tmp1, tau5, tau6, 1);
  }
}

}  // namespace r2d3c
