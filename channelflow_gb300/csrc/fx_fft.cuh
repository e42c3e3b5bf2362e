// FFTs on 64-bit fixed point (fx.cuh), composite radices up to 8 in registers.
#pragma once

#include <utility>

#include "fft.cuh"
#include "fx.cuh"
#include "fx_plan.h"

// Constants of the butterflies, split as above (2^62 times the value, rounded).
namespace fxk {
constexpr long long kR = 3260954456333195553ll;   // sqrt(1/2)
constexpr long long kH = 3993837246235628775ll;   // sqrt(3)/2
constexpr long long kC1 = 1425089352415399811ll;  // cos(2 pi/5)
constexpr long long kC2 = -3730932361629093763ll; // cos(4 pi/5)
constexpr long long kS1 = 4385974038932618941ll;  // sin(2 pi/5)
constexpr long long kS2 = 2710681029835013083ll;  // sin(4 pi/5)
constexpr long long kD1 = 2875339201863983833ll, kE1 = 3605561316464170519ll;  // cos, sin(2 pi/7)
constexpr long long kD2 = -1026196679933739317ll, kE2 = 4496061421583520199ll;  // cos, sin(4 pi/7)
constexpr long long kD3 = -4154985531143938469ll, kE3 = 2000935573311439104ll;  // cos, sin(6 pi/7)
template <long long C>
__device__ __forceinline__ long long mul(long long a) {
  constexpr int l = (int)(uint32_t)((unsigned long long)C & 0xffffffffull);
  constexpr int h = (int)((C - (long long)l) >> 32);
  return fx_mulc(a, h, l);
}
template <long long C>
__device__ __forceinline__ long long mul_sum(long long a) {
  constexpr int l = (int)(uint32_t)((unsigned long long)C & 0xffffffffull);
  constexpr int h = (int)((C - (long long)l) >> 32);
  return fx_mulc_sum(a, h, l);
}
template <long long C>
__device__ __forceinline__ fxc mul(fxc a) {
  return fxc{mul<C>(a.x), mul<C>(a.y)};
}
}  // namespace fxk

// a exp(-2 pi i M / N)
template <int N, int M>
__device__ __forceinline__ fxc fx_rot(fxc a) {
  if constexpr (M == 0) {
    return a;
  } else if constexpr (4 * M == N) {
    return fxc{a.y, -a.x};
  } else if constexpr (2 * M == N) {
    return fxc{-a.x, -a.y};
  } else if constexpr (4 * M == 3 * N) {
    return fxc{-a.y, a.x};
  } else if constexpr (8 * M % N == 0) {  // odd multiples of 45 degrees
    const long long p = fxk::mul_sum<fxk::kR>(a.x + a.y), q = fxk::mul_sum<fxk::kR>(a.y - a.x);
    if constexpr (8 * M == N) return fxc{p, q};
    if constexpr (8 * M == 3 * N) return fxc{q, -p};
    if constexpr (8 * M == 5 * N) return fxc{-p, -q};
    return fxc{-q, p};
  } else {
    static_assert(6 * M == N || 3 * M == N, "sixths of a turn");
    const long long hx = (a.x + 1) >> 1, hy = (a.y + 1) >> 1, sx = fxk::mul<fxk::kH>(a.x), sy = fxk::mul<fxk::kH>(a.y);
    return 6 * M == N ? fxc{hx + sy, hy - sx} : fxc{sy - hx, -hy - sx};
  }
}

// DFTs in registers, exp(-2 pi i n k / RAD).
template <int RAD>
struct FxDft;
template <>
struct FxDft<2> {
  static __device__ __forceinline__ void run(fxc* x) {
    const fxc t = x[0];
    x[0] = fx_add(t, x[1]);
    x[1] = fx_sub(t, x[1]);
  }
};
template <>
struct FxDft<4> {
  static __device__ __forceinline__ void run(fxc* x) {
    const fxc a0 = fx_add(x[0], x[2]), a1 = fx_sub(x[0], x[2]);
    const fxc a2 = fx_add(x[1], x[3]), a3 = fx_rot<4, 1>(fx_sub(x[1], x[3]));
    x[0] = fx_add(a0, a2);
    x[2] = fx_sub(a0, a2);
    x[1] = fx_add(a1, a3);
    x[3] = fx_sub(a1, a3);
  }
};
template <>
struct FxDft<3> {
  static __device__ __forceinline__ void run(fxc* x) {
    const fxc s = fx_add(x[1], x[2]), d = fx_sub(x[1], x[2]);
    const fxc m = fxc{x[0].x - ((s.x + 1) >> 1), x[0].y - ((s.y + 1) >> 1)};
    const fxc t = fx_rot<4, 1>(fxk::mul<fxk::kH>(d));
    x[0] = fx_add(x[0], s);
    x[1] = fx_add(m, t);
    x[2] = fx_sub(m, t);
  }
};
template <>
struct FxDft<5> {
  static __device__ __forceinline__ void run(fxc* x) {
    using namespace fxk;
    const fxc a1 = fx_add(x[1], x[4]), b1 = fx_sub(x[1], x[4]);
    const fxc a2 = fx_add(x[2], x[3]), b2 = fx_sub(x[2], x[3]);
    const fxc m1 = fx_add(x[0], fx_add(fxk::mul<kC1>(a1), fxk::mul<kC2>(a2)));
    const fxc m2 = fx_add(x[0], fx_add(fxk::mul<kC2>(a1), fxk::mul<kC1>(a2)));
    const fxc t1 = fx_rot<4, 1>(fx_add(fxk::mul<kS1>(b1), fxk::mul<kS2>(b2)));
    const fxc t2 = fx_rot<4, 1>(fx_sub(fxk::mul<kS2>(b1), fxk::mul<kS1>(b2)));
    x[0] = fx_add(x[0], fx_add(a1, a2));
    x[1] = fx_add(m1, t1);
    x[4] = fx_sub(m1, t1);
    x[2] = fx_add(m2, t2);
    x[3] = fx_sub(m2, t2);
  }
};
// X_o and X_{7-o}: x_0 + sum_r cos(2 pi o r / 7) (x_r + x_{7-r}) -+ i sin(2 pi o r / 7) (x_r - x_{7-r})
template <>
struct FxDft<7> {
  template <long long D1, long long D2, long long D3, long long E1, long long E2, long long E3>
  static __device__ __forceinline__ void pair(fxc x0, const fxc* a, const fxc* b, fxc& p, fxc& m) {
    const fxc c = fx_add(fx_add(x0, fxk::mul<D1>(a[0])), fx_add(fxk::mul<D2>(a[1]), fxk::mul<D3>(a[2])));
    const fxc s = fx_rot<4, 1>(fx_add(fxk::mul<E1>(b[0]), fx_add(fxk::mul<E2>(b[1]), fxk::mul<E3>(b[2]))));
    p = fx_add(c, s);
    m = fx_sub(c, s);
  }
  static __device__ __forceinline__ void run(fxc* x) {
    using namespace fxk;
    const fxc a[3] = {fx_add(x[1], x[6]), fx_add(x[2], x[5]), fx_add(x[3], x[4])};
    const fxc b[3] = {fx_sub(x[1], x[6]), fx_sub(x[2], x[5]), fx_sub(x[3], x[4])};
    const fxc x0 = x[0];
    x[0] = fx_add(x0, fx_add(a[0], fx_add(a[1], a[2])));
    pair<kD1, kD2, kD3, kE1, kE2, kE3>(x0, a, b, x[1], x[6]);
    pair<kD2, kD3, kD1, kE2, -kE3, -kE1>(x0, a, b, x[2], x[5]);
    pair<kD3, kD1, kD2, kE3, -kE1, kE2>(x0, a, b, x[3], x[4]);
  }
};
// A B points: X[k1 + A k2] = sum_n2 exp(-2 pi i n2 k1 / (A B)) (sum_n1 x[n1 B + n2] W_A^(n1 k1)) W_B^(n2 k2).
template <int A, int B>
struct FxDft2 {
  template <int N2, int... K1>
  static __device__ __forceinline__ void column(const fxc* x, fxc* y, std::integer_sequence<int, K1...>) {
    fxc t[A] = {x[K1 * B + N2]...};
    FxDft<A>::run(t);
    ((y[K1 * B + N2] = fx_rot<A * B, (N2 * K1) % (A * B)>(t[K1])), ...);
  }
  template <int... N2>
  static __device__ __forceinline__ void columns(const fxc* x, fxc* y, std::integer_sequence<int, N2...>) {
    (column<N2>(x, y, std::make_integer_sequence<int, A>{}), ...);
  }
  static __device__ __forceinline__ void run(fxc* x) {
    fxc y[A * B];
    columns(x, y, std::make_integer_sequence<int, B>{});
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      FxDft<B>::run(y + k1 * B);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) x[k1 + A * k2] = y[k1 * B + k2];
    }
  }
};
template <> struct FxDft<6> : FxDft2<2, 3> {};
template <> struct FxDft<8> : FxDft2<2, 4> {};

// One Stockham stage over nseq sequences (fft.cuh's formulation), the length and the points before the stage known at
// compile time (CL, CN) or not (0).  swin / swout: real and imaginary parts change places on the way in / out (an inverse
// transform is a forward one between two such swaps).
template <int RAD, int CL, int CN>
__device__ __forceinline__ void fx_stage(const fxc* src, fxc* dst, int nseq, int ss, int L, int Ns,
                                         const fxtw* __restrict__ twt, bool swin, bool swout, int tid, int nthr) {
  // neighbouring lanes on neighbouring sequences: their odd pitch keeps the strided accesses of every radix on different
  // banks, and they share their twiddle factors
  const int LR = (CL ? CL : L) / RAD, NS = CN ? CN : Ns, total = nseq * LR;
  const float invq = 1.0f / nseq, invn = 1.0f / NS;
  for (int idx = tid; idx < total; idx += nthr) {
    int q, j, kq, k;
    divmod_small(idx, nseq, invq, j, q);
    if constexpr (CN > 0)
      k = j % CN;
    else
      divmod_small(j, NS, invn, kq, k);
    const fxc* sp = src + q * ss + j;
    fxc x[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) {
      x[r] = sp[r * LR];
      if (CN <= 1 && swin) x[r] = fxc{x[r].y, x[r].x};
    }
    if (NS > 1) {
#pragma unroll
      for (int r = 1; r < RAD; ++r) x[r] = fx_cmul(x[r], __ldg(twt + k * (RAD - 1) + (r - 1)));
    }
    FxDft<RAD>::run(x);
    fxc* dp = dst + q * ss + (j - k) * RAD + k;
#pragma unroll
    for (int r = 0; r < RAD; ++r) {
      if (CN * RAD == CL && swout) x[r] = fxc{x[r].y, x[r].x};
      dp[r * NS] = x[r];
    }
  }
}

// Direct DFT of a larger prime radix: the butterfly's inputs are twiddled in place, then summed per output.
__device__ inline void fx_stage_prime(int Rr, fxc* src, fxc* dst, int nseq, int ss, int L, int Ns,
                                      const fxtw* __restrict__ twt, bool swin, bool swout, int tid, int nthr) {
  const fxtw* rt = twt + Ns * (Rr - 1);
  const int LR = L / Rr;
  for (int idx = tid; idx < nseq * LR; idx += nthr) {
    const int q = idx / LR, j = idx - q * LR, k = j % Ns;
    fxc* sp = src + q * ss + j;
    for (int r = 0; r < Rr; ++r) {
      fxc x = sp[r * LR];
      if (swin) x = fxc{x.y, x.x};
      if (k != 0 && r > 0) x = fx_cmul(x, __ldg(twt + k * (Rr - 1) + (r - 1)));
      sp[r * LR] = x;
    }
    fxc* dp = dst + q * ss + (j - k) * Rr + k;
    for (int o = 0; o < Rr; ++o) {
      fxc acc = sp[0];
      int e = 0;
      for (int r = 1; r < Rr; ++r) {
        e += o;
        if (e >= Rr) e -= Rr;
        acc = fx_add(acc, fx_cmul(sp[r * LR], __ldg(rt + e)));
      }
      dp[o * Ns] = swout ? fxc{acc.y, acc.x} : acc;
    }
  }
}

// nseq sequences (stride ss) at element offset a of the block's shared memory, ping-pong with b; returns the offset of
// the result.  All threads of the block; the caller has synchronised the inputs, the result is synchronised.  Not
// inlined: the kernels share one copy of the butterflies.  ANY: lengths with a factor of 7 or a larger prime, in
// kernels of their own (in the same kernel they cost the other lengths 3%).
template <bool ANY>
__device__ __noinline__ int fx_fft(int a, int b, int nseq, int ss, int L, unsigned long long rad,
                                       const fxtw* __restrict__ tw, bool inv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, nthr = blockDim.x;
  fxc* const base = reinterpret_cast<fxc*>(smem_raw);
  auto turn = [&](int R, int Ns) {  // after a stage
    tw += fx_stage_tw(R, Ns);
    __syncthreads();
    const int t = a;
    a = b;
    b = t;
  };
  if constexpr (!ANY) {
#define FX_STAGE(r, l, n) \
  fx_stage<r, l, n>(base + a, base + b, nseq, ss, l, n, tw, inv, inv, tid, nthr); \
  turn(r, n);
    switch (L) {  // the lengths of the usual grids, indices known at compile time (the radices of fx_plan)
      case 32: FX_STAGE(8, 32, 1) FX_STAGE(4, 32, 8) return a;
      case 48: FX_STAGE(8, 48, 1) FX_STAGE(6, 48, 8) return a;
      case 64: FX_STAGE(8, 64, 1) FX_STAGE(8, 64, 8) return a;
      case 96: FX_STAGE(6, 96, 1) FX_STAGE(4, 96, 6) FX_STAGE(4, 96, 24) return a;
      case 128: FX_STAGE(8, 128, 1) FX_STAGE(4, 128, 8) FX_STAGE(4, 128, 32) return a;
    }
#undef FX_STAGE
  }
  for (int Ns = 1; Ns < L; rad >>= 8) {
    const int R = (int)(rad & 255);
    const bool in = inv && Ns == 1, out = inv && Ns * R == L;
    switch (R) {
#define FX_CASE(r) \
  case r: fx_stage<r, 0, 0>(base + a, base + b, nseq, ss, L, Ns, tw, in, out, tid, nthr); break;
      FX_CASE(2) FX_CASE(3) FX_CASE(4) FX_CASE(5) FX_CASE(6) FX_CASE(8)
      default:
        if constexpr (ANY) {
          if (R == 7)
            fx_stage<7, 0, 0>(base + a, base + b, nseq, ss, L, Ns, tw, in, out, tid, nthr);
          else
            fx_stage_prime(R, base + a, base + b, nseq, ss, L, Ns, tw, in, out, tid, nthr);
        }
#undef FX_CASE
    }
    turn(R, Ns);
    Ns *= R;
  }
  return a;
}
