// 64-bit fixed-point FFTs for the FP64 path.
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition, but a 64-bit integer addition
// (IADD3 pair) in about 2 and a 32 x 32 -> 64 bit multiply-add (IMAD.WIDE) in about 5 (measured with a
// throughput probe).  An FFT is mostly additions, so the FP64 path's transforms run on integers: a sequence is
// scaled by one power of two such that the sum of the magnitudes of its elements stays below 2^61, which bounds
// every intermediate value of the transform, and rounded to integers.  Its rounding errors are a few units of
// 2^-61 of that sum, below those of the same FFT in FP64 (whose units are 2^-53 of the local values).
//
// Twiddle factors are fixed-point too: c = (h 2^32 + l) 2^-62 with signed 32-bit h, l.  A complex product with
// components a = ah 2^32 + al (al signed) sums the cross terms ah l + al h of both real products in one 64-bit
// accumulator, drops al l (below one unit) and takes six IMAD.WIDE per component.
#pragma once

#include "common.cuh"
#include "fft.cuh"

struct alignas(16) fxc {
  long long x, y;
};

// One twiddle factor: x = (x 2^32 + y) 2^-62 + i (z 2^32 + w) 2^-62.
typedef int4 fxtw;

__device__ __forceinline__ fxc fx_add(fxc a, fxc b) { return fxc{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fxc fx_sub(fxc a, fxc b) { return fxc{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ fxc fx_muli(fxc a, int sign) {  // sign * i * a
  return sign < 0 ? fxc{a.y, -a.x} : fxc{-a.y, a.x};
}
__device__ __forceinline__ long long fx_mw(int a, int b, long long c) { return (long long)a * b + c; }

// a w (sign < 0) or a conj(w) (sign > 0); |a.x| + |a.y| <= 2^61.
__device__ __forceinline__ fxc fx_cmul(fxc a, fxtw w, int sign) {
  const int xh = w.x, xl = w.y;
  const int yh = sign > 0 ? -w.z : w.z, yl = sign > 0 ? -w.w : w.w;
  const int nh = sign > 0 ? w.z : -w.z, nl = sign > 0 ? w.w : -w.w;
  const int al = (int)a.x, bl = (int)a.y;
  const int ah = (int)(a.x >> 32) + (int)((unsigned)al >> 31), bh = (int)(a.y >> 32) + (int)((unsigned)bl >> 31);
  const int a4 = ah << 2, b4 = bh << 2;
  const long long half = 1ll << 29;
  const long long mx = fx_mw(bl, nh, fx_mw(bh, nl, fx_mw(al, xh, fx_mw(ah, xl, half))));
  const long long my = fx_mw(al, yh, fx_mw(ah, yl, fx_mw(bl, xh, fx_mw(bh, xl, half))));
  return fxc{fx_mw(b4, nh, fx_mw(a4, xh, mx >> 30)), fx_mw(a4, yh, fx_mw(b4, xh, my >> 30))};
}

// a c for a real constant c = (h 2^32 + l) 2^-62, |a| <= 2^61.
__device__ __forceinline__ long long fx_mulc(long long a, int h, int l) {
  const int al = (int)a, ah = (int)(a >> 32) + (int)((unsigned)al >> 31);
  return fx_mw(ah << 2, h, fx_mw(al, h, fx_mw(ah, l, 1ll << 29)) >> 30);
}

// Host: the split of c (|c| <= 1).
inline void fx_split(long double c, int& h, int& l) {
  const long double s = c * 4611686018427387904.0L;  // 2^62
  long long v = (long long)(s < 0 ? s - 0.5L : s + 0.5L);
  l = (int)(uint32_t)(v & 0xffffffffll);
  if (l == INT32_MIN) {  // negated in the conjugate product: keep -l representable
    l += 1;
    v += 1;
  }
  h = (int)((v - l) >> 32);
}

// Constants of the radix-3 and radix-5 butterflies, split as above (2^62 times the value, rounded).
namespace fxk {
constexpr long long kH = 3993837246235628775ll;   // sqrt(3)/2
constexpr long long kC1 = 1425089352415399811ll;  // cos(2 pi/5)
constexpr long long kC2 = -3730932361629093763ll; // cos(4 pi/5)
constexpr long long kS1 = 4385974038932618941ll;  // sin(2 pi/5)
constexpr long long kS2 = 2710681029835013083ll;  // sin(4 pi/5)
template <long long C>
__device__ __forceinline__ long long mul(long long a) {
  constexpr int l = (int)(uint32_t)((unsigned long long)C & 0xffffffffull);
  constexpr int h = (int)((C - (long long)l) >> 32);
  return fx_mulc(a, h, l);
}
template <long long C>
__device__ __forceinline__ fxc mul(fxc a) {
  return fxc{mul<C>(a.x), mul<C>(a.y)};
}
}  // namespace fxk

template <int RAD>
__device__ __forceinline__ void fx_dft(fxc* x, int sign) {
  if constexpr (RAD == 2) {
    const fxc t = x[0];
    x[0] = fx_add(t, x[1]);
    x[1] = fx_sub(t, x[1]);
  } else if constexpr (RAD == 4) {
    const fxc a0 = fx_add(x[0], x[2]), a1 = fx_sub(x[0], x[2]);
    const fxc a2 = fx_add(x[1], x[3]), a3 = fx_muli(fx_sub(x[1], x[3]), sign);
    x[0] = fx_add(a0, a2);
    x[2] = fx_sub(a0, a2);
    x[1] = fx_add(a1, a3);
    x[3] = fx_sub(a1, a3);
  } else if constexpr (RAD == 3) {
    const fxc s = fx_add(x[1], x[2]), d = fx_sub(x[1], x[2]);
    const fxc m = fxc{x[0].x - ((s.x + 1) >> 1), x[0].y - ((s.y + 1) >> 1)};
    const fxc t = fx_muli(fxk::mul<fxk::kH>(d), sign);
    x[0] = fx_add(x[0], s);
    x[1] = fx_add(m, t);
    x[2] = fx_sub(m, t);
  } else {
    static_assert(RAD == 5, "radix");
    using namespace fxk;
    const fxc a1 = fx_add(x[1], x[4]), b1 = fx_sub(x[1], x[4]);
    const fxc a2 = fx_add(x[2], x[3]), b2 = fx_sub(x[2], x[3]);
    const fxc m1 = fx_add(x[0], fx_add(fxk::mul<kC1>(a1), fxk::mul<kC2>(a2)));
    const fxc m2 = fx_add(x[0], fx_add(fxk::mul<kC2>(a1), fxk::mul<kC1>(a2)));
    const fxc t1 = fx_muli(fx_add(fxk::mul<kS1>(b1), fxk::mul<kS2>(b2)), sign);
    const fxc t2 = fx_muli(fx_sub(fxk::mul<kS2>(b1), fxk::mul<kS1>(b2)), sign);
    x[0] = fx_add(x[0], fx_add(a1, a2));
    x[1] = fx_add(m1, t1);
    x[4] = fx_sub(m1, t1);
    x[2] = fx_add(m2, t2);
    x[3] = fx_sub(m2, t2);
  }
}

// One Stockham stage of radix RAD over nseq sequences (fft.cuh's formulation); L and Ns at run time.
template <int RAD>
__device__ __forceinline__ void fx_stage(const fxc* src, fxc* dst, int nseq, int ss, int L, int Ns,
                                         const fxtw* __restrict__ twt, int sign, int tid, int nthr) {
  const int LR = L / RAD, total = nseq * LR;
  const float invl = 1.0f / LR, invn = 1.0f / Ns;
  for (int idx = tid; idx < total; idx += nthr) {
    int q, j, kq, k;
    divmod_small(idx, LR, invl, q, j);
    divmod_small(j, Ns, invn, kq, k);
    const fxc* sp = src + q * ss + j;
    fxc x[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) x[r] = sp[r * LR];
    if (k != 0) {
#pragma unroll
      for (int r = 1; r < RAD; ++r) x[r] = fx_cmul(x[r], __ldg(twt + k * (RAD - 1) + (r - 1)), sign);
    }
    fx_dft<RAD>(x, sign);
    fxc* dp = dst + q * ss + (j - k) * RAD + k;
#pragma unroll
    for (int r = 0; r < RAD; ++r) dp[r * Ns] = x[r];
  }
}

// Any length of an FftPlan: nseq sequences (stride ss) from a, ping-pong with b; returns the buffer that holds the
// result.  All threads of the block; the caller has synchronised the inputs, the result is synchronised.
__device__ inline fxc* fx_fft_generic(fxc* a, fxc* b, int nseq, int ss, const FftPlan& p, const fxtw* __restrict__ tw,
                                      int sign, int tid, int nthr) {
  const int L = p.L;
  fxc *src = a, *dst = b;
  for (int s = 0; s < p.nst; ++s) {
    const int Rr = p.radix[s], Ns = p.Ns[s];
    const fxtw* twt = tw + p.twoff[s];
    switch (Rr) {
      case 2: fx_stage<2>(src, dst, nseq, ss, L, Ns, twt, sign, tid, nthr); break;
      case 3: fx_stage<3>(src, dst, nseq, ss, L, Ns, twt, sign, tid, nthr); break;
      case 4: fx_stage<4>(src, dst, nseq, ss, L, Ns, twt, sign, tid, nthr); break;
      case 5: fx_stage<5>(src, dst, nseq, ss, L, Ns, twt, sign, tid, nthr); break;
      default: {
        // direct DFT of a larger prime radix: the butterfly's inputs are twiddled in place, then summed per output
        const fxtw* rt = tw + p.rootoff[s];
        const int LR = L / Rr;
        for (int idx = tid; idx < nseq * LR; idx += nthr) {
          const int q = idx / LR, j = idx - q * LR, k = j % Ns;
          fxc* sp = src + q * ss + j;
          if (k != 0)
            for (int r = 1; r < Rr; ++r) sp[r * LR] = fx_cmul(sp[r * LR], __ldg(twt + k * (Rr - 1) + (r - 1)), sign);
          fxc* dp = dst + q * ss + (j - k) * Rr + k;
          for (int o = 0; o < Rr; ++o) {
            fxc acc = sp[0];
            int e = 0;
            for (int r = 1; r < Rr; ++r) {
              e += o;
              if (e >= Rr) e -= Rr;
              acc = fx_add(acc, fx_cmul(sp[r * LR], __ldg(rt + e), sign));
            }
            dp[o * Ns] = acc;
          }
        }
      }
    }
    __syncthreads();
    fxc* t = src;
    src = dst;
    dst = t;
  }
  return src;
}

// Compile-time length (the radix order of the host plan: 4s, one 2, 3s, 5s).
template <int L, int Ns, int TWOFF>
__device__ __forceinline__ fxc* fx_fft_fixed(fxc* src, fxc* dst, int nseq, int ss, const fxtw* __restrict__ tw, int sign,
                                             int tid, int nthr) {
  if constexpr (Ns >= L) {
    return src;
  } else {
    constexpr int RAD = RadixOf<L / Ns>::v, LR = L / RAD;
    const int total = nseq * LR;
    for (int idx = tid; idx < total; idx += nthr) {
      const int q = idx / LR, j = idx - q * LR, k = j % Ns;
      const fxc* sp = src + q * ss + j;
      fxc x[RAD];
#pragma unroll
      for (int r = 0; r < RAD; ++r) x[r] = sp[r * LR];
      if constexpr (Ns > 1) {
#pragma unroll
        for (int r = 1; r < RAD; ++r) x[r] = fx_cmul(x[r], __ldg(tw + TWOFF + k * (RAD - 1) + (r - 1)), sign);
      }
      fx_dft<RAD>(x, sign);
      fxc* dp = dst + q * ss + (j - k) * RAD + k;
#pragma unroll
      for (int r = 0; r < RAD; ++r) dp[r * Ns] = x[r];
    }
    __syncthreads();
    return fx_fft_fixed<L, Ns * RAD, TWOFF + Ns * (RAD - 1)>(dst, src, nseq, ss, tw, sign, tid, nthr);
  }
}

__device__ inline fxc* fx_fft(fxc* a, fxc* b, int nseq, int ss, const FftPlan& p, const fxtw* __restrict__ tw, int sign,
                              int tid, int nthr) {
  switch (p.L) {
    case 32: return fx_fft_fixed<32, 1, 0>(a, b, nseq, ss, tw, sign, tid, nthr);
    case 48: return fx_fft_fixed<48, 1, 0>(a, b, nseq, ss, tw, sign, tid, nthr);
    case 64: return fx_fft_fixed<64, 1, 0>(a, b, nseq, ss, tw, sign, tid, nthr);
    case 96: return fx_fft_fixed<96, 1, 0>(a, b, nseq, ss, tw, sign, tid, nthr);
    case 128: return fx_fft_fixed<128, 1, 0>(a, b, nseq, ss, tw, sign, tid, nthr);
    default: return fx_fft_generic(a, b, nseq, ss, p, tw, sign, tid, nthr);
  }
}

// ---------------------------------------------------------------------------
// Scaling.  A line of doubles becomes integers v = round(x 2^K); K from the largest exponent of the line and a
// 17-bit estimate (rounded up) of the sum of magnitudes.  FX_NAN marks a line with an infinite or NaN element
// (its outputs are NaN), FX_ZERO a line of zeros.
// ---------------------------------------------------------------------------
constexpr int FX_NAN = -(1 << 24), FX_ZERO = 1 << 22;

// exponent key of x: ordered like |x|, zero only for x = 0
__device__ __forceinline__ unsigned fx_key(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) | (unsigned)(__double2loint(x) != 0);
}
__device__ __forceinline__ int fx_exp_of_key(unsigned key) { return max((int)(key >> 20), 1); }

// |x| in units of 2^(emax - 1039), rounded up
__device__ __forceinline__ unsigned fx_mag(double x, int emax) {
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
  const int e = (int)(h >> 20);
  const unsigned m = (h & 0xfffffu) | (e ? 0x100000u : 0u);
  return (m >> min(4 + emax - max(e, 1), 31)) + 1u;
}
// K of a line (value = v 2^-K) from its magnitude sum S > 0 (units 2^(emax - 1039)): the magnitudes of its integers
// sum to less than 2^lim.
__device__ __forceinline__ int fx_line_K(int emax, unsigned S, int lim) {
  return min(lim - (32 - __clz(S)) - (emax - 1039), 1083 - emax);  // the bound holds for lines of subnormals only
}
// round(x 2^K), K from fx_line_K of the line (lim <= 61, so the shift is at least 2)
__device__ __forceinline__ long long fx_quant(double x, int K) {
  const int hi = __double2hiint(x);
  const int e = (hi >> 20) & 0x7ff;
  unsigned long long m = ((unsigned long long)((hi & 0xfffff) | (e ? 0x100000 : 0)) << 32) | (unsigned)__double2loint(x);
  const int r = min(1085 - K - max(e, 1), 64);  // m 2^10 >> r
  m = ((m << 10) >> (r - 1)) + 1 >> 1;
  const long long s = (long long)hi >> 63;  // sign
  return ((long long)m ^ s) - s;
}
// v 2^-K, rounded to nearest even, without the conversion instruction
__device__ __forceinline__ double fx_to_double(long long v, int K) {
  if (v == 0) return K <= FX_NAN / 2 ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
  unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
  const int lz = __clzll((long long)u);
  const int E = 1085 - lz - K;  // biased exponent - 1
  if (E < 0 || E > 2044) {      // rare: results near the ends of the exponent range
    if (K <= FX_NAN / 2) return __longlong_as_double(0x7ff8000000000000ll);
    return scalbn(__ll2double_rn(v), -K);
  }
  u <<= lz;
  const unsigned r = (((unsigned)u & 0x7ffu) + ((unsigned)(u >> 11) & 1u) + 0x3ffu) >> 11;
  const unsigned long long b = ((unsigned long long)(unsigned)E << 52) + (u >> 11) + r;
  return __longlong_as_double((long long)(b | ((unsigned long long)v & 0x8000000000000000ull)));
}
// v 2^-K
__device__ __forceinline__ double fx_double(long long v, int K) {
  if (K < -900 || K > 1000) {  // rare: NaN lines, zero lines, results near the ends of the exponent range
    if (K <= FX_NAN / 2) return __longlong_as_double(0x7ff8000000000000ll);
    if (v == 0) return 0.0;
    return scalbn(__ll2double_rn(v), -K);
  }
  const double d = __ll2double_rn(v);
  return v == 0 ? 0.0 : __hiloint2double(__double2hiint(d) - (K << 20), __double2loint(d));
}
