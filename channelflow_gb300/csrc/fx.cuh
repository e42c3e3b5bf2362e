// 64-bit fixed-point arithmetic for the FP64 path (FFTs: fx_fft.cuh).
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition, but a 64-bit integer addition
// (IADD3 pair) in about 2 and a 32 x 32 -> 64 bit multiply-add (IMAD.WIDE) in 8 to 11 (measured with a
// throughput probe, 8 warps a sub-partition).  An FFT is mostly additions, so the FP64 path's transforms run on integers: a sequence is
// scaled by one power of two such that the sum of the magnitudes of its elements (real plus imaginary) stays below
// 2^61, which bounds the modulus of every intermediate value of the transform, and rounded to integers.  Its rounding
// errors are a few units of 2^-61 of that sum: up to FX_LMAX points (fx_plan.h) below those of the same FFT in FP64, whose
// units are 2^-53 of the local values.
//
// Twiddle factors are fixed-point too: c = (h 2^32 + l) 2^-62 with signed 32-bit h, l.  A complex product with
// components a = ah 2^32 + al (al signed) sums the cross terms ah l + al h of both real products in one 64-bit
// accumulator, drops al l (below one unit) and takes six IMAD.WIDE per component.
#pragma once

#include "common.cuh"

struct alignas(16) fxc {
  long long x, y;
};

// One twiddle factor: x = (x 2^32 + y) 2^-62 + i (z 2^32 + w) 2^-62.
typedef int4 fxtw;

__device__ __forceinline__ fxc fx_add(fxc a, fxc b) { return fxc{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fxc fx_sub(fxc a, fxc b) { return fxc{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ long long fx_mw(int a, int b, long long c) { return (long long)a * b + c; }

// a w; |a.x|, |a.y| < 2^61 (of a modulus below 2^61, so that the result's components are too).
__device__ __forceinline__ fxc fx_cmul(fxc a, fxtw w) {
  const int xh = w.x, xl = w.y, yh = w.z, yl = w.w, nh = -w.z, nl = -w.w;
  const int al = (int)a.x, bl = (int)a.y;
  const int ah = (int)(a.x >> 32) + (int)((unsigned)al >> 31), bh = (int)(a.y >> 32) + (int)((unsigned)bl >> 31);
  const int a4 = ah << 2, b4 = bh << 2;
  const long long half = 1ll << 29;
  const long long mx = fx_mw(bl, nh, fx_mw(bh, nl, fx_mw(al, xh, fx_mw(ah, xl, half))));
  const long long my = fx_mw(al, yh, fx_mw(ah, yl, fx_mw(bl, xh, fx_mw(bh, xl, half))));
  return fxc{fx_mw(b4, nh, fx_mw(a4, xh, mx >> 30)), fx_mw(a4, yh, fx_mw(b4, xh, my >> 30))};
}

// a c for a real constant c = (h 2^32 + l) 2^-62, |a| < 2^61.
__device__ __forceinline__ long long fx_mulc(long long a, int h, int l) {
  const int al = (int)a, ah = (int)(a >> 32) + (int)((unsigned)al >> 31);
  return fx_mw(ah << 2, h, fx_mw(al, h, fx_mw(ah, l, 1ll << 29)) >> 30);
}

// The same for |a| < 2^62: the sum of both components of a number whose modulus is below 2^61 reaches sqrt(2) 2^61, which
// four times its high half would carry out of 32 bits.  The product is shifted instead.
__device__ __forceinline__ long long fx_mulc_sum(long long a, int h, int l) {
  const int al = (int)a, ah = (int)(a >> 32) + (int)((unsigned)al >> 31);
  return ((long long)ah * h << 2) + (fx_mw(al, h, fx_mw(ah, l, 1ll << 29)) >> 30);
}

// a b 2^-64 for |a|, |b| < 2^61, without the product of the low halves (below one unit).
__device__ __forceinline__ long long fx_mulhi(long long a, long long b) {
  const int al = (int)a, bl = (int)b;
  const int ah = (int)(a >> 32) + (int)((unsigned)al >> 31), bh = (int)(b >> 32) + (int)((unsigned)bl >> 31);
  return fx_mw(ah, bh, fx_mw(al, bh, (long long)ah * bl) >> 32);
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
