// The fixed-point FFTs of the FP64 path (csrc/fx.cuh, fx_fft.cuh, fx_plan.h) compiled for the host: the arithmetic is
// plain integer C++, so one "thread" runs a block's stages.  Built as a shared library by tests/test_fx_host.py.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

using std::max;
using std::min;

struct Dim {
  int x, y, z;
};
static const Dim threadIdx{0, 0, 0}, blockDim{1, 1, 1};
static void __syncthreads() {}
template <class T>
static T __ldg(const T* p) {
  return *p;
}
static int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
static int __clz(unsigned v) { return v ? __builtin_clz(v) : 32; }
static int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
template <class T, class S>
static T bits(S s) {
  static_assert(sizeof(T) == sizeof(S), "bits");
  T t;
  std::memcpy(&t, &s, sizeof t);
  return t;
}
static int __double2hiint(double x) { return (int)(bits<long long>(x) >> 32); }
static int __double2loint(double x) { return (int)bits<long long>(x); }
static double __hiloint2double(int hi, int lo) { return bits<double>((long long)hi << 32 | (unsigned)lo); }
static double __longlong_as_double(long long v) { return bits<double>(v); }
static double __ll2double_rn(long long v) { return (double)v; }
static float __int2float_rn(int v) { return (float)v; }
static int __float2int_rz(float v) { return (int)v; }

static size_t __cvta_generic_to_shared(const void*) { return 0; }

#undef __shared__
#undef __noinline__
#define __noinline__
#define __shared__
alignas(16) unsigned char smem_raw[2 * 16 * (8192 + 1)];

#include "fx_fft.cuh"

// FFT of one complex line of length L (in and out interleaved), scaled as the x passes scale a column.
extern "C" void fx_line(int L, int inverse, const double* in, double* out) {
  fxc* a = reinterpret_cast<fxc*>(smem_raw);
  const FxPlan p = fx_plan(L);
  const std::vector<int> tw = fx_twiddles(L);
  unsigned key = 0, S = 0;
  for (int i = 0; i < 2 * L; ++i) key = max(key, fx_key(in[i]));
  const int emax = fx_exp_of_key(key);
  for (int i = 0; i < 2 * L; ++i) S += fx_mag(in[i], emax);
  const int K = key == 0 ? FX_ZERO : fx_line_K(emax, S, 61);
  for (int i = 0; i < L; ++i)
    a[i] = key == 0 ? fxc{0, 0} : fxc{fx_quant(in[2 * i], K), fx_quant(in[2 * i + 1], K)};
  const fxtw* t = reinterpret_cast<const fxtw*>(tw.data());
  const fxc* r = a + (p.any ? fx_fft<true>(0, L + 1, 1, L + 1, L, p.rad, t, inverse != 0)
                            : fx_fft<false>(0, L + 1, 1, L + 1, L, p.rad, t, inverse != 0));
  for (int i = 0; i < L; ++i) {
    out[2 * i] = fx_double(r[i].x, K);
    out[2 * i + 1] = fx_double(r[i].y, K);
  }
}
