// Plans and tables of the fixed-point FFTs (fx_fft.cuh), on the host.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <vector>

// Longest line on fixed point; longer ones take FP64 arithmetic (fft.cuh).  The scale allows for the sum of magnitudes,
// so the error of flat data grows with the length, that of a double-precision FFT only with the root of its logarithm.
// Relative rms error of flat lines, the worst of their amplitudes within a power of two, fixed point / double: 128
// 6.9e-17 / 1.9e-16, 300 2.2e-16 / 2.6e-16, 336 2.0e-16 / 2.3e-16, 360 2.4e-16 / 2.4e-16, 512 2.6e-16 / 2.1e-16, 1024
// 4.9e-16 / 2.3e-16, 3000 1.5e-15 / 2.6e-16.  Lines with decaying spectra are the more exact on fixed point at every
// length.
constexpr int FX_LMAX = 336;

// Stages of a transform of length L: up to eight radices, eight bits each, first stage lowest.  Radices with a
// butterfly in registers, or primes above 7 (direct DFT, roots behind the stage's twiddles).  Fewest stages first: each
// costs a pass through shared memory and L (1 - 1 / radix) twiddle products (128 = 8 x 4 x 4: 192 and eighth turns,
// 4 x 4 x 4 x 2: 256).  Radices up to 8 keep a kernel within 64 registers and four blocks an SM; up to 10 in 80
// registers were level or slower, up to 16 in 128 registers 20-30% slower (z pass 128x97x128 158 us).
struct FxPlan {
  int L;
  bool any;  // a radix of 7 or a larger prime
  unsigned long long rad;
};
__host__ __device__ constexpr bool fx_composite(int r) {
  return r >= 2 && r <= 8;
}
// twiddle entries of stage (radix R, Ns points before it)
__host__ __device__ constexpr int fx_stage_tw(int R, int Ns) { return Ns * (R - 1) + (fx_composite(R) ? 0 : R); }

// The split c = (h 2^32 + l) 2^-62 (|c| <= 1).
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

// Fewest stages, then the smallest radices, largest first; primes above 7 last.
inline void fx_search(int m, int maxr, unsigned long long cur, int n, int sum, int& bn, int& bsum, unsigned long long& best) {
  if (m == 1) {
    if (n < bn || (n == bn && sum < bsum)) {
      bn = n;
      bsum = sum;
      best = cur;
    }
    return;
  }
  if (n + 1 > bn) return;
  for (int r = std::min(maxr, m); r >= 2; --r)
    if (m % r == 0 && fx_composite(r)) fx_search(m / r, r, cur | (unsigned long long)r << (8 * n), n + 1, sum + r, bn, bsum, best);
}

inline FxPlan fx_plan(int L) {
  static std::atomic<unsigned long long> known[8192];  // a function of L alone
  if (L < 8192)
    if (const unsigned long long k = known[L].load(std::memory_order_relaxed)) return FxPlan{L, k >> 63 != 0, k & ~(1ull << 63)};
  int m = L, np = 0, primes[8];
  for (int p = 11; p <= m; p += 2)
    while (m % p == 0 && p % 3 && p % 5 && p % 7) {
      primes[np++] = p;
      m /= p;
    }
  int bn = 8, bsum = 0;
  unsigned long long best = 0;
  fx_search(m, 8, 0, 0, 0, bn, bsum, best);
  for (int i = 0; i < np; ++i) best |= (unsigned long long)primes[i] << (8 * (bn + i));
  bool any = false;
  for (unsigned long long r = best; r; r >>= 8) any = any || (r & 255) == 7 || (r & 255) > 8;
  if (L < 8192) known[L].store(best | (unsigned long long)any << 63, std::memory_order_relaxed);
  return FxPlan{L, any, best};
}

// Per stage: exp(-2 pi i k r / (Ns R)) at [k (R - 1) + r - 1], then a prime's roots exp(-2 pi i e / R).
inline std::vector<int> fx_twiddles(int L) {
  std::vector<int> t;
  auto push = [&](long long m, long long n) {
    const long double x = 2 * 3.14159265358979323846264338327950288L * (long double)(m % n) / (long double)n;
    const bool cz = 4 * (m % n) == n || 4 * (m % n) == 3 * n, sz = 2 * (m % n) % n == 0;
    int v[4];
    fx_split(cz ? 0.0L : cosl(x), v[0], v[1]);
    fx_split(sz ? 0.0L : -sinl(x), v[2], v[3]);
    t.insert(t.end(), v, v + 4);
  };
  unsigned long long rad = fx_plan(L).rad;
  for (int Ns = 1; Ns < L; rad >>= 8) {
    const int R = (int)(rad & 255);
    for (int k = 0; k < Ns; ++k)
      for (int r = 1; r < R; ++r) push((long long)k * r, (long long)Ns * R);
    if (!fx_composite(R))
      for (int e = 0; e < R; ++e) push(e, R);
    Ns *= R;
  }
  if (t.empty()) t.resize(4);
  return t;
}
