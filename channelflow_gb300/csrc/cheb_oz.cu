// Chebyshev transforms of FP64 lines on the tensor cores, by exact integer products.
//
// out[n][l] = sum_j M[n][j] in[j][l] for every real line l (the inverse transform M = T with T[j][n] = cos(pi n j /
// (N-1)), the forward transform F of chebyfft, chebyshev.cpp:262-284, and DF, its derivative).  A line is scaled by a
// power of two such that its magnitudes sum to less than 2^61 and rounded to integers X (fx.cuh); a matrix row is
// scaled to a largest magnitude in (1/2, 1] and rounded to 62 bits.  Both are written in seven balanced digits of
// nine bits (-256 .. 255; FP16 holds them exactly), most significant first; products of digits i and j weigh
// 2^-9(i + j), the 28 pairs with i + j <= 6 are kept.  All pairs of one weight and all K points sum into one FP32
// accumulator of tensor memory below 2^24 (checked for every matrix row at set-up), so every sum is exact and the
// result carries about 2^-59 of the line's sum of magnitudes, whatever the order of the sums.
// (Error-free splitting of a matrix product into digit products: Ozaki, Ogita, Oishi and Rump, 2012.)  The bound of the
// check holds for every Ny from 3 to 144 but 116, 122, 134-136, 138, 141 and 143.
//
// Parity: the even and odd coefficients are two systems of half the size (T[N-1-j][n] = (-1)^n T[j][n]): the inverse
// transform multiplies each parity's coefficients and combines y_j = E_j + O_j, y_{N-1-j} = E_j - O_j; the forward
// transforms fold x_j +- x_{N-1-j} first.  The derivative of an inverse transform is taken before it, d_n = d_{n+2} + 2
// (n+1) x_{n+1} in integers with 32 fraction bits, rounded once: coefficients rounded before their weights would be off
// by up to N^2 units at the walls.  Relative error of N(u) for mean profiles with flat spectra, rounded before / here /
// dense FP64 products: Ny = 49 4.3e-15 / 1.5e-16 / 4.8e-16, 97 2.6e-14 / 1.2e-16 / 6.0e-16, 139 8.9e-14 / 1.9e-16 /
// 3.9e-16; FP64 step 128x97x128 519 -> 525 us.
//
// One CTA: 128 lines (the M rows of the MMA) of one job.  K runs in stages of two steps of 16 through a ring: 512
// threads quantise 32 points of every line and write the digits as seven K-major operands a step (no swizzle: 8 x
// 16-byte core matrices), the bulk-copy engine brings the matrix digits; one thread issues the products.  The
// digits of the matrix lie side by side as N columns, so digit i of the lines meets all its digits j <= 6 - i in at most
// two MMAs, whose accumulators start at column i NT (weight i + j).  Two CTAs cannot share an SM (tensor memory: 7 NT
// + 8 columns; shared memory).
//
// Measured against FP64 arithmetic, which the FP64 pipe bounds (one warp instruction per 64 cycles).  128x97x128: curl
// and inverse transforms 190 us (FFT form) -> 68 us and 10 us more in the x pass, which forms the vorticity; forward 91
// -> 56 us.  72x57x90, skew-symmetric: gradient 107 -> 28 us, forward with divergence 484 -> 43 us.  Ny = 35, 190 modes:
// 29 -> 17 us and 24 -> 11 us (10 and 8 with k_cheb_oz_few).  FlowField y transform 128x97x128: 1340 -> 83 and 96 us.
// Relative error of one transform 5e-17 (FP64 products 2e-16 ... 5e-16).  Bound by instruction issue and latency of the
// digits and the sums (16 warps an SM).  256 threads (and K steps of 16): 102 and 70 us.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "fx.cuh"
#include "kernels.h"

namespace {

constexpr int OZ_THREADS = 512, OZ_LINES = 128, OZ_DIGITS = 7;
constexpr int OZ_ASTAGE = OZ_DIGITS * OZ_LINES * 16 * 2;  // bytes of the line digits of one K step

__host__ __device__ constexpr int oz_bstage(int NT) { return (OZ_DIGITS * NT + 8) * 32; }

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// Shared-memory matrix descriptor: K-major, no swizzle, leading / stride byte offsets 128 / 256, version 1.
__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, int acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}
// Bounded wait (false: it ran out).
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  for (int w = 0; w < (1 << 20); ++w) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

struct OzArgs {
  GridDev g;  // modes of the complex lines (wavenumbers, (0,0) mode); unused by jobs without them
  int N, NT, nlines, split;
  int ring, spill;  // stages in the ring; inverse: the first parity's results wait in the output array
  unsigned ld;
  double dscale;  // 2 / (b - a)
  OzTables t;
  int* err;
  OzJob job[OZ_MAX_JOBS];
};

// Magnitude sum of a line, in units of 2^(e - 1043) with e the largest exponent met so far.
struct OzSum {
  unsigned long long S = 0;
  int e = 1;
  unsigned nz = 0;
  __device__ __forceinline__ void add(double x, unsigned w) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    const int xe = (int)(h >> 20), ex = max(xe, 1);
    nz |= h | (unsigned)__double2loint(x);
    if (ex > e) {
      S = (S >> min(ex - e, 63)) + 1;
      e = ex;
    }
    const unsigned m = (h & 0xfffffu) | (xe ? 0x100000u : 0u);
    S += (unsigned long long)((m >> min(e - ex, 31)) + 1u) * w;
  }
};

// An integer with 32 fraction bits.
struct OzFix {
  long long i;
  unsigned f;
};
__device__ __forceinline__ OzFix oz_add(OzFix a, OzFix b) {
  const unsigned f = a.f + b.f;
  return OzFix{a.i + b.i + (f < b.f), f};
}
__device__ __forceinline__ long long oz_round(OzFix a) { return a.i + (a.f >> 31); }
__device__ __forceinline__ OzFix oz_half(OzFix a) { return OzFix{a.i >> 1, (a.f >> 1) | ((unsigned)a.i << 31)}; }
// w x 2^K for 0 <= w < 2^10 and K from oz_scale of a line whose scale counts x with at least this weight (the product is
// below 2^61 and its shift at least -8), without what lies below 2^-32
__device__ __forceinline__ OzFix oz_term(double x, int K, unsigned w) {
  const int hi = __double2hiint(x);
  const int e = (hi >> 20) & 0x7ff;
  const unsigned long long m = ((unsigned long long)((hi & 0xfffff) | (e ? 0x100000 : 0)) << 32) | (unsigned)__double2loint(x);
  const unsigned long long p = m * w;  // below 2^63
  const int s = 1075 - K - max(e, 1);  // p 2^-s
  const long long i = (long long)(s < 0 ? p << -s : p >> min(s, 63));
  const unsigned f = (unsigned)(s < 32 ? p << (32 - s) : p >> min(s - 32, 63));
  return hi < 0 ? OzFix{-i - (f != 0), 0u - f} : OzFix{i, f};
}

// Seven digits (most significant first) of the eight integers x[0..7], |x| < 2^61, as FP16 pairs; copies 32 rows apart.
template <int COPIES>
__device__ __forceinline__ void oz_store(unsigned char* dst, const long long (&x)[8]) {
  constexpr unsigned long long OFF = 0x4020100804020100ull;  // 256 in every digit
  unsigned lo[8], hi[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const unsigned long long v = (unsigned long long)x[e] + OFF;
    lo[e] = (unsigned)v;
    hi[e] = (unsigned)(v >> 32);
  }
  const __half2 bias = __floats2half2_rn(-1280.0f, -1280.0f);  // 0x6400 + u is 1024 + u
#pragma unroll
  for (int d = 0; d < OZ_DIGITS; ++d) {
    const int b = 9 * (OZ_DIGITS - 1 - d);
    unsigned w[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      unsigned a0, a1;
      if (b + 9 <= 32) {
        a0 = lo[2 * p] >> b;
        a1 = b <= 16 ? lo[2 * p + 1] << (16 - b) : lo[2 * p + 1] >> (b - 16);
      } else if (b < 32) {
        a0 = __funnelshift_r(lo[2 * p], hi[2 * p], b);
        a1 = __funnelshift_r(lo[2 * p + 1], hi[2 * p + 1], b - 16);
      } else {
        const int c = b - 32;
        a0 = hi[2 * p] >> c;
        a1 = c <= 16 ? hi[2 * p + 1] << (16 - c) : hi[2 * p + 1] >> (c - 16);
      }
      const unsigned u = (a0 & 0x1ffu) | (a1 & 0x1ff0000u) | 0x64006400u;
      const __half2 h = __hadd2(*reinterpret_cast<const __half2*>(&u), bias);
      w[p] = *reinterpret_cast<const unsigned*>(&h);
    }
#pragma unroll
    for (int c = 0; c < COPIES; ++c)
      *reinterpret_cast<uint4*>(dst + d * (OZ_LINES * 32) + c * 1024) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// sum_s r_s 2^(9 (6 - s) - 8) of the exact FP32 sums r
__device__ __forceinline__ long long oz_sum(const uint32_t (&r)[OZ_DIGITS]) {
  int d[OZ_DIGITS];
#pragma unroll
  for (int s = 0; s < OZ_DIGITS; ++s) d[s] = __float2int_rn(__uint_as_float(r[s]));
  long long x = (long long)(2 * d[5] + ((d[6] + 128) >> 8));
  x = fx_mw(d[4], 1 << 10, x);
  x = fx_mw(d[3], 1 << 19, x);
  x = fx_mw(d[2], 1 << 28, x);
  x += (long long)((unsigned long long)(((unsigned)d[0] << 14) + ((unsigned)d[1] << 5)) << 32);
  return x;
}

// K of a line (fx_line_K) from the sums of its four quarters, stride apart
__device__ __forceinline__ int oz_scale(const unsigned long long* sS, const int* sE, int stride) {
  int e = 1;
  bool nz = false;
  for (int i = 0; i < 4; ++i) {
    const int ei = sE[i * stride];
    e = max(e, ei & 0xffff);
    nz = nz || (ei & 0x10000);
  }
  unsigned long long S = 4;
  for (int i = 0; i < 4; ++i) S += sS[i * stride] >> min(e - (sE[i * stride] & 0xffff), 63);
  if (!nz) return FX_ZERO;
  if (e == 2047) return FX_NAN;
  return min(61 - (64 - __clzll((long long)S)) - (e - 1043), 1083 - e);
}

// A line of a job: its wavenumbers, its base flow and its points.  FP64 instructions take the whole warp's slot even where
// no lane needs them: the rare ones stand behind branches over whole groups of points.
template <bool INV>
struct OzLine {
  const OzJob& job;
  const double *src = nullptr, *base = nullptr;
  double kx = 0.0, kz = 0.0, shift = 0.0;
  unsigned ld;
  int N, gl;
  bool act, hasb, fd = false;
  __device__ __forceinline__ OzLine(const OzArgs& a, const OzJob& j, int gl_, bool act_)
      : job(j), ld(a.ld), N(a.N), gl(gl_), act(act_) {
    const int m = min(gl, a.nlines - 1) >> 1;
    if (job.gx || job.pkx) {
      const int ikx = mode_kx(a.g, m), ikz = mode_kz(a.g, m);
      const double sg = gl & 1 ? 2.0 * M_PI : -2.0 * M_PI;  // i k f: re = -k f_im, im = k f_re
      kx = ikx == a.g.kxmax ? 0.0 : sg * ikx / a.g.Lx;
      kz = ikz == a.g.kzmax ? 0.0 : sg * ikz / a.g.Lz;
    }
    if (job.base || job.shift != 0.0) {
      if (act && !(gl & 1) && mode_kx(a.g, m) == 0 && mode_kz(a.g, m) == 0) {
        if (job.base) base = job.base + (size_t)job.bstride * mode_field(a.g, m);
        shift = job.shift;
      }
    }
    hasb = __any_sync(0xffffffffu, base != nullptr || shift != 0.0);
  }
  // v[i] = point n0 + i dn of the line, i < cnt, else zero
  __device__ __forceinline__ void load8(double (&v)[8], int n0, int dn, int cnt) const {
    unsigned o = (unsigned)n0 * ld + gl;
#pragma unroll
    for (int i = 0; i < 8; ++i, o += (unsigned)dn * ld) v[i] = src && i < cnt ? src[o] : 0.0;
    if constexpr (INV) {
      if (hasb) {
        for (int i = 0; i < 8; ++i)
          if (i < cnt) {
            if (base) v[i] += base[n0 + i * dn];
            if (n0 + i * dn == 0) v[i] -= shift;
          }
      }
    } else if (!fd && job.pkx) {
      double px[8], pz[8];
      o = (unsigned)n0 * ld + (gl ^ 1);
#pragma unroll
      for (int i = 0; i < 8; ++i, o += (unsigned)dn * ld) {
        px[i] = i < cnt ? job.pkx[o] : 0.0;
        pz[i] = i < cnt ? job.pkz[o] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = fma(job.wF, v[i], job.wK * fma(kx, px[i], kz * pz[i]));
    }
  }
  // magnitudes of every fourth point
  __device__ __forceinline__ void magnitudes(OzSum& sum, int quarter) const {
    if (act)
      for (int n0 = quarter; n0 < N; n0 += 32) {
        double v[8];
        load8(v, n0, 4, (N - n0 + 3) >> 2);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int n = n0 + 4 * i;
          if (n < N && !(INV && job.deriv && n == 0)) sum.add(v[i], INV && job.deriv ? (unsigned)n * (n + 1) : 1u);
        }
      }
  }
};

template <bool INV>
__global__ void __launch_bounds__(OZ_THREADS, 1) k_cheb_oz(const __grid_constant__ OzArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int N = a.N, NT = a.NT;
  const OzJob& job = a.job[blockIdx.y];
  const int bst = oz_bstage(NT);
  const int ring = a.ring;
  unsigned char* As = smem;
  unsigned char* Bs = As + ring * 2 * OZ_ASTAGE;
  unsigned long long* sS = reinterpret_cast<unsigned long long*>(Bs + ring * 2 * bst);  // [512]
  int* sE = reinterpret_cast<int*>(sS + OZ_THREADS);                                    // [512]
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sE + OZ_THREADS);  // [2] matrix digits landed, [2] stage consumed
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 4);
  long long* Ev = reinterpret_cast<long long*>(tslot + 4);  // [NT][128] results of the first parity
  const int tid = threadIdx.x, warp = tid >> 5;
  const int line = tid & (OZ_LINES - 1), h = tid >> 7;  // four threads a line
  const int gl = blockIdx.x * OZ_LINES + line;
  const bool act = gl < a.nlines;
  const unsigned ld = a.ld;
  uint32_t tcols = 32;
  while ((int)tcols < OZ_DIGITS * NT + 8) tcols *= 2;

  if (tid == 0) {
    for (int i = 0; i < 4; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(mbar + i)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)), "r"(tcols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tslot;
  pdl_wait();  // the previous kernel's output is read from here on
  pdl_trigger();

  OzLine<INV> ln(a, job, gl, act);
  const double kx = ln.kx, kz = ln.kz;
  const bool emit_scale = INV && job.deriv && a.dscale != 1.0, emit_grad = INV && job.gx != nullptr;

  bool ok = true;
  uint32_t late = 0, lpar = 0;  // thread 0: barrier and parity of a copy given up; none is started after it
  int t = 0;  // K steps issued so far (ring position)
  const int nstage = INV || !job.pd ? 1 : 2;
  const int q0 = a.split ? (int)blockIdx.z : 0, q1 = a.split ? q0 + 1 : 2;  // parities of this CTA
  for (int sg = 0; sg < nstage; ++sg) {
    const bool fd = !INV && sg == 1;  // derivative of the forward transform
    const OzMatrix& M = INV ? a.t.T : (fd ? a.t.DF : a.t.F);
    ln.src = fd ? job.pd : job.in;
    ln.fd = fd;
    // scale of the line: its four threads sum the magnitudes of every fourth point
    OzSum sum;
    ln.magnitudes(sum, h);
    sS[tid] = sum.S;
    sE[tid] = sum.e | (sum.nz ? 0x10000 : 0);
    __syncthreads();
    const int K = oz_scale(sS + line, sE + line, OZ_LINES);
    __syncthreads();  // sS, sE are free
    const bool live = act && K != FX_ZERO && K != FX_NAN;
    for (int p = q0; p < q1; ++p) {
      const int q = fd ? 1 - p : p;  // input parity; a CTA's outputs stay of parity p
      const int KR = q ? N / 2 : (N + 1) / 2, KS = (KR + 15) / 16;
      const unsigned char* Mg = reinterpret_cast<const unsigned char*>(M.digits) + (q ? (size_t)(((N + 1) / 2 + 15) / 16) * bst : 0);
      OzFix carry{0, 0};  // running derivative
      const int last = (KS - 1) / 2;
      for (int pr = last; pr >= 0; --pr, ++t) {
        const int st = t % ring, use = t / ring, nks = min(KS - 2 * pr, 2);
        const uint32_t full = smem_u32(mbar + st), done = smem_u32(mbar + 2 + st);
        if (use > 0 && !mbar_wait(done, (uint32_t)((use - 1) & 1))) ok = false;
        if (tid == 0 && !late) {
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(full), "r"((uint32_t)(nks * bst))
                       : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                           smem_u32(Bs + st * 2 * bst)),
                       "l"(Mg + (size_t)2 * pr * bst), "r"((uint32_t)(nks * bst)), "r"(full)
                       : "memory");
        }
        const int k0 = 32 * pr + 8 * h;  // this thread's eight points
        long long x[8];
        double v[8];
        if constexpr (INV) {
          const int n0 = 2 * k0 + q + (job.deriv ? 1 : 0);
          ln.load8(v, n0, 2, live ? (N - n0 + 1) >> 1 : 0);
          if (job.deriv) {  // suffix sums: within the thread's points, then over the line's other threads
            OzFix d[8], acc{0, 0};
#pragma unroll
            for (int e = 7; e >= 0; --e) {
              if (live) acc = oz_add(acc, oz_term(v[e], K, 2 * (n0 + 2 * e)));
              d[e] = acc;
            }
            sS[tid] = (unsigned long long)acc.i;
            sE[tid] = (int)acc.f;
            __syncthreads();
            OzFix above = carry;
#pragma unroll
            for (int i = 3; i >= 0; --i) {
              const OzFix ti{(long long)sS[i * OZ_LINES + line], (unsigned)sE[i * OZ_LINES + line]};
              if (i > h) above = oz_add(above, ti);
              carry = oz_add(carry, ti);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) d[e] = oz_add(d[e], above);
            if (n0 == 1) d[0] = oz_half(d[0]);
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = oz_round(d[e]);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = live ? fx_quant(v[e], K) : 0;
          }
        } else {
          double w[8];
          ln.load8(v, k0, 1, live ? KR - k0 : 0);
          ln.load8(w, N - 1 - k0, -1, live ? N / 2 - k0 : 0);  // the middle point stands alone
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const long long xv = live ? fx_quant(v[e], K) : 0, xw = live ? fx_quant(w[e], K) : 0;
            x[e] = q ? xv - xw : xv + xw;
          }
        }
        if ((h >> 1) < nks)
          oz_store<1>(As + (st * 2 + (h >> 1)) * OZ_ASTAGE + (line >> 3) * 256 + (h & 1) * 128 + (line & 7) * 16, x);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        if (tid == 0) {
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          if (!late && mbar_wait(full, (uint32_t)(use & 1))) {
            for (int k = 0; k < nks; ++k) {
              const uint32_t a0 = smem_u32(As + (st * 2 + k) * OZ_ASTAGE), b0 = smem_u32(Bs + (st * 2 + k) * bst);
              for (int i = 0; i < OZ_DIGITS; ++i) {
                // columns of digits 0 .. 6 - i; eight more where that is no multiple of 16 (they fall past the last weight)
                const int cols = (NT * (OZ_DIGITS - i) + 15) & ~15;
                for (int c0 = 0; c0 < cols; c0 += 256) {
                  const int nc = min(cols - c0, 256);
                  const uint32_t idesc = (1u << 4) | ((uint32_t)(nc >> 3) << 17) | ((uint32_t)(OZ_LINES >> 4) << 24);
                  mma_f16(tmem + (uint32_t)(i * NT + c0), oz_desc(a0 + i * (OZ_LINES * 32)), oz_desc(b0 + c0 * 32), idesc,
                          pr != last || k != 0 || i != 0);
                }
              }
            }
          } else {
            ok = false;
            if (!late) {
              late = full;
              lpar = (uint32_t)(use & 1);
            }
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(done)
                       : "memory");
        }
      }
      if (!mbar_wait(smem_u32(mbar + 2 + (t - 1) % ring), (uint32_t)(((t - 1) / ring) & 1))) ok = false;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      // epilogue: this thread's line is TMEM lane 32 (warp % 4) + lane; columns in units of 8, shared out over h
      const int rows = INV ? (N + 1) / 2 : (p ? N / 2 : (N + 1) / 2);
      const int* rexp = M.rexp + p * NT;
      for (int cu = h; cu * 8 < rows; cu += 4) {
        uint32_t r[OZ_DIGITS][8];
#pragma unroll
        for (int s = 0; s < OZ_DIGITS; ++s) {
          const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(s * NT + 8 * cu);
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                       : "=r"(r[s][0]), "=r"(r[s][1]), "=r"(r[s][2]), "=r"(r[s][3]), "=r"(r[s][4]), "=r"(r[s][5]),
                         "=r"(r[s][6]), "=r"(r[s][7])
                       : "r"(ta));
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        long long v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t w[OZ_DIGITS];
#pragma unroll
          for (int s = 0; s < OZ_DIGITS; ++s) w[s] = r[s][c];
          v[c] = oz_sum(w);
        }
        const int r0 = 8 * cu, nr = min(8, rows - r0);
        if constexpr (INV) {
          // the even part waits in shared memory or in the output array (written and read by this thread)
          long long* E = a.spill ? reinterpret_cast<long long*>(job.out) + (unsigned)r0 * ld + gl : Ev + r0 * OZ_LINES + line;
          const unsigned es = a.spill ? ld : OZ_LINES;
          const bool eok = act || !a.spill;
          if (p == 0) {
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (eok && c < nr) E[c * es] = v[c];
            continue;
          }
          double y[2][8];
          long long ew[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) ew[c] = eok && c < nr ? E[c * es] : 0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const long long ev = ew[c];
            y[0][c] = fx_to_double(r0 + c < N / 2 ? ev + v[c] : ev, K);
            y[1][c] = fx_to_double(ev - v[c], K);
          }
          if (emit_scale) {
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int c = 0; c < 8; ++c) y[i][c] *= a.dscale;
          }
          const int nr2 = min(8, N / 2 - r0);  // rows with a mirrored point
          if (act) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              if (c < nr) job.out[(unsigned)(r0 + c) * ld + gl] = y[0][c];
              if (c < nr2) job.out[(unsigned)(N - 1 - r0 - c) * ld + gl] = y[1][c];
            }
          }
          if (emit_grad) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const double y0 = __shfl_xor_sync(0xffffffffu, y[0][c], 1), y1 = __shfl_xor_sync(0xffffffffu, y[1][c], 1);
              const unsigned o0 = (unsigned)(r0 + c) * ld + gl, o1 = (unsigned)(N - 1 - r0 - c) * ld + gl;
              if (act && c < nr) {
                job.gx[o0] = kx * y0;
                job.gz[o0] = kz * y0;
              }
              if (act && c < nr2) {
                job.gx[o1] = kx * y1;
                job.gz[o1] = kz * y1;
              }
            }
          }
        } else {
          double y[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) y[c] = fx_to_double(v[c], c < nr ? K + rexp[r0 + c] : 0);
          if (job.inplace && p == 0) {
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (c < nr) Ev[(r0 + c) * OZ_LINES + line] = __double_as_longlong(y[c]);
            continue;
          }
          if (fd) {
            double f[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) f[c] = act && c < nr ? job.out[(unsigned)(2 * (r0 + c) + p) * ld + gl] : 0.0;
#pragma unroll
            for (int c = 0; c < 8; ++c) y[c] = fma(job.wD, y[c], f[c]);
          }
          if (act) {
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (c < nr) job.out[(unsigned)(2 * (r0 + c) + p) * ld + gl] = y[c];
          }
        }
      }
      if (!INV && job.inplace && p == 1 && act)
        for (int cu = h; cu * 8 < (N + 1) / 2; cu += 4)
          for (int row = 8 * cu; row < min(8 * cu + 8, (N + 1) / 2); ++row)
            job.out[(unsigned)(2 * row) * ld + gl] = __longlong_as_double(Ev[row * OZ_LINES + line]);
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    }
    __syncthreads();  // sS, sE of the next stage
  }
  if (!ok) {  // copies and products that are still under way end before their memory is given back (bounded again)
    if (a.err) *static_cast<volatile int*>(a.err) = 1;
    if (late) mbar_wait(late, lpar);
    mbar_wait(smem_u32(mbar + 2 + (t - 1) % ring), (uint32_t)(((t - 1) / ring) & 1));
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tcols));
}

// ---------------------------------------------------------------------------
// The same transforms of few lines of up to 64 points.  A CTA takes 32 lines of one job and both parities.  Its lines
// stand four times in the MMA's 128 rows, once per quarter of tensor memory (a warp reads one quarter only), so that its 16
// warps share out the digits (a warp: 8 points of one parity) and the sums (a warp: OZ_COLS columns).  The line scales are
// summed as in k_cheb_oz and the products are exact: the results are the same bits.
// Where k_cheb_oz has a few CTAs its time is one CTA's: issue slots 42% active, 3000 instructions a warp.  Ny = 35, 190
// modes: inverse with curl 17.6 -> 10.0 us, forward 10.3 -> 8.1 us; FP64 steps 24x17x24 72.6 -> 64.4 us, 32x33x32 79.4 ->
// 70.6 us, 40x41x40 96.8 -> 87.6 us.
// ---------------------------------------------------------------------------
constexpr int OZ_LS = 32;

template <int C>
__device__ __forceinline__ void oz_load(uint32_t ta, uint32_t* r) {
  if constexpr (C == 4) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(ta));
  } else {
    static_assert(C == 2, "columns a warp");
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(ta));
  }
}

// C sums from the accumulators at ta (seven weights NT columns apart)
template <int C>
__device__ __forceinline__ void oz_sums(uint32_t ta, int NT, long long (&v)[C]) {
  uint32_t r[OZ_DIGITS][C];
#pragma unroll
  for (int s = 0; s < OZ_DIGITS; ++s) oz_load<C>(ta + (uint32_t)(s * NT), r[s]);
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int c = 0; c < C; ++c) {
    uint32_t w[OZ_DIGITS];
#pragma unroll
    for (int s = 0; s < OZ_DIGITS; ++s) w[s] = r[s][c];
    v[c] = oz_sum(w);
  }
}

template <bool INV>
__global__ void __launch_bounds__(OZ_THREADS, 1) k_cheb_oz_few(const __grid_constant__ OzArgs a) {
  constexpr int C = INV ? 2 : 4;  // columns a warp
  extern __shared__ __align__(128) unsigned char smem[];
  const int N = a.N, NT = a.NT;
  const OzJob& job = a.job[blockIdx.y];
  const int bst = oz_bstage(NT);
  unsigned char* As = smem;                                                               // [parity][K step]
  unsigned char* Bs = As + 4 * OZ_ASTAGE;                                                 // [parity's K steps]
  unsigned long long* sS = reinterpret_cast<unsigned long long*>(Bs + 4 * bst);           // [256]
  int* sE = reinterpret_cast<int*>(sS + 8 * OZ_LS);                                       // [256]
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sE + 8 * OZ_LS);                           // matrix landed, products done
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 2);
  const int tid = threadIdx.x, warp = tid >> 5, line = tid & 31;
  const int gl = blockIdx.x * OZ_LS + line;
  const bool act = gl < a.nlines;
  const unsigned ld = a.ld;
  const int acols = OZ_DIGITS * NT + 8;  // accumulators of a parity
  uint32_t tcols = 32;
  while ((int)tcols < 2 * acols) tcols *= 2;
  const int KR[2] = {(N + 1) / 2, N / 2}, KS[2] = {(KR[0] + 15) / 16, (KR[1] + 15) / 16};
  const uint32_t full = smem_u32(mbar), done = smem_u32(mbar + 1);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(mbar + i)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)), "r"(tcols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tslot;
  pdl_wait();  // the previous kernel's output is read from here on
  pdl_trigger();
  OzLine<INV> ln(a, job, gl, act);

  bool ok = true;
  int late = -1;  // thread 0: stage of a copy given up; none is started after it
  const int nstage = INV || !job.pd ? 1 : 2;
  for (int sg = 0; sg < nstage; ++sg) {
    const bool fd = !INV && sg == 1;
    const OzMatrix& M = INV ? a.t.T : (fd ? a.t.DF : a.t.F);
    ln.src = fd ? job.pd : job.in;
    ln.fd = fd;
    if (tid == 0 && late < 0) {  // the previous stage's products have read their matrix
      const uint32_t bytes = (uint32_t)((KS[0] + KS[1]) * bst);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(full), "r"(bytes) : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                       smem_u32(Bs)),
                   "l"(M.digits), "r"(bytes), "r"(full)
                   : "memory");
    }
    if (warp < 4) {
      OzSum sum;
      ln.magnitudes(sum, warp);
      sS[tid] = sum.S;
      sE[tid] = sum.e | (sum.nz ? 0x10000 : 0);
    }
    __syncthreads();
    const int K = oz_scale(sS + line, sE + line, OZ_LS);
    const bool live = act && K != FX_ZERO && K != FX_NAN;
    __syncthreads();  // sS, sE are free

    const int q = (warp >> 2) & 1, part = warp & 3, k0 = 8 * part;  // warps 0 ... 7: digits of 8 points of input parity q
    long long x[8];
    OzFix d[8];  // derivative
    if (warp < 8) {
      double v[8];
      if constexpr (INV) {
        const int n0 = 2 * k0 + q + (job.deriv ? 1 : 0);
        ln.load8(v, n0, 2, live ? (N - n0 + 1) >> 1 : 0);
        if (job.deriv) {
          OzFix acc{0, 0};
#pragma unroll
          for (int e = 7; e >= 0; --e) {
            if (live) acc = oz_add(acc, oz_term(v[e], K, 2 * (n0 + 2 * e)));
            d[e] = acc;
          }
          sS[tid] = (unsigned long long)acc.i;
          sE[tid] = (int)acc.f;
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = live ? fx_quant(v[e], K) : 0;
        }
      } else {
        double w[8];
        ln.load8(v, k0, 1, live ? KR[q] - k0 : 0);
        ln.load8(w, N - 1 - k0, -1, live ? N / 2 - k0 : 0);  // the middle point stands alone
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const long long xv = live ? fx_quant(v[e], K) : 0, xw = live ? fx_quant(w[e], K) : 0;
          x[e] = q ? xv - xw : xv + xw;
        }
      }
    }
    if (INV && job.deriv) {
      __syncthreads();
      if (warp < 8) {
        OzFix above{0, 0};
        for (int i = part + 1; i < 4; ++i) {
          const int o = (4 * q + i) * OZ_LS + line;
          above = oz_add(above, OzFix{(long long)sS[o], (unsigned)sE[o]});
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] = oz_add(d[e], above);
        if (2 * k0 + q == 0) d[0] = oz_half(d[0]);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = oz_round(d[e]);
      }
    }
    if (warp < 8 && (part >> 1) < KS[q])
      oz_store<4>(As + (2 * q + (part >> 1)) * OZ_ASTAGE + (line >> 3) * 256 + (part & 1) * 128 + (line & 7) * 16, x);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      if (late < 0 && mbar_wait(full, (uint32_t)(sg & 1))) {
        for (int iq = 0; iq < 2; ++iq) {
          const uint32_t acc = tmem + (uint32_t)((fd ? 1 - iq : iq) * acols);
          for (int k = 0; k < KS[iq]; ++k) {
            const uint32_t a0 = smem_u32(As + (2 * iq + k) * OZ_ASTAGE), b0 = smem_u32(Bs + (iq * KS[0] + k) * bst);
            for (int i = 0; i < OZ_DIGITS; ++i) {
              const int nc = (NT * (OZ_DIGITS - i) + 15) & ~15;
              const uint32_t idesc = (1u << 4) | ((uint32_t)(nc >> 3) << 17) | ((uint32_t)(OZ_LINES >> 4) << 24);
              mma_f16(acc + (uint32_t)(i * NT), oz_desc(a0 + i * (OZ_LINES * 32)), oz_desc(b0), idesc, k != 0 || i != 0);
            }
          }
        }
      } else {
        ok = false;
        if (late < 0) late = sg;
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(done) : "memory");
    }
    if (!mbar_wait(done, (uint32_t)(sg & 1))) ok = false;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    if constexpr (INV) {
      for (int r0 = C * warp; r0 < KR[0]; r0 += C * 16) {
        long long ev[C], od[C];
        oz_sums<C>(tq + r0, NT, ev);
        oz_sums<C>(tq + acols + r0, NT, od);
        double y[2][C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          y[0][c] = fx_to_double(r0 + c < N / 2 ? ev[c] + od[c] : ev[c], K);
          y[1][c] = fx_to_double(ev[c] - od[c], K);
        }
        if (job.deriv && a.dscale != 1.0) {
#pragma unroll
          for (int c = 0; c < C; ++c) {
            y[0][c] *= a.dscale;
            y[1][c] *= a.dscale;
          }
        }
        const unsigned o0 = (unsigned)r0 * ld + gl, o1 = (unsigned)(N - 1 - r0) * ld + gl;
        const bool w0[2] = {act && r0 < KR[0], act && r0 + 1 < KR[0]}, w1[2] = {act && r0 < N / 2, act && r0 + 1 < N / 2};
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (w0[c]) job.out[o0 + c * ld] = y[0][c];
          if (w1[c]) job.out[o1 - c * ld] = y[1][c];
        }
        if (job.gx) {
#pragma unroll
          for (int c = 0; c < C; ++c) {
            const double y0 = __shfl_xor_sync(0xffffffffu, y[0][c], 1), y1 = __shfl_xor_sync(0xffffffffu, y[1][c], 1);
            if (w0[c]) {
              job.gx[o0 + c * ld] = ln.kx * y0;
              job.gz[o0 + c * ld] = ln.kz * y0;
            }
            if (w1[c]) {
              job.gx[o1 - c * ld] = ln.kx * y1;
              job.gz[o1 - c * ld] = ln.kz * y1;
            }
          }
        }
      }
    } else {
      const int p = warp >> 3, rows = KR[p];
      const int* rexp = M.rexp + p * NT;
      for (int r0 = C * (warp & 7); r0 < rows; r0 += C * 8) {
        long long v[C];
        oz_sums<C>(tq + (uint32_t)(p * acols + r0), NT, v);
        double y[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool in = act && r0 + c < rows;
          y[c] = fx_to_double(v[c], r0 + c < rows ? K + rexp[r0 + c] : 0);
          double* out = job.out + (unsigned)(2 * (r0 + c) + p) * ld + gl;
          if (fd && in) y[c] = fma(job.wD, y[c], *out);
          if (in) *out = y[c];
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();  // sS, sE, accumulators of the next stage
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  }
  if (!ok) {  // copies and products that are still under way end before their memory is given back (bounded again)
    if (a.err) *static_cast<volatile int*>(a.err) = 1;
    if (late >= 0) mbar_wait(full, (uint32_t)late);
    mbar_wait(done, (uint32_t)(nstage - 1));
  }
  __syncwarp();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tcols));
}

int oz_nt(int N) { return ((N + 1) / 2 + 7) & ~7; }

uint16_t half_of_int(int d) {  // exact: |d| <= 256
  if (d == 0) return 0;
  const int m = d < 0 ? -d : d;
  int e = 0;
  while (m >> (e + 1)) ++e;
  return (uint16_t)((d < 0 ? 0x8000 : 0) | ((e + 15) << 10) | ((m << (10 - e)) & 0x3ff));
}

size_t oz_smem(int N, int ring, bool held) {
  const int NT = oz_nt(N);
  return ring * 2 * (size_t)(OZ_ASTAGE + oz_bstage(NT)) + OZ_THREADS * 12 + 4 * 8 + 16 +
         (held ? (size_t)NT * OZ_LINES * 8 : 0);
}

// Whether k_cheb_oz_few runs: both parities' accumulators within tensor memory (Ny <= 64) and, beside 152 SMs, CTAs for one
// wave (forward: k_cheb_oz splits its parities over CTAs) or one and a half (inverse).  FP64 steps with k_cheb_oz and with
// this: inverse of 155 CTAs (48x49x48) 97.9 and 94.0 us, of 220 (54x33x60) 102.8 and 102.1; forward of 186 CTAs (72x49x64)
// 124.4 and 130.1; both beyond the lines (72x33x54: 159 and 265 CTAs) 109.4 and 112.5.
bool oz_few(bool inverse, int N, int nlines, int njobs) {
  return 2 * (OZ_DIGITS * oz_nt(N) + 8) <= 512 &&
         (long)((nlines + OZ_LS - 1) / OZ_LS) * njobs <= (inverse ? 152 * 3 / 2 : 152);
}

template <bool INV>
cudaError_t run_oz_few(OzArgs& a, int njobs, cudaStream_t st) {
  static const bool attr = [] {
    cudaFuncSetAttribute(k_cheb_oz_few<INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return true;
  }();
  (void)attr;
  const size_t smem = 4 * (size_t)(OZ_ASTAGE + oz_bstage(a.NT)) + OZ_LS * (8 * 8 + 8 * 4) + 2 * 8 + 16;
  return launch_pdl(k_cheb_oz_few<INV>, dim3((a.nlines + OZ_LS - 1) / OZ_LS, njobs), dim3(OZ_THREADS), smem, st, a);
}

template <bool INV>
cudaError_t run_oz(OzArgs& a, int njobs, bool inplace, cudaStream_t st) {
  static const bool attr = [] {
    cudaFuncSetAttribute(k_cheb_oz<INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return true;
  }();
  (void)attr;
  // Two stages overlap the digits with the products.  Beside them the first parity's results fit in shared memory up to
  // Ny = 111; beyond, they wait in the output array, or one stage is given up where that is the input.
  bool held = INV || inplace;
  a.ring = 2;
  a.spill = 0;
  if (held && oz_smem(a.N, 2, true) > 227 * 1024) {
    if (INV && !inplace) {
      a.spill = 1;
      held = false;
    } else {
      a.ring = 1;
    }
  }
  return launch_pdl(k_cheb_oz<INV>, dim3((a.nlines + OZ_LINES - 1) / OZ_LINES, njobs, a.split ? 2 : 1), dim3(OZ_THREADS),
                    oz_smem(a.N, a.ring, held), st, a);
}

}  // namespace

size_t oz_matrix_bytes(int N) {
  const int k0 = ((N + 1) / 2 + 15) / 16, k1 = (N / 2 + 15) / 16;
  return (size_t)(k0 + k1) * oz_bstage(oz_nt(N));
}

// Digits [input parity][K step][digit and row][16 points] in the operand layout, row exponents [output parity][NT].
bool oz_matrix(int N, int kind, std::vector<uint16_t>& digits, std::vector<int>& rexp) {
  const int NT = oz_nt(N), bst = oz_bstage(NT);
  if (N < 3 || NT > 72) return false;
  typedef __int128 i128;
  std::vector<long long> ct(2 * (N - 1));  // cos(pi i / (N-1)) 2^62
  for (int i = 0; i < 2 * (N - 1); ++i) {
    const int r = std::min(i, 2 * (N - 1) - i), f = std::min(r, N - 1 - r);  // first quadrant
    const long double c = 4 * f == 2 * (N - 1) ? 0.0L : cosl(3.14159265358979323846264338327950288L * f / (N - 1));
    ct[i] = llroundl(ldexpl(f == r ? c : -c, 62));
  }
  digits.assign(oz_matrix_bytes(N) / 2, 0);
  rexp.assign(2 * NT, 0);
  size_t off = 0;
  for (int q = 0; q < 2; ++q) {
    const int KR = q ? N / 2 : (N + 1) / 2, KS = (KR + 15) / 16;
    const int opar = kind == OZ_DF ? 1 - q : q;
    const int rows = kind == OZ_T ? (N + 1) / 2 : (opar ? N / 2 : (N + 1) / 2);
    std::vector<i128> run(KR, 0), v(KR);
    // forward matrices without their factor 1 / (2 (N - 1)), times 2^62; DF by the recurrence of diff, from the top
    auto fwd = [&](int n, int j) {
      return (i128)ct[(long long)n * j % (2 * (N - 1))] * ((n == 0 || n == N - 1) ? 1 : 2) * ((j == 0 || j == N - 1) ? 1 : 2);
    };
    for (int r = rows - 1; r >= 0; --r) {
      const int n = 2 * r + opar;
      i128 big = 0;
      for (int k = 0; k < KR; ++k) {
        if (kind == OZ_T) {
          v[k] = ct[(long long)(2 * k + q) * r % (2 * (N - 1))];
        } else if (kind == OZ_F) {
          v[k] = fwd(n, k);
        } else {
          if (n + 1 < N) run[k] += fwd(n + 1, k) * (2 * (n + 1));
          v[k] = n == 0 ? run[k] / 2 : run[k];
        }
        big = std::max(big, v[k] < 0 ? -v[k] : v[k]);
      }
      // rows scaled by 2^-e to a largest magnitude in (1/2, 1]; T not, both parities of a point share its scale
      const i128 den = kind == OZ_T ? 1 : 2 * (N - 1), one = (i128)1 << 62;
      int e = 0;
      if (kind != OZ_T && big > 0) {
        while (big > (den << e) * one) ++e;
        while (e <= 0 && (big << (1 - e)) <= den * one) --e;
      }
      rexp[opar * NT + r] = -e;
      long long sum[OZ_DIGITS] = {0};
      for (int k = 0; k < KR; ++k) {
        const i128 num = e < 0 ? v[k] << -e : v[k], d2 = den << (e > 0 ? e : 0);
        long long x = (long long)((num + (num < 0 ? -d2 : d2) / 2) / d2);
        int dg[OZ_DIGITS];
        for (int s = OZ_DIGITS - 1; s > 0; --s) {
          dg[s] = (int)((x + 256) & 511) - 256;
          x = (x - dg[s]) >> 9;
        }
        dg[0] = (int)x;
        for (int s = 0; s < OZ_DIGITS; ++s) {
          sum[s] += dg[s] < 0 ? -dg[s] : dg[s];
          const int row = s * NT + r;
          digits[off / 2 + (size_t)(k >> 4) * (bst / 2) + (row >> 3) * 128 + ((k >> 3) & 1) * 64 + (row & 7) * 8 + (k & 7)] =
              half_of_int(dg[s]);
        }
      }
      // exact FP32 accumulation: every weight's sum of products below 2^24.  The line's digits are at most 256; their
      // leading ones sum to at most 128 + K over a line (sum of magnitudes below 2^61) and meet digit 6 of the row.
      long long tot = 128 + KR;
      for (int s = 0; s < OZ_DIGITS - 1; ++s) tot += sum[s];
      if (tot * 256 >= (1ll << 24)) return false;
    }
    off += (size_t)KS * bst;
  }
  return true;
}

cudaError_t launch_cheb_oz(const GridDev& g, int N, bool inverse, int nlines, size_t ld, const OzTables& t, const OzJob* jobs,
                           int njobs, int* err, cudaStream_t st) {
  if (njobs < 1 || njobs > OZ_MAX_JOBS || N != t.N || ld * (size_t)N >= (1ull << 32)) return cudaErrorInvalidValue;
  OzArgs a{};
  a.g = g;
  a.N = N;
  a.NT = oz_nt(N);
  a.nlines = nlines;
  a.ld = (unsigned)ld;
  a.dscale = 2.0 / (g.b - g.a);
  a.t = t;
  a.err = err;
  bool inplace = false;
  for (int i = 0; i < njobs; ++i) {
    if (jobs[i].inplace && jobs[i].pd) return cudaErrorInvalidValue;  // the held parity has no derivative term
    a.job[i] = jobs[i];
    inplace = inplace || jobs[i].inplace;
  }
  if (oz_few(inverse, N, nlines, njobs)) return inverse ? run_oz_few<true>(a, njobs, st) : run_oz_few<false>(a, njobs, st);
  if (inverse) return run_oz<true>(a, njobs, inplace, st);
  a.split = !inplace;  // the forward parities are independent: one CTA each
  return run_oz<false>(a, njobs, inplace, st);
}
