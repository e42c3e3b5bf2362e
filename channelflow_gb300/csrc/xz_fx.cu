// x and z passes of the FP64 path on 64-bit integers (fx.cuh): the x inverse and forward FFTs of the solved
// columns of one y-plane and component, and the z pass (c2r, the nonlinear form's products, r2c).  Arrays in and
// out are the FP64 arrays of the generic passes (k_xinv, k_zphys, k_xfwd), in the same layout.
//
// Every line is scaled on its own: a column of the x passes, each real row of the z pass (two rows share a complex
// sequence, with a scale each).
//
// Measured against the same passes in FP64 arithmetic, which the FP64 pipe bounds (one warp instruction per 64 cycles),
// at 128x97x128: z pass 340 -> 116 us, x inverse 134 -> 55 us (65 us with the vorticity formed in it), x forward 76 -> 29
// us; 192x129x160: z pass 1138 -> 353 us; bound here by integer issue.  Against radices 4, 2, 3, 5 alone: z pass 123 ->
// 116 us at 128x97x128, 402 -> 353 us at 192x129x160, 170 -> 143 us at 72x57x90 (skew-symmetric form).
// Relative error of N(u) against extended precision: 1.5e-16 ... 2.5e-16 at 32x9x32 (FP64 arithmetic 2.7e-16 ...
// 8.8e-16), for spectra from 0.5^(|kx|+|kz|) to flat.
#include "fx_fft.cuh"
#include "kernels.h"

namespace {

constexpr int FX_THREADS = 256;

__device__ __forceinline__ double fx_raw(long long v) { return __longlong_as_double(v); }

// Scales the raw doubles of one complex column (elements pos(i), i < n, all others zero) to integers in place; one
// warp.  Returns K.
template <class POS>
__device__ __forceinline__ int fx_scale_column(fxc* col, int n, POS pos, int lane) {
  unsigned key = 0;
  for (int i = lane; i < n; i += 32) {
    const fxc v = col[pos(i)];
    key = max(key, max(fx_key(fx_raw(v.x)), fx_key(fx_raw(v.y))));
  }
  key = __reduce_max_sync(0xffffffffu, key);
  const int emax = fx_exp_of_key(key);
  unsigned S = 0;
  for (int i = lane; i < n; i += 32) {
    const fxc v = col[pos(i)];
    S += fx_mag(fx_raw(v.x), emax) + fx_mag(fx_raw(v.y), emax);
  }
  S = __reduce_add_sync(0xffffffffu, S);
  const int K = fx_line_K(emax, S, 61);
  for (int i = lane; i < n; i += 32) {
    const fxc v = col[pos(i)];
    col[pos(i)] = key == 0 ? fxc{0, 0} : fxc{fx_quant(fx_raw(v.x), K), fx_quant(fx_raw(v.y), K)};
  }
  return key == 0 ? FX_ZERO : (emax == 2047 ? FX_NAN : K);
}

// Vorticity component c - 3 of a mode (wavenumbers kx, kz) at one point, W (component stride cs) = u, v, w, dw/dy, -,
// du/dy:  omega = (dw/dy - i kz v, i kz u - i kx w, i kx v - du/dy).
__device__ __forceinline__ double2 fx_vorticity(int c, const double2* W, size_t cs, double kx, double kz) {
  if (c == 4) {
    const double2 u = W[0], w = W[2 * cs];
    return make_double2(kx * w.y - kz * u.y, kz * u.x - kx * w.x);
  }
  const double2 v = W[cs], d = W[c * cs];
  if (c == 3) return make_double2(fma(kz, v.y, d.x), fma(-kz, v.x, d.y));
  return make_double2(fma(-kx, v.y, -d.x), fma(kx, v.x, -d.y));
}

__global__ void k_curl_points(GridDev g, double2* W) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, ny = blockIdx.y;
  if (i >= g.Md) return;
  const int ix = i / g.NKz, iz = i - ix * g.NKz;
  const size_t cs = (size_t)g.Ny * g.Md;
  double2* w = W + (size_t)ny * g.Md + i;
  const double kx = 2.0 * M_PI / g.Lx * (ix <= g.Kx ? ix : ix - g.NKx), kz = 2.0 * M_PI / g.Lz * iz;
  for (int c = 3; c < 6; ++c) w[c * cs] = fx_vorticity(c, w, cs, kx, kz);
}

template <bool ANY>
__global__ void __launch_bounds__(FX_THREADS, 4) k_xinv_fx(GridDev g, FxPlan px, const fxtw* __restrict__ tw,
                                                        const double2* __restrict__ W, double2* __restrict__ X, int czc,
                                                        int curl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_wait();  // launched with launch_pdl: the previous kernel's output is read from here on
  const int ss = g.Nx + 1;
  const int iz0 = blockIdx.z * czc, nc = min(czc, g.NKz - iz0);
  const float invc = 1.0f / nc;
  fxc* a = reinterpret_cast<fxc*>(smem_raw);
  fxc* b = a + (size_t)czc * ss;
  double* skx = reinterpret_cast<double*>(b + (size_t)czc * ss);  // wavenumbers (curl)
  double* skz = skx + (curl ? g.NKx : 0);
  int* sK = reinterpret_cast<int*>(skz + (curl ? czc : 0));
  const int ny = blockIdx.x, c = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double2* src = W + ((size_t)c * g.Ny + ny) * g.Md;
  const int Kx = g.Kx, NKx = g.NKx, Nx = g.Nx;
  if (curl && c >= 3) {
    for (int i = tid; i < NKx; i += FX_THREADS) skx[i] = 2.0 * M_PI * (i <= Kx ? i : i - NKx) / g.Lx;
    for (int i = tid; i < nc; i += FX_THREADS) skz[i] = 2.0 * M_PI * (iz0 + i) / g.Lz;
    __syncthreads();
  }
#pragma unroll 4
  for (int i = tid; i < NKx * nc; i += FX_THREADS) {
    int ix, jz;
    divmod_small(i, nc, invc, ix, jz);
    double2 v = src[ix * g.NKz + iz0 + jz];
    if (curl && c >= 3) v = fx_vorticity(c, W + (size_t)ny * g.Md + ix * g.NKz + iz0 + jz, (size_t)g.Ny * g.Md,
                                         skx[ix], skz[jz]);
    a[jz * ss + (ix <= Kx ? ix : Nx + ix - NKx)] = fxc{__double_as_longlong(v.x), __double_as_longlong(v.y)};
  }
  {
    const int G = Nx - NKx;  // the unsolved wavenumbers
    const float invg = 1.0f / G;
    for (int i = tid; i < nc * G; i += FX_THREADS) {
      int jz, p;
      divmod_small(i, G, invg, jz, p);
      a[jz * ss + Kx + 1 + p] = fxc{0, 0};
    }
  }
  __syncthreads();
  for (int jz = warp; jz < nc; jz += FX_THREADS / 32) {
    const int K = fx_scale_column(a + jz * ss, NKx, [=](int i) { return i <= Kx ? i : Nx + i - NKx; }, lane);
    if (lane == 0) sK[jz] = K;
  }
  __syncthreads();
  const fxc* r = a + fx_fft<ANY>(0, czc * ss, nc, ss, px.L, px.rad, tw, true);
  double2* dst = X + ((size_t)c * g.Ny + ny) * (size_t)Nx * g.NKz;
  for (int i = tid; i < Nx * nc; i += FX_THREADS) {
    int x, jz;
    divmod_small(i, nc, invc, x, jz);
    const fxc v = r[jz * ss + x];
    const int K = sK[jz];
    dst[x * g.NKz + iz0 + jz] = make_double2(fx_double(v.x, K), fx_double(v.y, K));
  }
}

template <bool ANY>
__global__ void __launch_bounds__(FX_THREADS, 4) k_xfwd_fx(GridDev g, FxPlan px, const fxtw* __restrict__ tw,
                                                        const double2* __restrict__ Z, double2* __restrict__ F,
                                                        double scale, int czc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_wait();  // launched with launch_pdl: the previous kernel's output is read from here on
  const int ss = g.Nx + 1;
  const int iz0 = blockIdx.z * czc, nc = min(czc, g.NKz - iz0);
  const float invc = 1.0f / nc;
  fxc* a = reinterpret_cast<fxc*>(smem_raw);
  fxc* b = a + (size_t)czc * ss;
  int* sK = reinterpret_cast<int*>(b + (size_t)czc * ss);
  const int ny = blockIdx.x, c = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double2* src = Z + ((size_t)c * g.Ny + ny) * (size_t)g.Nx * g.NKz;
#pragma unroll 4
  for (int i = tid; i < g.Nx * nc; i += FX_THREADS) {
    int x, jz;
    divmod_small(i, nc, invc, x, jz);
    const double2 v = src[x * g.NKz + iz0 + jz];
    a[jz * ss + x] = fxc{__double_as_longlong(v.x), __double_as_longlong(v.y)};
  }
  __syncthreads();
  for (int jz = warp; jz < nc; jz += FX_THREADS / 32) {
    const int K = fx_scale_column(a + jz * ss, g.Nx, [](int i) { return i; }, lane);
    if (lane == 0) sK[jz] = K;
  }
  __syncthreads();
  const fxc* r = a + fx_fft<ANY>(0, czc * ss, nc, ss, px.L, px.rad, tw, false);
  double2* dst = F + ((size_t)c * g.Ny + ny) * g.Md;
#pragma unroll 4
  for (int i = tid; i < g.NKx * nc; i += FX_THREADS) {
    int ix, jz;
    divmod_small(i, nc, invc, ix, jz);
    const fxc v = r[jz * ss + (ix <= g.Kx ? ix : g.Nx + ix - g.NKx)];
    const int K = sK[jz];
    dst[ix * g.NKz + iz0 + jz] = make_double2(fx_double(v.x, K) * scale, fx_double(v.y, K) * scale);
  }
}

// ---------------------------------------------------------------------------
// z pass.  Real sequence k of the block (row r = k / NC, component c = k % NC) is half of complex sequence k / 2.
// ---------------------------------------------------------------------------
template <int FORM>
struct FxForm;
template <>
struct FxForm<NL_ROTATIONAL> { static constexpr int NC = 6, NO = 3; };
template <>
struct FxForm<NL_CONVECTION> { static constexpr int NC = 12, NO = 3; };
template <>
struct FxForm<NL_DIVERGENCE> { static constexpr int NC = 3, NO = 6; };
template <>
struct FxForm<NL_SKEW> { static constexpr int NC = 12, NO = 9; };

// Products of the form: output o is the sum of its terms c[a] c[b] (sub: minus).
struct FxTerm {
  int a, b;
  bool sub;
};
template <int FORM>
__host__ __device__ constexpr int fx_nterm(int o) {
  return FORM == NL_ROTATIONAL ? 2 : ((FORM == NL_CONVECTION || (FORM == NL_SKEW && o < 3)) ? 3 : 1);
}
template <int FORM>
__host__ __device__ constexpr FxTerm fx_term(int o, int t) {
  if (FORM == NL_ROTATIONAL) {  // omega x u, c = u, v, w, ox, oy, oz
    const int j = (o + 1) % 3, k = (o + 2) % 3;
    return t == 0 ? FxTerm{3 + j, k, false} : FxTerm{3 + k, j, true};
  }
  if (FORM == NL_CONVECTION || (FORM == NL_SKEW && o < 3)) return FxTerm{t, 3 + 3 * o + t, false};  // u_j d u_o / d x_j
  const int q = FORM == NL_SKEW ? o - 3 : o;  // uu, uv, uw, vv, vw, ww
  return FxTerm{q < 3 ? 0 : (q < 5 ? 1 : 2), q < 3 ? q : (q < 5 ? q - 2 : 2), false};
}

__device__ __forceinline__ unsigned fx_absbits(long long v) {
  const int h = (int)(v >> 32);
  return (unsigned)(h ^ (h >> 31));
}
__device__ __forceinline__ long long fx_round_shift(long long v, int s) {  // v 2^s
  return s >= 0 ? v << s : ((v >> (min(-s, 63) - 1)) + 1) >> 1;
}

template <int FORM, bool ANY>
__global__ void __launch_bounds__(FX_THREADS, 4) k_zphys_fx(GridDev g, FxPlan pz, const fxtw* __restrict__ tw, int RP,
                                                         const double2* __restrict__ X, double2* __restrict__ Z) {
  constexpr int NC = FxForm<FORM>::NC, NO = FxForm<FORM>::NO;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_wait();  // launched with launch_pdl: the previous kernel's output is read from here on
  const int Nz = g.Nz, ss = Nz + 1, NKz = g.NKz;
  const int nseq = ((NC > NO ? NC : NO) * RP) / 2;
  const int ninv = NC * RP / 2, nfwd = NO * RP / 2;
  fxc* A = reinterpret_cast<fxc*>(smem_raw);
  fxc* B = A + (size_t)nseq * ss;
  int* sK = reinterpret_cast<int*>(B + (size_t)nseq * ss);  // exponent K of every component's row (normalised)
  int* sN = sK + 2 * nseq;                                  // left shift that normalises it
  int* sF = sN + 2 * nseq;                                  // exponent K of every output's row
  const int ny = blockIdx.y, x0 = blockIdx.x * RP;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t plane = (size_t)g.Nx * NKz;
  const float invk = 1.0f / NKz;
  {
    // the pack below writes bins 0..NKz-1 and Nz-NKz+1..Nz-1 of every inverse sequence: zero the gap
    const int G = Nz - 2 * NKz + 1;
    const float invg = 1.0f / G;
    for (int i = tid; i < ninv * G; i += FX_THREADS) {
      int sq, z;
      divmod_small(i, G, invg, sq, z);
      A[(size_t)sq * ss + NKz + z] = fxc{0, 0};
    }
  }
  // raw doubles of the two rows a, b of a sequence: bin iz holds a's coefficient, bin Nz - iz b's, bin 0 both
#pragma unroll 4
  for (int i = tid; i < ninv * NKz; i += FX_THREADS) {
    int s, iz;
    divmod_small(i, NKz, invk, s, iz);
    const int k0 = 2 * s, k1 = 2 * s + 1;
    const int r0 = k0 / NC, c0 = k0 % NC, r1 = k1 / NC, c1 = k1 % NC;
    double2 ca = make_double2(0, 0), cb = make_double2(0, 0);
    if (x0 + r0 < g.Nx) ca = X[((size_t)c0 * g.Ny + ny) * plane + (size_t)(x0 + r0) * NKz + iz];
    if (x0 + r1 < g.Nx) cb = X[((size_t)c1 * g.Ny + ny) * plane + (size_t)(x0 + r1) * NKz + iz];
    fxc* sq = A + (size_t)s * ss;
    if (iz == 0) {
      sq[0] = fxc{__double_as_longlong(ca.x), __double_as_longlong(cb.x)};
    } else {
      sq[iz] = fxc{__double_as_longlong(ca.x), __double_as_longlong(ca.y)};
      sq[Nz - iz] = fxc{__double_as_longlong(cb.x), __double_as_longlong(cb.y)};
    }
  }
  __syncthreads();
  for (int s = warp; s < ninv; s += FX_THREADS / 32) {
    fxc* sq = A + (size_t)s * ss;
    unsigned ka = 0, kb = 0;
    for (int iz = lane; iz < NKz; iz += 32) {
      const fxc p = sq[iz];
      if (iz == 0) {
        ka = fx_key(fx_raw(p.x));
        kb = fx_key(fx_raw(p.y));
      } else {
        const fxc q = sq[Nz - iz];
        ka = max(ka, max(fx_key(fx_raw(p.x)), fx_key(fx_raw(p.y))));
        kb = max(kb, max(fx_key(fx_raw(q.x)), fx_key(fx_raw(q.y))));
      }
    }
    ka = __reduce_max_sync(0xffffffffu, ka);
    kb = __reduce_max_sync(0xffffffffu, kb);
    const int ea = fx_exp_of_key(ka), eb = fx_exp_of_key(kb);
    unsigned Sa = 0, Sb = 0;  // every coefficient but the mean appears twice in the sequence
    for (int iz = lane; iz < NKz; iz += 32) {
      const fxc p = sq[iz];
      if (iz == 0) {
        Sa = fx_mag(fx_raw(p.x), ea);
        Sb = fx_mag(fx_raw(p.y), eb);
      } else {
        const fxc q = sq[Nz - iz];
        Sa += 2 * (fx_mag(fx_raw(p.x), ea) + fx_mag(fx_raw(p.y), ea));
        Sb += 2 * (fx_mag(fx_raw(q.x), eb) + fx_mag(fx_raw(q.y), eb));
      }
    }
    Sa = __reduce_add_sync(0xffffffffu, Sa);
    Sb = __reduce_add_sync(0xffffffffu, Sb);
    const int Ka = fx_line_K(ea, Sa, 60), Kb = fx_line_K(eb, Sb, 60);
    for (int iz = lane; iz < NKz; iz += 32) {
      const fxc p = sq[iz];
      if (iz == 0) {
        sq[0] = fxc{ka ? fx_quant(fx_raw(p.x), Ka) : 0, kb ? fx_quant(fx_raw(p.y), Kb) : 0};
      } else {
        const fxc q = sq[Nz - iz];
        const long long ax = ka ? fx_quant(fx_raw(p.x), Ka) : 0, ay = ka ? fx_quant(fx_raw(p.y), Ka) : 0;
        const long long bx = kb ? fx_quant(fx_raw(q.x), Kb) : 0, by = kb ? fx_quant(fx_raw(q.y), Kb) : 0;
        sq[iz] = fxc{ax - by, ay + bx};       // A_k + i B_k
        sq[Nz - iz] = fxc{ax + by, bx - ay};  // conj(A_k) + i conj(B_k)
      }
    }
    if (lane == 0) {
      sK[2 * s] = ka == 0 ? FX_ZERO : (ea == 2047 ? FX_NAN : Ka);
      sK[2 * s + 1] = kb == 0 ? FX_ZERO : (eb == 2047 ? FX_NAN : Kb);
    }
  }
  __syncthreads();
  fxc* P = A + fx_fft<ANY>(0, nseq * ss, ninv, ss, pz.L, pz.rad, tw, true);
  fxc* Q = P == A ? B : A;
  // normalise every component by its largest value: the scale above allows for the sum of magnitudes
  for (int s = warp; s < ninv; s += FX_THREADS / 32) {
    const fxc* sq = P + (size_t)s * ss;
    unsigned mx = 0, my = 0;
    for (int z = lane; z < Nz; z += 32) {
      const fxc v = sq[z];
      mx |= fx_absbits(v.x);
      my |= fx_absbits(v.y);
    }
    mx = __reduce_or_sync(0xffffffffu, mx);
    my = __reduce_or_sync(0xffffffffu, my);
    if (lane < 2) {
      const int n = max(__clz(lane == 0 ? mx : my) - 3, 0);  // |v| < 2^61 after the shift
      sN[2 * s + lane] = n;
      sK[2 * s + lane] += n;
    }
  }
  __syncthreads();
  for (int i = tid; i < RP * Nz; i += FX_THREADS) {
    const int r = i / Nz, z = i - r * Nz;
    long long c[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const int k = r * NC + q;
      const fxc* v = P + (size_t)(k >> 1) * ss + z;
      c[q] = ((k & 1) ? v->y : v->x) << sN[k];
    }
    const int* Kr = sK + r * NC;
#pragma unroll
    for (int o = 0; o < NO; ++o) {
      constexpr int MT = 3;
      int kt[MT], km = INT32_MAX;
#pragma unroll
      for (int t = 0; t < MT; ++t)
        if (t < fx_nterm<FORM>(o)) {
          kt[t] = Kr[fx_term<FORM>(o, t).a] + Kr[fx_term<FORM>(o, t).b];
          km = min(km, kt[t]);
        }
      long long f = 0;
#pragma unroll
      for (int t = 0; t < MT; ++t)
        if (t < fx_nterm<FORM>(o)) {
          const long long p = fx_mulhi(c[fx_term<FORM>(o, t).a], c[fx_term<FORM>(o, t).b]) >> min(kt[t] - km, 63);
          f = fx_term<FORM>(o, t).sub ? f - p : f + p;
        }
      const int k = r * NO + o;
      long long* q = reinterpret_cast<long long*>(Q + (size_t)(k >> 1) * ss + z);
      q[k & 1] = f;
      if (z == 0) sF[k] = km - 64;
    }
  }
  __syncthreads();
  // scale every output row to the sum of its magnitudes (2^60 per half)
  for (int s = warp; s < nfwd; s += FX_THREADS / 32) {
    fxc* sq = Q + (size_t)s * ss;
    unsigned Sx = 0, Sy = 0;
    for (int z = lane; z < Nz; z += 32) {
      const fxc v = sq[z];
      Sx += (fx_absbits(v.x) >> 8) + 1;  // units 2^40
      Sy += (fx_absbits(v.y) >> 8) + 1;
    }
    Sx = __reduce_add_sync(0xffffffffu, Sx);
    Sy = __reduce_add_sync(0xffffffffu, Sy);
    const int sx = 20 - (32 - __clz(Sx)), sy = 20 - (32 - __clz(Sy));
    for (int z = lane; z < Nz; z += 32) {
      const fxc v = sq[z];
      sq[z] = fxc{fx_round_shift(v.x, sx), fx_round_shift(v.y, sy)};
    }
    if (lane == 0) {
      sF[2 * s] += sx;
      sF[2 * s + 1] += sy;
    }
  }
  __syncthreads();
  const fxc* G = A + fx_fft<ANY>((int)(Q - A), (int)(P - A), nfwd, ss, pz.L, pz.rad, tw, false);
#pragma unroll 2
  for (int i = tid; i < nfwd * NKz; i += FX_THREADS) {
    int s, iz;
    divmod_small(i, NKz, invk, s, iz);
    const fxc* sq = G + (size_t)s * ss;
    const fxc zk = sq[iz], zm = sq[iz == 0 ? 0 : Nz - iz];
    const int k0 = 2 * s, k1 = 2 * s + 1;
    const int r0 = k0 / NO, o0 = k0 % NO, r1 = k1 / NO, o1 = k1 % NO;
    const int K0 = sF[k0] + 1, K1 = sF[k1] + 1;  // + 1: half the sum
    if (x0 + r0 < g.Nx)
      Z[((size_t)o0 * g.Ny + ny) * plane + (size_t)(x0 + r0) * NKz + iz] =
          make_double2(fx_double(zk.x + zm.x, K0), fx_double(zk.y - zm.y, K0));
    if (x0 + r1 < g.Nx)
      Z[((size_t)o1 * g.Ny + ny) * plane + (size_t)(x0 + r1) * NKz + iz] =
          make_double2(fx_double(zk.y + zm.y, K1), fx_double(zm.x - zk.x, K1));
  }
}

// ---------------------------------------------------------------------------
// Whole-FlowField passes (transforms.cu), in place: every mode, Nyquist included.
// ---------------------------------------------------------------------------

// Complex FFT along x of columns [z0, z0 + cols) of one plane [x][Mz]; plane blockIdx.x, column chunk blockIdx.y.
template <bool ANY>
__global__ void __launch_bounds__(FX_THREADS, 4) k_field_x(int Nx, int Mz, int cols, FxPlan px, const fxtw* __restrict__ tw,
                                                        int sign, double scale, double2* __restrict__ data) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ss = Nx + 1, z0 = blockIdx.y * cols, nc = min(cols, Mz - z0);
  const float invc = 1.0f / nc;
  fxc* a = reinterpret_cast<fxc*>(smem_raw);
  fxc* b = a + (size_t)cols * ss;
  int* sK = reinterpret_cast<int*>(b + (size_t)cols * ss);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* plane = data + blockIdx.x * (size_t)Nx * Mz + z0;
#pragma unroll 4
  for (int i = tid; i < Nx * nc; i += FX_THREADS) {
    int x, c;
    divmod_small(i, nc, invc, x, c);
    const double2 v = plane[(size_t)x * Mz + c];
    a[c * ss + x] = fxc{__double_as_longlong(v.x), __double_as_longlong(v.y)};
  }
  __syncthreads();
  for (int c = warp; c < nc; c += FX_THREADS / 32) {
    const int K = fx_scale_column(a + c * ss, Nx, [](int i) { return i; }, lane);
    if (lane == 0) sK[c] = K;
  }
  __syncthreads();
  const fxc* r = a + fx_fft<ANY>(0, cols * ss, nc, ss, px.L, px.rad, tw, sign > 0);
#pragma unroll 2
  for (int i = tid; i < Nx * nc; i += FX_THREADS) {
    int x, c;
    divmod_small(i, nc, invc, x, c);
    const fxc v = r[c * ss + x];
    plane[(size_t)x * Mz + c] = make_double2(fx_double(v.x, sK[c]) * scale, fx_double(v.y, sK[c]) * scale);
  }
}

// z transform of x rows, two real rows per complex sequence, with a scale each.  Rows of Nzpad = Nz + 2 doubles;
// c2r (INV): Nz / 2 + 1 complex in (the imaginary parts of the first and last are not used), Nz reals out, the padding
// zero; r2c: the reverse.
template <bool INV, bool ANY>
__global__ void __launch_bounds__(FX_THREADS, 4) k_field_z(long long nrows, int Nz, int seqs, FxPlan pz,
                                                        const fxtw* __restrict__ tw, double* __restrict__ data) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ss = Nz + 1, Mz = Nz / 2 + 1, Nzpad = 2 * Mz;
  fxc* a = reinterpret_cast<fxc*>(smem_raw);
  fxc* b = a + (size_t)seqs * ss;
  int* sK = reinterpret_cast<int*>(b + (size_t)seqs * ss);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long row0 = 2ll * seqs * blockIdx.x;
  const int nr = (int)min((long long)(2 * seqs), nrows - row0), ns = (nr + 1) / 2;  // an odd last row pairs with zeros
  double* rows = data + row0 * Nzpad;
  const float invz = 1.0f / Nz, invm = 1.0f / Mz;
  if (INV) {
    // bin k < Mz of row 2 s at k, of row 2 s + 1 at Nz - k (the ends: both real parts in one element)
#pragma unroll 2
    for (int i = tid; i < ns * Mz; i += FX_THREADS) {
      int s, k;
      divmod_small(i, Mz, invm, s, k);
      const double2 p = reinterpret_cast<const double2*>(rows + (size_t)(2 * s) * Nzpad)[k];
      const double2 q = 2 * s + 1 < nr ? reinterpret_cast<const double2*>(rows + (size_t)(2 * s + 1) * Nzpad)[k]
                                       : make_double2(0, 0);
      fxc* sq = a + (size_t)s * ss;
      if (k == 0 || 2 * k == Nz) {
        sq[k] = fxc{__double_as_longlong(p.x), __double_as_longlong(q.x)};
      } else {
        sq[k] = fxc{__double_as_longlong(p.x), __double_as_longlong(p.y)};
        sq[Nz - k] = fxc{__double_as_longlong(q.x), __double_as_longlong(q.y)};
      }
    }
  } else {
#pragma unroll 2
    for (int i = tid; i < ns * Nz; i += FX_THREADS) {
      int s, z;
      divmod_small(i, Nz, invz, s, z);
      const double p = rows[(size_t)(2 * s) * Nzpad + z];
      const double q = 2 * s + 1 < nr ? rows[(size_t)(2 * s + 1) * Nzpad + z] : 0.0;
      a[(size_t)s * ss + z] = fxc{__double_as_longlong(p), __double_as_longlong(q)};
    }
  }
  __syncthreads();
  for (int s = warp; s < ns; s += FX_THREADS / 32) {
    fxc* sq = a + (size_t)s * ss;
    const int n = INV ? Mz : Nz;
    // raw values of element i: row 0's in p, row 1's in q; ends: real values only
    auto get = [&](int i, double (&p)[2], double (&q)[2]) {
      const fxc v = sq[i];
      const bool real = !INV || i == 0 || 2 * i == Nz;
      const fxc w = real ? fxc{v.y, 0} : sq[Nz - i];
      p[0] = fx_raw(v.x);
      p[1] = real ? 0.0 : fx_raw(v.y);
      q[0] = fx_raw(w.x);
      q[1] = real ? 0.0 : fx_raw(w.y);
    };
    unsigned ka = 0, kb = 0;
    for (int i = lane; i < n; i += 32) {
      double p[2], q[2];
      get(i, p, q);
      ka = max(ka, max(fx_key(p[0]), fx_key(p[1])));
      kb = max(kb, max(fx_key(q[0]), fx_key(q[1])));
    }
    ka = __reduce_max_sync(0xffffffffu, ka);
    kb = __reduce_max_sync(0xffffffffu, kb);
    const int ea = fx_exp_of_key(ka), eb = fx_exp_of_key(kb);
    unsigned Sa = 0, Sb = 0;  // a c2r coefficient appears twice in the sequence
    for (int i = lane; i < n; i += 32) {
      double p[2], q[2];
      get(i, p, q);
      Sa += fx_mag(p[0], ea) + fx_mag(p[1], ea);
      Sb += fx_mag(q[0], eb) + fx_mag(q[1], eb);
    }
    Sa = __reduce_add_sync(0xffffffffu, Sa) * (INV ? 2 : 1);
    Sb = __reduce_add_sync(0xffffffffu, Sb) * (INV ? 2 : 1);
    const int Ka = fx_line_K(ea, Sa, 60), Kb = fx_line_K(eb, Sb, 60);
    for (int i = lane; i < n; i += 32) {
      double p[2], q[2];
      get(i, p, q);
      const long long ax = ka ? fx_quant(p[0], Ka) : 0, ay = ka ? fx_quant(p[1], Ka) : 0;
      const long long bx = kb ? fx_quant(q[0], Kb) : 0, by = kb ? fx_quant(q[1], Kb) : 0;
      if (!INV || i == 0 || 2 * i == Nz) {
        sq[i] = fxc{ax, bx};
      } else {
        sq[i] = fxc{ax - by, ay + bx};       // A_k + i B_k
        sq[Nz - i] = fxc{ax + by, bx - ay};  // conj(A_k) + i conj(B_k)
      }
    }
    if (lane == 0) {
      sK[2 * s] = ka == 0 ? FX_ZERO : (ea == 2047 ? FX_NAN : Ka);
      sK[2 * s + 1] = kb == 0 ? FX_ZERO : (eb == 2047 ? FX_NAN : Kb);
    }
  }
  __syncthreads();
  const fxc* G = a + fx_fft<ANY>(0, seqs * ss, ns, ss, pz.L, pz.rad, tw, INV);
  if (INV) {
#pragma unroll 2
    for (int i = tid; i < ns * Nz; i += FX_THREADS) {
      int s, z;
      divmod_small(i, Nz, invz, s, z);
      const fxc v = G[(size_t)s * ss + z];
      rows[(size_t)(2 * s) * Nzpad + z] = fx_double(v.x, sK[2 * s]);
      if (2 * s + 1 < nr) rows[(size_t)(2 * s + 1) * Nzpad + z] = fx_double(v.y, sK[2 * s + 1]);
    }
    for (int i = tid; i < 2 * nr; i += FX_THREADS) rows[(size_t)(i >> 1) * Nzpad + Nz + (i & 1)] = 0.0;
  } else {
#pragma unroll 2
    for (int i = tid; i < ns * Mz; i += FX_THREADS) {
      int s, k;
      divmod_small(i, Mz, invm, s, k);
      const fxc zk = G[(size_t)s * ss + k], zm = G[(size_t)s * ss + (k == 0 ? 0 : Nz - k)];
      const int K0 = sK[2 * s] + 1, K1 = sK[2 * s + 1] + 1;  // + 1: half the sum
      reinterpret_cast<double2*>(rows + (size_t)(2 * s) * Nzpad)[k] =
          make_double2(fx_double(zk.x + zm.x, K0), fx_double(zk.y - zm.y, K0));
      if (2 * s + 1 < nr)
        reinterpret_cast<double2*>(rows + (size_t)(2 * s + 1) * Nzpad)[k] =
            make_double2(fx_double(zk.y + zm.y, K1), fx_double(zm.x - zk.x, K1));
    }
  }
}

template <int FORM>
cudaError_t run_zphys_fx(const GridDev& g, const FftPlan& pz, const fxtw* tw, int RP, const double2* X, double2* Z,
                         cudaStream_t st) {
  static const bool attr = [] {
    cudaFuncSetAttribute(k_zphys_fx<FORM, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    cudaFuncSetAttribute(k_zphys_fx<FORM, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return true;
  }();
  (void)attr;
  const FxPlan p = fx_plan(pz.L);
  return launch_pdl(p.any ? k_zphys_fx<FORM, true> : k_zphys_fx<FORM, false>, dim3((g.Nx + RP - 1) / RP, g.Ny), dim3(FX_THREADS),
                    zphys_smem_bytes<double>(g, FORM, RP), st, g, p, tw, RP, X, Z);
}

size_t xfx_smem(const GridDev& g, int czc, bool curl) {
  return xfft_smem_bytes<double>(g, czc) + sizeof(int) * czc + (curl ? sizeof(double) * (g.NKx + czc) : 0);
}

}  // namespace

// Shared memory of n sequences of length L with their exponents (two per sequence).
static size_t field_smem(int L, int n) { return (2 * sizeof(fxc) * (size_t)(L + 1) + 2 * sizeof(int)) * n; }

cudaError_t launch_field_x(int Nx, int Mz, int nplanes, const void* tw, int sign, double scale,
                           cpx<double>* data, cudaStream_t st) {
  static const bool attr = [] {
    cudaFuncSetAttribute(k_field_x<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    cudaFuncSetAttribute(k_field_x<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return true;
  }();
  (void)attr;
  int cols = 1;  // about 64 KB of columns: three blocks an SM
  while (cols < Mz && cols < 16 && field_smem(Nx, cols + 1) <= 64 * 1024) ++cols;
  const FxPlan p = fx_plan(Nx);
  const auto k = p.any ? k_field_x<true> : k_field_x<false>;
  k<<<dim3(nplanes, (Mz + cols - 1) / cols), FX_THREADS, field_smem(Nx, cols), st>>>(Nx, Mz, cols, p, (const fxtw*)tw, sign,
                                                                                     scale, (double2*)data);
  return cudaGetLastError();
}

cudaError_t launch_field_z(long long nrows, int Nz, bool inverse, const void* tw, double* data,
                           cudaStream_t st) {
  static const bool attr = [] {
    for (auto k : {k_field_z<false, false>, k_field_z<false, true>, k_field_z<true, false>, k_field_z<true, true>})
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return true;
  }();
  (void)attr;
  int seqs = 1;
  while (seqs < 16 && field_smem(Nz, seqs + 1) <= 64 * 1024) ++seqs;
  const unsigned nb = (unsigned)((nrows + 2 * seqs - 1) / (2 * seqs));
  const FxPlan p = fx_plan(Nz);
  const auto k = inverse ? (p.any ? k_field_z<true, true> : k_field_z<true, false>)
                         : (p.any ? k_field_z<false, true> : k_field_z<false, false>);
  k<<<nb, FX_THREADS, field_smem(Nz, seqs), st>>>(nrows, Nz, seqs, p, (const fxtw*)tw, data);
  return cudaGetLastError();
}

cudaError_t launch_xinv_fx(const GridDev& g, const FftPlan& px, const void* tw, const cpx<double>* W, cpx<double>* X,
                           int ncomp, int czc, bool curl, cudaStream_t st) {
  static const bool attr = [] {
    cudaFuncSetAttribute(k_xinv_fx<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    cudaFuncSetAttribute(k_xinv_fx<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return true;
  }();
  (void)attr;
  const FxPlan p = fx_plan(px.L);
  return launch_pdl(p.any ? k_xinv_fx<true> : k_xinv_fx<false>, dim3(g.Ny, ncomp, (g.NKz + czc - 1) / czc), dim3(FX_THREADS),
                    xfx_smem(g, czc, curl), st, g, p, (const fxtw*)tw, (const double2*)W, (double2*)X, czc, (int)curl);
}

cudaError_t launch_curl_points(const GridDev& g, cpx<double>* W, cudaStream_t st) {
  k_curl_points<<<dim3((g.Md + 127) / 128, g.Ny), 128, 0, st>>>(g, (double2*)W);
  return cudaGetLastError();
}

cudaError_t launch_xfwd_fx(const GridDev& g, const FftPlan& px, const void* tw, const cpx<double>* Z, cpx<double>* F,
                           int ncomp, int czc, cudaStream_t st) {
  static const bool attr = [] {
    cudaFuncSetAttribute(k_xfwd_fx<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    cudaFuncSetAttribute(k_xfwd_fx<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return true;
  }();
  (void)attr;
  const double scale = 1.0 / ((double)g.Nx * (double)g.Nz);
  const FxPlan p = fx_plan(px.L);
  return launch_pdl(p.any ? k_xfwd_fx<true> : k_xfwd_fx<false>, dim3(g.Ny, ncomp, (g.NKz + czc - 1) / czc), dim3(FX_THREADS),
                    xfx_smem(g, czc, false), st, g, p, (const fxtw*)tw, (const double2*)Z, (double2*)F, scale, czc);
}

cudaError_t launch_zphys_fx(const GridDev& g, int form, const FftPlan& pz, const void* tw, int RP, const cpx<double>* X,
                            cpx<double>* Z, cudaStream_t st) {
  const fxtw* t = (const fxtw*)tw;
  const double2* x = (const double2*)X;
  double2* z = (double2*)Z;
  if (RP < 2 || RP % 2) return cudaErrorInvalidValue;  // whole pairs of output rows
  switch (form) {
    case NL_ROTATIONAL: return run_zphys_fx<NL_ROTATIONAL>(g, pz, t, RP, x, z, st);
    case NL_CONVECTION: return run_zphys_fx<NL_CONVECTION>(g, pz, t, RP, x, z, st);
    case NL_DIVERGENCE: return run_zphys_fx<NL_DIVERGENCE>(g, pz, t, RP, x, z, st);
    case NL_SKEW: return run_zphys_fx<NL_SKEW>(g, pz, t, RP, x, z, st);
    default: return cudaErrorInvalidValue;
  }
}
