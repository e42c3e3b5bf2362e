// FlowField transforms on the GPU: makePhysical / makeSpectral and their
// xz and y halves, on a whole FlowField buffer in the reference's serial
// layout (every mode, Nyquist included), FP64.
//
// Reference functions restated (channelflow project paths):
//   FlowField::makeSpectral_xz / makePhysical_xz   channelflow/flowfield.cpp:1850-1886
//       (FFTW r2c / c2r over (x, z) per (y, component), 1/(Nx Nz) on the forward transform)
//   FlowField::makeSpectral_y / makePhysical_y     channelflow/flowfield.cpp:1888-1987
//       (REDFT00 along y per (x, z, component); chebyfft/ichebyfft scaling, chebyshev.cpp:262-303)
//   FlowField::makeSpectral / makePhysical         channelflow/flowfield.cpp:1989-1997
//   the (xzstate, ystate) bookkeeping              channelflow/flowfield.h:280-282
//
// Buffer layout (flowfield.h:370-400): Nd*Ny*Nx*Nzpad doubles, Nzpad = 2*(Nz/2+1).
//   xz-physical:  real u(nx, ny, nz, i) at nz + Nzpad*(nx + Nx*(ny + Ny*i)), nz < Nz
//   xz-spectral:  complex u(mx, my, mz, i) at mz + Mz*(mx + Nx*(my + Ny*i)), Mz = Nz/2+1
// The y transforms act on the reals along y (stride Nx*Nzpad) in either xz state, so a y transform of an
// xz-spectral field transforms the real and imaginary parts of every mode.
//
// Kernels (not on the DNS step's hot path, which keeps only solved modes and fuses its transforms into the
// nonlinear pass):
//   launch_cheb_oz (cheb_oz.cu)  y-lines on the tensor cores, in place; where Ny is not covered:
//   k_cheb_full   dense Ny x Ny FP64 product per y-line, 32 x 32 output tiles staged through shared memory
//   launch_field_x (xz_fx.cu)  complex FFT along x of kz columns of one (y, component) plane, in place
//   launch_field_z (xz_fx.cu)  z transform of x rows: c2r (Hermitian completion, FFTW's convention of taking only the
//                 real parts of the kz = 0 and Nz/2 terms) or r2c, in place
//   k_long_x, k_long_z  the same of lines longer than FX_LMAX (fx_plan.h), in FP64 arithmetic (fft.cuh), the more exact
//                 there
// The FFTs run on 64-bit integers (fx.cuh); against the same passes in FP64 arithmetic, 128x97x128, three components:
// z 247 -> 51 us, x 135 -> 48 us.
#include "../../include/cfgpu.h"
#include "kernels.h"

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <string>
#include <vector>

bool cfgpu_fft_plan(int L, FftPlan& p, std::vector<std::complex<long double>>& tw);

namespace {

int tf_fail(int code, const std::string& m) { return cfgpu_record_error(code, m); }

#define TF_CK(x)                                                                                  \
  do {                                                                                            \
    cudaError_t e_ = (x);                                                                         \
    if (e_ != cudaSuccess) return tf_fail(CFGPU_ECUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

constexpr int TF_MAX = 3071;  // longest x or z line (96 KB of shared memory with its copy)
constexpr int CT = 32;  // tile edge of the Chebyshev product

// out[c][j][l] = sum_n M[j][n] in[c][n][l] for j < N, l < nl; blocks: (line tiles, row tiles, components).
__global__ void __launch_bounds__(256) k_cheb_full(int N, int nl, size_t cs, const double* __restrict__ M,
                                                   const double* __restrict__ in, double* __restrict__ out) {
  __shared__ double sM[CT][CT + 1];
  __shared__ double sX[CT][CT + 1];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads, 4 rows each
  const int l = blockIdx.x * CT + tx;
  const int j0 = blockIdx.y * CT;
  const double* src = in + blockIdx.z * cs;
  double* dst = out + blockIdx.z * cs;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int n0 = 0; n0 < N; n0 += CT) {
    for (int r = ty; r < CT; r += 8) {
      const int j = j0 + r, n = n0 + tx;
      sM[r][tx] = (j < N && n < N) ? M[(size_t)j * N + n] : 0.0;
      const int nn = n0 + r;
      sX[r][tx] = (nn < N && l < nl) ? src[(size_t)nn * nl + l] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < CT; ++k) {
      const double x = sX[k][tx];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = fma(sM[ty + 8 * q][k], x, acc[q]);
    }
    __syncthreads();
  }
  if (l < nl)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = j0 + ty + 8 * q;
      if (j < N) dst[(size_t)j * nl + l] = acc[q];
    }
}

// Complex FFT along x of columns [z0, z0 + cols) of one plane [x][Mz]; plane blockIdx.x, column chunk blockIdx.y.
__global__ void __launch_bounds__(256) k_long_x(int Nx, int Mz, int cols, FftPlan px, const cpx<double>* __restrict__ tw,
                                                int sign, double scale, cpx<double>* __restrict__ data) {
  extern __shared__ unsigned char smem_raw[];
  const int ss = Nx + 1, z0 = blockIdx.y * cols, nc = min(cols, Mz - z0);
  cpx<double>* a = reinterpret_cast<cpx<double>*>(smem_raw);
  cpx<double>* b = a + (size_t)cols * ss;
  cpx<double>* plane = data + blockIdx.x * (size_t)Nx * Mz + z0;
  for (int i = threadIdx.x; i < nc * Nx; i += blockDim.x) {
    const int x = i / nc, c = i - x * nc;
    a[c * ss + x] = plane[(size_t)x * Mz + c];
  }
  __syncthreads();
  fft_batch<double>(a, b, nc, ss, px, tw, sign);
  for (int i = threadIdx.x; i < nc * Nx; i += blockDim.x) {
    const int x = i / nc, c = i - x * nc;
    plane[(size_t)x * Mz + c] = cscale(a[c * ss + x], scale);
  }
}

// z transform of rows of Nz + 2 doubles, `rows` a block: c2r (inverse, Hermitian completion) or r2c.
__global__ void __launch_bounds__(256) k_long_z(long long nrows, int Nz, int rows, FftPlan pz,
                                                const cpx<double>* __restrict__ tw, int inverse, double* __restrict__ data) {
  extern __shared__ unsigned char smem_raw[];
  const int Mz = Nz / 2 + 1, Nzpad = 2 * Mz, ss = Nz + 1;
  cpx<double>* a = reinterpret_cast<cpx<double>*>(smem_raw);
  cpx<double>* b = a + (size_t)rows * ss;
  const long long row0 = (long long)rows * blockIdx.x;
  const int nr = (int)min((long long)rows, nrows - row0);
  double* first = data + row0 * Nzpad;
  for (int i = threadIdx.x; i < nr * Nz; i += blockDim.x) {
    const int r = i / Nz, k = i - r * Nz, m = k < Mz ? k : Nz - k;
    const double* row = first + (size_t)r * Nzpad;
    if (inverse)  // only the real parts of the first and last coefficient
      a[r * ss + k] = cmk<double>(row[2 * m], k == 0 || 2 * k == Nz ? 0.0 : (k < Mz ? row[2 * m + 1] : -row[2 * m + 1]));
    else
      a[r * ss + k] = cmk<double>(row[k], 0.0);
  }
  __syncthreads();
  fft_batch<double>(a, b, nr, ss, pz, tw, inverse ? +1 : -1);
  for (int i = threadIdx.x; i < nr * Nzpad; i += blockDim.x) {
    const int r = i / Nzpad, z = i - r * Nzpad;
    const cpx<double>* s = a + r * ss;
    first[(size_t)r * Nzpad + z] = inverse ? (z < Nz ? s[z].x : 0.0) : (z & 1 ? s[z >> 1].y : s[z >> 1].x);
  }
}

long double cospi_frac(long long m, long long d) {  // cos(pi m / d), argument reduced over the integers
  long long r = m % (2 * d);
  if (r < 0) r += 2 * d;
  return cosl(3.14159265358979323846264338327950288L * (long double)r / (long double)d);
}

}  // namespace

struct cfgpu_flowfield_s {
  int Nx = 0, Ny = 0, Nz = 0, Nd = 0;
  double Lx = 0, Lz = 0, a = -1, b = 1;
  int xzstate = CFGPU_SPECTRAL, ystate = CFGPU_SPECTRAL;
  size_t n = 0;  // doubles
  double* data = nullptr;
  double* work = nullptr;
  OzTables oz{};  // N = 0: Ny not covered, dense products with Mfwd, Minv
  unsigned char* ozblock = nullptr;
  double* Mfwd = nullptr;  // [n][j] chebyfft
  double* Minv = nullptr;  // [j][n] ichebyfft
  void* twx = nullptr;  // fx_twiddles up to FX_LMAX, complex doubles of the plan beyond
  void* twz = nullptr;
  FftPlan px{}, pz{};
  cudaStream_t st = nullptr;
  int* waiterr = nullptr;  // cfgpu_wait_flag
};

namespace {

template <typename T>
int tf_upload(const std::vector<T>& h, T** d, cudaStream_t st) {
  TF_CK(cudaMalloc((void**)d, h.size() * sizeof(T)));
  TF_CK(cudaMemcpyAsync(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, st));
  return CFGPU_OK;
}

int y_transform(cfgpu_flowfield f, bool to_spectral) {
  if (f->Ny < 2) return CFGPU_OK;
  const int nl = f->Nx * 2 * (f->Nz / 2 + 1);
  const size_t cs = (size_t)f->Ny * nl;
  if (f->oz.N) {
    GridDev g{};
    g.b = 1;
    g.a = -1;
    for (int c0 = 0; c0 < f->Nd; c0 += OZ_MAX_JOBS) {
      OzJob job[OZ_MAX_JOBS] = {};
      const int nj = std::min(OZ_MAX_JOBS, f->Nd - c0);
      for (int c = 0; c < nj; ++c) {
        job[c].in = job[c].out = f->data + (c0 + c) * cs;
        job[c].inplace = 1;
      }
      TF_CK(launch_cheb_oz(g, f->Ny, !to_spectral, nl, nl, f->oz, job, nj, f->waiterr, f->st));
    }
    return CFGPU_OK;
  }
  dim3 grid((nl + CT - 1) / CT, (f->Ny + CT - 1) / CT, f->Nd);
  k_cheb_full<<<grid, 256, 0, f->st>>>(f->Ny, nl, cs, to_spectral ? f->Mfwd : f->Minv, f->data, f->work);
  TF_CK(cudaGetLastError());
  TF_CK(cudaMemcpyAsync(f->data, f->work, f->n * sizeof(double), cudaMemcpyDeviceToDevice, f->st));
  return CFGPU_OK;
}

// Lines beside their copies in about 96 KB of shared memory, at most 16 a block.
int long_lines(int L) { return std::min(16, (int)(96 * 1024 / (2 * sizeof(cpx<double>) * (L + 1)))); }

bool long_attr() {
  static const bool attr = [] {
    cudaFuncSetAttribute(k_long_x, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    cudaFuncSetAttribute(k_long_z, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    return true;
  }();
  return attr;
}

cudaError_t x_pass(cfgpu_flowfield f, int sign, double scale) {
  const int Mz = f->Nz / 2 + 1, planes = f->Ny * f->Nd;
  cpx<double>* data = reinterpret_cast<cpx<double>*>(f->data);
  if (f->Nx <= FX_LMAX) return launch_field_x(f->Nx, Mz, planes, f->twx, sign, scale, data, f->st);
  long_attr();
  const int cols = std::min(Mz, long_lines(f->Nx));
  k_long_x<<<dim3(planes, (Mz + cols - 1) / cols), 256, 2 * sizeof(cpx<double>) * (size_t)cols * (f->Nx + 1), f->st>>>(
      f->Nx, Mz, cols, f->px, (const cpx<double>*)f->twx, sign, scale, data);
  return cudaGetLastError();
}

cudaError_t z_pass(cfgpu_flowfield f, bool inverse) {
  const long long nrows = (long long)f->Ny * f->Nd * f->Nx;
  if (f->Nz <= FX_LMAX) return launch_field_z(nrows, f->Nz, inverse, f->twz, f->data, f->st);
  long_attr();
  const int rows = long_lines(f->Nz);
  k_long_z<<<(unsigned)((nrows + rows - 1) / rows), 256, 2 * sizeof(cpx<double>) * (size_t)rows * (f->Nz + 1), f->st>>>(
      nrows, f->Nz, rows, f->pz, (const cpx<double>*)f->twz, inverse, f->data);
  return cudaGetLastError();
}

int xz_transform(cfgpu_flowfield f, bool to_spectral) {
  if (f->Nx > TF_MAX || f->Nz > TF_MAX) return tf_fail(CFGPU_ENOTSUP, "Nx or Nz too large for the shared-memory FFT");
  if (to_spectral) {
    TF_CK(z_pass(f, false));
    TF_CK(x_pass(f, -1, 1.0 / ((double)f->Nx * f->Nz)));
  } else {
    TF_CK(x_pass(f, +1, 1.0));
    TF_CK(z_pass(f, true));
  }
  return CFGPU_OK;
}

// Twiddles of lines of length L (plan and its table tw).
int line_twiddles(int L, const std::vector<std::complex<long double>>& tw, void** dst, cudaStream_t st) {
  std::vector<cpx<double>> t;
  if (L <= FX_LMAX) {
    const std::vector<int> q = fx_twiddles(L);  // (x, y, z, w) of an entry in two doubles' place
    t.resize(q.size() / 4);
    std::memcpy((void*)t.data(), q.data(), q.size() * sizeof(int));
  } else {
    for (const auto& w : tw) t.push_back(cmk<double>((double)w.real(), (double)w.imag()));
  }
  const int e = tf_upload(t, (cpx<double>**)dst, st);
  if (e == CFGPU_OK) TF_CK(cudaStreamSynchronize(st));  // t is a local
  return e;
}

int finish(cfgpu_flowfield f, int st) {
  if (st != CFGPU_OK) {
    (void)cudaStreamSynchronize(f->st);
    return st;
  }
  TF_CK(cudaStreamSynchronize(f->st));
  return cfgpu_wait_status(f->waiterr);
}

}  // namespace

extern "C" {

cfgpu_status cfgpu_flowfield_create(const cfgpu_grid* g, int Nd, cfgpu_flowfield* out) {
  if (!g || !out || Nd < 1 || g->Nx < 2 || g->Nz < 2 || g->Ny < 2 || g->Nx % 2 || g->Nz % 2 || !(g->b > g->a) ||
      g->Lx <= 0 || g->Lz <= 0)
    return tf_fail(CFGPU_EINVAL, "bad argument");
  *out = nullptr;
  auto* f = new cfgpu_flowfield_s();
  f->Nx = g->Nx;
  f->Ny = g->Ny;
  f->Nz = g->Nz;
  f->Nd = Nd;
  f->Lx = g->Lx;
  f->Lz = g->Lz;
  f->a = g->a;
  f->b = g->b;
  f->n = (size_t)Nd * g->Ny * g->Nx * 2 * (g->Nz / 2 + 1);
  std::vector<std::complex<long double>> twx, twz;
  int st = CFGPU_OK;
  if (!cfgpu_fft_plan(g->Nx, f->px, twx) || !cfgpu_fft_plan(g->Nz, f->pz, twz))
    st = tf_fail(CFGPU_ENOTSUP, "Nx and Nz must factor into primes <= " + std::to_string(FFT_MAX_RADIX));
  if (st == CFGPU_OK && cudaStreamCreateWithFlags(&f->st, cudaStreamNonBlocking) != cudaSuccess)
    st = tf_fail(CFGPU_ECUDA, "cudaStreamCreate failed");
  if (st == CFGPU_OK) st = cfgpu_wait_flag(&f->waiterr);
  if (st == CFGPU_OK) {
    cudaError_t e = cudaMalloc((void**)&f->data, f->n * sizeof(double));
    if (e == cudaSuccess) e = cudaMemsetAsync(f->data, 0, f->n * sizeof(double), f->st);
    if (e != cudaSuccess) st = tf_fail(CFGPU_ENOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  if (st == CFGPU_OK) {
    const int N = g->Ny;
    std::vector<uint16_t> dg[2];
    std::vector<int> re[2];
    std::vector<unsigned char> oz;
    std::vector<double> Mf, Mi;
    if (f->n / Nd < (1ull << 32) && oz_matrix(N, OZ_T, dg[0], re[0]) && oz_matrix(N, OZ_F, dg[1], re[1])) {
      const size_t mb = oz_matrix_bytes(N), rb = re[0].size() * sizeof(int);
      oz.resize(2 * (mb + rb));
      for (int k = 0; k < 2; ++k) {
        std::memcpy(oz.data() + k * mb, dg[k].data(), mb);
        std::memcpy(oz.data() + 2 * mb + k * rb, re[k].data(), rb);
      }
      st = tf_upload(oz, &f->ozblock, f->st);
      f->oz.N = N;
      f->oz.T = OzMatrix{f->ozblock, (const int*)(f->ozblock + 2 * mb)};
      f->oz.F = OzMatrix{f->ozblock + mb, (const int*)(f->ozblock + 2 * mb + rb)};
    } else {
      Mf.resize((size_t)N * N);
      Mi.resize((size_t)N * N);
      for (int n = 0; n < N; ++n)
        for (int j = 0; j < N; ++j) {
          const long double cn = (n == 0 || n == N - 1) ? 0.5L : 1.0L;
          const long double w = (j == 0 || j == N - 1) ? 1.0L : 2.0L;
          Mf[(size_t)n * N + j] = (double)(w * cn * cospi_frac((long long)n * j, N - 1) / (N - 1));
          Mi[(size_t)j * N + n] = (double)cospi_frac((long long)n * j, N - 1);
        }
      if (cudaMalloc((void**)&f->work, f->n * sizeof(double)) != cudaSuccess)
        st = tf_fail(CFGPU_ENOMEM, "cudaMalloc: work array");
      if (st == CFGPU_OK) st = tf_upload(Mf, &f->Mfwd, f->st);
      if (st == CFGPU_OK) st = tf_upload(Mi, &f->Minv, f->st);
    }
    if (st == CFGPU_OK) st = line_twiddles(f->Nx, twx, &f->twx, f->st);
    if (st == CFGPU_OK) st = line_twiddles(f->Nz, twz, &f->twz, f->st);
    // the host vectors go out of scope: wait for the copies
    if (st == CFGPU_OK && cudaStreamSynchronize(f->st) != cudaSuccess) st = tf_fail(CFGPU_ECUDA, "stream sync");
  }
  if (st != CFGPU_OK) {
    cfgpu_flowfield_destroy(f);
    return st;
  }
  *out = f;
  return CFGPU_OK;
}

cfgpu_status cfgpu_flowfield_destroy(cfgpu_flowfield f) {
  if (!f) return CFGPU_OK;
  if (f->st) cudaStreamSynchronize(f->st);
  cudaFree(f->data);
  cudaFree(f->work);
  cudaFree(f->ozblock);
  cudaFree(f->Mfwd);
  cudaFree(f->Minv);
  cudaFree(f->twx);
  cudaFree(f->twz);
  cfgpu_wait_flag_free(f->waiterr);
  if (f->st) cudaStreamDestroy(f->st);
  delete f;
  return CFGPU_OK;
}

cfgpu_status cfgpu_flowfield_size(cfgpu_flowfield f, long long* ndoubles) {
  if (!f || !ndoubles) return tf_fail(CFGPU_EINVAL, "bad argument");
  *ndoubles = (long long)f->n;
  return CFGPU_OK;
}

cfgpu_status cfgpu_flowfield_data(cfgpu_flowfield f, double** device_ptr) {
  if (!f || !device_ptr) return tf_fail(CFGPU_EINVAL, "bad argument");
  *device_ptr = f->data;
  return CFGPU_OK;
}

cfgpu_status cfgpu_flowfield_upload(cfgpu_flowfield f, const double* host, int xzstate, int ystate) {
  if (!f || !host || (xzstate != CFGPU_SPECTRAL && xzstate != CFGPU_PHYSICAL) ||
      (ystate != CFGPU_SPECTRAL && ystate != CFGPU_PHYSICAL))
    return tf_fail(CFGPU_EINVAL, "bad argument");
  TF_CK(cudaMemcpyAsync(f->data, host, f->n * sizeof(double), cudaMemcpyHostToDevice, f->st));
  TF_CK(cudaStreamSynchronize(f->st));
  *f->waiterr = 0;  // whole new data
  f->xzstate = xzstate;
  f->ystate = ystate;
  return CFGPU_OK;
}

cfgpu_status cfgpu_flowfield_download(cfgpu_flowfield f, double* host) {
  if (!f || !host) return tf_fail(CFGPU_EINVAL, "bad argument");
  TF_CK(cudaMemcpyAsync(host, f->data, f->n * sizeof(double), cudaMemcpyDeviceToHost, f->st));
  TF_CK(cudaStreamSynchronize(f->st));
  return cfgpu_wait_status(f->waiterr);
}

cfgpu_status cfgpu_flowfield_inject_wait_error(cfgpu_flowfield f) {
  if (!f) return tf_fail(CFGPU_EINVAL, "bad argument");
  *f->waiterr = 1;
  return CFGPU_OK;
}

cfgpu_status cfgpu_flowfield_state(cfgpu_flowfield f, int* xzstate, int* ystate) {
  if (!f || !xzstate || !ystate) return tf_fail(CFGPU_EINVAL, "bad argument");
  *xzstate = f->xzstate;
  *ystate = f->ystate;
  return CFGPU_OK;
}

cfgpu_status cfgpu_flowfield_make_spectral_xz(cfgpu_flowfield f) {
  if (!f) return tf_fail(CFGPU_EINVAL, "bad argument");
  if (f->xzstate == CFGPU_SPECTRAL) return CFGPU_OK;
  const int st = finish(f, xz_transform(f, true));
  if (st == CFGPU_OK) f->xzstate = CFGPU_SPECTRAL;
  return st;
}

cfgpu_status cfgpu_flowfield_make_physical_xz(cfgpu_flowfield f) {
  if (!f) return tf_fail(CFGPU_EINVAL, "bad argument");
  if (f->xzstate == CFGPU_PHYSICAL) return CFGPU_OK;
  const int st = finish(f, xz_transform(f, false));
  if (st == CFGPU_OK) f->xzstate = CFGPU_PHYSICAL;
  return st;
}

cfgpu_status cfgpu_flowfield_make_spectral_y(cfgpu_flowfield f) {
  if (!f) return tf_fail(CFGPU_EINVAL, "bad argument");
  if (f->ystate == CFGPU_SPECTRAL) return CFGPU_OK;
  const int st = finish(f, y_transform(f, true));
  if (st == CFGPU_OK) f->ystate = CFGPU_SPECTRAL;
  return st;
}

cfgpu_status cfgpu_flowfield_make_physical_y(cfgpu_flowfield f) {
  if (!f) return tf_fail(CFGPU_EINVAL, "bad argument");
  if (f->ystate == CFGPU_PHYSICAL) return CFGPU_OK;
  const int st = finish(f, y_transform(f, false));
  if (st == CFGPU_OK) f->ystate = CFGPU_PHYSICAL;
  return st;
}

// makeSpectral: xz first, then y; makePhysical: y first, then xz (flowfield.cpp:1989-1997).
cfgpu_status cfgpu_flowfield_make_spectral(cfgpu_flowfield f) {
  cfgpu_status s = cfgpu_flowfield_make_spectral_xz(f);
  return s == CFGPU_OK ? cfgpu_flowfield_make_spectral_y(f) : s;
}

cfgpu_status cfgpu_flowfield_make_physical(cfgpu_flowfield f) {
  cfgpu_status s = cfgpu_flowfield_make_physical_y(f);
  return s == CFGPU_OK ? cfgpu_flowfield_make_physical_xz(f) : s;
}

}  // extern "C"
