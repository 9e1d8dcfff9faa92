// ep_noalloc.cu - the k-space convolution of poten() for callers that
// cannot allocate device memory.
//
// Some callers can't call cudaMalloc: a Fortran or C host that runs inside
// a framework owning the whole device memory pool (the framework hands out
// buffers, and any allocation behind its back breaks its accounting or
// fails), or code running while a CUDA graph is being captured, where a
// fresh allocation is not allowed.  ep_convolve_noalloc gives them the
// density convolution out = IFFT(FFT(in) * K) / N that poten() applies with
// the coarse-graining, Lennard-Jones and alpha_s kernels, using only the
// buffers the caller passes plus the fixed scratch array below.
//
// The scratch is a file-scope __device__ array: every GPU that loads the
// library holds it (EP_NOALLOC_SCRATCH_BYTES) until the process exits.  In
// host code the array's name is only a host-side stand-in, so its device
// address is looked up once per device with cudaGetSymbolAddress.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "../../include/eff_pot.h"
#include "ep_kernels.cuh"
#include "ep_xw.cuh"
#include "ep_yz.cuh"

namespace {

// Largest half spectrum: (nx/2+1)*ny*nz <= 33*64*64 (a 64^3 grid); axes of
// at most 320 points.
constexpr long long kMaxHalf = 33LL * 64 * 64;
constexpr int kMaxAxis = 320;
constexpr long long kScratchElems = 2 * kMaxHalf;

static __device__ __align__(256) double2 g_noalloc_scratch[kScratchElems];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
double2* g_scratch_addr[kMaxDevices] = {};
const double2* g_roots_addr[kMaxDevices] = {};

// Roots exp(-2 pi i k / n), k < n, of every axis length, as a constant table of
// the library (89 KB): three kernels a call computed them before, three
// of eight launches.  With the per-length X, Y and Z kernels a call takes 41 us
// at 32^3 (57 before) and 51 at 30 x 54 x 64 (78): its five launches.  Each angle is reduced to its octant and the sine or
// cosine series summed there in long double, then rounded.
constexpr bool axis_len(int n) {
  if (n < 2) return false;
  while (n % 2 == 0) n /= 2;
  while (n % 3 == 0) n /= 3;
  while (n % 5 == 0) n /= 5;
  return n == 1;
}
constexpr int roots_at(int n) {
  int at = 0;
  for (int m = 2; m < n; ++m)
    if (axis_len(m)) at += m;
  return at;
}
constexpr int kRoots = roots_at(kMaxAxis + 1);
constexpr long double sin_series(long double x) {
  long double t = x, s = 0.0L;
  for (int i = 1; i < 14; ++i) {
    s += t;
    t *= -x * x / ((2.0L * i) * (2.0L * i + 1.0L));
  }
  return s;
}
constexpr long double cos_series(long double x) {
  long double t = 1.0L, s = 0.0L;
  for (int i = 1; i < 14; ++i) {
    s += t;
    t *= -x * x / ((2.0L * i - 1.0L) * (2.0L * i));
  }
  return s;
}
struct Roots {
  double v[2 * kRoots];
};
constexpr Roots make_roots() {
  Roots r{};
  int at = 0;
  for (int n = 2; n <= kMaxAxis; ++n) {
    if (!axis_len(n)) continue;
    for (int k = 0; k < n; ++k, ++at) {
      // angle 2 pi k / n = q pi/2 + (pi/2) (f / n), 0 <= f < n
      const int q = 4 * k / n, f = 4 * k - q * n;
      const long double half = 1.57079632679489661923132169163975144L;
      const bool up = 2 * f > n;
      const long double x = half * (up ? n - f : f) / n;
      const double a = (double)(up ? sin_series(x) : cos_series(x)), b = (double)(up ? cos_series(x) : sin_series(x));
      const double co = q == 0 ? a : q == 1 ? -b : q == 2 ? -a : b;
      const double si = q == 0 ? b : q == 1 ? a : q == 2 ? -b : -a;
      r.v[2 * at] = co;
      r.v[2 * at + 1] = -si;
    }
  }
  return r;
}
static __device__ const __align__(16) Roots g_noalloc_roots = make_roots();

// Backward c2r along x of every line, scaled by 1/N, into a real array.
__global__ void k_noalloc_xinv(Geo g, const double2* __restrict__ spec, double* __restrict__ out,
                               const __grid_constant__ FftPlan p2, const double2* __restrict__ twx, double scale, int nl) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nx = g.nx;
  XSmem<double> S(smraw, nl, nx);
  const long long nlines = (long long)g.ny * g.nz;
  const long long line0 = (long long)blockIdx.x * nl;
  const int nlv = (int)min((long long)nl, nlines - line0);
  for (int i = threadIdx.x; i < nx; i += blockDim.x) S.tw[i] = twx[i];
  __syncthreads();
  x_inverse<double>(spec, line0, nlv, nl, nx, g.nxh, S, p2, scale, S.R);
  for (int e = threadIdx.x; e < nlv * nx; e += blockDim.x) out[line0 * nx + e] = S.R[e];
}

size_t x_smem_of(int nl, int nx) {
  return 2 * (size_t)nl * (nx / 2 + 1) * sizeof(double2) + (size_t)nx * sizeof(double2) + (size_t)nl * nx * sizeof(double);
}
size_t l_smem_of(int LT, int n, int nbuf) {
  return (size_t)nbuf * LT * (n + 1) * sizeof(double2) + (size_t)n * sizeof(double2) + (size_t)LT * sizeof(long long);
}

// Once per device, with that device current: the device addresses of the
// scratch array and the roots and the shared-memory limits of the general
// kernels.
int device_setup(int dev, double2** out, const double2** roots) {
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (g_scratch_addr[dev]) {
    *out = g_scratch_addr[dev];
    *roots = g_roots_addr[dev];
    return EP_OK;
  }
  void *ptr = nullptr, *rp = nullptr;
  if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr ||
      cudaGetSymbolAddress(&rp, g_noalloc_roots) != cudaSuccess || !rp) {
    cudaGetLastError();
    return EP_ERR_CUDA;
  }
  const int big = 220 * 1024;
  if (cudaFuncSetAttribute(k_x1<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) != cudaSuccess ||
      cudaFuncSetAttribute(k_c2c<double, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) != cudaSuccess ||
      cudaFuncSetAttribute(k_c2c<double, +1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) != cudaSuccess ||
      cudaFuncSetAttribute(k_zconv<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) != cudaSuccess ||
      cudaFuncSetAttribute(k_noalloc_xinv, cudaFuncAttributeMaxDynamicSharedMemorySize, big) != cudaSuccess) {
    cudaGetLastError();
    return EP_ERR_CUDA;
  }
  g_roots_addr[dev] = static_cast<const double2*>(rp);
  g_scratch_addr[dev] = static_cast<double2*>(ptr);
  *out = g_scratch_addr[dev];
  *roots = g_roots_addr[dev];
  return EP_OK;
}

cudaError_t launch(const void* fn, dim3 grid, int threads, void** args, size_t smem, cudaStream_t st) {
  return cudaLaunchKernel(fn, grid, dim3((unsigned)threads), args, smem, st);
}
constexpr size_t kDefaultSmem = 48 * 1024;  // above it a kernel needs its limit raised

}  // namespace

extern "C" int ep_convolve_noalloc(const double* d_in, const double* d_kernel, double* d_out, int nx, int ny,
                                   int nz, void* stream) {
  if (!d_in || !d_kernel || !d_out) return EP_ERR_INVALID_ARG;
  // the X passes read pairs of d_in
  if ((uintptr_t)d_in % 16 || (uintptr_t)d_kernel % 8 || (uintptr_t)d_out % 8) return EP_ERR_INVALID_ARG;
  if (nx % 2 || !axis_len(nx) || !axis_len(ny) || !axis_len(nz)) return EP_ERR_BAD_GRID;
  const long long half = (long long)(nx / 2 + 1) * ny * nz;
  if (half > kMaxHalf || nx > kMaxAxis || ny > kMaxAxis || nz > kMaxAxis) return EP_ERR_UNSUPPORTED;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return EP_ERR_NO_DEVICE;
  }
  double2* scratch = nullptr;
  const double2* roots = nullptr;
  int r = device_setup(dev, &scratch, &roots);
  if (r) return r;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double2* S = scratch;
  double2* Tsp = scratch + kMaxHalf;
  const double2 *twx = roots + roots_at(nx), *twy = roots + roots_at(ny), *twz = roots + roots_at(nz);
  Geo g{nx, ny, nz, nx / 2 + 1, (long long)nx * ny * nz, half};
  long long nlines = (long long)ny * nz;
  double scale = 1.0 / ((double)nx * ny * nz);
  cudaError_t e = cudaSuccess;
  // X forward, Y forward, Z with the product, Y backward, X backward: the
  // kernels of each axis' length, or the general engine
  const XWKernels* kx = xw_kernels<double>(nx / 2);
  // k_xw_c2r stores pairs: a d_out that is not 16-byte aligned (a slice of a
  // host's pool) takes the general engine's last pass, which stores doubles
  const XWKernels* ko = (uintptr_t)d_out % 16 ? nullptr : kx;
  const YZKernels *ky = yz_kernels<double>(ny), *kz = yz_kernels<double>(nz);
  FftPlan p2{}, pY{}, pZ{};
  int nl = 16, LT = 16, LZ = 16;
  if (!kx || !ko) {
    make_plan(nx / 2, p2);
    while (nl > 1 && x_smem_of(nl, nx) > 110 * 1024) nl /= 2;
  }
  if (!ky) {
    make_plan(ny, pY);
    while (LT > 1 && l_smem_of(LT, ny, 2) > 110 * 1024) LT /= 2;
  }
  if (!kz) {
    make_plan(nz, pZ);
    while (LZ > 1 && l_smem_of(LZ, nz, 3) > 110 * 1024) LZ /= 2;
  }
  // (the X kernels' rows stay under the default limit)
  if (ky && ky->line_bytes + ky->tw_bytes > kDefaultSmem) e = yz_limit_c2c(*ky);
  if (e == cudaSuccess && kz && kz->line_bytes + kz->tw_bytes > kDefaultSmem) e = yz_limit_conv(*kz);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return EP_ERR_CUDA;
  }
  auto grid_x = [&](const XWKernels* k) {
    const int lines = k ? k->lines : nl;
    return dim3((unsigned)((nlines + lines - 1) / lines));
  };
  if (kx) {
    Phys ph{};
    FdW<double> fd{};
    XWArgs<double> a{};
    a.den = d_in;
    a.out[0] = S;
    a.twx = twx;
    void* args[] = {&nlines, &ph, &fd, &a};
    e = launch(kx->x[0], grid_x(kx), kx->threads, args, kx->smem[0], st);
  } else {
    k_x1<double><<<grid_x(nullptr), 256, x_smem_of(nl, nx), st>>>(g, d_in, S, p2, twx, nl);
  }
  Arr8<double> ay{};
  LineSet ly{(long long)g.nxh, (long long)g.nxh * ny, (long long)g.nxh, (long long)g.nxh * nz};
  auto pass_y = [&](double2* a, int dir) {
    ay.a[0] = a;
    if (ky) {
      void* args[] = {&ay, &ly, &twy};
      if (e == cudaSuccess)
        e = launch(ky->c2c[dir < 0 ? 0 : 1], dim3((unsigned)((ly.nlines + ky->lines - 1) / ky->lines)), ky->threads,
                   args, ky->line_bytes + ky->tw_bytes, st);
      return;
    }
    const dim3 grid((unsigned)((ly.nlines + LT - 1) / LT));
    if (dir < 0) k_c2c<double, -1><<<grid, 256, l_smem_of(LT, ny, 2), st>>>(ay, ly, pY, twy, LT);
    else k_c2c<double, +1><<<grid, 256, l_smem_of(LT, ny, 2), st>>>(ay, ly, pY, twy, LT);
  };
  pass_y(S, -1);
  ConvSpec<double> cs{};
  cs.in[0] = S;
  cs.out[0][0] = Tsp;
  cs.ker[0][0] = d_kernel;
  cs.nout[0] = 1;
  LineSet lz{(long long)g.nxh * ny, 0, (long long)g.nxh * ny, (long long)g.nxh * ny};
  if (kz) {
    void* args[] = {&cs, &lz, &twz};
    if (e == cudaSuccess)
      e = launch(kz->conv, dim3((unsigned)((lz.nlines + kz->lines - 1) / kz->lines)), kz->threads, args,
                 kz->line_bytes + kz->tw_bytes, st);
  } else {
    k_zconv<double><<<dim3((unsigned)((lz.nlines + LZ - 1) / LZ)), 256, l_smem_of(LZ, nz, 3), st>>>(cs, lz, pZ, twz, LZ);
  }
  pass_y(Tsp, +1);
  if (ko) {
    const double2* spec = Tsp;
    void* args[] = {&nlines, &spec, &d_out, &twx, &scale};
    if (e == cudaSuccess) e = launch(ko->c2r, grid_x(ko), ko->threads, args, ko->smem[3], st);
  } else {
    k_noalloc_xinv<<<grid_x(nullptr), 256, x_smem_of(nl, nx), st>>>(g, Tsp, d_out, p2, twx, scale, nl);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return EP_ERR_CUDA;
  }
  if (cudaGetLastError() != cudaSuccess) return EP_ERR_CUDA;
  return EP_OK;
}
