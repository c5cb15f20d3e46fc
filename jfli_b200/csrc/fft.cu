// 3D real FFT passes for sm_100a: r2c along z, complex column passes along y and x,
// and c2r along z. The x pass carries a k-space operator so that
//   forward x FFT -> operator -> inverse x FFT
// happens in one read and one write of the half spectrum (Poisson solve, initial
// condition filter), or so that the forward x FFT feeds the P(k) histogram without
// writing the spectrum back at all.
//
// Pass structure of a Poisson solve on an [nx][ny][nz] mesh (M = nx*ny*nz cells):
//   rfft_z   : read 4M B real,     write 8(M/2+...) B half spectrum
//   cols(y)  : read+write the half spectrum
//   x_op     : read+write the half spectrum (forward x, multiply, inverse x)
//   cols(y)^-1
//   irfft_z  : read the half spectrum, write 4M B real
#include <cmath>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "fft_passes.cuh"
#include "internal.h"

namespace jfli {

// ---------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------
bool make_fft_plan(int n, FftPlan* p) {
  if (n < 2) return false;
  int m = n, a = 0, b = 0;
  while (m % 2 == 0) {
    m /= 2;
    ++a;
  }
  while (m % 3 == 0) {
    m /= 3;
    ++b;
  }
  if (m != 1) return false;
  p->n = n;
  p->nst = 0;
  while (a >= 3) {
    p->radix[p->nst++] = 8;
    a -= 3;
  }
  if (a == 2) p->radix[p->nst++] = 4;
  if (a == 1) p->radix[p->nst++] = 2;
  for (int i = 0; i < b; ++i) p->radix[p->nst++] = 3;
  return p->nst <= kMaxRadixStages;
}

bool fft_axis_supported(int n) {
  FftPlan p;
  return n >= 2 && n <= kFftTileElems && make_fft_plan(n, &p);
}

bool mesh_fft_supported(int nx, int ny, int nz) {
  return nz % 2 == 0 && nz >= 4 && fft_axis_supported(nx) && fft_axis_supported(ny) && fft_axis_supported(nz / 2);
}

void* device_table(const void* host, size_t bytes) {
  // An allocation is refused while a stream is captured, by this thread or (global mode) another, but
  // in relaxed mode: without it a length first met in a capture would fail.
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  void* d = nullptr;
  cudaStream_t s = nullptr;
  bool ok = cudaMalloc(&d, bytes) == cudaSuccess &&
            cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMemcpyAsync(d, host, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaStreamSynchronize(s) == cudaSuccess;
  if (s) cudaStreamDestroy(s);
  if (!ok && d) cudaFree(d);
  cudaThreadExchangeStreamCaptureMode(&mode);
  return ok ? d : nullptr;
}

// ---- twiddle tables w_n^m = exp(-2 pi i m / n), one per (device, n), built once on the host
static std::mutex g_tw_mutex;
static std::map<std::pair<int, int>, float2*> g_tw_tables;

const float2* twiddle_table(int n) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_tw_mutex);
  auto key = std::make_pair(dev, n);
  auto it = g_tw_tables.find(key);
  if (it != g_tw_tables.end()) return it->second;
  std::vector<float2> h(n);
  for (int m = 0; m < n; ++m) {
    const double ang = 2.0 * M_PI * (double)m / (double)n;
    h[m] = make_float2((float)std::cos(ang), (float)-std::sin(ang));
  }
  float2* d = static_cast<float2*>(device_table(h.data(), sizeof(float2) * n));
  if (!d) return nullptr;
  g_tw_tables[key] = d;
  return d;
}

static PkArgs pk_args(const MeshDims& d, const float* kedges, int nedges, const float* box, float norm,
                      double* partials) {
  PkArgs a;
  a.nx = d.nx;
  a.ny = d.ny;
  a.nz = d.nz;
  a.kedges = kedges;
  a.nedges = nedges;
  a.cx = (float)(2.0 * M_PI / (double)box[0]);
  a.cy = (float)(2.0 * M_PI / (double)box[1]);
  a.cz = (float)(2.0 * M_PI / (double)box[2]);
  a.norm = norm;
  a.partials = partials;
  return a;
}

cudaError_t rfft3d_forward(const float* in, float2* spec, const MeshDims& d, float sub, cudaStream_t s) {
  const cudaError_t e = launch_forward_zy(in, spec, d, sub, s);
  if (e != cudaSuccess) return e;
  return launch_cols(-1, spec, x_geom(d), d.spec_elems(), d.batch, s);
}

// 2D r2c of (ny, nz) maps: the z and y passes of rfft3d_forward on a mesh with nx = 1
cudaError_t rfft2d_forward(const float* in, float2* spec, const MeshDims& d, cudaStream_t s) {
  return launch_forward_zy(in, spec, d, 0.0f, s);
}

cudaError_t rfft3d_inverse(float2* spec, float* out, const MeshDims& d, float scale, cudaStream_t s) {
  const cudaError_t e = launch_cols(1, spec, x_geom(d), d.spec_elems(), d.batch, s);
  if (e != cudaSuccess) return e;
  return launch_inverse_yz(spec, out, d, scale, s);
}

// real mesh -> (forward 3D FFT, k-space op, inverse 3D FFT) -> real mesh. `mixed`: see reg_fft_length
template <class Op>
static cudaError_t filter_chain(const float* in, float2* spec, float* out, const MeshDims& d, float sub, const Op& op,
                                cudaStream_t s, float* clear = nullptr, bool mixed = true) {
  cudaError_t e = launch_forward_zy(in, spec, d, sub, s, clear, mixed);
  if (e != cudaSuccess) return e;
  e = launch_x_op(spec, d, op, s, mixed);
  if (e != cudaSuccess) return e;
  return launch_inverse_yz(spec, out, d, 1.0f, s, mixed);
}

cudaError_t poisson_potential(const float* rho, float2* spec, float* pot, const MeshDims& d, float rho_mean,
                              float scale, cudaStream_t s, float* clear, bool mixed) {
  PoissonOp op;
  op.nx = d.nx;
  op.ny = d.ny;
  op.nz = d.nz;
  op.norm = scale / ((float)d.nx * (float)d.ny * (float)d.nz);
  return filter_chain(rho, spec, pot, d, rho_mean, op, s, clear, mixed);
}

cudaError_t pgd_potential(const float* rho, float2* spec, float* pot, const MeshDims& d, float rho_mean, float kl,
                          float ks, float scale, cudaStream_t s) {
  return mixed_pgd_potential(rho, spec, pot, d, rho_mean, kl, ks, 0.f, 1.f, scale, s);
}

cudaError_t mixed_pgd_potential(const float* rho, float2* spec, float* pot, const MeshDims& d, float rho_mean,
                                float kl, float ks, float c0, float c1, float scale, cudaStream_t s) {
  PgdOp op;
  op.nx = d.nx;
  op.ny = d.ny;
  op.nz = d.nz;
  op.norm = scale / ((float)d.nx * (float)d.ny * (float)d.nz);
  op.kl2 = kl * kl;
  op.ks4 = ks * ks * ks * ks;
  op.c0 = c0;
  op.c1 = c1;
  return filter_chain(rho, spec, pot, d, rho_mean, op, s);
}

cudaError_t ic_filter(const float* noise, float2* spec, float* out, const MeshDims& d, const float* ktab,
                      const float* ptab, int ntab, const float* box, int zero_mode_one, cudaStream_t s,
                      const float* dptab) {
  IcOp op;
  op.dptab = dptab;
  op.nx = d.nx;
  op.ny = d.ny;
  op.nz = d.nz;
  op.ktab = ktab;
  op.ptab = ptab;
  op.ntab = ntab;
  op.lx = box[0];
  op.ly = box[1];
  op.lz = box[2];
  op.factor = (float)(((double)d.nx * d.ny * d.nz) / ((double)box[0] * box[1] * box[2]));
  op.norm = 1.0f / ((float)d.nx * (float)d.ny * (float)d.nz);
  op.zero_mode_one = zero_mode_one;
  return filter_chain(noise, spec, out, d, 0.0f, op, s, nullptr, false);
}

cudaError_t power_adjoint(const float* mesh, float2* spec, float* out, const MeshDims& d, const float* kedges,
                          const float* weights, int nedges, const float* box, cudaStream_t s) {
  PkAdjOp op;
  op.nx = d.nx;
  op.ny = d.ny;
  op.nz = d.nz;
  op.kedges = kedges;
  op.weights = weights;
  op.nedges = nedges;
  op.cx = (float)(2.0 * M_PI / (double)box[0]);
  op.cy = (float)(2.0 * M_PI / (double)box[1]);
  op.cz = (float)(2.0 * M_PI / (double)box[2]);
  op.norm = 1.0f / ((float)d.nx * (float)d.ny * (float)d.nz);
  return filter_chain(mesh, spec, out, d, 0.0f, op, s);
}

cudaError_t power_poles_adjoint(const float* mesh, float2* spec, float* out, const MeshDims& d, const float* kedges,
                                const float* weights, int nedges, const int* ells, int nell, const float* box,
                                const float* los, int cplx, cudaStream_t s) {
  PkAdjOp op;
  op.nx = d.nx;
  op.ny = d.ny;
  op.nz = d.nz;
  op.kedges = kedges;
  op.weights = weights;
  op.nedges = nedges;
  op.cx = (float)(2.0 * M_PI / (double)box[0]);
  op.cy = (float)(2.0 * M_PI / (double)box[1]);
  op.cz = (float)(2.0 * M_PI / (double)box[2]);
  op.norm = 1.0f / ((float)d.nx * (float)d.ny * (float)d.nz);
  op.nell = nell;
  op.cplx = cplx;
  for (int e = 0; e < nell && e < kMaxAdjPoles; ++e) op.ells[e] = ells[e];
  op.lx = los[0];
  op.ly = los[1];
  op.lz = los[2];
  return filter_chain(mesh, spec, out, d, 0.0f, op, s);
}

cudaError_t power_partials(const float* mesh, float2* spec, double* partials, const MeshDims& d, const float* kedges,
                           int nedges, const float* box, float norm, cudaStream_t s) {
  const cudaError_t e = launch_forward_zy(mesh, spec, d, 0.0f, s);
  if (e != cudaSuccess) return e;
  return launch_x_pk(spec, d, pk_args(d, kedges, nedges, box, norm, partials), s);
}

// ---------------------------------------------------------------------------------
// P(k) without any allocation, for callers that cannot allocate device memory.
//
// The half spectrum and the per-CTA histogram partials live in one file-scope device
// array of kNoAllocScratchBytes. The transforms use the shared-memory Stockham kernels,
// which build their twiddles in the kernel, so no twiddle table is created either.
// ---------------------------------------------------------------------------------
constexpr size_t kNoAllocScratchBytes = 11u << 20;  // 11 MiB: a 128^3 spectrum plus its partials
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
static std::mutex g_noalloc_mutex;
static void* g_noalloc_ptr[kNoAllocMaxDevices];  // device -> address of g_noalloc_scratch on it
static void* g_noalloc_ctx[kNoAllocMaxDevices];  // the context that address belongs to

// The calling thread's current driver context (cuCtxGetCurrent through the runtime's
// driver entry point, so the library needs no link to libcuda), or nullptr.
static void* current_context() {
  using GetCurrent = int (*)(void**);
  static GetCurrent fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<GetCurrent>(f);
  }();
  void* ctx = nullptr;
  if (fn == nullptr || fn(&ctx) != 0) return nullptr;
  return ctx;
}

// Device address of the scratch array on the current device. The first call on a device
// looks it up with cudaGetSymbolAddress (with that device current); later calls reuse it.
// The address is tied to the device's context: a new context on the device (after
// cudaDeviceReset, for instance) gets a new lookup, so no call uses a stale address.
cudaError_t noalloc_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  void* ctx = g_noalloc_ptr[dev] ? current_context() : nullptr;
  if (g_noalloc_ptr[dev] == nullptr || ctx == nullptr || ctx != g_noalloc_ctx[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);  // makes the device's primary context current
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[dev] = p;
    g_noalloc_ctx[dev] = current_context();
  }
  *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

size_t noalloc_scratch_bytes() { return kNoAllocScratchBytes; }

cudaError_t power_partials_noalloc(const float* mesh, float2* spec, double* partials, const MeshDims& d,
                                   const float* kedges, int nedges, const float* box, float norm, cudaStream_t s) {
  // the shared-memory Stockham passes, which build their twiddles in the kernel
  cudaError_t e = rfft_z_generic(mesh, spec, d, 0.0f, s);
  if (e != cudaSuccess) return e;
  e = cols_generic(-1, spec, y_geom(d), d.spec_elems(), d.batch, s);
  if (e != cudaSuccess) return e;
  // forward x feeding the histogram
  return x_pk_generic(spec, d, pk_args(d, kedges, nedges, box, norm, partials), s);
}

}  // namespace jfli
