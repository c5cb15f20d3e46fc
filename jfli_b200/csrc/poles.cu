// Cross spectra and Legendre multipoles of P(k) (reference _src/power/_compute.py:68-119,
// _power with mesh2 and/or multipoles != 0).
//
// The reference bins the full complex grid: w_l = (2l + 1) L_l(mu) with mu = (k . los) / |k|
// (0 at k = 0), and sums Re and Im of w_l F1 conj(F2) per bin (|F|^2 for an auto spectrum).
// Here the meshes go through this library's r2c (the half spectrum, [nx][ny][nz/2 + 1]) and
// every element with 0 < kz < nz/2 also adds its conjugate partner (-k; for real meshes
// F(-k) = conj F(k)) with the partner's own wavevector, so the sums are those of the full
// grid, odd multipoles and imaginary parts included. |k| and the bin are formed as the
// monopole kernel forms them (kspace_ops.cuh PkTile); mu with the reference's float32 order
// (x, y, z products summed, then divided by |k|); L_l by the reference's recurrence in FP32.
// Per-CTA FP64 sums: [2 nell + 2][nedges + 1] = for each l (Re, Im), then mode count, sum |k|.
#include "binning.cuh"
#include "common.cuh"
#include "internal.h"
#include "kspace_ops.cuh"

namespace jfli {

constexpr int kPolesThreads = 256;
constexpr int kMaxPoles = 8;

struct PolesArgs {
  int nx, ny, nz, nedges, nell;
  float cx, cy, cz, lx, ly, lz, norm;
  int ells[kMaxPoles], lmax;  // lmax: the largest of ells
  int strip;                  // |ky| values a thread walks
};

// The multipole weights (2l + 1) L_l(mu) of the listed multipoles in FP32, by legendre_f32's
// recurrence run once up to the largest.
template <int NELL>
__device__ __forceinline__ void pole_weights(const PolesArgs& a, float mu, float (&w)[NELL]) {
  float p0 = 1.f, p1 = mu;
#pragma unroll
  for (int e = 0; e < NELL; ++e) w[e] = a.ells[e] == 0 ? 1.f : mu;
  for (int n = 2; n <= a.lmax; ++n) {
    const float pn = __fdiv_rn(__fsub_rn(__fmul_rn(__fmul_rn((float)(2 * n - 1), mu), p1), __fmul_rn((float)(n - 1), p0)),
                               (float)n);
    p0 = p1;
    p1 = pn;
#pragma unroll
    for (int e = 0; e < NELL; ++e)
      if (a.ells[e] == n) w[e] = pn;
  }
#pragma unroll
  for (int e = 0; e < NELL; ++e) w[e] = __fmul_rn((float)(2 * a.ells[e] + 1), w[e]);
}

// Sums of one thread's current bin: per multipole Re (and, for a cross spectrum, Im; an auto
// spectrum's F conj(F) has no imaginary part), then |k|, and the modes.
template <int NELL, bool CROSS>
struct PoleSums {
  static constexpr int NV = (CROSS ? 2 : 1) * NELL;
  double v[NV], k;
  unsigned n;

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = 0.0;
    k = 0.0;
    n = 0;
  }
};

// Bytes of one histogram column: the sums above per bin and a count.
__host__ __device__ inline size_t poles_column_bytes(int nedges, int nell, bool cross) {
  return (size_t)(nedges + 1) * ((size_t)((cross ? 2 : 1) * nell + 1) * sizeof(double) + sizeof(unsigned));
}
constexpr size_t kPolesHistBudget = 48u << 10;

__host__ __device__ inline int poles_columns(int nedges, int nell, bool cross) {
  return histogram_columns(poles_column_bytes(nedges, nell, cross), kPolesHistBudget);
}

// A thread holds one kz and one |kx| and walks a strip of |ky|: its up to four half-spectrum
// elements (+-kx, +-ky, kz) share |k| bit for bit, and |k| grows slowly along the strip, so
// the bin is looked up and the sums are flushed to shared memory a few times per strip
// (binning.cuh). Lanes hold consecutive kz, so the loads are coalesced. An element with
// 0 < kz < nz/2 also stands for its conjugate partner -k in the other half: its mu is -mu and
// L_l(-mu) = (-1)^l L_l(mu) bit for bit, except on a Nyquist plane of x or y, whose
// frequency is -n/2 for both.
//
// The strip is the longest of 16, 8, ..., 1 that still gives every thread of the grid work
// (a 64^3 mesh has 1089 (|kx|, kz) pairs for the grid's 75776 threads).
constexpr int kPolesStrip = 16;

template <int NELL, bool CROSS>
__global__ void __launch_bounds__(kPolesThreads) k_power_poles(const float2* __restrict__ spec1,
                                                               const float2* __restrict__ spec2, PolesArgs a,
                                                               const float* __restrict__ kedges,
                                                               double* __restrict__ partials) {
  extern __shared__ double hist[];  // [NV + 1][bins][cols] FP64, [bins][cols] counts, the edges
  using Sums = PoleSums<NELL, CROSS>;
  constexpr int NV = Sums::NV;
  const int nb = a.nedges + 1;
  const int cols = poles_columns(a.nedges, NELL, CROSS);
  const int plane = nb * cols;
  unsigned* count = reinterpret_cast<unsigned*>(hist + (size_t)(NV + 1) * plane);
  float* edges = reinterpret_cast<float*>(count + plane);
  for (int i = threadIdx.x; i < (NV + 1) * plane; i += blockDim.x) hist[i] = 0.0;
  for (int i = threadIdx.x; i < plane; i += blockDim.x) count[i] = 0;
  for (int i = threadIdx.x; i < a.nedges; i += blockDim.x) edges[i] = kedges[i];
  __syncthreads();
  const int hz = a.nz / 2 + 1, hx = a.nx / 2 + 1, hy = a.ny / 2 + 1;
  const long long nel = (long long)a.nx * a.ny * hz;
  const long long b = blockIdx.y;
  spec1 += b * nel;
  spec2 += b * nel;
  const int column = (threadIdx.x & 31) & (cols - 1);
  const int strips = (hy + a.strip - 1) / a.strip;
  const long long items = (long long)hx * strips * hz;
  Sums acc;
  acc.clear();
  auto flush = [&](int bin) {
    if (acc.n == 0) return;
    double* h = hist + bin * cols + column;
#pragma unroll
    for (int i = 0; i < NV; ++i) atomicAdd(h + (size_t)i * plane, acc.v[i]);
    atomicAdd(h + (size_t)NV * plane, acc.k);
    atomicAdd(count + bin * cols + column, acc.n);
  };
  for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < items;
       it += (long long)gridDim.x * blockDim.x) {
    const int iz = (int)(it % hz);
    const long long r = it / hz;
    const int j0 = (int)(r % strips) * a.strip, jx = (int)(r / strips);
    const int j1 = min(hy, j0 + a.strip);
    const bool inner = iz > 0 && 2 * iz < a.nz;  // its conjugate partner lies in the other half
    const float az = __fmul_rn(a.cz, (float)signed_freq(iz, a.nz));
    const float az2 = __fmul_rn(az, az), azl = __fmul_rn(az, a.lz);
    const float ax1 = __fmul_rn(a.cx, (float)signed_freq(jx, a.nx));
    const float ax2 = __fmul_rn(ax1, ax1);
    const int xs = (jx == 0 || 2 * jx == a.nx) ? 1 : 2;
    BinCursor cur;
    acc.clear();
    for (int jy = j0; jy < j1; ++jy) {
      const float ay1 = __fmul_rn(a.cy, (float)signed_freq(jy, a.ny));
      const float kmag = __fsqrt_rn(__fadd_rn(__fadd_rn(ax2, __fmul_rn(ay1, ay1)), az2));
      if (!cur.holds(kmag)) {
        flush(cur.bin);
        acc.clear();
        cur.move(kmag, edges, a.nedges);
      }
      const int ys = (jy == 0 || 2 * jy == a.ny) ? 1 : 2;
      for (int q = 0; q < xs * ys; ++q) {
        const bool mx = q >= ys, my = ys == 2 && (q & 1);  // the mirrored index along x, y
        const int ix = mx ? a.nx - jx : jx, iy = my ? a.ny - jy : jy;
        const float ax = mx ? -ax1 : ax1, ay = my ? -ay1 : ay1;
        const long long e = ((long long)ix * a.ny + iy) * hz + iz;
        const float2 f = __ldg(spec1 + e);
        const float2 g = CROSS ? __ldg(spec2 + e) : f;
        // F1 conj(F2) * norm
        const double cre = ((double)f.x * g.x + (double)f.y * g.y) * (double)a.norm;
        const double cim = CROSS ? ((double)f.y * g.x - (double)f.x * g.y) * (double)a.norm : 0.0;
        const float dot = __fadd_rn(__fadd_rn(__fmul_rn(ax, a.lx), __fmul_rn(ay, a.ly)), azl);
        float w[NELL];
        pole_weights<NELL>(a, kmag == 0.f ? 0.f : __fdiv_rn(dot, kmag), w);
        if (!inner) {
#pragma unroll
          for (int m = 0; m < NELL; ++m) {
            acc.v[m] += (double)w[m] * cre;
            if (CROSS) acc.v[NELL + m] += (double)w[m] * cim;
          }
        } else if (2 * ix != a.nx && 2 * iy != a.ny) {
#pragma unroll
          for (int m = 0; m < NELL; ++m) {
            // w + w' and w - w' of the pair (w' = +-w): 2 w or 0
            const double even = (a.ells[m] & 1) ? 0.0 : 2.0 * (double)w[m];
            acc.v[m] += even * cre;
            if (CROSS) acc.v[NELL + m] += (2.0 * (double)w[m] - even) * cim;
          }
        } else {
          const float px = 2 * ix == a.nx ? ax : -ax, py = 2 * iy == a.ny ? ay : -ay;
          const float dotp = __fadd_rn(__fadd_rn(__fmul_rn(px, a.lx), __fmul_rn(py, a.ly)), __fmul_rn(-az, a.lz));
          float wp[NELL];
          pole_weights<NELL>(a, __fdiv_rn(dotp, kmag), wp);
#pragma unroll
          for (int m = 0; m < NELL; ++m) {
            acc.v[m] += ((double)w[m] + (double)wp[m]) * cre;
            if (CROSS) acc.v[NELL + m] += ((double)w[m] - (double)wp[m]) * cim;
          }
        }
      }
      const unsigned modes = (unsigned)(xs * ys) * (inner ? 2u : 1u);
      acc.n += modes;
      acc.k += (double)modes * (double)kmag;
    }
    flush(cur.bin);
  }
  __syncthreads();
  // [2 nell + 2][nb] per CTA: (Re, Im) per multipole, mode count, sum |k|; columns in order
  double* out = partials + (b * gridDim.x + blockIdx.x) * (long long)(2 * NELL + 2) * nb;
  for (int i = threadIdx.x; i < (2 * NELL + 2) * nb; i += blockDim.x) {
    const int q = i / nb, bin = i - q * nb;
    double s = 0.0;
    if (q == 2 * NELL) {
      for (int c = 0; c < cols; ++c) s += (double)count[bin * cols + c];
    } else if (q == 2 * NELL + 1 || !(q & 1) || CROSS) {
      const int v = q == 2 * NELL + 1 ? NV : ((q & 1) ? NELL + q / 2 : q / 2);
      for (int c = 0; c < cols; ++c) s += hist[(size_t)v * plane + bin * cols + c];
    }
    out[i] = s;
  }
}

template <int NELL, bool CROSS>
static cudaError_t launch_poles(const float2* spec1, const float2* spec2, const PolesArgs& a, const float* kedges,
                                double* partials, int ctas, int batch, cudaStream_t s) {
  const size_t smem = poles_columns(a.nedges, NELL, CROSS) * poles_column_bytes(a.nedges, NELL, CROSS) +
                      sizeof(float) * a.nedges;
  cudaError_t e = cudaFuncSetAttribute(k_power_poles<NELL, CROSS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  k_power_poles<NELL, CROSS><<<dim3(ctas, batch), kPolesThreads, smem, s>>>(spec1, spec2, a, kedges, partials);
  note_launch();
  return cudaGetLastError();
}

int power_poles_ctas(const MeshDims& d) {
  const long long nel = d.spec_elems();
  long long c = (nel + kPolesThreads - 1) / kPolesThreads;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const long long cap = (long long)nsm * 2;
  return (int)(c < cap ? (c < 1 ? 1 : c) : cap);
}

cudaError_t power_poles(const float* mesh1, const float* mesh2, const MeshDims& d, const float* kedges, int nedges,
                        const float* box, const float* los, const int* ells, int nell, float2* spec1, float2* spec2,
                        double* partials, double* out, cudaStream_t s) {
  cudaError_t e = rfft3d_forward(mesh1, spec1, d, 0.0f, s);
  if (e == cudaSuccess && mesh2) e = rfft3d_forward(mesh2, spec2, d, 0.0f, s);
  if (e != cudaSuccess) return e;
  PolesArgs a;
  a.nx = d.nx;
  a.ny = d.ny;
  a.nz = d.nz;
  a.nedges = nedges;
  a.nell = nell;
  a.cx = (float)(2.0 * M_PI / (double)box[0]);
  a.cy = (float)(2.0 * M_PI / (double)box[1]);
  a.cz = (float)(2.0 * M_PI / (double)box[2]);
  a.lx = los[0];
  a.ly = los[1];
  a.lz = los[2];
  a.norm = 1.0f / ((float)d.nx * (float)d.ny * (float)d.nz);
  a.lmax = 0;
  for (int i = 0; i < kMaxPoles; ++i) {
    a.ells[i] = i < nell ? ells[i] : 0;
    if (a.ells[i] > a.lmax) a.lmax = a.ells[i];
  }
  const int ctas = power_poles_ctas(d);
  const int nq = 2 * nell + 2;
  const long long threads = (long long)ctas * kPolesThreads, hx = d.nx / 2 + 1, hy = d.ny / 2 + 1;
  a.strip = kPolesStrip;
  while (a.strip > 1 && hx * d.hz() * ((hy + a.strip - 1) / a.strip) < threads) a.strip >>= 1;
  e = cudaErrorInvalidValue;
  switch (nell) {
#define JFLI_POLES(N_)                                                                             \
  case N_:                                                                                         \
    e = mesh2 ? launch_poles<N_, true>(spec1, spec2, a, kedges, partials, ctas, d.batch, s)        \
              : launch_poles<N_, false>(spec1, spec1, a, kedges, partials, ctas, d.batch, s);      \
    break;
    JFLI_POLES(1) JFLI_POLES(2) JFLI_POLES(3) JFLI_POLES(4) JFLI_POLES(5) JFLI_POLES(6) JFLI_POLES(7) JFLI_POLES(8)
#undef JFLI_POLES
  }
  if (e != cudaSuccess) return e;
  return sums_finalize(partials, ctas, nq * (nedges + 1), out, d.batch, s);
}

}  // namespace jfli
