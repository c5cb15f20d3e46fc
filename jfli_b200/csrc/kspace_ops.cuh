// k-space operators applied inside the x pass of the 3D FFT (see fft.cu).
//
// Wavenumbers follow the particle-mesh convention of JaxPM's `fftk`
// (k_i = 2*pi*fftfreq(n_i), radians per cell) for the Poisson/PGD kernels, and the
// physical convention of jax-fli's `_initialize_pk` (k_i = 2*pi*fftfreq(n_i)*n_i/L_i,
// h/Mpc) for P(k) and initial conditions.
#pragma once

#include "binning.cuh"
#include "common.cuh"

namespace jfli {

// k_i^2 for bin i of an axis of length n, rounded to float like fftk's float32 table.
__device__ __forceinline__ float k_rad_per_cell(int i, int n) {
  return (float)(6.283185307179586476925 * (double)signed_freq(i, n) / (double)n);
}

// Poisson potential: pot_k = delta_k * (-1/k^2) * norm, k = 0 -> 0.
// Follows JaxPM `invlaplace_kernel` (reference call site pm/solvers.py:22 via pm_forces).
struct PoissonOp {
  int nx, ny, nz;
  float norm;
  static size_t smem_bytes(const PoissonOp& op) { return sizeof(float) * op.nx; }
  __device__ void prologue(float* sm, int) const {
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
      const float k = k_rad_per_cell(i, nx);
      sm[i] = k * k;
    }
    __syncthreads();
  }
  __device__ float2 apply(float2 v, int kx, int ky, int kz, float* sm, int) const {
    const float k1 = k_rad_per_cell(ky, ny);
    const float k2 = k_rad_per_cell(kz, nz);
    const float kk = sm[kx] + k1 * k1 + k2 * k2;
    const float g = (kk == 0.f) ? 0.f : -1.f / kk;
    return cscale(v, g * norm);
  }
};

// PGD short-range potential (reference pm/correction.py:177-189), optionally mixed with the
// Poisson potential:
// pot_k = delta_k * (-1/k^2) * (c0 + c1 exp(-kl^2/k^2) exp(-k^4/ks^4)) * norm, k = 0 -> 0.
// (c0, c1) = (0, 1) is the PGD potential; (kick, boost) the combined potential whose force
// is a reversible step's kick plus SharpeningKernel's velocity boost at the same positions
// (reference pm/solvers.py:292-318, pm/correction.py:214-333).
struct PgdOp {
  int nx, ny, nz;
  float norm, kl2, ks4;
  float c0 = 0.f, c1 = 1.f;
  static size_t smem_bytes(const PgdOp& op) { return sizeof(float) * op.nx; }
  __device__ void prologue(float* sm, int) const {
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
      const float k = k_rad_per_cell(i, nx);
      sm[i] = k * k;
    }
    __syncthreads();
  }
  __device__ float2 apply(float2 v, int kx, int ky, int kz, float* sm, int) const {
    const float k1 = k_rad_per_cell(ky, ny);
    const float k2 = k_rad_per_cell(kz, nz);
    const float kk = sm[kx] + k1 * k1 + k2 * k2;
    if (kk == 0.f) return make_float2(0.f, 0.f);
    const float range = expf(-kl2 / kk) * expf(-(kk * kk) / ks4);
    return cscale(v, (-1.f / kk) * (c0 + c1 * range) * norm);
  }
};

// Linear interpolation with end extrapolation on a tabulated P(k), the behaviour of
// jax_cosmo's `interp` used by JaxPM `interpolate_power_spectrum`
// (reference call site initial.py:171-173; infer/dist.py:50-53).
__device__ __forceinline__ float interp_table(float x, const float* xp, const float* fp, int n) {
  // first index with xp[i] >= x (searchsorted, side="left")
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (xp[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  int i = lo - 1;
  i = i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
  const float slope = (fp[i + 1] - fp[i]) / (xp[i + 1] - xp[i]);
  return fp[i] + (x - xp[i]) * slope;
}

// interp_table with the slope of the segment it used (the derivative of the linear
// interpolation, end segments extrapolated as in the value).
__device__ __forceinline__ float interp_table_d(float x, const float* xp, const float* fp, int n, float& slope) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (xp[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  int i = lo - 1;
  i = i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
  slope = (fp[i + 1] - fp[i]) / (xp[i + 1] - xp[i]);
  return fp[i] + (x - xp[i]) * slope;
}

// Gaussian initial conditions (reference initial.py:175-182):
// field_k *= sqrt(P(|k|) * M / V) * norm, |k| in h/Mpc. `zero_mode_one` reproduces the
// k = 0 guard of infer/dist.py:68.
struct IcOp {
  int nx, ny, nz;
  const float* ktab;
  const float* ptab;
  int ntab;
  float lx, ly, lz;  // box side lengths L_i
  float factor;      // M / V
  float norm;        // 1 / M
  int zero_mode_one;
  // Tangent mode (dptab != null): the derivative of the multiplier along a change dptab
  // of the table, interp(dptab) * factor / (2 sqrt(P)) (0 where P <= 0 and at the
  // k = 0 guard), used for gradients with respect to the cosmology behind P(k).
  const float* dptab = nullptr;
  // Shared memory: kx [nx], the tables k, P [ntab], the segments' slopes or in tangent mode dP
  // [ntab], the buckets' starts, and the buckets' shift and base.
  //
  // A search from the ends of the table per mode (seven dependent reads for 128 points) and the
  // division of its slope took longer than the transform. The slopes are made once per CTA, and
  // k's bits above `shift` (eighths of an octave or coarser, so that the table's span fits) give
  // a bucket whose first and last index are tabulated: a logarithmic table has about one point
  // to a bucket. The index, and so the result, is the same. 384^3: 380 -> 287 us (Poisson 171).
  static constexpr int kBuckets = 256;
  static size_t smem_bytes(const IcOp& op) {
    return sizeof(float) * (op.nx + 3 * op.ntab) + sizeof(unsigned short) * (kBuckets + 2) + 2 * sizeof(int);
  }
  __device__ void prologue(float* sm, int) const {
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
      sm[i] = k_rad_per_cell(i, nx) / lx * (float)nx;
    }
    float* xp = sm + nx;
    float* fp = xp + ntab;
    for (int i = threadIdx.x; i < ntab; i += blockDim.x) {
      xp[i] = ktab[i];
      fp[i] = ptab[i];
      if (dptab) fp[ntab + i] = dptab[i];
    }
    __syncthreads();
    if (!dptab)
      for (int i = threadIdx.x; i + 1 < ntab; i += blockDim.x)
        fp[ntab + i] = (fp[i + 1] - fp[i]) / (xp[i + 1] - xp[i]);
    unsigned short* start = reinterpret_cast<unsigned short*>(fp + 2 * ntab);
    // bucket 1 starts from the second k of the table: the first may be 0
    const int first = __float_as_int(fmaxf(xp[1], 0.f)), span = __float_as_int(fmaxf(xp[ntab - 1], 0.f)) - first;
    int shift = 20;
    while ((span >> shift) > kBuckets - 4) ++shift;
    const int base = first >> shift;
    if (threadIdx.x == 0) {
      int* at = reinterpret_cast<int*>(start + kBuckets + 2);
      at[0] = shift;
      at[1] = base - 1;
    }
    for (int b = threadIdx.x; b <= kBuckets; b += blockDim.x)
      start[b] = (unsigned short)(b == 0          ? 0
                                  : b == kBuckets ? ntab
                                                  : search(__int_as_float((base + b - 1) << shift), xp, 0, ntab));
    __syncthreads();
  }
  // first index in [lo, hi) with xp[i] >= x, or hi
  static __device__ __forceinline__ int search(float x, const float* xp, int lo, int hi) {
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (xp[mid] < x)
        lo = mid + 1;
      else
        hi = mid;
    }
    return lo;
  }
  __device__ float2 apply(float2 v, int kx, int ky, int kz, float* sm, int) const {
    const float ax = sm[kx];
    const float ay = k_rad_per_cell(ky, ny) / ly * (float)ny;
    const float az = k_rad_per_cell(kz, nz) / lz * (float)nz;
    const float kmag = sqrtf(ax * ax + ay * ay + az * az);
    const float *xp = sm + nx, *fp = xp + ntab;
    const unsigned short* start = reinterpret_cast<const unsigned short*>(fp + 2 * ntab);
    const int* at = reinterpret_cast<const int*>(start + kBuckets + 2);
    const int b = min(max((__float_as_int(kmag) >> at[0]) - at[1], 0), kBuckets - 1);
    const int i = min(max(search(kmag, xp, start[b], start[b + 1]) - 1, 0), ntab - 2);
    const float slope = dptab ? (fp[i + 1] - fp[i]) / (xp[i + 1] - xp[i]) : fp[ntab + i];
    float pk = (fp[i] + (kmag - xp[i]) * slope) * factor;
    if (dptab) {
      const float dpk = interp_table(kmag, xp, fp + ntab, ntab) * factor;
      float m = pk > 0.f ? dpk / (2.0f * sqrtf(pk)) : 0.f;
      if (zero_mode_one && kmag == 0.f) m = 0.f;
      return cscale(v, m * norm);
    }
    if (zero_mode_one && kmag == 0.f) pk = 1.f;
    return cscale(v, sqrtf(pk) * norm);
  }
};

// Power spectrum histogram (reference _src/power/_compute.py:23-119): |delta_k|^2 with
// ortho normalisation binned by digitize(|k|, kedges) over the full grid. The half
// spectrum stores each mode with 0 < kz < nz/2 once for itself and its conjugate
// partner, so those modes count twice. Sums are kept in FP64.
struct PkArgs {
  int nx, ny, nz;
  const float* kedges;
  int nedges;
  float cx, cy, cz;  // 2*pi / L_i
  float norm;        // 1 / M for norm="ortho"
  double* partials;  // [batch][nctas][3][nedges+1]
};

constexpr size_t kPkHistBudget = 24u << 10;  // bytes of histogram columns (one column always fits)

__host__ __device__ inline int pk_hist_columns(int nedges) {
  return histogram_columns((size_t)(nedges + 1) * 20, kPkHistBudget);
}
// shared memory of the histogram, the edges and the tile's column constants
__host__ __device__ inline size_t pk_smem_bytes(int nedges, int columns) {
  return (size_t)pk_hist_columns(nedges) * (nedges + 1) * 20 + sizeof(float) * ((size_t)nedges + 3 * (size_t)columns) + 8;
}

// A CTA's part of the histogram: [nedges + 1][cols] sums of power and of |k| (FP64) and mode
// counts (32 bits: a mesh has fewer than 2^32 modes), the edges, and per column of the tile
// (ky^2, kz^2, weight).
struct PkTile {
  double *power, *ksum;
  unsigned* count;
  float *edges, *column;
  int cols;

  __device__ PkTile(const PkArgs& a, void* sm) {
    cols = pk_hist_columns(a.nedges);
    const size_t n = (size_t)cols * (a.nedges + 1);
    power = reinterpret_cast<double*>(sm);
    ksum = power + n;
    count = reinterpret_cast<unsigned*>(ksum + n);
    edges = reinterpret_cast<float*>(count + n);
    column = edges + a.nedges;
  }
  __device__ void clear(const PkArgs& a) {
    for (int i = threadIdx.x; i < cols * (a.nedges + 1); i += blockDim.x) {
      power[i] = 0.0;
      ksum[i] = 0.0;
      count[i] = 0;
    }
    for (int i = threadIdx.x; i < a.nedges; i += blockDim.x) edges[i] = a.kedges[i];
  }
  // tile columns c0 .. c0 + w - 1, column = ky hz + kz (one past the last has weight 0)
  __device__ void set_columns(const PkArgs& a, int c0, int w, int ncols, int hz) {
    for (int c = threadIdx.x; c < w; c += blockDim.x) {
      const int col = c0 + c;
      const int ky = col / hz, kz = col - ky * hz;
      // |k| with the rounding of the reference's float32 grid: no FMA contraction, sum in
      // x, y, z order, correctly rounded sqrt (decides the bin of modes on an edge)
      const float ay = __fmul_rn(a.cy, (float)signed_freq(ky, a.ny));
      const float az = __fmul_rn(a.cz, (float)signed_freq(kz, a.nz));
      column[3 * c + 0] = __fmul_rn(ay, ay);
      column[3 * c + 1] = __fmul_rn(az, az);
      column[3 * c + 2] = col < ncols ? ((kz == 0 || 2 * kz == a.nz) ? 1.f : 2.f) : 0.f;
    }
  }
  __device__ __forceinline__ float kmag(float ax2, int c) const {
    return __fsqrt_rn(__fadd_rn(__fadd_rn(ax2, column[3 * c]), column[3 * c + 1]));
  }
  __device__ __forceinline__ void flush(int bin, double p, double k, unsigned n) {
    const int i = bin * cols + ((threadIdx.x & 31) & (cols - 1));
    atomicAdd(power + i, p);
    atomicAdd(ksum + i, k);
    atomicAdd(count + i, n);
  }
  // Bins a transformed tile buf[e * pitch + c] (element e < n of column c < w), pitch odd.
  // The modes e and n - e have the same |k| bit for bit and are taken together. Lanes run
  // along e (no bank conflicts); a thread walks `span` successive columns. The element
  // e = n / 2 has no partner and would leave a row of one lane, so the lanes of the last
  // warps take it, one column each.
  __device__ __forceinline__ void add(const PkArgs& a, const float2* buf, int pitch, int n, int w) {
    const int rows = (n + 1) / 2;
    const int groups = max(1, min(w, (int)blockDim.x / rows));
    const int span = (w + groups - 1) / groups;
    for (int i = threadIdx.x; i < rows * groups; i += blockDim.x) {
      const int grp = i / rows, e = i - grp * rows;
      const float ax = __fmul_rn(a.cx, (float)e), ax2 = __fmul_rn(ax, ax);
      const float2* lower = buf + e * pitch;
      const float2* upper = buf + (n - e) * pitch;  // read only when e > 0
      BinCursor cur;
      double p = 0.0, ks = 0.0;
      unsigned cnt = 0;
      const int c1 = min(w, (grp + 1) * span);
      for (int c = grp * span; c < c1; ++c) {
        const float wt = column[3 * c + 2];
        if (wt == 0.f) break;
        const float k = kmag(ax2, c);
        if (!cur.holds(k)) {
          if (cnt) flush(cur.bin, p * (double)a.norm, ks, cnt);
          cur.move(k, edges, a.nedges);
          p = ks = 0.0;
          cnt = 0;
        }
        const float2 f = lower[c];
        double q = (double)f.x * f.x + (double)f.y * f.y;
        float m = wt;
        if (e > 0) {
          const float2 g = upper[c];
          q += (double)g.x * g.x + (double)g.y * g.y;
          m += wt;
        }
        p += (double)wt * q;
        ks += (double)m * (double)k;
        cnt += (unsigned)m;
      }
      if (cnt) flush(cur.bin, p * (double)a.norm, ks, cnt);
    }
    if ((n & 1) == 0) {
      const int c = (int)blockDim.x - 1 - (int)threadIdx.x;
      if (c < w && column[3 * c + 2] > 0.f) {
        const float wt = column[3 * c + 2];
        const float ax = __fmul_rn(a.cx, (float)(n / 2));
        const float k = kmag(__fmul_rn(ax, ax), c);
        const float2 f = buf[(n / 2) * pitch + c];
        flush(digitize(k, edges, a.nedges), (double)wt * ((double)f.x * f.x + (double)f.y * f.y) * (double)a.norm,
              (double)wt * (double)k, (unsigned)wt);
      }
    }
  }
  // the CTA's sums, columns added in order; called after a barrier
  __device__ void store(const PkArgs& a, int batch, int cta, int nctas) {
    const int nb = a.nedges + 1;
    double* dst = a.partials + ((long long)batch * nctas + cta) * 3 * nb;
    for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) {
      const int q = i / nb, bin = i - q * nb;
      double s = 0.0;
      for (int c = 0; c < cols; ++c) {
        const int at = bin * cols + c;
        s += q == 0 ? power[at] : (q == 1 ? (double)count[at] : ksum[at]);
      }
      dst[i] = s;
    }
  }
};

// Adjoint of P(k) with respect to the mesh: mode k is scaled by weights[bin(k)] * norm,
// bin(k) = digitize(|k|, kedges) with the same |k| rounding as the histogram, so that the inverse
// transform gives dL/dmesh = sum over bins of dL/dP_b * dP_b/dmesh when
// weights[b] = 2 * dL/dP_b * prod(L/N) / count_b (0 for the dropped under/overflow bins).
// L_l(mu) by the reference's recurrence, in FP32 (the multipole weights (2l + 1) L_l(mu) of
// the reference's _power, _src/power/_compute.py:96-103)
__device__ __forceinline__ float legendre_f32(int ell, float mu) {
  if (ell == 0) return 1.f;
  if (ell == 1) return mu;
  float p0 = 1.f, p1 = mu;
  for (int n = 2; n <= ell; ++n) {
    const float pn = __fdiv_rn(__fsub_rn(__fmul_rn(__fmul_rn((float)(2 * n - 1), mu), p1), __fmul_rn((float)(n - 1), p0)),
                               (float)n);
    p0 = p1;
    p1 = pn;
  }
  return p1;
}

constexpr int kMaxAdjPoles = 8;

// Adjoint of the binned P(k) sums: out = irfft(rfft(mesh) * w(k) / M). Monopole (nell = 0):
// w(k) = weights[bin(|k|)]. Multipoles of an auto spectrum (nell > 0): the mode's weight is
// sum over the multipoles e of weights[e][bin] (2l_e + 1) L_l_e(mu), mu = (k . los) / |k|,
// and w(k) its mean over the mode and its conjugate partner (a real mesh's gradient sees
// only that Hermitian part). The partner's signed frequencies are the mode's negated, except
// along an axis where the mode sits on the Nyquist plane (index n/2, frequency -n/2 for
// both): there mu is not -mu, and odd multipoles of an auto spectrum do not vanish.
// Cross spectra (cplx = 1): weights holds the real then the imaginary parts, nell x (nedges +
// 1) each, of a complex per-bin factor c; the Hermitian part of c w(k) is the multiplier:
// Re(c) (w(k) + w(partner)) / 2 + i Im(c) (w(k) - w(partner)) / 2.
struct PkAdjOp {
  int nx, ny, nz;
  const float* kedges;
  const float* weights;  // nedges + 1
  int nedges;
  float cx, cy, cz;  // 2*pi / L_i
  float norm;        // 1 / M (inverse transform)
  int nell = 0;      // multipoles: weights holds nell x (nedges + 1) (twice that when cplx)
  int cplx = 0;
  int ells[kMaxAdjPoles] = {};
  float lx = 0.f, ly = 0.f, lz = 1.f;  // unit line of sight
  static size_t smem_bytes(const PkAdjOp& op) {
    return sizeof(float) * (op.nedges + (op.cplx ? 2 : 1) * (op.nell > 0 ? op.nell : 1) * (op.nedges + 1));
  }
  __device__ void prologue(float* sm, int) const {
    const int nw = (cplx ? 2 : 1) * (nell > 0 ? nell : 1) * (nedges + 1);
    for (int i = threadIdx.x; i < nedges; i += blockDim.x) sm[i] = kedges[i];
    for (int i = threadIdx.x; i < nw; i += blockDim.x) sm[nedges + i] = weights[i];
    __syncthreads();
  }
  __device__ float2 apply(float2 v, int kx, int ky, int kz, float* sm, int) const {
    const float ax = __fmul_rn(cx, (float)signed_freq(kx, nx));
    const float ay = __fmul_rn(cy, (float)signed_freq(ky, ny));
    const float az = __fmul_rn(cz, (float)signed_freq(kz, nz));
    const float kmag = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(ax, ax), __fmul_rn(ay, ay)), __fmul_rn(az, az)));
    int lo = 0, hi = nedges;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (sm[mid] <= kmag)
        lo = mid + 1;
      else
        hi = mid;
    }
    if (nell == 0) return cscale(v, sm[nedges + lo] * norm);
    const float dot = __fadd_rn(__fadd_rn(__fmul_rn(ax, lx), __fmul_rn(ay, ly)), __fmul_rn(az, lz));
    const float mu = kmag == 0.f ? 0.f : __fdiv_rn(dot, kmag);
    const float px = 2 * kx == nx ? ax : -ax, py = 2 * ky == ny ? ay : -ay, pz = 2 * kz == nz ? az : -az;
    const float dotp = __fadd_rn(__fadd_rn(__fmul_rn(px, lx), __fmul_rn(py, ly)), __fmul_rn(pz, lz));
    const float mup = kmag == 0.f ? 0.f : __fdiv_rn(dotp, kmag);
    float w = 0.f, wo = 0.f;
    const int im0 = nedges + nell * (nedges + 1);
    for (int e = 0; e < nell; ++e) {
      const float f = (float)(2 * ells[e] + 1);
      const float a = __fmul_rn(f, legendre_f32(ells[e], mu)), b = __fmul_rn(f, legendre_f32(ells[e], mup));
      w += sm[nedges + e * (nedges + 1) + lo] * (0.5f * (a + b));
      if (cplx) wo += sm[im0 + e * (nedges + 1) + lo] * (0.5f * (a - b));
    }
    if (!cplx) return cscale(v, w * norm);
    return make_float2((v.x * w - v.y * wo) * norm, (v.x * wo + v.y * w) * norm);
  }
};

}  // namespace jfli
