// z passes of the 3D FFT: r2c and c2r along the contiguous axis.
#include "fft_engine.cuh"
#include "fft_passes.cuh"
#include "fft_reg.cuh"
#include "internal.h"
#include "smem_async.cuh"

namespace jfli {

// ---------------------------------------------------------------------------------
// r2c along z: a CTA owns `rows` (a power of two) consecutive z-rows. Each row of nz
// reals is read as nh = nz/2 complex pairs (x[2j] + i x[2j+1]), transformed with an
// nh-point FFT and untangled into the nh+1 non-redundant outputs. `sub` is subtracted
// from every input (it only changes the k = 0 mode and keeps FP32 headroom for the
// fluctuations of a density of mean `sub`).
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(kFftThreads) k_rfft_z(const float* __restrict__ in, float2* __restrict__ out,
                                                        int nrows, int nz, int rows, FftPlan pl, float sub,
                                                        long long in_bstride, long long out_bstride) {
  extern __shared__ float2 sm[];
  const int nh = nz >> 1;
  const int hz = nh + 1;
  const int P = rows + 1;
  float2* bufa = sm;
  float2* bufb = bufa + (size_t)hz * P;
  float2* tw = bufb + (size_t)hz * P;
  float2* tw2 = tw + nh;
  in += (long long)blockIdx.y * in_bstride;
  out += (long long)blockIdx.y * out_bstride;
  const int row0 = blockIdx.x * rows;

  fill_twiddles(tw, nh);
  for (int m = threadIdx.x; m <= nh; m += blockDim.x) {
    double s, c;
    sincospi((double)m / (double)nh, &s, &c);
    tw2[m] = make_float2((float)c, (float)-s);  // exp(-2 pi i m / nz)
  }
  const float2* in2 = reinterpret_cast<const float2*>(in);
  const int E = rows * nh;
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int r = idx / nh;
    const int j = idx - r * nh;
    const int row = row0 + r;
    float2 z = make_float2(0.f, 0.f);
    if (row < nrows) {
      z = in2[(long long)row * nh + j];
      z.x -= sub;
      z.y -= sub;
    }
    bufa[j * P + r] = z;
  }
  __syncthreads();
  const float2* res = tile_fft<-1>(bufa, bufb, P, fft_ilog2(rows), pl, tw);
  const int E2 = rows * hz;
  for (int idx = threadIdx.x; idx < E2; idx += blockDim.x) {
    const int r = idx / hz;
    const int k = idx - r * hz;
    const int row = row0 + r;
    if (row >= nrows) continue;
    const float2 zk = res[(k == nh ? 0 : k) * P + r];
    const float2 zm = res[(k == 0 ? 0 : nh - k) * P + r];
    const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    const float2 d = make_float2(zk.x - zm.x, zk.y + zm.y);  // zk - conj(zm)
    const float2 o = make_float2(0.5f * d.y, -0.5f * d.x);   // d / (2i)
    out[(long long)row * hz + k] = cadd(e, cmul(tw2[k], o));
  }
}

// ---------------------------------------------------------------------------------
// c2r along z (unnormalised; callers fold 1/M into the k-space operator or pass
// `scale`). Reads nh+1 half-spectrum entries per row, re-tangles them into nh complex
// values, inverse-transforms and writes nz reals.
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(kFftThreads) k_irfft_z(const float2* __restrict__ in, float* __restrict__ out,
                                                         int nrows, int nz, int rows, FftPlan pl, float scale,
                                                         long long in_bstride, long long out_bstride) {
  extern __shared__ float2 sm[];
  const int nh = nz >> 1;
  const int hz = nh + 1;
  const int P = rows + 1;
  float2* bufa = sm;
  float2* bufb = bufa + (size_t)hz * P;
  float2* tw = bufb + (size_t)hz * P;
  float2* tw2 = tw + nh;
  in += (long long)blockIdx.y * in_bstride;
  out += (long long)blockIdx.y * out_bstride;
  const int row0 = blockIdx.x * rows;

  fill_twiddles(tw, nh);
  for (int m = threadIdx.x; m <= nh; m += blockDim.x) {
    double s, c;
    sincospi((double)m / (double)nh, &s, &c);
    tw2[m] = make_float2((float)c, (float)s);  // exp(+2 pi i m / nz)
  }
  const int E2 = rows * hz;
  for (int idx = threadIdx.x; idx < E2; idx += blockDim.x) {
    const int r = idx / hz;
    const int k = idx - r * hz;
    const int row = row0 + r;
    bufb[k * P + r] = (row < nrows) ? in[(long long)row * hz + k] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  // Z[k] = (X[k] + conj X[nh-k]) + i (X[k] - conj X[nh-k]) exp(+2 pi i k / nz)
  const int E = rows * nh;
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int k = idx / rows;
    const int r = idx - k * rows;
    const float2 xk = bufb[k * P + r];
    const float2 xm = bufb[(nh - k) * P + r];
    const float2 e = make_float2(xk.x + xm.x, xk.y - xm.y);
    const float2 d = cmul(make_float2(xk.x - xm.x, xk.y + xm.y), tw2[k]);
    bufa[k * P + r] = make_float2(e.x - d.y, e.y + d.x);
  }
  __syncthreads();
  const float2* res = tile_fft<1>(bufa, bufb, P, fft_ilog2(rows), pl, tw);
  float2* out2 = reinterpret_cast<float2*>(out);
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int r = idx / nh;
    const int j = idx - r * nh;
    const int row = row0 + r;
    if (row < nrows) out2[(long long)row * nh + j] = cscale(res[j * P + r], scale);
  }
}

// Shared-memory layout of the register row passes, without bank conflicts. A half warp's 16
// eight-byte accesses are served at once when their indices differ mod 16.
//   * exchange buffer: stage 1 has t across the lanes, so its t stride YS is odd; stage 2 has kb
//     and then the row across the lanes, so the row stride is Q mod 16 (kb + Q r = tid).
//   * transformed rows (r2c): the row stride ZS is Q mod 16 for the same reason.
//   * stage-1 twiddles w^(t kb) are laid out by (kb, t) from Q = 12 on: read from the plain table
//     the stride kb costs up to 8 passes (384^3 c2r 93.9 -> 90.7 us; with Q = 8 the fill costs
//     as much as it saves, 256^3 c2r 26.6 and 27.5).
// And the r2c output takes the pair (k, N - k) per thread, whose two inputs are the same. r2c
// with all of it: 256^3 35.2 -> 31.7 us, 384^3 120 -> 106, 512^3 230 -> 205; c2r 384^3 98 -> 91.
template <int N>
struct RowSmem {
  static constexpr int P = Split<N>::P, Q = Split<N>::Q, R = RowCfg<N>::R;
  static constexpr int mod16(int least) { return least + ((Q - least) % 16 + 16) % 16; }
  static constexpr int YS = Q | 1;
  static constexpr int S = mod16(P * YS);
  static constexpr int ZS = mod16(N + 1);
  static constexpr bool kStaged = Q >= 12;
  static constexpr int TWS = kStaged ? (Q - 1) * P : 0;  // w^(t kb), kb = 1 .. Q - 1
  static constexpr int r2c = N + N + 1 + TWS + R * (S > ZS ? S : ZS);
  static constexpr int XB = R * (N + 1 > S ? N + 1 : S);
  static constexpr int c2r = XB + N + N + 1 + TWS;
};

template <int P>
__device__ __forceinline__ float2 stage_twiddle(const float2* __restrict__ twg, int m) {
  return twg[(m % P) * (m / P + 1)];
}
// r2c along z, nh = nz/2 = N complex per row, R rows per CTA.
// With `clear` (the input mesh itself) each input value is overwritten with 0 by the thread
// that read it, so a density mesh comes out cleared for the next paint.
template <int N>
__global__ void __launch_bounds__(RowCfg<N>::T) k_rfft_z_reg(const float* in, float2* __restrict__ out,
                                                             int nrows, float sub, const float2* __restrict__ twg,
                                                             const float2* __restrict__ twg2, long long in_b,
                                                             long long out_b, float* clear) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, R = RowCfg<N>::R, T = RowCfg<N>::T;
  constexpr int S = RowSmem<N>::S, YS = RowSmem<N>::YS, ZS = RowSmem<N>::ZS;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* tw2 = tw + N;       // N+1 entries: exp(-2 pi i k / (2N))
  float2* tws = tw2 + N + 1;  // stage-1 twiddles
  float2* ybuf = tws + RowSmem<N>::TWS;  // rows of stride S; reused for the Z rows (stride ZS)
  in += (long long)blockIdx.y * in_b;
  out += (long long)blockIdx.y * out_b;
  if (clear) clear += (long long)blockIdx.y * in_b;
  const int tid = threadIdx.x;
  grid_wait();
  for (int m = tid; m < N; m += T) tw[m] = twg[m];
  for (int m = tid; m <= N; m += T) tw2[m] = twg2[m];
  for (int m = tid; m < RowSmem<N>::TWS; m += T) tws[m] = stage_twiddle<P>(twg, m);
  __syncthreads();
  const int row0 = blockIdx.x * R;
  const float2* in2 = reinterpret_cast<const float2*>(in);
  for (int w = tid; w < R * P; w += T) {
    const int t = w % P, r = w / P;
    const int row = row0 + r;
    float2 u[Q];
    if (row < nrows) {
      const float2* src = in2 + (long long)row * N + t;
#pragma unroll
      for (int m = 0; m < Q; ++m) {
        const float2 z = src[P * m];
        u[m] = make_float2(z.x - sub, z.y - sub);
      }
      if (clear) {
        float2* dst = reinterpret_cast<float2*>(clear) + (long long)row * N + t;
#pragma unroll
        for (int m = 0; m < Q; ++m) dst[P * m] = make_float2(0.f, 0.f);
      }
    } else {
#pragma unroll
      for (int m = 0; m < Q; ++m) u[m] = make_float2(0.f, 0.f);
    }
    RegDFT<Q, -1, P>::run(u, tw);
#pragma unroll
    for (int kb = 0; kb < Q; ++kb)
      ybuf[r * S + t * YS + kb] = (kb == 0) ? u[0] : cmul(u[kb], RowSmem<N>::kStaged ? tws[(kb - 1) * P + t] : tw[t * kb]);
  }
  __syncthreads();
  const int kb = tid % Q, r = tid / Q;
  float2 u[P];
#pragma unroll
  for (int t = 0; t < P; ++t) u[t] = ybuf[r * S + t * YS + kb];
  RegDFT<P, -1, Q>::run(u, tw);
  __syncthreads();
#pragma unroll
  for (int ka = 0; ka < P; ++ka) ybuf[r * ZS + kb + Q * ka] = u[ka];
  __syncthreads();
  const auto untangle = [](float2 zk, float2 zm, float2 w) {
    const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    const float2 d = make_float2(zk.x - zm.x, zk.y + zm.y);
    const float2 o = make_float2(0.5f * d.y, -0.5f * d.x);
    return cadd(e, cmul(w, o));
  };
  grid_release();
  constexpr int H = N / 2 + 1;
  for (int w = tid; w < R * H; w += T) {
    const int rr = w / H;
    const int k = w - rr * H;
    const int row = row0 + rr;
    if (row >= nrows) continue;
    const float2 zk = ybuf[rr * ZS + k];
    const float2 zm = ybuf[rr * ZS + (k == 0 ? 0 : N - k)];
    float2* dst = out + (long long)row * (N + 1);
    dst[k] = untangle(zk, zm, tw2[k]);
    if (2 * k != N) dst[N - k] = untangle(zm, zk, tw2[N - k]);
  }
}

// c2r along z (unnormalised times `scale`). A CTA's input rows are one contiguous block; its
// threads bring it into shared memory with asynchronous 16-byte copies, so the whole block is
// in flight at once (a loop of loads, each waited for before its store, left the pass at 2.0
// TB/s: 384^3 222 -> 98 us (91 with RowSmem), 256^3 41.5 -> 26.6 us, 64^3 6.0 -> 3.7 us).
template <int N>
__global__ void __launch_bounds__(RowCfg<N>::T) k_irfft_z_reg(const float2* __restrict__ in, float* __restrict__ out,
                                                              int nrows, float scale, const float2* __restrict__ twg,
                                                              const float2* __restrict__ twg2, long long in_b,
                                                              long long out_b) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, R = RowCfg<N>::R, T = RowCfg<N>::T;
  constexpr int S = RowSmem<N>::S, YS = RowSmem<N>::YS;
  constexpr int IT = (R * P + T - 1) / T;  // stage-1 items per thread
  extern __shared__ __align__(16) float2 sm[];
  float2* xbuf = sm;  // R*(N+1) input rows, then (aliased) the R*S exchange buffer
  float2* ybuf = xbuf;
  float2* tw = sm + RowSmem<N>::XB;
  float2* tw2 = tw + N;
  float2* tws = tw2 + N + 1;  // stage-1 twiddles
  in += (long long)blockIdx.y * in_b;
  out += (long long)blockIdx.y * out_b;
  const int tid = threadIdx.x;
  const int row0 = blockIdx.x * R;
  const int have = min(R, nrows - row0) * (N + 1);  // rows past the last are not read
  const float2* src = in + (long long)row0 * (N + 1);
  grid_wait();
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    for (int w = tid; w < have / 2; w += T) copy_async<16>(xbuf + 2 * w, src + 2 * w);
    if ((have & 1) && tid == 0) copy_async<8>(xbuf + have - 1, src + have - 1);
  } else {
    for (int w = tid; w < have; w += T) copy_async<8>(xbuf + w, src + w);
  }
  for (int m = tid; m < N; m += T) tw[m] = twg[m];
  for (int m = tid; m <= N; m += T) tw2[m] = twg2[m];
  for (int m = tid; m < RowSmem<N>::TWS; m += T) tws[m] = stage_twiddle<P>(twg, m);
  copy_async_wait();
  __syncthreads();
  float2 u1[IT][Q];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int w = tid + it * T;
    if (w >= R * P) continue;
    const int t = w % P, r = w / P;
#pragma unroll
    for (int m = 0; m < Q; ++m) {
      const int e = t + P * m;
      const float2 xk = xbuf[r * (N + 1) + e];
      const float2 xm = xbuf[r * (N + 1) + N - e];
      const float2 ee = make_float2(xk.x + xm.x, xk.y - xm.y);
      const float2 dd = cmul(make_float2(xk.x - xm.x, xk.y + xm.y), conjf2(tw2[e]));
      u1[it][m] = make_float2(ee.x - dd.y, ee.y + dd.x);
    }
    RegDFT<Q, 1, P>::run(u1[it], tw);
  }
  __syncthreads();  // every input row has been read; the exchange buffer may overwrite it
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int w = tid + it * T;
    if (w >= R * P) continue;
    const int t = w % P, r = w / P;
#pragma unroll
    for (int kb = 0; kb < Q; ++kb)
      ybuf[r * S + t * YS + kb] = (kb == 0) ? u1[it][0] : cmul(u1[it][kb], conjf2(RowSmem<N>::kStaged ? tws[(kb - 1) * P + t] : tw[t * kb]));
  }
  __syncthreads();
  grid_release();
  const int kb = tid % Q, r = tid / Q;
  const int row = row0 + r;
  float2 u[P];
#pragma unroll
  for (int t = 0; t < P; ++t) u[t] = ybuf[r * S + t * YS + kb];
  RegDFT<P, 1, Q>::run(u, tw);
  if (row < nrows) {
    float2* dst = reinterpret_cast<float2*>(out) + (long long)row * N + kb;
#pragma unroll
    for (int ka = 0; ka < P; ++ka) dst[Q * ka] = cscale(u[ka], scale);
  }
}

template <int N>
static cudaError_t rfft_z_reg(const float* in, float2* out, const MeshDims& d, float sub, cudaStream_t s,
                              float* clear) {
  constexpr int R = RowCfg<N>::R, T = RowCfg<N>::T;
  const float2* tw = twiddle_table(N);
  const float2* tw2 = twiddle_table(2 * N);
  if (!tw || !tw2) return cudaErrorMemoryAllocation;
  const int nrows = d.nx * d.ny;
  const size_t smem = (size_t)RowSmem<N>::r2c * sizeof(float2);
  cudaFuncSetAttribute(k_rfft_z_reg<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_next(overlap_starts(d.cells() * d.batch), k_rfft_z_reg<N>, dim3((nrows + R - 1) / R, d.batch), T, smem, s, in,
              out, nrows, sub, tw, tw2, d.cells(), d.spec_elems(), clear);
  note_launch();
  return cudaGetLastError();
}

template <int N>
static cudaError_t irfft_z_reg(const float2* in, float* out, const MeshDims& d, float scale, cudaStream_t s) {
  constexpr int R = RowCfg<N>::R, T = RowCfg<N>::T;
  const float2* tw = twiddle_table(N);
  const float2* tw2 = twiddle_table(2 * N);
  if (!tw || !tw2) return cudaErrorMemoryAllocation;
  const int nrows = d.nx * d.ny;
  const size_t smem = (size_t)RowSmem<N>::c2r * sizeof(float2);
  cudaFuncSetAttribute(k_irfft_z_reg<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_next(overlap_starts(d.cells() * d.batch), k_irfft_z_reg<N>, dim3((nrows + R - 1) / R, d.batch), T, smem, s, in,
              out, nrows, scale, tw, tw2, d.spec_elems(), d.cells());
  note_launch();
  return cudaGetLastError();
}

// ---- launchers: register kernels, or the shared-memory Stockham pass for the remaining lengths
cudaError_t rfft_z_generic(const float* in, float2* out, const MeshDims& d, float sub, cudaStream_t s) {
  FftPlan pl;
  make_fft_plan(d.nz / 2, &pl);
  const int nrows = d.nx * d.ny;
  const int rows = z_rows_per_cta(d.nz);
  const int nh = d.nz / 2;
  const size_t smem = ((size_t)2 * (nh + 1) * (rows + 1) + nh + nh + 1) * sizeof(float2);
  dim3 grid((nrows + rows - 1) / rows, d.batch);
  cudaFuncSetAttribute(k_rfft_z, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_rfft_z<<<grid, kFftThreads, smem, s>>>(in, out, nrows, d.nz, rows, pl, sub, d.cells(), d.spec_elems());
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_rfft_z(const float* in, float2* out, const MeshDims& d, float sub, cudaStream_t s,
                          float* clear, bool mixed) {
  switch (reg_fft_length(d.nz / 2, mixed)) {
#define JFLI_CASE(N_) \
  case N_:            \
    return rfft_z_reg<N_>(in, out, d, sub, s, clear);
    JFLI_REG_SIZES(JFLI_CASE)
    JFLI_MIXED_SIZES(JFLI_CASE)
#undef JFLI_CASE
    default:
      break;
  }
  cudaError_t e = rfft_z_generic(in, out, d, sub, s);
  if (e == cudaSuccess && clear) e = cudaMemsetAsync(clear, 0, sizeof(float) * (size_t)d.cells() * d.batch, s);
  return e;
}

cudaError_t launch_irfft_z(const float2* in, float* out, const MeshDims& d, float scale, cudaStream_t s,
                           bool mixed) {
  switch (reg_fft_length(d.nz / 2, mixed)) {
#define JFLI_CASE(N_) \
  case N_:            \
    return irfft_z_reg<N_>(in, out, d, scale, s);
    JFLI_REG_SIZES(JFLI_CASE)
    JFLI_MIXED_SIZES(JFLI_CASE)
#undef JFLI_CASE
    default:
      break;
  }
  FftPlan pl;
  make_fft_plan(d.nz / 2, &pl);
  const int nrows = d.nx * d.ny;
  const int rows = z_rows_per_cta(d.nz);
  const int nh = d.nz / 2;
  const size_t smem = ((size_t)2 * (nh + 1) * (rows + 1) + nh + nh + 1) * sizeof(float2);
  dim3 grid((nrows + rows - 1) / rows, d.batch);
  cudaFuncSetAttribute(k_irfft_z, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_irfft_z<<<grid, kFftThreads, smem, s>>>(in, out, nrows, d.nz, rows, pl, scale, d.spec_elems(), d.cells());
  note_launch();
  return cudaGetLastError();
}

}  // namespace jfli
