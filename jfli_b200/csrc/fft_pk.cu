// x pass of the 3D FFT that feeds the P(k) histogram.
#include "cic.cuh"
#include "fft_engine.cuh"
#include "fft_passes.cuh"
#include "fft_reg.cuh"
#include "internal.h"

namespace jfli {

// Forward x pass feeding the P(k) histogram, for the remaining lengths (k_x_pk_reg).
__global__ void __launch_bounds__(kFftThreads) k_fft_x_pk(const float2* __restrict__ data, ColGeom g, FftPlan pl,
                                                          PkArgs a, long long bstride) {
  extern __shared__ float2 sm[];
  const int pitch = g.w | 1;
  float2* bufa = sm;
  float2* bufb = bufa + (size_t)g.n * pitch;
  float2* tw = bufb + (size_t)g.n * pitch;
  PkTile tile(a, tw + g.n);
  data += (long long)blockIdx.y * bstride;
  const int wl = fft_ilog2(g.w);
  fill_twiddles(tw, g.n);
  tile.clear(a);
  const int tiles = (g.ncols + g.w - 1) / g.w;
  const int E = g.n * g.w;
  for (int it = blockIdx.x; it < tiles; it += gridDim.x) {
    const int c0 = it * g.w;
    __syncthreads();
    tile.set_columns(a, c0, g.w, g.ncols, g.hz);
    for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
      const int e = idx >> wl, cc = idx & (g.w - 1);
      const int c = c0 + cc;
      bufa[e * pitch + cc] = (c < g.ncols) ? data[(long long)c + (long long)e * g.stride] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const float2* res = tile_fft<-1>(bufa, bufb, pitch, wl, pl, tw);
    tile.add(a, res, pitch, g.n, g.w);
  }
  __syncthreads();
  tile.store(a, blockIdx.y, blockIdx.x, gridDim.x);
}

// Forward x pass feeding the P(k) histogram (nothing is written back). A CTA takes tiles
// blockIdx.x, blockIdx.x + gridDim.x, ... and keeps one histogram over all of them, so the
// partials it leaves are a few hundred rows whatever the mesh. Between the transform and
// the binning the tile goes through shared memory once more, element-major with an odd
// pitch, because a thread walks neighbouring modes and the registers hold kx at stride Q.
// 512^3, 32 bins: 2.80 -> 0.38 ms beside 0.25 ms for the bare pass; the second kernel
// (spectra.cu) 0.95 -> 0.005 ms, as it reads 592 partials instead of 8224.
template <int N>
__global__ void __launch_bounds__(ColCfg<N>::T) k_x_pk_reg(const float2* __restrict__ data, ColGeom g,
                                                           const float2* __restrict__ twg, PkArgs a,
                                                           long long bstride) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, W = ColCfg<N>::W, T = ColCfg<N>::T, PW = W + 1;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* ybuf = sm + N;
  PkTile tile(a, ybuf + N * PW);
  data += (long long)blockIdx.y * bstride;
  const int tid = threadIdx.x;
  for (int m = tid; m < N; m += T) tw[m] = twg[m];
  tile.clear(a);
  const int tiles = (g.ncols + W - 1) / W;
  for (int it = blockIdx.x; it < tiles; it += gridDim.x) {
    const int c0 = it * W;
    __syncthreads();  // the tables are written, the previous tile is binned
    tile.set_columns(a, c0, W, g.ncols, g.hz);
    for (int w = tid; w < W * P; w += T) {
      const int c = w % W, t = w / W;
      const int col = c0 + c;
      float2 u[Q];
      if (col < g.ncols) {
        const float2* src = data + col + (long long)t * g.stride;
#pragma unroll
        for (int m = 0; m < Q; ++m) u[m] = src[(long long)(P * m) * g.stride];
      } else {
#pragma unroll
        for (int m = 0; m < Q; ++m) u[m] = make_float2(0.f, 0.f);
      }
      RegDFT<Q, -1, P>::run(u, tw);
#pragma unroll
      for (int kb = 0; kb < Q; ++kb)
        ybuf[(kb * P + t) * PW + c] = (kb == 0) ? u[0] : cmul(u[kb], twid<-1>(tw, t * kb));
    }
    __syncthreads();
    const int c = tid % W, kb = tid / W;
    float2 u[P];
#pragma unroll
    for (int t = 0; t < P; ++t) u[t] = ybuf[(kb * P + t) * PW + c];
    RegDFT<P, -1, Q>::run(u, tw);
    __syncthreads();
#pragma unroll
    for (int ka = 0; ka < P; ++ka) ybuf[(kb + Q * ka) * PW + c] = u[ka];
    __syncthreads();
    tile.add(a, ybuf, PW, N, W);
  }
  __syncthreads();
  tile.store(a, blockIdx.y, blockIdx.x, gridDim.x);
}

// CTAs of the P(k) x pass: enough tiles each that the histogram's set-up and the partials
// are small beside the transforms, few enough that all are resident at once.
constexpr int kPkCtasPerSm = 4;

static int pk_tiles(const MeshDims& d, int w) { return (x_geom(d).ncols + w - 1) / w; }
static int pk_cap(int tiles) {
  const int cap = kPkCtasPerSm * sm_count();
  return tiles < cap ? tiles : cap;
}

// (the workspace was sized by the tiles of the first list's lengths and of the shared-memory
// pass, which are at least as many as the partials now written)
int x_pass_ctas(const MeshDims& d) {
  const int w = reg_col_w(d.nx, true);
  return pk_tiles(d, w ? w : x_geom(d).w);
}
int pk_ctas(const MeshDims& d) {
  const int w = reg_col_w(d.nx);
  return pk_cap(pk_tiles(d, w ? w : x_geom(d).w));
}
int noalloc_x_pass_ctas(const MeshDims& d) { return pk_tiles(d, x_geom(d).w); }
int noalloc_pk_ctas(const MeshDims& d) { return pk_cap(pk_tiles(d, x_geom(d).w)); }

template <int N>
static cudaError_t x_pk_reg(const float2* data, const MeshDims& d, const PkArgs& a, cudaStream_t s) {
  constexpr int W = ColCfg<N>::W, T = ColCfg<N>::T;
  const float2* tw = twiddle_table(N);
  if (!tw) return cudaErrorMemoryAllocation;
  const size_t smem = ((size_t)N + (size_t)N * (W + 1)) * sizeof(float2) + pk_smem_bytes(a.nedges, W);
  cudaError_t e = cudaFuncSetAttribute(k_x_pk_reg<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_x_pk_reg<N><<<dim3(pk_ctas(d), d.batch), T, smem, s>>>(data, x_geom(d), tw, a, d.spec_elems());
  note_launch();
  return cudaGetLastError();
}

cudaError_t x_pk_generic(const float2* data, const MeshDims& d, const PkArgs& a, cudaStream_t s) {
  const ColGeom g = x_geom(d);
  FftPlan pl;
  make_fft_plan(g.n, &pl);
  const size_t smem = ((size_t)2 * g.n * (g.w | 1) + g.n) * sizeof(float2) +
                      pk_smem_bytes(a.nedges, g.w);
  cudaError_t e = cudaFuncSetAttribute(k_fft_x_pk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_fft_x_pk<<<dim3(noalloc_pk_ctas(d), d.batch), kFftThreads, smem, s>>>(data, g, pl, a, d.spec_elems());
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_x_pk(const float2* data, const MeshDims& d, const PkArgs& a, cudaStream_t s) {
  switch (d.nx) {
#define JFLI_CASE(N_) \
  case N_:            \
    return x_pk_reg<N_>(data, d, a, s);
    JFLI_REG_SIZES(JFLI_CASE)
    JFLI_MIXED_SIZES(JFLI_CASE)
#undef JFLI_CASE
    default:
      return x_pk_generic(data, d, a, s);
  }
}

}  // namespace jfli
