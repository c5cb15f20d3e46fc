// Complex column passes of the 3D FFT (along y, and along x without an operator).
#include "fft_engine.cuh"
#include "fft_passes.cuh"
#include "fft_reg.cuh"
#include "internal.h"

namespace jfli {

// ---------------------------------------------------------------------------------
// Column pass (used for y, and for x without an operator).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ long long col_addr(const ColGeom& g, int c, int e) {
  const int o = c / g.hz;
  return (long long)o * g.outer_stride + (c - o * g.hz) + (long long)e * g.stride;
}

template <int SIGN>
__global__ void __launch_bounds__(kFftThreads) k_fft_cols(float2* __restrict__ data, ColGeom g, FftPlan pl,
                                                          long long bstride) {
  extern __shared__ float2 sm[];
  float2* bufa = sm;
  float2* bufb = bufa + (size_t)g.n * g.w;
  float2* tw = bufb + (size_t)g.n * g.w;
  data += (long long)blockIdx.y * bstride;
  const int c0 = blockIdx.x * g.w;
  const int wl = fft_ilog2(g.w);
  fill_twiddles(tw, g.n);
  const int E = g.n * g.w;
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int e = idx >> wl;
    const int c = c0 + (idx & (g.w - 1));
    bufa[idx] = (c < g.ncols) ? data[col_addr(g, c, e)] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const float2* res = tile_fft<SIGN>(bufa, bufb, g.w, wl, pl, tw);
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int e = idx >> wl;
    const int c = c0 + (idx & (g.w - 1));
    if (c < g.ncols) data[col_addr(g, c, e)] = res[idx];
  }
}

__device__ __forceinline__ long long col_base(const ColGeom& g, int c) {
  const int o = c / g.hz;
  return (long long)o * g.outer_stride + (c - o * g.hz);
}

template <int N, int SIGN>
__global__ void __launch_bounds__(ColCfg<N>::T) k_cols_reg(float2* __restrict__ data, ColGeom g,
                                                           const float2* __restrict__ twg, long long bstride) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, W = ColCfg<N>::W, T = ColCfg<N>::T;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* ybuf = sm + N;
  data += (long long)blockIdx.y * bstride;
  const int tid = threadIdx.x;
  grid_wait();
  for (int m = tid; m < N; m += T) tw[m] = twg[m];
  __syncthreads();
  const int c0 = blockIdx.x * W;
  for (int w = tid; w < W * P; w += T) {
    const int c = w % W, t = w / W;
    const int col = c0 + c;
    float2 u[Q];
    if (col < g.ncols) {
      const float2* src = data + col_base(g, col) + (long long)t * g.stride;
#pragma unroll
      for (int m = 0; m < Q; ++m) u[m] = src[(long long)(P * m) * g.stride];
    } else {
#pragma unroll
      for (int m = 0; m < Q; ++m) u[m] = make_float2(0.f, 0.f);
    }
    RegDFT<Q, SIGN, P>::run(u, tw);
#pragma unroll
    for (int kb = 0; kb < Q; ++kb)
      ybuf[(kb * P + t) * W + c] = (kb == 0) ? u[0] : cmul(u[kb], twid<SIGN>(tw, t * kb));
  }
  __syncthreads();
  grid_release();
  const int c = tid % W, kb = tid / W;
  float2 u[P];
#pragma unroll
  for (int t = 0; t < P; ++t) u[t] = ybuf[(kb * P + t) * W + c];
  RegDFT<P, SIGN, Q>::run(u, tw);
  const int col = c0 + c;
  if (col < g.ncols) {
    float2* dst = data + col_base(g, col) + (long long)kb * g.stride;
#pragma unroll
    for (int ka = 0; ka < P; ++ka) dst[(long long)(Q * ka) * g.stride] = u[ka];
  }
}

template <int N, int SIGN>
static cudaError_t cols_reg(float2* data, const ColGeom& g, long long bstride, int batch, cudaStream_t s) {
  constexpr int W = ColCfg<N>::W, T = ColCfg<N>::T;
  const float2* tw = twiddle_table(N);
  if (!tw) return cudaErrorMemoryAllocation;
  const size_t smem = ((size_t)N + (size_t)N * W) * sizeof(float2);
  cudaFuncSetAttribute(k_cols_reg<N, SIGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_next(overlap_starts(2 * bstride * batch), k_cols_reg<N, SIGN>, dim3((g.ncols + W - 1) / W, batch), T, smem, s,
              data, g, tw, bstride);
  note_launch();
  return cudaGetLastError();
}

template <int SIGN>
static cudaError_t cols_generic_sign(float2* data, const ColGeom& g, long long bstride, int batch, cudaStream_t s) {
  FftPlan pl;
  make_fft_plan(g.n, &pl);
  const size_t smem = ((size_t)2 * g.n * g.w + g.n) * sizeof(float2);
  dim3 grid((g.ncols + g.w - 1) / g.w, batch);
  cudaFuncSetAttribute(k_fft_cols<SIGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_fft_cols<SIGN><<<grid, kFftThreads, smem, s>>>(data, g, pl, bstride);
  note_launch();
  return cudaGetLastError();
}

template <int SIGN>
static cudaError_t cols_sign(float2* data, const ColGeom& g, long long bstride, int batch, cudaStream_t s, bool mixed) {
  switch (reg_fft_length(g.n, mixed)) {
#define JFLI_CASE(N_) \
  case N_:            \
    return cols_reg<N_, SIGN>(data, g, bstride, batch, s);
    JFLI_REG_SIZES(JFLI_CASE)
    JFLI_MIXED_SIZES(JFLI_CASE)
#undef JFLI_CASE
    default:
      break;
  }
  return cols_generic_sign<SIGN>(data, g, bstride, batch, s);
}

cudaError_t launch_cols(int sign, float2* data, const ColGeom& g, long long bstride, int batch, cudaStream_t s,
                        bool mixed) {
  return sign < 0 ? cols_sign<-1>(data, g, bstride, batch, s, mixed) : cols_sign<1>(data, g, bstride, batch, s, mixed);
}

cudaError_t cols_generic(int sign, float2* data, const ColGeom& g, long long bstride, int batch, cudaStream_t s) {
  return sign < 0 ? cols_generic_sign<-1>(data, g, bstride, batch, s) : cols_generic_sign<1>(data, g, bstride, batch, s);
}

}  // namespace jfli
