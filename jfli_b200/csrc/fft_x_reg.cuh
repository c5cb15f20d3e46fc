// Register-resident x pass with a k-space operator (fft_x.cu and fft_x_mixed.cu): forward x FFT,
// operator, inverse x FFT in one read and one write of the half spectrum.
#pragma once

#include "fft_passes.cuh"

namespace jfli {

template <int N, class Op>
__global__ void __launch_bounds__(ColCfg<N>::T) k_x_op_reg(float2* __restrict__ data, ColGeom g,
                                                           const float2* __restrict__ twg, Op op, long long bstride) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, W = ColCfg<N>::W, T = ColCfg<N>::T;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* ybuf = sm + N;
  float* opsm = reinterpret_cast<float*>(ybuf + N * W);
  const int batch = blockIdx.y;
  data += (long long)batch * bstride;
  const int tid = threadIdx.x;
  grid_wait();
  for (int m = tid; m < N; m += T) tw[m] = twg[m];
  op.prologue(opsm, batch);  // ends with __syncthreads()
  const int c0 = blockIdx.x * W;
  // forward stage 1
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
      ybuf[(kb * P + t) * W + c] = (kb == 0) ? u[0] : cmul(u[kb], twid<-1>(tw, t * kb));
  }
  __syncthreads();
  // forward stage 2: this thread holds X[kb + Q ka], ka < P
  const int c = tid % W, kb = tid / W;
  const int col = c0 + c;
  float2 u[P];
#pragma unroll
  for (int t = 0; t < P; ++t) u[t] = ybuf[(kb * P + t) * W + c];
  RegDFT<P, -1, Q>::run(u, tw);
  if (col < g.ncols) {
    const int ky = col / g.hz;
    const int kz = col - ky * g.hz;
#pragma unroll
    for (int ka = 0; ka < P; ++ka) u[ka] = op.apply(u[ka], kb + Q * ka, ky, kz, opsm, batch);
  }
  __syncthreads();
  // inverse stage 1': t' = kb holds x'[t' + Q m'] = u[m'], m' < P
  RegDFT<P, 1, Q>::run(u, tw);
#pragma unroll
  for (int k1 = 0; k1 < P; ++k1) ybuf[(k1 * Q + kb) * W + c] = (k1 == 0) ? u[0] : cmul(u[k1], twid<1>(tw, kb * k1));
  __syncthreads();
  grid_release();
  // inverse stage 2': items (c, k1), k1 < P
  for (int w = tid; w < W * P; w += T) {
    const int cc = w % W, k1 = w / W;
    const int col2 = c0 + cc;
    float2 v[Q];
#pragma unroll
    for (int t = 0; t < Q; ++t) v[t] = ybuf[(k1 * Q + t) * W + cc];
    RegDFT<Q, 1, P>::run(v, tw);
    if (col2 < g.ncols) {
      float2* dst = data + col2 + (long long)k1 * g.stride;
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) dst[(long long)(P * k2) * g.stride] = v[k2];
    }
  }
}

template <int N, class Op>
static cudaError_t x_op_reg(float2* data, const ColGeom& g, const Op& op, long long bstride, int batch,
                            cudaStream_t s) {
  constexpr int W = ColCfg<N>::W, T = ColCfg<N>::T;
  const float2* tw = twiddle_table(N);
  if (!tw) return cudaErrorMemoryAllocation;
  const size_t smem = ((size_t)N + (size_t)N * W) * sizeof(float2) + Op::smem_bytes(op);
  cudaFuncSetAttribute(k_x_op_reg<N, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_next(overlap_starts(2 * bstride * batch), k_x_op_reg<N, Op>, dim3((g.ncols + W - 1) / W, batch), T, smem, s,
              data, g, tw, op, bstride);
  note_launch();
  return cudaGetLastError();
}

}  // namespace jfli
