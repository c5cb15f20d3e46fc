// x pass of the 3D FFT with a k-space operator: TMA-staged, register and shared-memory forms.
#include <atomic>
#include <type_traits>

#include "fft_engine.cuh"
#include "fft_passes.cuh"
#include "fft_tma.cuh"
#include "fft_x_reg.cuh"
#include "internal.h"

namespace jfli {

// ---------------------------------------------------------------------------------
// x pass with a k-space operator. Columns are (ky, kz) pairs, c = ky*hz + kz, and the
// transform runs over kx with stride ny*hz. Op is applied between the forward and the
// inverse transform.
// ---------------------------------------------------------------------------------
template <class Op>
__global__ void __launch_bounds__(kFftThreads) k_fft_x_op(float2* __restrict__ data, ColGeom g, FftPlan pl, Op op,
                                                          long long bstride) {
  extern __shared__ float2 sm[];
  float2* bufa = sm;
  float2* bufb = bufa + (size_t)g.n * g.w;
  float2* tw = bufb + (size_t)g.n * g.w;
  float* opsm = reinterpret_cast<float*>(tw + g.n);
  const int batch = blockIdx.y;
  data += (long long)batch * bstride;
  const int c0 = blockIdx.x * g.w;
  const int wl = fft_ilog2(g.w);
  fill_twiddles(tw, g.n);
  op.prologue(opsm, batch);
  const int E = g.n * g.w;
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int e = idx >> wl;
    const int c = c0 + (idx & (g.w - 1));
    bufa[idx] = (c < g.ncols) ? data[(long long)c + (long long)e * g.stride] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2* res = tile_fft<-1>(bufa, bufb, g.w, wl, pl, tw);
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int e = idx >> wl;
    const int c = c0 + (idx & (g.w - 1));
    if (c < g.ncols) {
      const int ky = c / g.hz;
      res[idx] = op.apply(res[idx], e, ky, c - ky * g.hz, opsm, batch);
    }
  }
  __syncthreads();
  res = tile_fft<1>(res, res == bufa ? bufb : bufa, g.w, wl, pl, tw);
  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    const int e = idx >> wl;
    const int c = c0 + (idx & (g.w - 1));
    if (c < g.ncols) data[(long long)c + (long long)e * g.stride] = res[idx];
  }
}

// ---- TMA-staged x pass
static std::atomic<int> g_x_pass_mode{1};  // 0 register pass, 1 TMA-staged pass (default)

void set_x_pass_mode(int mode) { g_x_pass_mode.store(mode); }
int x_pass_mode() { return g_x_pass_mode.load(); }

cudaError_t device_status(unsigned* out, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_jfli_status, sizeof(unsigned));
  if (e == cudaSuccess && reset) {
    const unsigned zero = 0;
    e = cudaMemcpyToSymbol(g_jfli_status, &zero, sizeof(unsigned));
  }
  return e;
}

bool x_pass_tensor_map(CUtensorMap* map, const float2* spec, const MeshDims& d, int w) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode encode = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Encode>(f);
  }();
  if (encode == nullptr || ((uintptr_t)spec % 16) != 0) return false;
  const cuuint64_t inner = 2ull * (cuuint64_t)d.ny * (cuuint64_t)d.hz();  // floats of one x plane
  const cuuint64_t plane_bytes = inner * sizeof(float);
  const cuuint64_t batch_bytes = (cuuint64_t)d.spec_elems() * sizeof(float2);
  if (plane_bytes % 16 != 0 || batch_bytes % 16 != 0 || (2 * w * sizeof(float)) % 16 != 0) return false;
  const cuuint64_t dims[3] = {inner, (cuuint64_t)d.nx, (cuuint64_t)d.batch};
  const cuuint64_t strides[2] = {plane_bytes, batch_bytes};
  const cuuint32_t box[3] = {(cuuint32_t)(2 * w), (cuuint32_t)(d.nx > kTmaBoxRows ? kTmaBoxRows : d.nx), 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float2*>(spec), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int N, class Op>
static cudaError_t x_op_tma(float2* data, const MeshDims& d, const Op& op, bool* done, cudaStream_t s) {
  *done = false;
  constexpr int W = ColCfg<N>::W, T = ColCfg<N>::T;
  if (N % TmaCfg<N>::ROWS != 0) return cudaSuccess;
  CUtensorMap map;
  if (!x_pass_tensor_map(&map, data, d, W)) return cudaSuccess;
  const float2* tw = twiddle_table(N);
  if (!tw) return cudaErrorMemoryAllocation;
  const ColGeom g = x_geom(d);
  const size_t smem = TmaCfg<N>::tile_bytes * 2 + sizeof(float2) * (size_t)N + Op::smem_bytes(op);
  cudaError_t e = cudaFuncSetAttribute(k_x_op_tma<N, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  launch_next(overlap_starts(d.cells() * d.batch), k_x_op_tma<N, Op>, dim3((g.ncols + W - 1) / W, d.batch), T, smem, s,
              map, g, tw, op);
  note_launch();
  *done = true;
  return cudaGetLastError();
}

template <class Op>
static cudaError_t x_op(float2* data, const MeshDims& d, const Op& op, cudaStream_t s, bool mixed) {
  const ColGeom g = x_geom(d);
  if (x_pass_mode() == 1) {
    bool done = false;
    cudaError_t e = cudaSuccess;
    switch (g.n) {
#define JFLI_CASE(N_)                            \
  case N_:                                       \
    e = x_op_tma<N_, Op>(data, d, op, &done, s); \
    break;
      JFLI_REG_SIZES(JFLI_CASE)
#undef JFLI_CASE
      default:
        break;
    }
    if (e != cudaSuccess || done) return e;
  }
  switch (g.n) {
#define JFLI_CASE(N_) \
  case N_:            \
    return x_op_reg<N_, Op>(data, g, op, d.spec_elems(), d.batch, s);
    JFLI_REG_SIZES(JFLI_CASE)
#undef JFLI_CASE
    default:
      break;
  }
  if constexpr (std::is_same_v<Op, PoissonOp>) {
    if (mixed) {
      bool done = false;
      const cudaError_t e = launch_x_op_mixed(data, d, op, &done, s);
      if (done || e != cudaSuccess) return e;
    }
  }
  FftPlan pl;
  make_fft_plan(g.n, &pl);
  const size_t smem = ((size_t)2 * g.n * g.w + g.n) * sizeof(float2) + Op::smem_bytes(op);
  dim3 grid((g.ncols + g.w - 1) / g.w, d.batch);
  cudaFuncSetAttribute(k_fft_x_op<Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_fft_x_op<Op><<<grid, kFftThreads, smem, s>>>(data, g, pl, op, d.spec_elems());
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_x_op(float2* data, const MeshDims& d, const PoissonOp& op, cudaStream_t s, bool mixed) {
  return x_op(data, d, op, s, mixed);
}
cudaError_t launch_x_op(float2* data, const MeshDims& d, const PgdOp& op, cudaStream_t s, bool mixed) {
  return x_op(data, d, op, s, mixed);
}
cudaError_t launch_x_op(float2* data, const MeshDims& d, const IcOp& op, cudaStream_t s, bool mixed) {
  return x_op(data, d, op, s, mixed);
}
cudaError_t launch_x_op(float2* data, const MeshDims& d, const PkAdjOp& op, cudaStream_t s, bool mixed) {
  return x_op(data, d, op, s, mixed);
}

}  // namespace jfli
