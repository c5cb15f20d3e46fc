// The z and y passes of small square planes (ny = nz = 32 to 144) in one kernel, one CTA per x
// plane: forward r2c along z and the transform along y, inverse y and c2r along z. The plane's half
// spectrum (5 to 101 KB) stays in shared memory between them, so it is written, or read, once
// where two passes move it three times, and a Poisson solve has three kernels in place of five.
// Each transform is the one of the separate passes (same splits, same tables, same order), and
// so are the bits.
//
// One such mesh is in L2 and its passes are bound by the latency of a kernel that starts,
// loads, exchanges and stores; a batch of them by bandwidth. Poisson solve, two passes -> one,
// of 1 and 16 meshes: 32^3 12.4 -> 7.5 us and 24.7 -> 14.9, 64^3 18.3 -> 13.4 and 42.8 -> 33.3, 96^3
// 29.5 -> 27.5 and 134 -> 113, 128^3 36.9 -> 28.9 and 284 -> 266. Larger planes (192^2: 184 KB)
// leave one CTA per SM and more planes than SMs, and oblong ones would need a kernel per pair
// of lengths.
#include "fft_passes.cuh"

namespace jfli {

template <int NY>
struct PlaneCfg {
  static constexpr int N = NY / 2, HZ = N + 1;
  static constexpr int PZ = Split<N>::P, QZ = Split<N>::Q, PY = Split<NY>::P, QY = Split<NY>::Q;
  static constexpr int T = NY <= 64 ? 8 * NY : 4 * NY;
  static_assert(T % PZ == 0 && T % QZ == 0, "a row's threads work in the same turn");
  // rows of the tile: QZ mod 16 entries apart, so that neither exchange along z has bank conflicts
  static constexpr int mod16(int least) { return least + ((QZ - least) % 16 + 16) % 16; }
  static constexpr int YS = QZ | 1;
  static constexpr int RS = mod16(PZ * YS > HZ ? PZ * YS : HZ);
  static constexpr size_t smem = sizeof(float2) * ((size_t)NY * RS + N + HZ + NY);
};

template <int NY>
struct PlaneSmem {
  float2 *tile, *twz, *tw2, *twy;
  __device__ __forceinline__ PlaneSmem(float2* sm, const float2* __restrict__ twzg, const float2* __restrict__ tw2g,
                                       const float2* __restrict__ twyg) {
    using C = PlaneCfg<NY>;
    tile = sm;
    twz = tile + NY * C::RS;
    tw2 = twz + C::N;
    twy = tw2 + C::HZ;
    for (int m = threadIdx.x; m < C::N; m += C::T) twz[m] = twzg[m];
    for (int m = threadIdx.x; m < C::HZ; m += C::T) tw2[m] = tw2g[m];
    for (int m = threadIdx.x; m < NY; m += C::T) twy[m] = twyg[m];
  }
};

template <int NY>
__global__ void __launch_bounds__(PlaneCfg<NY>::T) k_planes_forward(const float* in, float2* __restrict__ out, float sub,
                                                                    const float2* __restrict__ twzg,
                                                                    const float2* __restrict__ tw2g,
                                                                    const float2* __restrict__ twyg, long long in_b,
                                                                    long long out_b, float* clear) {
  using C = PlaneCfg<NY>;
  constexpr int N = C::N, HZ = C::HZ, PZ = C::PZ, QZ = C::QZ, PY = C::PY, QY = C::QY, T = C::T, RS = C::RS, YS = C::YS;
  extern __shared__ float2 sm[];
  grid_wait();
  const PlaneSmem<NY> s(sm, twzg, tw2g, twyg);
  float2* tile = s.tile;
  const int tid = threadIdx.x;
  const long long plane = blockIdx.y * in_b + (long long)blockIdx.x * NY * NY;
  const float2* in2 = reinterpret_cast<const float2*>(in + plane);
  float2* clear2 = clear ? reinterpret_cast<float2*>(clear + plane) : nullptr;
  out += blockIdx.y * out_b + (long long)blockIdx.x * NY * HZ;
  __syncthreads();
  // z, stage 1
  for (int w = tid; w < NY * PZ; w += T) {
    const int t = w % PZ, r = w / PZ;
    float2 u[QZ];
#pragma unroll
    for (int m = 0; m < QZ; ++m) {
      const float2 v = in2[r * N + t + PZ * m];
      u[m] = make_float2(v.x - sub, v.y - sub);
    }
    if (clear2) {
#pragma unroll
      for (int m = 0; m < QZ; ++m) clear2[r * N + t + PZ * m] = make_float2(0.f, 0.f);
    }
    RegDFT<QZ, -1, PZ>::run(u, s.twz);
#pragma unroll
    for (int kb = 0; kb < QZ; ++kb)
      tile[r * RS + t * YS + kb] = (kb == 0) ? u[0] : cmul(u[kb], twid<-1>(s.twz, t * kb));
  }
  __syncthreads();
  // z, stage 2, in place: the rows of one turn are read before they are written
  for (int w0 = 0; w0 < NY * QZ; w0 += T) {
    const int w = w0 + tid, kb = w % QZ, r = w / QZ;
    const bool on = w < NY * QZ;
    float2 u[PZ];
    if (on) {
#pragma unroll
      for (int t = 0; t < PZ; ++t) u[t] = tile[r * RS + t * YS + kb];
      RegDFT<PZ, -1, QZ>::run(u, s.twz);
    }
    __syncthreads();
    if (on) {
#pragma unroll
      for (int ka = 0; ka < PZ; ++ka) tile[r * RS + kb + QZ * ka] = u[ka];
    }
  }
  __syncthreads();
  // half spectrum of the packed rows, in place: a thread owns the pair (k, N - k)
  const auto untangle = [](float2 zk, float2 zm, float2 w) {
    const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    const float2 d = make_float2(zk.x - zm.x, zk.y + zm.y);
    const float2 o = make_float2(0.5f * d.y, -0.5f * d.x);
    return cadd(e, cmul(w, o));
  };
  constexpr int H = N / 2 + 1;
  for (int w = tid; w < NY * H; w += T) {
    const int r = w / H, k = w - r * H;
    float2* row = tile + r * RS;
    const float2 zk = row[k], zm = row[k == 0 ? 0 : N - k];
    row[k] = untangle(zk, zm, s.tw2[k]);
    if (2 * k != N) row[N - k] = untangle(zm, zk, s.tw2[N - k]);
  }
  __syncthreads();
  // y, stage 1, in place
  constexpr int IT = (HZ * PY + T - 1) / T;
  float2 v[IT][QY];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int w = tid + it * T;
    if (w >= HZ * PY) continue;
    const int c = w % HZ, t = w / HZ;
#pragma unroll
    for (int m = 0; m < QY; ++m) v[it][m] = tile[(t + PY * m) * RS + c];
    RegDFT<QY, -1, PY>::run(v[it], s.twy);
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int w = tid + it * T;
    if (w >= HZ * PY) continue;
    const int c = w % HZ, t = w / HZ;
#pragma unroll
    for (int kb = 0; kb < QY; ++kb)
      tile[(kb * PY + t) * RS + c] = (kb == 0) ? v[it][0] : cmul(v[it][kb], twid<-1>(s.twy, t * kb));
  }
  __syncthreads();
  grid_release();
  // y, stage 2, to memory
  for (int w = tid; w < HZ * QY; w += T) {
    const int c = w % HZ, kb = w / HZ;
    float2 u[PY];
#pragma unroll
    for (int t = 0; t < PY; ++t) u[t] = tile[(kb * PY + t) * RS + c];
    RegDFT<PY, -1, QY>::run(u, s.twy);
#pragma unroll
    for (int ka = 0; ka < PY; ++ka) out[(kb + QY * ka) * HZ + c] = u[ka];
  }
}

template <int NY>
__global__ void __launch_bounds__(PlaneCfg<NY>::T) k_planes_inverse(const float2* __restrict__ in,
                                                                    float* __restrict__ out, float scale,
                                                                    const float2* __restrict__ twzg,
                                                                    const float2* __restrict__ tw2g,
                                                                    const float2* __restrict__ twyg, long long in_b,
                                                                    long long out_b) {
  using C = PlaneCfg<NY>;
  constexpr int N = C::N, HZ = C::HZ, PZ = C::PZ, QZ = C::QZ, PY = C::PY, QY = C::QY, T = C::T, RS = C::RS, YS = C::YS;
  extern __shared__ float2 sm[];
  grid_wait();
  const PlaneSmem<NY> s(sm, twzg, tw2g, twyg);
  float2* tile = s.tile;
  const int tid = threadIdx.x;
  in += blockIdx.y * in_b + (long long)blockIdx.x * NY * HZ;
  float2* out2 = reinterpret_cast<float2*>(out + blockIdx.y * out_b + (long long)blockIdx.x * NY * NY);
  __syncthreads();
  // y, stage 1, from memory
  for (int w = tid; w < HZ * PY; w += T) {
    const int c = w % HZ, t = w / HZ;
    float2 u[QY];
#pragma unroll
    for (int m = 0; m < QY; ++m) u[m] = in[(t + PY * m) * HZ + c];
    RegDFT<QY, 1, PY>::run(u, s.twy);
#pragma unroll
    for (int kb = 0; kb < QY; ++kb)
      tile[(kb * PY + t) * RS + c] = (kb == 0) ? u[0] : cmul(u[kb], twid<1>(s.twy, t * kb));
  }
  __syncthreads();
  // y, stage 2, in place
  constexpr int IT = (HZ * QY + T - 1) / T;
  float2 v[IT][PY];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int w = tid + it * T;
    if (w >= HZ * QY) continue;
    const int c = w % HZ, kb = w / HZ;
#pragma unroll
    for (int t = 0; t < PY; ++t) v[it][t] = tile[(kb * PY + t) * RS + c];
    RegDFT<PY, 1, QY>::run(v[it], s.twy);
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int w = tid + it * T;
    if (w >= HZ * QY) continue;
    const int c = w % HZ, kb = w / HZ;
#pragma unroll
    for (int ka = 0; ka < PY; ++ka) tile[(kb + QY * ka) * RS + c] = v[it][ka];
  }
  __syncthreads();
  // z: packed rows and stage 1, in place
  for (int w0 = 0; w0 < NY * PZ; w0 += T) {
    const int w = w0 + tid, t = w % PZ, r = w / PZ;
    const bool on = w < NY * PZ;
    float2 u[QZ];
    if (on) {
#pragma unroll
      for (int m = 0; m < QZ; ++m) {
        const int e = t + PZ * m;
        const float2 xk = tile[r * RS + e], xm = tile[r * RS + N - e];
        const float2 ee = make_float2(xk.x + xm.x, xk.y - xm.y);
        const float2 dd = cmul(make_float2(xk.x - xm.x, xk.y + xm.y), conjf2(s.tw2[e]));
        u[m] = make_float2(ee.x - dd.y, ee.y + dd.x);
      }
      RegDFT<QZ, 1, PZ>::run(u, s.twz);
    }
    __syncthreads();
    if (on) {
#pragma unroll
      for (int kb = 0; kb < QZ; ++kb)
        tile[r * RS + t * YS + kb] = (kb == 0) ? u[0] : cmul(u[kb], twid<1>(s.twz, t * kb));
    }
  }
  __syncthreads();
  grid_release();
  // z, stage 2, to memory
  for (int w = tid; w < NY * QZ; w += T) {
    const int kb = w % QZ, r = w / QZ;
    float2 u[PZ];
#pragma unroll
    for (int t = 0; t < PZ; ++t) u[t] = tile[r * RS + t * YS + kb];
    RegDFT<PZ, 1, QZ>::run(u, s.twz);
#pragma unroll
    for (int ka = 0; ka < PZ; ++ka) out2[r * N + kb + QZ * ka] = cscale(u[ka], scale);
  }
}

template <int NY>
static cudaError_t planes_forward(const float* in, float2* out, const MeshDims& d, float sub, cudaStream_t s,
                                  float* clear) {
  const float2 *twz = twiddle_table(NY / 2), *tw = twiddle_table(NY);
  if (!twz || !tw) return cudaErrorMemoryAllocation;
  cudaError_t e = cudaFuncSetAttribute(k_planes_forward<NY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)PlaneCfg<NY>::smem);
  if (e != cudaSuccess) return e;
  launch_next(overlap_starts(d.cells() * d.batch), k_planes_forward<NY>, dim3(d.nx, d.batch), PlaneCfg<NY>::T,
              PlaneCfg<NY>::smem, s, in, out, sub, twz, tw, tw, d.cells(), d.spec_elems(), clear);
  note_launch();
  return cudaGetLastError();
}

template <int NY>
static cudaError_t planes_inverse(const float2* in, float* out, const MeshDims& d, float scale, cudaStream_t s) {
  const float2 *twz = twiddle_table(NY / 2), *tw = twiddle_table(NY);
  if (!twz || !tw) return cudaErrorMemoryAllocation;
  cudaError_t e = cudaFuncSetAttribute(k_planes_inverse<NY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)PlaneCfg<NY>::smem);
  if (e != cudaSuccess) return e;
  launch_next(overlap_starts(d.cells() * d.batch), k_planes_inverse<NY>, dim3(d.nx, d.batch), PlaneCfg<NY>::T,
              PlaneCfg<NY>::smem, s, in, out, scale, twz, tw, tw, d.spec_elems(), d.cells());
  note_launch();
  return cudaGetLastError();
}

#define JFLI_PLANE_SIZES(X) X(32) X(48) X(64) X(96) X(128)
#define JFLI_MIXED_PLANE_SIZES(X) X(36) X(54) X(72) X(108) X(144)

cudaError_t launch_forward_zy(const float* in, float2* spec, const MeshDims& d, float sub, cudaStream_t s, float* clear,
                              bool mixed) {
  if (d.ny == d.nz) {
    switch (reg_fft_length(d.ny, mixed)) {
#define JFLI_CASE(N_) \
  case N_:            \
    return planes_forward<N_>(in, spec, d, sub, s, clear);
      JFLI_PLANE_SIZES(JFLI_CASE)
      JFLI_MIXED_PLANE_SIZES(JFLI_CASE)
#undef JFLI_CASE
      default:
        break;
    }
  }
  const cudaError_t e = launch_rfft_z(in, spec, d, sub, s, clear, mixed);
  return e != cudaSuccess ? e : launch_cols(-1, spec, y_geom(d), d.spec_elems(), d.batch, s, mixed);
}

cudaError_t launch_inverse_yz(float2* spec, float* out, const MeshDims& d, float scale, cudaStream_t s, bool mixed) {
  if (d.ny == d.nz) {
    switch (reg_fft_length(d.ny, mixed)) {
#define JFLI_CASE(N_) \
  case N_:            \
    return planes_inverse<N_>(spec, out, d, scale, s);
      JFLI_PLANE_SIZES(JFLI_CASE)
      JFLI_MIXED_PLANE_SIZES(JFLI_CASE)
#undef JFLI_CASE
      default:
        break;
    }
  }
  const cudaError_t e = launch_cols(1, spec, y_geom(d), d.spec_elems(), d.batch, s, mixed);
  return e != cudaSuccess ? e : launch_irfft_z(spec, out, d, scale, s, mixed);
}

}  // namespace jfli
