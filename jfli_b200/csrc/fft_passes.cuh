// Shared by the files of the 3D FFT (fft.cu and fft_*.cu): the sizes with register kernels,
// the geometry of the column passes, and the launchers each file provides.
#pragma once

#include "common.cuh"
#include "fft_reg.cuh"
#include "internal.h"
#include "kspace_ops.cuh"

namespace jfli {

// Lengths with register kernels. The first list also has the TMA-staged x pass and every
// k-space operator; the second, the remaining 2^a 3^b lengths of common meshes (any even mesh
// axis 2^a 3^b from 32 to 768, and half of it), has the register column, row, Poisson,
// and P(k) passes (fft_x_mixed.cu), and takes the shared-memory Stockham pass for the other
// operators. The Stockham passes go through shared memory once per radix and build their
// twiddles with FP64 sincospi in every CTA: the five passes of a 216 x 144 x 324 Poisson solve
// took 345 us with them and take 115 with registers.
#define JFLI_REG_SIZES(X) \
  X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512) X(768) X(1024)
#define JFLI_MIXED_SIZES(X)                                                                                \
  X(18) X(27) X(36) X(54) X(72) X(81) X(108) X(144) X(162) X(216) X(243) X(288) X(324) X(432) X(486) X(576) \
      X(648)

inline __host__ __device__ int pow2_floor(int v) {
  int p = 1;
  while (p * 2 <= v) p *= 2;
  return p;
}
inline int z_rows_per_cta(int nz) { return pow2_floor(kFftTileElems / (nz / 2)); }
inline int col_tile_width(int n) {
  int w = kFftTileElems / n;
  if (w > 16) w = 16;
  return w < 1 ? 1 : pow2_floor(w);
}

inline ColGeom y_geom(const MeshDims& d) {
  ColGeom g;
  g.n = d.ny;
  g.hz = d.hz();
  g.ncols = d.nx * g.hz;
  g.w = col_tile_width(g.n);
  g.stride = g.hz;
  g.outer_stride = (long long)d.ny * g.hz;
  return g;
}

inline ColGeom x_geom(const MeshDims& d) {
  ColGeom g;
  g.n = d.nx;
  g.hz = d.hz();
  g.ncols = d.ny * g.hz;
  g.w = col_tile_width(g.n);
  g.stride = (long long)d.ny * g.hz;
  g.outer_stride = g.hz;
  return g;
}

// Columns per tile of the register x pass of length n (0: no register kernels); `first`: the
// first list alone.
inline int reg_col_w(int n, bool first = false) {
  switch (n) {
#define JFLI_CASE(N_) \
  case N_:            \
    return ColCfg<N_>::W;
    JFLI_REG_SIZES(JFLI_CASE)
#undef JFLI_CASE
#define JFLI_CASE(N_) \
  case N_:            \
    return first ? 0 : ColCfg<N_>::W;
    JFLI_MIXED_SIZES(JFLI_CASE)
#undef JFLI_CASE
    default:
      return 0;
  }
}

// The length a launcher looks up its register kernels by: with `mixed` false the second list
// counts as unsupported (-1), so that those axes take the Stockham pass. The initial-condition
// filter and the LPT solves ask for that. Their results place every particle near a grid point,
// on one side or the other of a CIC cell face, where the derivative of the force jumps, and the
// two kinds of pass round differently (3e-7 of the field): with the mixed lengths in them the
// gradient of a 108^3 or 144^3 run through 12 to 20 steps moves by 5e-5 to 4e-4 of its norm, where
// repeats of one build differ by 2e-6 to 7e-5 (atomics). In the solves of the steps and of the
// reverse sweep, where the atomics reorder the density anyway, it moves by no more than that.
// The LPT adjoint places no particle and takes the register passes (its phi1 then rounds apart from
// the forward call's, 3e-7).
inline int reg_fft_length(int n, bool mixed) {
  if (mixed) return n;
  switch (n) {
#define JFLI_CASE(N_) case N_:
    JFLI_MIXED_SIZES(JFLI_CASE)
#undef JFLI_CASE
    return -1;
    default:
      return n;
  }
}

__device__ __forceinline__ int fft_ilog2(int v) { return 31 - __clz(v); }

// ---- fft.cu
bool make_fft_plan(int n, FftPlan* p);
const float2* twiddle_table(int n);
// ---- fft_z.cu. `clear`: the input mesh, set to 0 once it has been read (nullptr: left as it is);
// `mixed`: see reg_fft_length
cudaError_t launch_rfft_z(const float* in, float2* out, const MeshDims& d, float sub, cudaStream_t s,
                          float* clear = nullptr, bool mixed = true);
cudaError_t launch_irfft_z(const float2* in, float* out, const MeshDims& d, float scale, cudaStream_t s,
                           bool mixed = true);
// the shared-memory r2c pass, which needs no table
cudaError_t rfft_z_generic(const float* in, float2* out, const MeshDims& d, float sub, cudaStream_t s);
// ---- fft_cols.cu
cudaError_t launch_cols(int sign, float2* data, const ColGeom& g, long long bstride, int batch, cudaStream_t s,
                        bool mixed = true);
cudaError_t cols_generic(int sign, float2* data, const ColGeom& g, long long bstride, int batch, cudaStream_t s);
// ---- fft_planes.cu: r2c along z and forward y, inverse y and c2r along z, in one kernel or two
cudaError_t launch_forward_zy(const float* in, float2* spec, const MeshDims& d, float sub, cudaStream_t s,
                              float* clear = nullptr, bool mixed = true);
cudaError_t launch_inverse_yz(float2* spec, float* out, const MeshDims& d, float scale, cudaStream_t s,
                              bool mixed = true);
// ---- fft_x.cu, fft_x_mixed.cu
cudaError_t launch_x_op(float2* data, const MeshDims& d, const PoissonOp& op, cudaStream_t s, bool mixed);
cudaError_t launch_x_op(float2* data, const MeshDims& d, const PgdOp& op, cudaStream_t s, bool mixed);
cudaError_t launch_x_op(float2* data, const MeshDims& d, const IcOp& op, cudaStream_t s, bool mixed);
cudaError_t launch_x_op(float2* data, const MeshDims& d, const PkAdjOp& op, cudaStream_t s, bool mixed);
cudaError_t launch_x_op_mixed(float2* data, const MeshDims& d, const PoissonOp& op, bool* done, cudaStream_t s);
// ---- fft_pk.cu
cudaError_t launch_x_pk(const float2* data, const MeshDims& d, const PkArgs& a, cudaStream_t s);
cudaError_t x_pk_generic(const float2* data, const MeshDims& d, const PkArgs& a, cudaStream_t s);

}  // namespace jfli
