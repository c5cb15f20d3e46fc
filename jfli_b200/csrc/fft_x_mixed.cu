// Register x passes of the mixed lengths (JFLI_MIXED_SIZES) for the Poisson solve.
#include "fft_x_reg.cuh"

namespace jfli {

cudaError_t launch_x_op_mixed(float2* data, const MeshDims& d, const PoissonOp& op, bool* done, cudaStream_t s) {
  const ColGeom g = x_geom(d);
  *done = true;
  switch (g.n) {
#define JFLI_CASE(N_) \
  case N_:            \
    return x_op_reg<N_, PoissonOp>(data, g, op, d.spec_elems(), d.batch, s);
    JFLI_MIXED_SIZES(JFLI_CASE)
#undef JFLI_CASE
    default:
      *done = false;
      return cudaSuccess;
  }
}

}  // namespace jfli
