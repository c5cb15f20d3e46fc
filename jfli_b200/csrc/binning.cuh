// Binned FP64 sums of the power-spectrum kernels (PkTile in kspace_ops.cuh for fft_pk.cu, poles.cu).
//
// A thread walks modes whose |k| changes slowly (successive kz columns at one kx, or
// successive ky at one kz), keeps the sums of the current bin in registers and adds them to
// the CTA's shared histogram only when the bin changes. The shared FP64 addition is a
// compare-and-swap loop that serialises the lanes that meet on one address, so the
// histogram has up to 32 columns and lane L adds to column L % columns; the columns are
// summed in order at the end. (One addition per mode, aggregated over the warp by bin with
// double shuffles, took 2.80 ms of the 512^3 spectrum's x pass; a segmented shuffle
// reduction over runs of lanes 0.66 ms; this form 0.38 ms, of which the transform is 0.25.)
#pragma once

#include "common.cuh"

namespace jfli {

// numpy.digitize(right=False): the number of edges <= x (ascending edges).
__device__ __forceinline__ int digitize(float x, const float* edges, int nedges) {
  int lo = 0, hi = nedges;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (edges[mid] <= x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// The bin a thread is in, with its edges in registers.
struct BinCursor {
  int bin = -1;  // -1: none yet
  float lo, hi;

  // The last bin has no upper edge (NaN): it holds infinity too, and move never looks past it.
  __device__ __forceinline__ bool holds(float x) const { return bin >= 0 && x >= lo && !(x >= hi); }
  // move to x's bin; the next one up is tried before the search
  __device__ __forceinline__ void move(float x, const float* edges, int nedges) {
    if (bin >= 0 && x >= hi && (bin + 1 == nedges || x < edges[bin + 1]))
      ++bin;
    else
      bin = digitize(x, edges, nedges);
    lo = bin > 0 ? edges[bin - 1] : -INFINITY;
    hi = bin < nedges ? edges[bin] : NAN;
  }
};

// Columns of a histogram whose single column takes `bytes`: the largest power of two up to
// 32 that fits `budget`.
inline __host__ __device__ int histogram_columns(size_t bytes, size_t budget) {
  int c = 32;
  while (c > 1 && (size_t)c * bytes > budget) c >>= 1;
  return c;
}

}  // namespace jfli
