// Spherical harmonic transform of HEALPix ring maps (FP64), the two stages of healpy's
// anafast (reference _src/power/_compute.py:175-191): the ring transforms along phi, which
// take a map to per-ring Fourier coefficients F[r][m] (m = 0..lmax, phase e^{-i m phi_0}
// applied) and back, and the O(lmax^2 x rings) Legendre stages between F and a_lm:
//
//   analysis:  a_lm  = w * sum_r lambda_lm(theta_r) F[r][m]
//   synthesis: G[r][m] = sum_l a_lm lambda_lm(theta_r)
//
// lambda_lm are the orthonormal associated Legendre functions with the Condon-Shortley
// phase. a_lm is packed by m: a[m][l - m], offset m (lmax + 1) - m (m - 1) / 2.
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace jfli {

__host__ __device__ __forceinline__ long long alm_offset(int m, int lmax) {
  return (long long)m * (lmax + 1) - (long long)m * (m - 1) / 2;
}

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }

// ---- Legendre stages ----------------------------------------------------------------
//
// Both are FP64-arithmetic bound (a B200 SM issues 64 FP64 FMAs a clock). Per (l, m) and ring
// the least is the recursion step and two multiply-adds of the sum, and two properties cut
// the rings and the step to their least form:
//   * lambda_lm(pi - theta) = (-1)^(l+m) lambda_lm(theta): a ring and its mirror image take one
//     recursion, on the sum (l - m even) or difference (odd) of their coefficients.
//   * with lambda_l = alpha_l mu_l, alpha_l = (a_l / a_(l-1)) alpha_(l-2) and a_l = sqrt((4 l^2
//     - 1) / (l^2 - m^2)), the three-term recursion lambda_l = a_l (z lambda_(l-1) -
//     lambda_(l-2) / a_(l-1)) becomes mu_l = (A_l z) mu_(l-1) - mu_(l-2), A_l = a_(l-1)
//     alpha_(l-1) / alpha_(l-2): one multiplication and one FMA per ring. alpha stays within
//     about [0.1, 1] and multiplies the finished sums (analysis) or a_lm (synthesis).
// So a pair of rings costs 4 FP64 instructions per l. A thread keeps RP pairs in registers
// (independent chains cover the FP64 latency), a CTA holds one m and up to 32 RP pairs per
// warp, with successive rings in a warp.
//
// Where lambda_mm underflows the recursion runs on values scaled by 2^(400 k) and k drops as
// they grow; a ring adds to the sums only at k = 0 (below, its lambda is under 2^-140). The
// scale is looked at every 8 l, over which a value grows by less than 2^60.
//
// The tables of one m (A_l and alpha_l) are made for 32 l per warp at a time, all warps at once,
// and the CTA's sums of those l are finished together: three barriers per super-tile. (One
// warp making the next 32 l's while the others worked had them wait for it at every table.)
//
// 1 B200, nside 1024, lmax 3000 (8190 x 4.5M (ring, l, m)): analysis 31.9 -> 3.6 ms, synthesis
// 19.4 -> 3.4 ms against one ring per thread with a three-multiplication recursion and, in the
// analysis, one shared-memory reduction per ring and l; FP64 floor of the form above 2.1 ms.
constexpr int kLTile = 32;    // l per table
constexpr int kLChunk = 8;    // l between looks at the scale
constexpr int kRowTile = 16;  // l between reductions over a warp
constexpr int kScaleBits = 400;

constexpr int kLegendreWarps = 4;  // at most

// A_l and alpha_l of the super-tile's l, and the products that the warps' tiles end on
struct LegendreTables {
  double A[kLegendreWarps * kLTile], alpha[kLegendreWarps * kLTile];
  double2 ends[kLegendreWarps];
};

// a_l^2 / a_(l-1)^2 (l > m + 1)
__device__ __forceinline__ double legendre_ratio(int l, int m) {
  const double d = (double)l, e = d - 1.0;
  return ((4.0 * d * d - 1.0) * ((double)(l - 1 - m) * (double)(l - 1 + m))) /
         (((double)(l - m) * (double)(l + m)) * (4.0 * e * e - 1.0));
}

// Tables of a super-tile of 32 l per warp from s0 (s0 - m a multiple of 32), warp w making those
// of l = s0 + 32 w + lane: alpha_l^2 is the product of the ratios of equal parity (a scan over
// lanes of a stride of two, then over the warps' tiles, then the carry of the super-tiles
// before), A_l = a_(l-1) alpha_(l-1) / alpha_(l-2) from the same products, so that their
// accumulated rounding cancels in lambda (the closed form A_l = a_(m+1) alpha_(l-1)^2 would
// need no second division, but lets it in: 1.5e-12 of lambda at l = 700 against 2e-14).
// carry: alpha^2 of the last two l before s0, the same in every thread. Two barriers inside,
// the first before the tables are overwritten, the second after they are written.
__device__ __forceinline__ void legendre_tables(LegendreTables& t, int s0, int m, double2& carry) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int l = s0 + kLTile * warp + lane;
  double q = l > m + 1 ? legendre_ratio(l, m) : 1.0;  // alpha_m = alpha_(m+1) = 1
#pragma unroll
  for (int off = 2; off < 32; off <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, q, off);
    if (lane >= off) q *= v;
  }
  if (lane == 30) t.ends[warp].x = q;
  if (lane == 31) t.ends[warp].y = q;
  __syncthreads();
  double2 c = carry;  // alpha^2 of the last two l before this warp's tile
  for (int w = 0; w < warps; ++w) {
    if (w == warp) c = carry;
    carry.x *= t.ends[w].x;
    carry.y *= t.ends[w].y;
  }
  q *= (lane & 1) ? c.y : c.x;
  double p1 = __shfl_up_sync(0xffffffffu, q, 1), p2 = __shfl_up_sync(0xffffffffu, q, 2);
  if (lane == 0) {
    p1 = c.y;
    p2 = c.x;
  } else if (lane == 1) {
    p2 = c.y;
  }
  const double e = (double)(l - 1);
  t.A[kLTile * warp + lane] =
      sqrt(l > m + 1 ? ((4.0 * e * e - 1.0) * p1) / (((double)(l - 1 - m) * (double)(l - 1 + m)) * p2)
                     : 2.0 * m + 3.0);  // lambda_(m+1) = a_(m+1) z lambda_mm
  t.alpha[kLTile * warp + lane] = sqrt(q);
  __syncthreads();
}

// ln of the normalisation of lambda_mm without its sign: ln sqrt((1 / 4 pi) prod_(k=1..m) (2k
// + 1) / 2k), summed over the CTA's threads in a fixed order.
__device__ __forceinline__ double legendre_lognorm(int m, double* scratch) {
  double s = 0.0;
  for (int k = 1 + threadIdx.x; k <= m; k += blockDim.x) s += log1p(0.5 / (double)k);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = s;
  __syncthreads();
  s = 0.0;
  for (int w = 0; w < (int)blockDim.x / 32; ++w) s += scratch[w];
  __syncthreads();
  return 0.5 * (s - 2.5310242469692907);  // ln 4 pi
}

// One ring (pair) of a thread: z, the last two mu, and the scale k (see above). Every l, the
// first included, is one step: a step that is skipped at l = m costs selects at all others.
struct LegendreRing {
  double z, prev, cur;
  int k;

  __device__ __forceinline__ void start(int m, double zr, double lognorm) {
    z = zr;
    prev = 0.0;
    const double s2 = (1.0 - zr) * (1.0 + zr);
    const double v = m == 0 ? lognorm : lognorm + 0.5 * m * log(s2);  // s2 = 0: -inf, lambda = 0
    const double step = kScaleBits * 0.69314718055994530942;
    k = v < -0.5 * step ? (int)fmin(1e6, ceil((-0.5 * step - v) / step)) : 0;
    // before l = m: the step to it gives A z 0 - prev = lambda_mm
    cur = 0.0;
    prev = exp(v + k * step);
    if (!(m & 1)) prev = -prev;
  }
  __device__ __forceinline__ void rescale() {
    if (k > 0 && fabs(cur) > 0x1p200) {
      cur *= 0x1p-400;
      prev *= 0x1p-400;
      --k;
    }
  }
  // (cur, prev) <- (A z cur - prev, cur)
  __device__ __forceinline__ void step(double A) {
    const double n = fma(A * z, cur, -prev);
    prev = cur;
    cur = n;
  }
};

// Ring pairs of a CTA: pair p is rings p and nrings - 1 - p (the same ring in the middle).
// z need not be mirror symmetric: a CTA that finds a pair whose z differ from mirror images by
// more than rounding takes the two hemispheres one after the other instead.
struct RingPairs {
  int nrings, pairs;
  __device__ __forceinline__ bool mirrored(const double* z, int first, int n) const {
    bool ok = true;
    for (int p = first + threadIdx.x; p < min(pairs, first + n); p += blockDim.x)
      ok = ok && fabs(z[p] + z[nrings - 1 - p]) <= 4e-16;
    return __syncthreads_and(ok);
  }
};

// Four warps at most: the warps of a CTA meet at every super-tile, and the pole-side ones have less
// to do (at nside 1024 one CTA of eight warps per m took 5.7 and 3.9 ms for the two stages,
// two of four 4.3 and 3.6; with the tables per super-tile 3.6 and 3.4).
constexpr int kLegendreThreads = 32 * kLegendreWarps;
template <int RP>
constexpr int kLegendreCtas = RP == 8 ? 3 : 6;  // resident per SM by registers (168 and 80)

// Analysis: a thread's sums over its pairs go through shared memory, 16 l at a time per warp: a
// lane stores one value per l and afterwards adds up half a row (the lanes of one l), so the
// reduction over a warp's rings costs four instructions per l.
// Its rows, part and tables take 44 KB with four warps, so that five CTAs of RP = 2 fit an SM.
template <int RP>
__global__ void __launch_bounds__(kLegendreThreads, kLegendreCtas<RP>) k_sht_analysis(const double2* __restrict__ F,
                                                                   const double* __restrict__ z, int nrings, int lmax,
                                                                   double w, double2* __restrict__ alm) {
  __shared__ LegendreTables tab;
  __shared__ double2 part[kLegendreWarps][kLegendreWarps * kLTile];
  extern __shared__ double2 rows[];  // per warp [16 l][33]
  const int m = blockIdx.x;
  F += (long long)blockIdx.z * nrings * (lmax + 1);
  alm += blockIdx.z * alm_offset(lmax + 1, lmax);
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2* row = rows + (size_t)warp * kRowTile * 33;
  const RingPairs rp{nrings, (nrings + 1) / 2};
  const int first = blockIdx.y * (blockDim.x * RP);
  const bool mirror = rp.mirrored(z, first, blockDim.x * RP);
  const double lognorm = legendre_lognorm(m, &part[0][0].x);
  const long long off = alm_offset(m, lmax);
  const long long fs = lmax + 1;
  for (int hemi = 0; hemi < (mirror ? 1 : 2); ++hemi) {
    LegendreRing r[RP];
    double2 even[RP], odd[RP];
#pragma unroll
    for (int j = 0; j < RP; ++j) {
      const int p = first + warp * (32 * RP) + 32 * j + lane;
      const int q = nrings - 1 - p;
      even[j] = odd[j] = make_double2(0.0, 0.0);
      double zr = 0.0;
      if (p < rp.pairs && !(hemi == 1 && p == q)) {
        if (mirror) {
          const double2 a = F[p * fs + m], b = p == q ? make_double2(0.0, 0.0) : F[q * fs + m];
          even[j] = zadd(a, b);
          odd[j] = zsub(a, b);
          zr = p == q ? z[p] : 0.5 * (z[p] - z[q]);
        } else {
          const int ring = hemi == 0 ? p : q;
          even[j] = odd[j] = F[ring * fs + m];
          zr = z[ring];
        }
      }
      r[j].start(m, zr, lognorm);
    }
    // 0, or NaN where a ring's coefficients are not finite: what a ring adds before its lambda counts
    double2 poison = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < RP; ++j) {
      poison.x += 0.0 * even[j].x + 0.0 * odd[j].x;
      poison.y += 0.0 * even[j].y + 0.0 * odd[j].y;
    }
    const bool poisoned = __any_sync(0xffffffffu, !(poison.x == 0.0 && poison.y == 0.0));
    double2 carry = make_double2(1.0, 1.0);
    for (int s0 = m; s0 <= lmax; s0 += kLTile * warps) {
      legendre_tables(tab, s0, m, carry);
      const int t2 = min(kLTile * warps, lmax + 1 - s0);
      for (int t1 = 0; t1 < t2; t1 += kRowTile) {
        bool any = poisoned;
        for (int t0 = t1; t0 < t1 + kRowTile; t0 += kLChunk) {
          int scaled = 0;
#pragma unroll
          for (int j = 0; j < RP; ++j) {
            r[j].rescale();
            scaled += r[j].k > 0;
          }
          const bool all_on = __all_sync(0xffffffffu, scaled == 0);
          const bool none_on = __all_sync(0xffffffffu, scaled == RP);
          if (!none_on) any = true;
          double2* out = row + (t0 - t1) * 33 + lane;
          auto chunk = [&](auto masked) {
            bool on[RP];
            if constexpr (masked) {
#pragma unroll
              for (int j = 0; j < RP; ++j) on[j] = r[j].k == 0;
            }
#pragma unroll
            for (int t = 0; t < kLChunk; ++t) {
              double2 sum = make_double2(0.0, 0.0);
#pragma unroll
              for (int j = 0; j < RP; ++j) {
                r[j].step(tab.A[t0 + t]);
                double v = r[j].cur;
                if constexpr (masked) v = on[j] ? v : 0.0;
                const double2 f = (t & 1) ? odd[j] : even[j];
                sum.x = fma(v, f.x, sum.x);
                sum.y = fma(v, f.y, sum.y);
              }
              out[t * 33] = sum;
            }
          };
          if (all_on) {
            chunk(std::false_type{});
          } else if (!none_on) {
            chunk(std::true_type{});
          } else {  // nothing to add yet
#pragma unroll
            for (int t = 0; t < kLChunk; ++t) {
#pragma unroll
              for (int j = 0; j < RP; ++j) r[j].step(tab.A[t0 + t]);
              out[t * 33] = poison;
            }
          }
        }
        __syncwarp();
        double2 sum = make_double2(0.0, 0.0);
        if (any) {
          const double2* in = row + (lane & 15) * 33 + (lane & 16);
#pragma unroll
          for (int i = 0; i < 16; ++i) sum = zadd(sum, in[i]);
        }
        sum.x += __shfl_xor_sync(0xffffffffu, sum.x, 16);
        sum.y += __shfl_xor_sync(0xffffffffu, sum.y, 16);
        if (lane < kRowTile) part[warp][t1 + lane] = sum;
        __syncwarp();  // row is free again
      }
      __syncthreads();
      const int l = s0 + threadIdx.x;
      if (l <= lmax) {
        double2 s = make_double2(0.0, 0.0);
        for (int i = 0; i < warps; ++i) s = zadd(s, part[i][threadIdx.x]);
        const double f = w * tab.alpha[threadIdx.x];
        double2* dst = alm + off + (l - m);
        if (gridDim.y > 1) {
          atomicAdd(&dst->x, f * s.x);
          atomicAdd(&dst->y, f * s.y);
        } else if (hemi == 0) {
          *dst = make_double2(f * s.x, f * s.y);
        } else {
          *dst = make_double2(dst->x + f * s.x, dst->y + f * s.y);
        }
      }
    }
  }
}

template <int RP>
__global__ void __launch_bounds__(kLegendreThreads, kLegendreCtas<RP>) k_sht_synthesis(const double2* __restrict__ alm,
                                                                    const double* __restrict__ z, int nrings, int lmax,
                                                                    double2* __restrict__ G) {
  __shared__ LegendreTables tab;
  __shared__ double2 a_tile[kLegendreWarps * kLTile];  // alpha_l a_lm
  __shared__ double scratch[kLegendreWarps];
  const int m = blockIdx.x;
  alm += blockIdx.z * alm_offset(lmax + 1, lmax);
  G += (long long)blockIdx.z * nrings * (lmax + 1);
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const RingPairs rp{nrings, (nrings + 1) / 2};
  const int first = blockIdx.y * (blockDim.x * RP);
  const bool mirror = rp.mirrored(z, first, blockDim.x * RP);
  const double lognorm = legendre_lognorm(m, scratch);
  const double2* a = alm + alm_offset(m, lmax);
  const long long fs = lmax + 1;
  for (int hemi = 0; hemi < (mirror ? 1 : 2); ++hemi) {
    LegendreRing r[RP];
    double2 even[RP], odd[RP];
#pragma unroll
    for (int j = 0; j < RP; ++j) {
      const int p = first + warp * (32 * RP) + 32 * j + lane;
      const int q = nrings - 1 - p;
      double zr = 0.0;
      if (p < rp.pairs) zr = mirror ? (p == q ? z[p] : 0.5 * (z[p] - z[q])) : z[hemi == 0 ? p : q];
      even[j] = odd[j] = make_double2(0.0, 0.0);
      r[j].start(m, zr, lognorm);
    }
    double2 carry = make_double2(1.0, 1.0);
    for (int s0 = m; s0 <= lmax; s0 += kLTile * warps) {
      legendre_tables(tab, s0, m, carry);
      {
        const int l = s0 + threadIdx.x;
        const double2 v = l <= lmax ? a[l - m] : make_double2(0.0, 0.0);
        const double f = tab.alpha[threadIdx.x];
        a_tile[threadIdx.x] = make_double2(f * v.x, f * v.y);
      }
      __syncthreads();
      const int t1 = min(kLTile * warps, lmax + 1 - s0);
      for (int t0 = 0; t0 < t1; t0 += kLChunk) {
        int scaled = 0;
#pragma unroll
        for (int j = 0; j < RP; ++j) {
          r[j].rescale();
          scaled += r[j].k > 0;
        }
        const bool all_on = __all_sync(0xffffffffu, scaled == 0);
        const bool none_on = __all_sync(0xffffffffu, scaled == RP);
        auto chunk = [&](auto masked) {
          bool on[RP];
          if constexpr (masked) {
#pragma unroll
            for (int j = 0; j < RP; ++j) on[j] = r[j].k == 0;
          }
#pragma unroll
          for (int t = 0; t < kLChunk; ++t) {
            const double2 c = a_tile[t0 + t];
#pragma unroll
            for (int j = 0; j < RP; ++j) {
              r[j].step(tab.A[t0 + t]);
              double v = r[j].cur;
              if constexpr (masked) v = on[j] ? v : 0.0;
              double2& s = (t & 1) ? odd[j] : even[j];
              s.x = fma(v, c.x, s.x);
              s.y = fma(v, c.y, s.y);
            }
          }
        };
        if (all_on) {
          chunk(std::false_type{});
        } else if (!none_on) {
          chunk(std::true_type{});
        } else {
#pragma unroll
          for (int t = 0; t < kLChunk; ++t)
#pragma unroll
            for (int j = 0; j < RP; ++j) r[j].step(tab.A[t0 + t]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < RP; ++j) {
      const int p = first + warp * (32 * RP) + 32 * j + lane;
      const int q = nrings - 1 - p;
      if (p >= rp.pairs) continue;
      const double2 sum = zadd(even[j], odd[j]);
      if (mirror) {
        G[p * fs + m] = sum;
        if (q != p) G[q * fs + m] = zsub(even[j], odd[j]);
      } else {
        G[(hemi == 0 ? p : q) * fs + m] = sum;
      }
    }
  }
}

// Pairs per thread and threads of a CTA. Eight pairs per thread (eight independent chains, the
// least reduction and table work per pair) for large maps; two for small ones, whose 3 nside
// CTAs do not fill the SMs for long and end on the serial chain of their first m, unless
// several maps go together. a_lm with three refinements, 2 against 8 pairs: nside 512 5.1 and
// 4.4 ms, nside 256 0.94 and 1.07 (two maps together 1.72 and 1.60, four 3.26 and 3.08), four of
// nside 128 0.69 and 0.85. With fewer m than kLegendreFill two pairs as well: C_l at nside 512, lmax 64 648
// and 694 us, lmax 200 758 and 806; nside 1024, lmax 200 2.69 and 2.67 ms, lmax 280 2.91 and 2.85.
constexpr int kLegendreFill = 222;

struct LegendreShape {
  int rp, threads, blocks;
};

static LegendreShape legendre_shape(int nrings, int lmax, int nmaps) {
  const int pairs = (nrings + 1) / 2;
  LegendreShape s;
  const bool fills = (long long)(lmax + 1) * nmaps >= kLegendreFill;
  s.rp = fills && (pairs >= 1024 || (pairs >= 512 && nmaps >= 2)) ? 8 : 2;
  int warps = (pairs + 32 * s.rp - 1) / (32 * s.rp);
  s.blocks = (warps + kLegendreWarps - 1) / kLegendreWarps;
  warps = (warps + s.blocks - 1) / s.blocks;
  s.threads = 32 * warps;
  return s;
}

// ---- ring transforms along phi ------------------------------------------------------
// RING geometry of ring r (0 = northernmost, i = r + 1): pixel count, first pixel, and the
// longitude of the first pixel centre, by which the transforms have phi. In the belt it is half a
// pixel from the painters' pixel centres (Gorski et al. 2005; ring_info_tab) on every ring, 0 where
// they have pi / (4 nside) and the other way around: C_l of a painted map falls short from l ~
// nside on (tests/test_sht_longitudes.py).
struct RingPhi {
  long long start;
  int n;
  double phi0;
};

__device__ __forceinline__ RingPhi ring_phi(int r, int nside) {
  const int i = r + 1;
  const long long npix = 12LL * nside * nside;
  RingPhi g;
  if (i < nside) {
    g.n = 4 * i;
    g.start = 2LL * i * (i - 1);
    g.phi0 = 3.14159265358979323846 / (4.0 * i);
  } else if (i <= 3 * nside) {
    g.n = 4 * nside;
    g.start = 2LL * nside * (nside - 1) + (long long)(i - nside) * 4 * nside;
    g.phi0 = ((i - nside + 1) % 2 == 1) ? 0.0 : 3.14159265358979323846 / (4.0 * nside);
  } else {
    const int j = 4 * nside - i;
    g.n = 4 * j;
    g.start = npix - 2LL * j * (j + 1);
    g.phi0 = 3.14159265358979323846 / (4.0 * j);
  }
  return g;
}

constexpr int kRingThreads = 128;
constexpr int kReseed = 64;  // exact phase every 64 terms; rotations in between

// e^{-i m phi_j}, phi_j = phi0 + 2 pi j / n, with the angle reduced exactly: (m j) mod n.
__device__ __forceinline__ double2 phase(int m, int j, int n, double phi0, double sign) {
  const long long q = ((long long)m * j) % n;
  const double ang = (double)m * phi0 + 6.283185307179586476925 * (double)q / (double)n;
  double sn, cs;
  sincos(ang, &sn, &cs);
  return make_double2(cs, sign * sn);
}

// Direct sums (where ring_fft does not hold):
// F[r][m] = sum_j f_j e^{-i m phi_j}, m = 0..lmax (aliasing for m >= n is the DFT's own).
// One block per (ring, 128 m); the ring's values staged in shared memory.
__global__ void __launch_bounds__(kRingThreads) k_ring_analysis(const double* __restrict__ map, int nside, int lmax,
                                                                double2* __restrict__ F) {
  extern __shared__ double ring[];
  const int r = blockIdx.y;
  map += blockIdx.z * 12LL * nside * nside;
  F += (long long)blockIdx.z * gridDim.y * (lmax + 1);
  const RingPhi g = ring_phi(r, nside);
  for (int j = threadIdx.x; j < g.n; j += blockDim.x) ring[j] = map[g.start + j];
  __syncthreads();
  const int m = blockIdx.x * kRingThreads + threadIdx.x;
  if (m > lmax) return;
  double2 step;  // e^{-i 2 pi m / n}
  {
    const double ang = 6.283185307179586476925 * (double)(m % g.n) / (double)g.n;
    double sn, cs;
    sincos(ang, &sn, &cs);
    step = make_double2(cs, -sn);
  }
  double sx = 0.0, sy = 0.0;
  for (int j0 = 0; j0 < g.n; j0 += kReseed) {
    double2 w = phase(m, j0, g.n, g.phi0, -1.0);
    const int j1 = min(j0 + kReseed, g.n);
    for (int j = j0; j < j1; ++j) {
      const double f = ring[j];
      sx += f * w.x;
      sy += f * w.y;
      w = make_double2(w.x * step.x - w.y * step.y, w.x * step.y + w.y * step.x);
    }
  }
  F[(long long)r * (lmax + 1) + m] = make_double2(sx, sy);
}

// f_j = Re G[r][0] + 2 sum_{m >= 1} Re(G[r][m] e^{i m phi_j}). One block per (ring, 128
// pixels); the ring's coefficients staged in shared memory.
__global__ void __launch_bounds__(kRingThreads) k_ring_synthesis(const double2* __restrict__ G, int nside, int lmax,
                                                                 double* __restrict__ map) {
  extern __shared__ double2 coef[];
  const int r = blockIdx.y;
  map += blockIdx.z * 12LL * nside * nside;
  G += (long long)blockIdx.z * gridDim.y * (lmax + 1);
  const RingPhi g = ring_phi(r, nside);
  for (int m = threadIdx.x; m <= lmax; m += blockDim.x) coef[m] = G[(long long)r * (lmax + 1) + m];
  __syncthreads();
  const int j = blockIdx.x * kRingThreads + threadIdx.x;
  if (j >= g.n) return;
  const double phij = g.phi0 + 6.283185307179586476925 * (double)j / (double)g.n;
  double2 step;  // e^{i phi_j}
  {
    double sn, cs;
    sincos(phij, &sn, &cs);
    step = make_double2(cs, sn);
  }
  double acc = 0.0;
  for (int m0 = 1; m0 <= lmax; m0 += kReseed) {
    double2 w = phase(m0, j, g.n, g.phi0, 1.0);
    const int m1 = min(m0 + kReseed, lmax + 1);
    for (int m = m0; m < m1; ++m) {
      acc += coef[m].x * w.x - coef[m].y * w.y;
      w = make_double2(w.x * step.x - w.y * step.y, w.x * step.y + w.y * step.x);
    }
  }
  map[g.start + j] = coef[0].x + 2.0 * acc;
}

// Rings with 4 nside pixels or fewer are transformed, where ring_fft holds, by an FP64 FFT in
// shared memory, one CTA per ring. A ring has n = 4 i pixels; its 2 i complex pairs (f_2j +
// i f_2j+1) split into two interleaved transforms of length i, which are plain radix-4 ones
// when i is a power of two and Bluestein convolutions of length M = 2^c >= 2 i - 1 otherwise
// (x_j c_j convolved with conj(c_j), c_j = e^{-i pi j^2 / i}, the chirp's index reduced
// exactly: j^2 mod 2 i). The transforms are decimation in frequency (natural -> digit
// reversed) and back in time, so nothing is permuted; the pointwise product does not see the
// order and a plain transform's outputs are picked up by their digit-reversed position.
// A ring is never mixed with another one: a NaN or a huge value stays in its ring.
//
// 1 B200, nside 1024, lmax 3000: analysis 19.4 -> 0.44 ms, synthesis 20.0 -> 0.42 ms against direct
// sums (npix x lmax terms). Those still serve larger nside, whose convolutions (M = 4096 and
// more, three arrays) leave one CTA per SM or none, and few coefficients (ring_fft): a warp of the
// sums has one per lane, so that their cost goes up every 32. FFT and direct sums, analysis and
// synthesis, in us: lmax 16, nside 256 26, 25 and 27, 17, 700 307, 131 and 325, 103, 1024 301, 320 and
// 333, 217; lmax 32, nside 384 77, 74 and 82, 46, 1024 303, 456 and 334, 305; lmax 64, nside 16 5.7, 3.3 and
// 6.3, 3.5, 64 6.8, 8.0 and 7.4, 5.1, 384 77, 103 and 82, 72, 700 307, 294 and 325, 229.
constexpr int kRingFftMax = 1024;

// Short rings are bound by the FFT's barriers, belts that are no power of two are convolutions.
static bool ring_fft(int nside, int lmax) {
  const bool convolved = (nside & (nside - 1)) != 0;
  const int least = nside < 64 ? 96 : (!convolved ? 32 : (nside <= 512 ? 64 : 96));
  return nside <= kRingFftMax && lmax >= least;
}
constexpr int kRingFftThreads = 256;

struct RingFft {
  int i, M, lg;   // sub-transform length, its FFT length 2^lg
  bool plain;     // M == i
  double2 *arr;   // [2][M]
  double2 *filt;  // [M + 1]: the chirp filter's spectrum (before that, free)
  double2 *tw;    // [M / 4]: e^{-2 pi i j / M}
  double2 *part;  // [kRingFftThreads]: the synthesis's partial sums of short rings
};

__host__ __device__ inline int ring_fft_length(int i) {
  if ((i & (i - 1)) == 0) return i;
  int M = 1;
  while (M < 2 * i - 1) M <<= 1;
  return M;
}
// shared memory for rings of up to 4 nside pixels
inline size_t ring_fft_smem(int nside) {
  int M = 1;
  for (int i = nside; i >= 1 && i > nside - 2; --i) {  // nside and nside - 1 cover the largest of both kinds
    const int L = ring_fft_length(i);
    if (L > M) M = L;
  }
  // the synthesis keeps the ring's 2 i + 1 folded coefficients in filt, whatever the kind
  const size_t filt = (size_t)(M > 2 * nside ? M : 2 * nside) + 1;
  return sizeof(double2) * ((size_t)2 * M + filt + M / 4 + kRingFftThreads);
}

__device__ __forceinline__ double2 cispi(double x) {  // e^{i pi x}
  double s, c;
  sincospi(x, &s, &c);
  return make_double2(c, s);
}

__device__ __forceinline__ double2 chirp(int j, int i) { return zconj(cispi((double)((j * j) % (2 * i)) / (double)i)); }

__device__ __forceinline__ RingFft ring_fft_setup(int i, double2* sm) {
  RingFft f;
  f.i = i;
  f.M = ring_fft_length(i);
  f.plain = f.M == i;
  f.lg = 31 - __clz(f.M);
  f.arr = sm;
  f.filt = sm + 2 * f.M;
  f.tw = f.filt + (max(f.M, 2 * i) + 1);
  f.part = f.tw + f.M / 4;
  for (int j = threadIdx.x; j < f.M / 4; j += blockDim.x) f.tw[j] = cispi(-2.0 * j / (double)f.M);
  return f;
}

// Forward DIF transforms of `count` consecutive arrays of length M = 2^lg, in place; ends with
// a barrier.
__device__ __forceinline__ void ring_fft_forward(double2* x, int count, int lg, const double2* tw) {
  int lq = lg - 2, step = 0;  // quarter 2^lq, twiddle stride 2^step
  for (; lq >= 0; lq -= 2, step += 2) {
    const int total = count << (lg - 2);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const int j = t & ((1 << lq) - 1);
      double2* p = x + (((t >> lq) << (lq + 2)) + j);
      const double2 a0 = p[0], a1 = p[1 << lq], a2 = p[2 << lq], a3 = p[3 << lq];
      const double2 s02 = zadd(a0, a2), d02 = zsub(a0, a2), s13 = zadd(a1, a3), d13 = zsub(a1, a3);
      const double2 w1 = tw[j << step], w2 = zmul(w1, w1);
      p[0] = zadd(s02, s13);
      p[1 << lq] = zmul(make_double2(d02.x + d13.y, d02.y - d13.x), w1);  // (d02 - i d13) w
      p[2 << lq] = zmul(zsub(s02, s13), w2);
      p[3 << lq] = zmul(make_double2(d02.x - d13.y, d02.y + d13.x), zmul(w2, w1));
    }
    __syncthreads();
  }
  if (lg & 1) {
    const int total = count << (lg - 1);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const double2 a = x[2 * t], b = x[2 * t + 1];
      x[2 * t] = zadd(a, b);
      x[2 * t + 1] = zsub(a, b);
    }
    __syncthreads();
  }
}

// The inverse of ring_fft_forward (unnormalised), digit reversed -> natural.
__device__ __forceinline__ void ring_fft_inverse(double2* x, int count, int lg, const double2* tw) {
  if (lg & 1) {
    const int total = count << (lg - 1);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const double2 a = x[2 * t], b = x[2 * t + 1];
      x[2 * t] = zadd(a, b);
      x[2 * t + 1] = zsub(a, b);
    }
    __syncthreads();
  }
  for (int lq = lg & 1; lq <= lg - 2; lq += 2) {
    const int step = lg - 2 - lq;
    const int total = count << (lg - 2);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const int j = t & ((1 << lq) - 1);
      double2* p = x + (((t >> lq) << (lq + 2)) + j);
      const double2 w1 = zconj(tw[j << step]), w2 = zmul(w1, w1);
      const double2 y0 = p[0], y1 = zmul(p[1 << lq], w1), y2 = zmul(p[2 << lq], w2), y3 = zmul(p[3 << lq], zmul(w2, w1));
      const double2 s02 = zadd(y0, y2), d02 = zsub(y0, y2), s13 = zadd(y1, y3), d13 = zsub(y1, y3);
      p[0] = zadd(s02, s13);
      p[1 << lq] = make_double2(d02.x - d13.y, d02.y + d13.x);  // d02 + i d13
      p[2 << lq] = zsub(s02, s13);
      p[3 << lq] = make_double2(d02.x + d13.y, d02.y - d13.x);
    }
    __syncthreads();
  }
}

// Where ring_fft_forward leaves frequency k.
__device__ __forceinline__ int digit_reversed(int k, int lg) {
  int pos = 0, left = lg;
  while (left >= 2) {
    left -= 2;
    pos |= (k & 3) << left;
    k >>= 2;
  }
  if (left == 1) pos |= k & 1;
  return pos;
}

// DFT of length 2 i of the values whose pairs (s_2j, s_2j+1) the caller put in (arr[0][j],
// arr[1][j]), j < i. Afterwards frequency k is at ring_fft_at(f, k). Starts and ends with a
// barrier; filt is overwritten.
__device__ __forceinline__ void ring_fft_run(const RingFft& f) {
  const int i = f.i, M = f.M;
  __syncthreads();
  if (f.plain) {
    ring_fft_forward(f.arr, 2, f.lg, f.tw);
  } else {
    for (int j = threadIdx.x; j < M; j += blockDim.x) {
      const bool in = j < i;
      const double2 c = chirp(in ? j : 0, i);
      f.arr[j] = in ? zmul(f.arr[j], c) : make_double2(0.0, 0.0);
      f.arr[M + j] = in ? zmul(f.arr[M + j], c) : make_double2(0.0, 0.0);
      const int b = in ? j : (M - j < i ? M - j : -1);
      f.filt[j] = b < 0 ? make_double2(0.0, 0.0) : zconj(chirp(b, i));
    }
    __syncthreads();
    ring_fft_forward(f.arr, 3, f.lg, f.tw);  // filt follows arr: transformed with it
    for (int j = threadIdx.x; j < M; j += blockDim.x) {
      const double2 b = f.filt[j];
      f.arr[j] = zmul(f.arr[j], b);
      f.arr[M + j] = zmul(f.arr[M + j], b);
    }
    __syncthreads();
    ring_fft_inverse(f.arr, 2, f.lg, f.tw);
  }
  const double scale = 1.0 / (double)M;
  for (int k = threadIdx.x; k < i; k += blockDim.x) {
    const int at = f.plain ? digit_reversed(k, f.lg) : k;
    double2 s0 = f.arr[at], s1 = f.arr[M + at];
    const double2 w = cispi(-(double)k / (double)i);  // e^{-2 pi i k / 2i}
    if (f.plain) {
      s1 = zmul(s1, w);
    } else {
      double2 c = chirp(k, i);
      c.x *= scale;
      c.y *= scale;
      s0 = zmul(s0, c);
      s1 = zmul(s1, zmul(c, w));
    }
    f.arr[at] = zadd(s0, s1);
    f.arr[M + at] = zsub(s0, s1);
  }
  __syncthreads();
}

__device__ __forceinline__ double2 ring_fft_at(const RingFft& f, int k) {
  const int half = k >= f.i;
  const int q = k - (half ? f.i : 0);
  return f.arr[half * f.M + (f.plain ? digit_reversed(q, f.lg) : q)];
}

// e^{-i m phi0}, phi0 = pi / n or 0
__device__ __forceinline__ double2 ring_phase(int m, const RingPhi& g) {
  if (g.phi0 == 0.0) return make_double2(1.0, 0.0);
  return cispi(-(double)(m % (2 * g.n)) / (double)g.n);
}

__global__ void __launch_bounds__(kRingFftThreads) k_ring_fft_analysis(const double* __restrict__ map, int nside,
                                                                       int lmax, double2* __restrict__ F) {
  extern __shared__ double2 sm2[];
  const int r = blockIdx.x;
  map += blockIdx.z * 12LL * nside * nside;
  F += (long long)blockIdx.z * gridDim.x * (lmax + 1);
  const RingPhi g = ring_phi(r, nside);
  const int n = g.n, h = n / 2;
  const RingFft f = ring_fft_setup(n / 4, sm2);
  const double* src = map + g.start;
  for (int j = threadIdx.x; j < h; j += blockDim.x)  // (f_2j, f_2j+1): ring starts and n are even
    f.arr[(j & 1) * f.M + (j >> 1)] = make_double2(src[2 * j], src[2 * j + 1]);
  ring_fft_run(f);
  double2* out = F + (long long)r * (lmax + 1);
  for (int m = threadIdx.x; m <= lmax; m += blockDim.x) {
    int k = m % n;
    const bool mirror = k > h;  // X[k] = conj X[n - k]
    if (mirror) k = n - k;
    const double2 a = ring_fft_at(f, k == h ? 0 : k), b = zconj(ring_fft_at(f, k == 0 ? 0 : h - k));
    const double2 e = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y + b.y));
    const double2 o = make_double2(0.5 * (a.y - b.y), -0.5 * (a.x - b.x));  // (a - b) / 2i
    double2 x = zadd(e, zmul(o, cispi(-2.0 * k / (double)n)));
    if (mirror) x = zconj(x);
    out[m] = zmul(x, ring_phase(m, g));
  }
}

__global__ void __launch_bounds__(kRingFftThreads) k_ring_fft_synthesis(const double2* __restrict__ G, int nside,
                                                                        int lmax, double* __restrict__ map) {
  extern __shared__ double2 sm2[];
  const int r = blockIdx.x;
  map += blockIdx.z * 12LL * nside * nside;
  G += (long long)blockIdx.z * gridDim.x * (lmax + 1);
  const RingPhi g = ring_phi(r, nside);
  const int n = g.n, h = n / 2;
  const RingFft f = ring_fft_setup(n / 4, sm2);
  const double2* src = G + (long long)r * (lmax + 1);
  // E[k], k = 0..h: the Hermitian part of the folded spectrum, (H[k] + conj H[n - k]) / 2 with
  // H[k] = sum over m = k, k + n, ... of c_m G[m] e^{i m phi0}, c_0 = 1 (real part), c_m = 2.
  // A ring with fewer frequencies than the CTA has threads gives each several threads, which
  // take every `groups`-th m and are added in order.
  const int nk = h + 1;
  const int groups = max(1, (int)blockDim.x / nk);
  double2* E = f.filt;
  double2* partial = f.part;  // [groups][nk]
  for (int t = threadIdx.x; t < groups * nk; t += blockDim.x) {
    const int grp = t / nk, k = t - grp * nk;
    double2 s = make_double2(0.0, 0.0);
    for (int m = k + grp * n; m <= lmax; m += groups * n) {
      double2 v = zmul(src[m], zconj(ring_phase(m, g)));
      if (m == 0) v = make_double2(0.5 * src[0].x, 0.0);
      s = zadd(s, v);
    }
    for (int m = (k == 0 ? n : n - k) + grp * n; m <= lmax; m += groups * n)
      s = zadd(s, zconj(zmul(src[m], zconj(ring_phase(m, g)))));
    if (k == 0 && grp == 0) s = zadd(s, make_double2(0.5 * src[0].x, 0.0));  // conj H[0]'s m = 0
    if (groups == 1)
      E[k] = s;
    else
      partial[t] = s;
  }
  __syncthreads();
  if (groups > 1) {
    for (int k = threadIdx.x; k < nk; k += blockDim.x) {
      double2 s = partial[k];
      for (int grp = 1; grp < groups; ++grp) s = zadd(s, partial[grp * nk + k]);
      E[k] = s;
    }
    __syncthreads();
  }
  // f_2j + i f_2j+1 = sum_k Z[k] e^{2 pi i j k / h}, Z[k] = (E[k] + conj E[h-k]) + i (E[k] - conj
  // E[h-k]) e^{2 pi i k / n}; the inverse transform as the conjugate of a forward one
  for (int k = threadIdx.x; k < h; k += blockDim.x) {
    const double2 a = E[k], b = zconj(E[h - k]);
    const double2 e = zadd(a, b), d = zmul(zsub(a, b), cispi(2.0 * k / (double)n));
    f.arr[(k & 1) * f.M + (k >> 1)] = make_double2(e.x - d.y, -(e.y + d.x));
  }
  ring_fft_run(f);
  double* dst = map + g.start;
  for (int j = threadIdx.x; j < h; j += blockDim.x) {
    const double2 v = ring_fft_at(f, j);
    dst[2 * j] = v.x;
    dst[2 * j + 1] = -v.y;
  }
}

cudaError_t sht_ring_analysis(const double* map, int nside, int lmax, double* F, cudaStream_t s, int nmaps) {
  const int nrings = 4 * nside - 1;
  double2* out = reinterpret_cast<double2*>(F);
  cudaError_t e;
  if (ring_fft(nside, lmax)) {
    const size_t smem = ring_fft_smem(nside);
    e = cudaFuncSetAttribute(k_ring_fft_analysis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_ring_fft_analysis<<<dim3(nrings, 1, nmaps), kRingFftThreads, smem, s>>>(map, nside, lmax, out);
  } else {
    const size_t smem = sizeof(double) * 4 * (size_t)nside;
    e = cudaFuncSetAttribute(k_ring_analysis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_ring_analysis<<<dim3((lmax + kRingThreads) / kRingThreads, nrings, nmaps), kRingThreads, smem, s>>>(map, nside,
                                                                                                          lmax, out);
  }
  note_launch();
  return cudaGetLastError();
}

cudaError_t sht_ring_synthesis(const double* G, int nside, int lmax, double* map, cudaStream_t s, int nmaps) {
  const int nrings = 4 * nside - 1;
  const double2* in = reinterpret_cast<const double2*>(G);
  cudaError_t e;
  if (ring_fft(nside, lmax)) {
    const size_t smem = ring_fft_smem(nside);
    e = cudaFuncSetAttribute(k_ring_fft_synthesis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_ring_fft_synthesis<<<dim3(nrings, 1, nmaps), kRingFftThreads, smem, s>>>(in, nside, lmax, map);
  } else {
    const size_t smem = sizeof(double2) * (size_t)(lmax + 1);
    e = cudaFuncSetAttribute(k_ring_synthesis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_ring_synthesis<<<dim3((4 * nside + kRingThreads - 1) / kRingThreads, nrings, nmaps), kRingThreads, smem, s>>>(
        in, nside, lmax, map);
  }
  note_launch();
  return cudaGetLastError();
}

template <int RP>
static cudaError_t analysis_launch(const LegendreShape& sh, const double* F, const double* z, int nrings, int lmax,
                                   double weight, double* alm, int nmaps, cudaStream_t s) {
  const size_t smem = sizeof(double2) * (size_t)(sh.threads / 32) * kRowTile * 33;
  cudaError_t e = cudaFuncSetAttribute(k_sht_analysis<RP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_sht_analysis<RP><<<dim3(lmax + 1, sh.blocks, nmaps), sh.threads, smem, s>>>(
      reinterpret_cast<const double2*>(F), z, nrings, lmax, weight, reinterpret_cast<double2*>(alm));
  note_launch();
  return cudaGetLastError();
}

cudaError_t sht_analysis(const double* F, const double* z, int nrings, int lmax, double weight, double* alm,
                         cudaStream_t s, int nmaps) {
  const LegendreShape sh = legendre_shape(nrings, lmax, nmaps);
  if (sh.blocks > 1) {  // the blocks of one m add to alm
    const cudaError_t e = cudaMemsetAsync(alm, 0, sizeof(double2) * (size_t)alm_offset(lmax + 1, lmax) * nmaps, s);
    if (e != cudaSuccess) return e;
  }
  if (sh.rp == 8) return analysis_launch<8>(sh, F, z, nrings, lmax, weight, alm, nmaps, s);
  return analysis_launch<2>(sh, F, z, nrings, lmax, weight, alm, nmaps, s);
}

cudaError_t sht_synthesis(const double* alm, const double* z, int nrings, int lmax, double* G, cudaStream_t s,
                          int nmaps) {
  const LegendreShape sh = legendre_shape(nrings, lmax, nmaps);
  const dim3 grid(lmax + 1, sh.blocks, nmaps);
  const double2* a = reinterpret_cast<const double2*>(alm);
  double2* out = reinterpret_cast<double2*>(G);
  if (sh.rp == 8)
    k_sht_synthesis<8><<<grid, sh.threads, 0, s>>>(a, z, nrings, lmax, out);
  else
    k_sht_synthesis<2><<<grid, sh.threads, 0, s>>>(a, z, nrings, lmax, out);
  note_launch();
  return cudaGetLastError();
}

// C_l = (Re a_l0 b_l0* + 2 sum_{m=1..l} Re a_lm b_lm*) / (2l + 1) (healpy alm2cl), FP64. A
// block takes 32 l; its 16 rows of threads each sum every 16th m (32 neighbouring l of one m
// are contiguous) and the rows are added in order, so the result is deterministic. (One
// thread per l left 3001 chains of dependent loads: 0.67 ms at lmax 3000, 0.05 ms now.)
constexpr int kClRows = 16;

__global__ void __launch_bounds__(32 * kClRows) k_sht_alm2cl(const double2* __restrict__ a,
                                                             const double2* __restrict__ b, int lmax,
                                                             double* __restrict__ cl) {
  __shared__ double sum[kClRows][33];
  const int l = blockIdx.x * 32 + threadIdx.x;
  double acc = 0.0;
  if (l <= lmax) {
#pragma unroll 4
    for (int m = 1 + threadIdx.y; m <= l; m += kClRows) {
      const long long o = alm_offset(m, lmax) + (l - m);
      const double2 x = a[o], y = b[o];
      acc += x.x * y.x + x.y * y.y;
    }
  }
  sum[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && l <= lmax) {
    acc = 0.0;
    for (int r = 0; r < kClRows; ++r) acc += sum[r][threadIdx.x];
    const double2 x0 = a[l], y0 = b[l];
    cl[l] = (x0.x * y0.x + x0.y * y0.y + 2.0 * acc) / (2.0 * l + 1.0);
  }
}

cudaError_t sht_alm2cl(const double* alm1, const double* alm2, int lmax, double* cl, cudaStream_t s) {
  k_sht_alm2cl<<<(lmax + 32) / 32, dim3(32, kClRows), 0, s>>>(reinterpret_cast<const double2*>(alm1),
                                                              reinterpret_cast<const double2*>(alm2 ? alm2 : alm1),
                                                              lmax, cl);
  note_launch();
  return cudaGetLastError();
}

}  // namespace jfli
