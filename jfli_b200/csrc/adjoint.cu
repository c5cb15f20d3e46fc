// Adjoint (vector-Jacobian) kernels of the PM force step and the reversible KKD update.
//
// The force on a particle at x is F_a(x) = R_x[M_a], the CIC readout R of the force mesh
// M_a = -D_a P (rho - mean), rho = sum_q W(x_q - .) the CIC density, P the Poisson
// operator (-1/k^2, k = 0 -> 0) and D_a the 4-point finite difference. For a cotangent u
// per particle the transpose J^T u of dF/dx has two parts:
//   * readout: u . grad_x R_x[M] = grad_x R_x[sum_a u_a M_a]    (corners combined first)
//   * density: grad_x R_x[rho_bar], rho_bar = sum_a (-D_a P)^T Ubar_a = P(div_FD Ubar),
//     Ubar_a = CIC paint of the particles with weights u_a (D_a^T = -D_a, P^T = P).
// The reversible step (reference pm/solvers.py:258-411, backward loop
// pm/integrate.py:288-535) is  v' = v + k F(x);  x' = x + d v'.  Its reverse recomputes
// x = x' - d v', F(x), v = v' - k F(x); its VJP is
//   lambda_v_total = lambda_v' + d lambda_x',   dL/dd = <lambda_x', v'>,
//   dL/dk = <lambda_v_total, F(x)>,   lambda_x = lambda_x' + k J^T lambda_v_total.
#include "cic.cuh"
#include "common.cuh"
#include "internal.h"

namespace jfli {

constexpr int kAdjThreads = 256;
constexpr int kAdjCtasPerSm = 8;

// Block-wide sum of two doubles; thread 0 returns the result.
__device__ __forceinline__ void block_sum2(double& a, double& b) {
  __shared__ double sa[kAdjThreads / 32], sb[kAdjThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sa[w] = a;
    sb[w] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = 0.0;
    b = 0.0;
    for (int i = 0; i < kAdjThreads / 32; ++i) {  // fixed order
      a += sa[i];
      b += sb[i];
    }
  }
}

// CIC deposit of the vector u on a float4 mesh [cell] = (u0, u1, u2, 0), one 16-byte vector
// atomic per corner where three meshes take three scalar ones. The lanes hold consecutive
// particles of one z row (the grid-stride loop; the active lanes a prefix of the warp),
// with deposit_lane_merged's z merge: when lane L's
// upper-z corners are lane L+1's lower-z corners, lane L+1 receives lane L's vector and its
// four upper-z weights and adds them to its own lower-z deposits (one vector atomic per
// shared cell instead of two).
__device__ __forceinline__ void deposit_vec4_lane_merged(float4* mesh, const PGrid& g, const Cic1& cx, const Cic1& cy,
                                                         const Cic1& cz, const float u[3]) {
  const unsigned mask = __activemask();
  const int lane = threadIdx.x & 31;
  const int xy0 = cx.i0 * g.yz + cy.i0 * g.nz;
  const int lo = xy0 + cz.i0, hi = xy0 + cz.i1;
  const int next_lo = __shfl_down_sync(mask, lo, 1);
  const int prev_hi = __shfl_up_sync(mask, hi, 1);
  const bool give = lane < 31 && ((mask >> (lane + 1)) & 1u) && next_lo == hi;
  const bool take = lane > 0 && ((mask >> (lane - 1)) & 1u) && prev_hi == lo;
  const float p0 = __shfl_up_sync(mask, u[0], 1), p1 = __shfl_up_sync(mask, u[1], 1),
              p2 = __shfl_up_sync(mask, u[2], 1);
  const int xo[2] = {cx.i0 * g.yz, cx.i1 * g.yz}, yo[2] = {cy.i0 * g.nz, cy.i1 * g.nz};
  const float wx[2] = {cx.w0, cx.w1}, wy[2] = {cy.w0, cy.w1};
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const float wab = wx[a] * wy[b];
      const float up = wab * cz.w1;
      const float recv = __shfl_up_sync(mask, up, 1);
      const float wl = wab * cz.w0;
      float4 low = make_float4(wl * u[0], wl * u[1], wl * u[2], 0.f);
      if (take) {
        low.x += recv * p0;
        low.y += recv * p1;
        low.z += recv * p2;
      }
      atomicAdd(mesh + (xo[a] + yo[b] + cz.i0), low);
      if (!give) atomicAdd(mesh + (xo[a] + yo[b] + cz.i1), make_float4(up * u[0], up * u[1], up * u[2], 0.f));
    }
}

// The upper-x corners of a lane's previous particle in the column walk, held back in registers:
// when the lane's next particle, one Lagrangian plane further in x, has its lower-x corners in
// the same four cells, both go out in one atomic per cell.
struct VecCarry {
  int xo, yo0, yo1, z0, z1;  // cell offsets of the 2 (y) x 2 (z) corners: x ny nz, y nz, z
  float w[4];                // weights [y][z]
  float u[3];
  bool valid;
};

// Deposit, for every lane of a full warp, the vectors v of the 2 (y) x 2 (z) corners of one x
// plane, with the z merge of deposit_vec4_lane_merged. Lanes with `on` false deposit nothing.
__device__ __forceinline__ void deposit_vec4_plane(float4* mesh, bool on, int xo, int yo0, int yo1, int z0, int z1,
                                                   const float v[4][3]) {
  const int lane = threadIdx.x & 31;
  const int lo = on ? xo + yo0 + z0 : -1;
  const int hi = on ? xo + yo0 + z1 : -2;
  const int next_lo = __shfl_down_sync(0xffffffffu, lo, 1);
  const int prev_hi = __shfl_up_sync(0xffffffffu, hi, 1);
  const bool give = on && lane < 31 && next_lo == hi;
  const bool take = on && lane > 0 && prev_hi == lo;
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    float low[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float recv = __shfl_up_sync(0xffffffffu, v[2 * b + 1][a], 1);
      low[a] = take ? v[2 * b][a] + recv : v[2 * b][a];
    }
    const int row = xo + (b ? yo1 : yo0);
    if (on) {
      atomicAdd(mesh + (row + z0), make_float4(low[0], low[1], low[2], 0.f));
      if (!give)
        atomicAdd(mesh + (row + z1), make_float4(v[2 * b + 1][0], v[2 * b + 1][1], v[2 * b + 1][2], 0.f));
    }
  }
}

__device__ __forceinline__ void vec_carry_deposit(float4* mesh, VecCarry& c) {
  float v[4][3];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int a = 0; a < 3; ++a) v[q][a] = c.w[q] * c.u[a];
  deposit_vec4_plane(mesh, c.valid, c.xo, c.yo0, c.yo1, c.z0, c.z1, v);
  c.valid = false;
}

// CIC deposit of u in the column walk (full warps, lanes on consecutive z particles of one row,
// successive calls of a lane on successive x planes): the lower-x plane now, with the carry
// when its cells are the same (otherwise the carry goes out alone), the upper-x plane later.
__device__ __forceinline__ void deposit_vec4_carried(float4* mesh, const PGrid& g, const Cic1& cx, const Cic1& cy,
                                                     const Cic1& cz, const float u[3], VecCarry& c) {
  const int xo0 = cx.i0 * g.yz, yo0 = cy.i0 * g.nz, yo1 = cy.i1 * g.nz;
  const float wyz[4] = {cy.w0 * cz.w0, cy.w0 * cz.w1, cy.w1 * cz.w0, cy.w1 * cz.w1};
  const bool same = c.valid && c.xo == xo0 && c.yo0 == yo0 && c.z0 == cz.i0;
  if (c.valid && !same) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      atomicAdd(mesh + (c.xo + (q & 2 ? c.yo1 : c.yo0) + (q & 1 ? c.z1 : c.z0)),
                make_float4(c.w[q] * c.u[0], c.w[q] * c.u[1], c.w[q] * c.u[2], 0.f));
  }
  float v[4][3];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      v[q][a] = cx.w0 * wyz[q] * u[a];
      if (same) v[q][a] += c.w[q] * c.u[a];
    }
  deposit_vec4_plane(mesh, true, xo0, yo0, yo1, cz.i0, cz.i1, v);
  c.xo = cx.i1 * g.yz;
  c.yo0 = yo0;
  c.yo1 = yo1;
  c.z0 = cz.i0;
  c.z1 = cz.i1;
#pragma unroll
  for (int q = 0; q < 4; ++q) c.w[q] = cx.w1 * wyz[q];
#pragma unroll
  for (int a = 0; a < 3; ++a) c.u[a] = u[a];
  c.valid = true;
}

// Reverse kick + first half of the VJP of one reversible step, at the un-drifted
// positions x (relative displacements). Per particle:
//   F = R_x[force];  <lambda_x, v'> -> partial[1];  u = lambda_v + drift * lambda_x;
//   <u, F> -> partial[0];  v = v' - kick F;  lambda_v = u;  ubar_a += W * u_a.
// partials holds 2 doubles per CTA and batch entry, summed in a fixed order later.
// ubar: three meshes [3][cells] (kVec4 false) or one float4 mesh [cells] (kVec4 true).
// The arithmetic of one particle, on its values in registers: x, v, lx (lambda_x), lv
// (lambda_v) in; x (un-drifted when undrift), v (un-kicked) and lv (= u) out.
template <bool kVec4>
__device__ __forceinline__ void unkick_core(float x[3], float v[3], const float lx[3], float lv[3], bool undrift,
                                            const float* __restrict__ force, float kick, float drift,
                                            float* __restrict__ ubar, const PGrid& g, int i, int j, int k, double& sk,
                                            double& sd, VecCarry* carry = nullptr) {
  if (undrift) {
#pragma unroll
    for (int a = 0; a < 3; ++a) x[a] += v[a] * -drift;
  }
  const Cic1 cx = cic_rel(i, x[0], g.nx), cy = cic_rel(j, x[1], g.ny), cz = cic_rel(k, x[2], g.nz);
  float f[3];
  gather_force_mesh(force, g, cx, cy, cz, f[0], f[1], f[2]);
  float u[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    sd += (double)lx[a] * (double)v[a];
    u[a] = lv[a] + drift * lx[a];
    sk += (double)u[a] * (double)f[a];
    v[a] = v[a] - f[a] * kick;
    lv[a] = u[a];
  }
  if (kVec4 && carry) {
    deposit_vec4_carried(reinterpret_cast<float4*>(ubar), g, cx, cy, cz, u, *carry);
  } else if (kVec4) {
    deposit_vec4_lane_merged(reinterpret_cast<float4*>(ubar), g, cx, cy, cz, u);
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) deposit(ubar + (size_t)a * g.np, g, cx, cy, cz, u[a]);
  }
}

// One particle with its own 4-byte loads and stores. With undrift (the float4 form of the
// reverse sweep over stored potentials), disp holds x' on entry: the particle is first
// un-drifted, x = x' - drift v', and x is written back.
template <bool kVec4>
__device__ __forceinline__ void unkick_particle(float* __restrict__ disp, bool undrift, float* __restrict__ vel,
                                                const float* __restrict__ lam_x, float* __restrict__ lam_v,
                                                const float* __restrict__ force, float kick, float drift,
                                                float* __restrict__ ubar, const PGrid& g, unsigned p, int i, int j,
                                                int k, double& sk, double& sd) {
  float x[3], v[3], lx[3], lv[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    x[a] = disp[3 * p + a];
    v[a] = vel[3 * p + a];
    lx[a] = lam_x[3 * p + a];
    lv[a] = lam_v[3 * p + a];
  }
  unkick_core<kVec4>(x, v, lx, lv, undrift, force, kick, drift, ubar, g, i, j, k, sk, sd);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (undrift) disp[3 * p + a] = x[a];
    vel[3 * p + a] = v[a];
    lam_v[3 * p + a] = lv[a];
  }
}

// The 32 particles of one z row (lane = z offset; the row's arrays start 16-byte aligned):
// lanes 0..23 move each array's 384 bytes as float4 with streaming loads and stores
// through the warp's shared buffers (4 x 24 float4), and every lane reads and writes its
// own 3 floats there (stride 3, no bank conflicts): one 16-byte instruction per array and
// row where the lanes' own accesses take three 4-byte ones.
template <bool kVec4>
__device__ __forceinline__ void unkick_row(float* __restrict__ disp, bool undrift, float* __restrict__ vel,
                                           const float* __restrict__ lam_x, float* __restrict__ lam_v,
                                           const float* __restrict__ force, float kick, float drift,
                                           float* __restrict__ ubar, const PGrid& g, unsigned p0, int i, int j, int k,
                                           int lane, float4 (*buf)[24], double& sk, double& sd, float4 row[4],
                                           bool more, VecCarry& carry) {
  float4* d4 = reinterpret_cast<float4*>(disp + 3ull * p0);
  float4* v4 = reinterpret_cast<float4*>(vel + 3ull * p0);
  const float4* x4 = reinterpret_cast<const float4*>(lam_x + 3ull * p0);
  float4* l4 = reinterpret_cast<float4*>(lam_v + 3ull * p0);
  if (lane < 24) {
    buf[0][lane] = row[0];
    buf[1][lane] = row[1];
    buf[2][lane] = row[2];
    buf[3][lane] = row[3];
    if (more) {  // the row of the next plane, on its way while this one is worked on
      const unsigned q = 3u * (unsigned)g.yz / 4u + (unsigned)lane;
      row[0] = __ldcs(d4 + q);
      row[1] = __ldcs(v4 + q);
      row[2] = __ldcs(x4 + q);
      row[3] = __ldcs(l4 + q);
    }
  }
  __syncwarp();
  float x[3], v[3], lx[3], lv[3];
  const float* f0 = reinterpret_cast<const float*>(buf[0]);
  const float* f1 = reinterpret_cast<const float*>(buf[1]);
  const float* f2 = reinterpret_cast<const float*>(buf[2]);
  const float* f3 = reinterpret_cast<const float*>(buf[3]);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    x[a] = f0[3 * lane + a];
    v[a] = f1[3 * lane + a];
    lx[a] = f2[3 * lane + a];
    lv[a] = f3[3 * lane + a];
  }
  __syncwarp();
  unkick_core<kVec4>(x, v, lx, lv, undrift, force, kick, drift, ubar, g, i, j, k, sk, sd, &carry);
  float* w0 = reinterpret_cast<float*>(buf[0]);
  float* w1 = reinterpret_cast<float*>(buf[1]);
  float* w3 = reinterpret_cast<float*>(buf[3]);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    w0[3 * lane + a] = x[a];
    w1[3 * lane + a] = v[a];
    w3[3 * lane + a] = lv[a];
  }
  __syncwarp();
  if (lane < 24) {
    if (undrift) __stcs(d4 + lane, buf[0][lane]);
    __stcs(v4 + lane, buf[1][lane]);
    __stcs(l4 + lane, buf[3][lane]);
  }
  __syncwarp();
}

constexpr int kAdjBrickY = 8, kAdjBrickZ = 32;
constexpr int kUnkickCtas = 2;        // resident per SM (128 registers)
constexpr int kUnkickStrideCtas = 3;  // of the grid-stride form (80)

// How walk_columns cuts the columns. Up to 2^22 cells the meshes that are gathered from and painted
// are in L2, and equal ranges of planes, one per resident CTA, leave no last round (0). Larger
// meshes are taken in slabs of 8 planes, so that columns that share lines meet in L2. Un-kick,
// ranges against slabs: 64^3 12.3 and 19.5 us, 128^3 67 and 73, 192^3 290 and 249, 256^3 717 and
// 611, 384^3 2450 and 2146. (The forward pass gains nothing from ranges: 64^3 10.0 us against
// 9.7 with bricks, 128^3 46.6 and 46.6.)
inline int walk_depth(const MeshDims& d) { return d.cells() * d.batch <= (1ll << 22) ? 0 : 8; }

// The columns of 8 (y) x 32 (z) cells of a mesh (ny a multiple of 8, nz of 32), in pieces for each
// CTA: run(first y, first z, first x, last x + 1). depth 0: the planes of all columns, one column
// after the other, cut into one range per CTA, equal to a plane; otherwise pieces of `depth`
// planes, all columns of a slab before the next slab (walk_depth).
template <class Run>
__device__ __forceinline__ void walk_columns(const PGrid& g, int depth, Run run) {
  const unsigned nx = (unsigned)g.nx, tz = (unsigned)g.nz / kAdjBrickZ, columns = tz * ((unsigned)g.ny / kAdjBrickY);
  unsigned t = blockIdx.x, last = depth ? columns * ((nx + depth - 1) / depth) : 0;
  if (!depth) {
    const unsigned long long planes = (unsigned long long)columns * nx;
    t = (unsigned)(planes * blockIdx.x / gridDim.x);
    last = (unsigned)(planes * (blockIdx.x + 1) / gridDim.x);
  }
  while (t < last) {
    unsigned col, i0, i1;
    if (depth) {
      col = t % columns;
      i0 = t / columns * depth;
      i1 = min(nx, i0 + depth);
      t += gridDim.x;
    } else {
      col = t / nx;
      i0 = t - col * nx;
      i1 = min(nx, i0 + (last - t));
      t += i1 - i0;
    }
    run((int)(col / tz) * kAdjBrickY, (int)(col % tz) * kAdjBrickZ, (int)i0, (int)i1);
  }
}


// Work order of the float4 form: when nz is a multiple of 32 and ny of 8, a CTA of 8 warps
// walks 8 (y) x 32 (z) columns of Lagrangian cells along x, each warp on one z row (the z merge
// of the deposit needs consecutive z in a warp), so that the rows and planes whose particles
// share CIC corners gather and deposit on one SM close in time (as the forward particle
// pass). Otherwise a grid-stride walk, which needs fewer registers: bounded like the column walk,
// with two CTAs per SM, it took 10.3 us for 48^3 against 9.1 with three (72^3 23.7 and 24.2).
//
// Bound by L1 (gathers and atomics of 16 bytes a lane). 128^3: 88 us with pieces of 8 planes over
// 1184 CTAs (2.3 rounds of the resident ones), 78 with equal ranges, 76.7 with the next row's
// loads ahead of this one (128 registers, two CTAs per SM), 67 with the x merge of VecCarry.
template <bool kVec4, bool kWalk>
__global__ void __launch_bounds__(kAdjThreads, kWalk ? kUnkickCtas : kUnkickStrideCtas) k_adj_unkick_paint(
    float* __restrict__ disp, int undrift, float* __restrict__ vel, const float* __restrict__ lam_x,
    float* __restrict__ lam_v, const float* __restrict__ force, float kick, float drift, float* __restrict__ ubar,
    double* __restrict__ partials, PGrid g, int depth) {
  const long long b = blockIdx.y;
  disp += b * g.np * 3;
  vel += b * g.np * 3;
  lam_x += b * g.np * 3;
  lam_v += b * g.np * 3;
  force += b * g.np * 4;
  ubar += b * g.np * (kVec4 ? 4 : 3);
  double sk = 0.0, sd = 0.0;
  __shared__ float4 rowbuf[kWalk ? kAdjBrickY : 1][4][24];  // per warp: disp, vel, lam_x, lam_v of one z row
  if (kWalk) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool staged = ((reinterpret_cast<uintptr_t>(disp) | reinterpret_cast<uintptr_t>(vel) |
                          reinterpret_cast<uintptr_t>(lam_x) | reinterpret_cast<uintptr_t>(lam_v)) & 15) == 0;
    walk_columns(g, depth, [&](int jc, int kc, int i0, int i1) {
      const int j = jc + w, k = kc + lane;
      VecCarry carry;
      carry.valid = false;
      float4 row[4];
      if (staged && lane < 24) {
        const unsigned p0 = ((unsigned)i0 * (unsigned)g.ny + (unsigned)j) * (unsigned)g.nz + (unsigned)(k - lane);
        row[0] = __ldcs(reinterpret_cast<const float4*>(disp + 3ull * p0) + lane);
        row[1] = __ldcs(reinterpret_cast<const float4*>(vel + 3ull * p0) + lane);
        row[2] = __ldcs(reinterpret_cast<const float4*>(lam_x + 3ull * p0) + lane);
        row[3] = __ldcs(reinterpret_cast<const float4*>(lam_v + 3ull * p0) + lane);
      }
      for (int i = i0; i < i1; ++i) {
        const unsigned p = ((unsigned)i * (unsigned)g.ny + (unsigned)j) * (unsigned)g.nz + (unsigned)k;
        if (staged)
          unkick_row<kVec4>(disp, undrift != 0, vel, lam_x, lam_v, force, kick, drift, ubar, g, p - (unsigned)lane,
                            i, j, k, lane, rowbuf[kWalk ? w : 0], sk, sd, row, i + 1 < i1,
                            carry);
        else
          unkick_particle<kVec4>(disp, undrift != 0, vel, lam_x, lam_v, force, kick, drift, ubar, g, p, i, j, k, sk,
                                 sd);
      }
      if (staged) vec_carry_deposit(reinterpret_cast<float4*>(ubar), carry);
    });
  } else {
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < g.np; p += gridDim.x * blockDim.x) {
      int i, j, k;
      particle_ijk(g, p, i, j, k);
      unkick_particle<kVec4>(disp, undrift != 0, vel, lam_x, lam_v, force, kick, drift, ubar, g, p, i, j, k, sk, sd);
    }
  }
  block_sum2(sk, sd);
  if (threadIdx.x == 0) {
    double* dst = partials + 2 * (b * gridDim.x + blockIdx.x);
    dst[0] = sk;
    dst[1] = sd;
  }
}

// CIC paint of a vector per particle (u, 3 floats, particle grid layout) onto a float4
// mesh, cleared by the caller: the cotangent paint of the PGD correction's adjoint.
__global__ void k_paint_vec4(const float* __restrict__ disp, const float* __restrict__ u, float* __restrict__ ubar,
                             PGrid g) {
  const long long b = blockIdx.y;
  disp += b * g.np * 3;
  u += b * g.np * 3;
  ubar += b * g.np * 4;
  for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < g.np; p += gridDim.x * blockDim.x) {
    int i, j, k;
    particle_ijk(g, p, i, j, k);
    const Cic1 cx = cic_rel(i, disp[3 * p + 0], g.nx), cy = cic_rel(j, disp[3 * p + 1], g.ny),
               cz = cic_rel(k, disp[3 * p + 2], g.nz);
    const float uu[3] = {u[3 * p + 0], u[3 * p + 1], u[3 * p + 2]};
    deposit_vec4_lane_merged(reinterpret_cast<float4*>(ubar), g, cx, cy, cz, uu);
  }
}

cudaError_t paint_vec4(const float* disp, const float* u, float* ubar, const MeshDims& d, cudaStream_t s) {
  k_paint_vec4<<<particle_grid_dims(d.cells(), d.batch, 256, 16), 256, 0, s>>>(disp, u, ubar, make_pgrid(d));
  note_launch();
  return cudaGetLastError();
}

// out(c) = [accumulate ? out(c) : 0] + sum_a D_a (alpha u_a + beta w_a)(c), with
// D_a f(c) = [8 (f(c+e_a) - f(c-e_a)) - (f(c+2e_a) - f(c-2e_a))] / 12. Component a of
// cell c is at index c * cell_stride + a * comp_stride (SoA meshes: 1, cells; AoS
// particle grids: 3, 1). w may be null.
__global__ void k_div_fd(const float* __restrict__ u, float alpha, const float* __restrict__ w, float beta,
                         long long cell_stride, long long comp_stride, int accumulate, float* __restrict__ out,
                         PGrid g) {
  grid_wait();
  const long long b = blockIdx.y;
  u += b * g.np * (cell_stride == 4 ? 4 : 3);
  if (w) w += b * g.np * 3;
  out += b * g.np;
  const float s = 1.0f / 12.0f;
  for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < g.np; p += gridDim.x * blockDim.x) {
    int c3[3];
    particle_ijk(g, p, c3[0], c3[1], c3[2]);
    const int n3[3] = {g.nx, g.ny, g.nz};
    const int st[3] = {g.yz, g.nz, 1};
    const int base = c3[0] * g.yz + c3[1] * g.nz + c3[2];
    float acc = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int rest = base - c3[a] * st[a];
      float v[4];
      const int off[4] = {-2, -1, 1, 2};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const long long q = (long long)(rest + wrap1(c3[a] + off[t], n3[a]) * st[a]);
        float val = alpha * u[q * cell_stride + a * comp_stride];
        if (w) val += beta * w[q * cell_stride + a * comp_stride];
        v[t] = val;
      }
      acc += (8.0f * (v[2] - v[1]) - (v[3] - v[0])) * s;
    }
    out[p] = accumulate ? out[p] + acc : acc;
  }
}

// The same of a float4 mesh (x, y, z, 0) with ny a multiple of 8 and nz of 32: CTAs of 8 x 32 threads
// walk columns along x. A thread loads its cell's 16 bytes once, three planes ahead, and keeps
// the x components of five planes in registers; the y and z components of a plane go through
// shared memory with two cells more on either side. The stencil form above loads 12 words, each
// 16 bytes from the next lane's, and is bound by L1. Stencil and this form: 64^3 4.4 and 5.3 us
// (few planes per CTA, each a round trip to L2), 96^3 10.0 and 8.4, 128^3 20.4 and 14.7, 192^3 62
// and 47, 256^3 164 and 100.
constexpr int kDivCtas = 5;  // resident per SM

__global__ void __launch_bounds__(kAdjThreads, kDivCtas) k_div_march(const float4* __restrict__ u, float alpha,
                                                                     int accumulate, float* __restrict__ out, PGrid g,
                                                                     int depth) {
  grid_wait();
  __shared__ float ys[2][kAdjBrickY + 4][kAdjBrickZ];
  __shared__ float zs[2][kAdjBrickY][kAdjBrickZ + 4];
  const long long b = blockIdx.y;
  u += b * g.np;
  out += b * g.np;
  const float s = 1.0f / 12.0f;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // threads 0..127 fetch the y halo (rows -2, -1, 8, 9), 128..159 the z halo (cells -2, -1, 32, 33)
  const bool hy = w < 4, hz = w == 4;
  const int hrow = w < 2 ? w : w + kAdjBrickY;  // row of ys
  const int zrow = lane >> 2, zcol = (lane & 3) < 2 ? (lane & 3) : (lane & 3) + kAdjBrickZ;
  walk_columns(g, depth, [&](int jc, int kc, int i0, int i1) {
    const int j = jc + w, k = kc + lane;
    const float4* cell = u + (j * g.nz + k);
    const float* halo = nullptr;
    if (hy) halo = &u[wrap1(jc + hrow - 2, g.ny) * g.nz + k].y;
    if (hz) halo = &u[(jc + zrow) * g.nz + wrap1(kc + zcol - 2, g.nz)].z;
    auto plane = [&](int i) { return (long long)wrap1(i, g.nx) * g.yz; };
    float xm2 = alpha * cell[plane(i0 - 2)].x, xm1 = alpha * cell[plane(i0 - 1)].x;
    float4 c0 = cell[plane(i0)], c1 = cell[plane(i0 + 1)], c2 = cell[plane(i0 + 2)];
    float h = halo ? halo[4 * plane(i0)] : 0.f;
    int buf = 0;
    for (int i = i0; i < i1; ++i, buf ^= 1) {
      const float4 next = i + 1 < i1 ? cell[plane(i + 3)] : c2;
      ys[buf][w + 2][lane] = alpha * c0.y;
      zs[buf][w][lane + 2] = alpha * c0.z;
      if (hy) ys[buf][hrow][lane] = alpha * h;
      if (hz) zs[buf][zrow][zcol] = alpha * h;
      if (halo && i + 1 < i1) h = halo[4 * plane(i + 1)];
      __syncthreads();  // the other buffer is written only after this plane's barrier
      float acc = (8.0f * (alpha * c1.x - xm1) - (alpha * c2.x - xm2)) * s;
      acc += (8.0f * (ys[buf][w + 3][lane] - ys[buf][w + 1][lane]) - (ys[buf][w + 4][lane] - ys[buf][w][lane])) * s;
      acc += (8.0f * (zs[buf][w][lane + 3] - zs[buf][w][lane + 1]) - (zs[buf][w][lane + 4] - zs[buf][w][lane])) * s;
      float* dst = out + (plane(i) + j * g.nz + k);
      *dst = accumulate ? *dst + acc : acc;
      xm2 = xm1;
      xm1 = alpha * c0.x;
      c0 = c1;
      c1 = c2;
      c2 = next;
    }
    __syncthreads();  // before the next piece writes a buffer that may still be read
  });
}

// lam_x += scale * grad_x R_x[h], h(corner) = rho_bar(corner) + sum_a u_a force_a(corner)
// (force AoS float4 per cell, as written by the force-mesh kernels),
// at relative positions disp. Either of rho_bar or (u, force) may be null. The gradient
// of the trilinear weights is one-sided at cell faces, like the derivative of the
// floor-based weights.
// The gradient of R_x[h] at one particle from its position x and vector u in registers:
// (gx, gy, gz) = grad_x R_x[rho_bar + sum_a u_a force_a].
__device__ __forceinline__ void adj_position_core(const float x[3], const float ua[3], bool use_u,
                                                  const float* __restrict__ rho_bar,
                                                  const float* __restrict__ force, const PGrid& g, int i, int j, int k,
                                                  float& gx, float& gy, float& gz) {
  const Cic1 cx = cic_rel(i, x[0], g.nx), cy = cic_rel(j, x[1], g.ny), cz = cic_rel(k, x[2], g.nz);
  const int xo[2] = {cx.i0 * g.yz, cx.i1 * g.yz}, yo[2] = {cy.i0 * g.nz, cy.i1 * g.nz}, zo[2] = {cz.i0, cz.i1};
  float h[2][2][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int bb = 0; bb < 2; ++bb)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int o = xo[a] + yo[bb] + zo[c];
        float v = rho_bar ? __ldg(rho_bar + o) : 0.f;
        if (use_u) {
          const float4 f = __ldg(reinterpret_cast<const float4*>(force) + o);
          v += ua[0] * f.x + ua[1] * f.y + ua[2] * f.z;
        }
        h[a][bb][c] = v;
      }
  const float wx[2] = {cx.w0, cx.w1}, wy[2] = {cy.w0, cy.w1}, wz[2] = {cz.w0, cz.w1};
  gx = 0.f;
  gy = 0.f;
  gz = 0.f;
#pragma unroll
  for (int bb = 0; bb < 2; ++bb)
#pragma unroll
    for (int c = 0; c < 2; ++c) gx += wy[bb] * wz[c] * (h[1][bb][c] - h[0][bb][c]);
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int c = 0; c < 2; ++c) gy += wx[a] * wz[c] * (h[a][1][c] - h[a][0][c]);
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int bb = 0; bb < 2; ++bb) gz += wx[a] * wy[bb] * (h[a][bb][1] - h[a][bb][0]);
}

__device__ __forceinline__ void adj_position_particle(const float* __restrict__ disp, const float* __restrict__ u,
                                                      const float* __restrict__ rho_bar,
                                                      const float* __restrict__ force, float scale,
                                                      float* __restrict__ lam_x, const PGrid& g, unsigned p, int i,
                                                      int j, int k) {
  const float x[3] = {disp[3 * p + 0], disp[3 * p + 1], disp[3 * p + 2]};
  const bool use_u = u && force;
  float ua[3] = {0.f, 0.f, 0.f};
  if (use_u) {
    ua[0] = u[3 * p + 0];
    ua[1] = u[3 * p + 1];
    ua[2] = u[3 * p + 2];
  }
  float gx, gy, gz;
  adj_position_core(x, ua, use_u, rho_bar, force, g, i, j, k, gx, gy, gz);
  lam_x[3 * p + 0] += scale * gx;
  lam_x[3 * p + 1] += scale * gy;
  lam_x[3 * p + 2] += scale * gz;
}

__global__ void __launch_bounds__(256) k_adj_position(const float* __restrict__ disp, const float* __restrict__ u,
                                                      const float* __restrict__ rho_bar,
                                                      const float* __restrict__ force, float scale,
                                                      float* __restrict__ lam_x, PGrid g) {
  const long long b = blockIdx.y;
  disp += b * g.np * 3;
  lam_x += b * g.np * 3;
  if (u) u += b * g.np * 3;
  if (force) force += b * g.np * 4;
  if (rho_bar) rho_bar += b * g.np;
  // (staging its rows through shared memory, as the un-kick does, measured 10% slower)
  for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < g.np; p += gridDim.x * blockDim.x) {
    int i, j, k;
    particle_ijk(g, p, i, j, k);
    adj_position_particle(disp, u, rho_bar, force, scale, lam_x, g, p, i, j, k);
  }
}

// ----------------------------------------------------------------------------------
static dim3 adj_grid(const MeshDims& d) { return particle_grid_dims(d.cells(), d.batch, kAdjThreads, kAdjCtasPerSm); }

// The grid of the float4 un-kick, whose partials sum_adjoint_partials adds up: its resident CTAs.
// No larger than adj_grid, the grid of the other form, all of whose partials the caller sums.
static bool unkick_walks(const MeshDims& d) { return d.nz % kAdjBrickZ == 0 && d.ny % kAdjBrickY == 0; }

static dim3 unkick_grid(const MeshDims& d) {
  const int ctas = unkick_walks(d) ? kUnkickCtas : kUnkickStrideCtas;
  const long long resident = max(1ll, (long long)ctas * sm_count() / d.batch);
  dim3 grid = adj_grid(d);
  if (resident < grid.x) grid.x = (unsigned)resident;
  return grid;
}

size_t adjoint_partials_count(const MeshDims& d) { return (size_t)2 * adj_grid(d).x * d.batch; }

// out[b][2] = sums of the per-CTA partials of batch entry b: each thread adds a strided
// slice, then a shared-memory tree in a fixed order (deterministic).
__global__ void __launch_bounds__(256) k_sum_partials(const double* __restrict__ partials, int nctas,
                                                      double* __restrict__ out) {
  grid_wait();
  __shared__ double sk[256], sd[256];
  const double* p = partials + 2ll * nctas * blockIdx.x;
  double a = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < nctas; i += 256) {
    a += p[2 * i];
    c += p[2 * i + 1];
  }
  sk[threadIdx.x] = a;
  sd[threadIdx.x] = c;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      sk[threadIdx.x] += sk[threadIdx.x + w];
      sd[threadIdx.x] += sd[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[2 * blockIdx.x] = sk[0];
    out[2 * blockIdx.x + 1] = sd[0];
  }
}

cudaError_t sum_adjoint_partials(const double* partials, const MeshDims& d, double* out, cudaStream_t s) {
  launch_next(overlap_starts(d.cells() * d.batch), k_sum_partials, d.batch, 256, 0, s, partials,
              (int)unkick_grid(d).x, out);
  note_launch();
  return cudaGetLastError();
}

cudaError_t adjoint_unkick_paint(const float* disp, float* vel, const float* lam_x, float* lam_v, const float* force,
                                 float kick, float drift, float* ubar, double* partials, const MeshDims& d,
                                 cudaStream_t s, bool vec4, float* undrift_disp) {
  // without undrift_disp the kernel only reads the positions
  float* dp = undrift_disp ? undrift_disp : const_cast<float*>(disp);
  const int undrift = undrift_disp != nullptr;
  cudaError_t e = cudaMemsetAsync(ubar, 0, sizeof(float) * (vec4 ? 4 : 3) * (size_t)d.cells() * d.batch, s);
  if (e != cudaSuccess) return e;
  if (vec4 && unkick_walks(d))
    k_adj_unkick_paint<true, true><<<unkick_grid(d), kAdjThreads, 0, s>>>(dp, undrift, vel, lam_x, lam_v, force, kick,
                                                                          drift, ubar, partials, make_pgrid(d),
                                                                          walk_depth(d));
  else if (vec4)
    k_adj_unkick_paint<true, false><<<unkick_grid(d), kAdjThreads, 0, s>>>(dp, undrift, vel, lam_x, lam_v, force, kick,
                                                                           drift, ubar, partials, make_pgrid(d), 0);
  else
    k_adj_unkick_paint<false, false><<<adj_grid(d), kAdjThreads, 0, s>>>(dp, undrift, vel, lam_x, lam_v, force, kick,
                                                                         drift, ubar, partials, make_pgrid(d), 0);
  note_launch();
  return cudaGetLastError();
}

cudaError_t divergence_fd(const float* u, float alpha, const float* w, float beta, int aos, int accumulate,
                          float* out, const MeshDims& d, cudaStream_t s) {
  // aos 0: three meshes; 1: particle grids (3 floats per cell); 2: float4 meshes
  const long long cell_stride = aos == 2 ? 4 : (aos ? 3 : 1);
  const long long comp_stride = aos ? 1 : d.cells();
  if (aos == 2 && w == nullptr && d.ny % kAdjBrickY == 0 && d.nz % kAdjBrickZ == 0 &&
      d.cells() * d.batch >= (1ll << 19)) {
    const long long planes = d.cells() / (kAdjBrickY * kAdjBrickZ);
    const long long resident = max(1ll, (long long)kDivCtas * sm_count() / d.batch);
    launch_next(overlap_starts(d.cells() * d.batch), k_div_march, dim3((unsigned)min(planes, resident), d.batch),
                kAdjThreads, 0, s, reinterpret_cast<const float4*>(u), alpha, accumulate, out, make_pgrid(d),
                walk_depth(d));
    note_launch();
    return cudaGetLastError();
  }
  launch_next(overlap_starts(d.cells() * d.batch), k_div_fd, particle_grid_dims(d.cells(), d.batch, 256, 16), 256, 0, s,
              u, alpha, w, beta, cell_stride, comp_stride, accumulate, out, make_pgrid(d));
  note_launch();
  return cudaGetLastError();
}

cudaError_t adjoint_position(const float* disp, const float* u, const float* rho_bar, const float* force, float scale,
                             float* lam_x, const MeshDims& d, cudaStream_t s) {
  k_adj_position<<<particle_grid_dims(d.cells(), d.batch, 256, 16), 256, 0, s>>>(disp, u, rho_bar, force, scale,
                                                                                lam_x, make_pgrid(d));
  note_launch();
  return cudaGetLastError();
}

}  // namespace jfli
