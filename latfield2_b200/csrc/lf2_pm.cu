// lf2_pm.cu -- kernels of the differentiable particle-mesh chain: CIC deposit
// and gather on particles kept in one order for a whole call (sorted by
// brick and cell when the call starts, no rebinning, so that gradients stay
// attached to their slots), the kick-drift update, a periodic 27-point
// stencil as the grid operator, the hand-written adjoints of all of them,
// and the permutations of the particle state into that order and of the
// gradients back.
//
//   deposit   rho(v)   += m_p / res^3 * W(v - x_p)            (scalarProjectionCIC)
//   gather    G_p       = sum_k W_k(x_p) F(corner_k)           (updateVel CIC kick)
//   kick      v_p      += dt * G_p
//   drift     off_p    += dt/res * v_p, carry into the cell    (move_particles_simple)
//   stencil   F_c(g)    = sum_o S[c][o] rho(g + o), o in {-1,0,1}^3
// with W = wx*wy*wz, wx = 1 - fx or fx, f the in-cell offset (cell units).
// Adjoints (gradients with respect to the inputs, given the output gradient):
//   deposit   dL/dm_p   = 1/res^3 * sum_k W_k gR(corner_k)
//             dL/df_p   = m_p/res^3 * sum_k dW_k/df gR(corner_k)
//   gather    gF(corner_k) += W_k gG_p          (a CIC deposit of gG)
//             dL/df_p  += sum_k dW_k/df (gG_p . F(corner_k))
//   stencil   gR(h)     = sum_c sum_o S[c][o] gF_c(h - o)
//             dL/dS[c][o] = sum_g gF_c(g) rho(g + o)
// dW/dfx = (bx ? 1 : -1) * wy * wz, etc.  Offsets and their gradients are in
// cell units; positions in box units are (cell + off) * res.  The force field
// F and its gradient are stored as one float4 (x, y, z, unused) per site, so
// that a corner is one 16-byte load and one vector atomic.
#include <cuda_runtime.h>

#include <algorithm>

#include "lf2_deposit_common.cuh"
#include "lf2_internal.h"

namespace lf2 {

namespace {

constexpr int PM_THREADS = 256;

inline int grid_for(int64_t n, int threads)
{
  int64_t g = (n + threads - 1) / threads;
  if (g > 148 * 32) g = 148 * 32;
  return (int)(g > 0 ? g : 1);
}

struct Corners {
  int32_t site[8];  // (a lattice has fewer than 2^31 sites)
  float w[8];
  float dw[8][3];
};

__device__ __forceinline__ void corners(const Geom& g, int32_t c, const float* off3, int64_t p,
                                        Corners& k)
{
  int x, y, z;
  cell_xyz(g, c, x, y, z);
  const int xs[2] = {x, x + 1 < g.n[0] ? x + 1 : 0};
  const int ys[2] = {y, y + 1 < g.n[1] ? y + 1 : 0};
  const int zs[2] = {z, z + 1 < g.n[2] ? z + 1 : 0};
  const float f[3] = {off3[3 * p], off3[3 * p + 1], off3[3 * p + 2]};
  const float h[3] = {1.0f - f[0], 1.0f - f[1], 1.0f - f[2]};
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int bx = (q >> 2) & 1, by = (q >> 1) & 1, bz = q & 1;
    const float wx = bx ? f[0] : h[0], wy = by ? f[1] : h[1], wz = bz ? f[2] : h[2];
    k.site[q] = (int32_t)site_index(g, xs[bx], ys[by], zs[bz]);
    k.w[q] = wx * wy * wz;
    k.dw[q][0] = (bx ? 1.0f : -1.0f) * wy * wz;
    k.dw[q][1] = (by ? 1.0f : -1.0f) * wx * wz;
    k.dw[q][2] = (bz ? 1.0f : -1.0f) * wx * wy;
  }
}

__global__ void k_pm_deposit(Geom g, int64_t np, const int32_t* __restrict__ cell,
                             const float* __restrict__ off3, const float* __restrict__ mass,
                             float gmass, float inv_vol, float* __restrict__ rho)
{
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
       p += (int64_t)gridDim.x * blockDim.x) {
    Corners k;
    corners(g, cell[p], off3, p, k);
    const float m = (mass ? mass[p] : gmass) * inv_vol;
#pragma unroll
    for (int q = 0; q < 8; q++) atomicAdd(&rho[k.site[q]], k.w[q] * m);
  }
}

// Fixed-point form of the chain's deposit (contexts in LF2_DEPOSIT_FIXED64):
// every corner's weight is the library's deterministic integer weight
// (fixed_corner, 2^-32 units), times the particle's mass relative to the
// largest mass M of the call in 2^-24 units; the integer sums (64-bit global
// atomics) do not depend on the order, and are converted once:
// rho += (float)sum * (M / res^3 * 2^-32).
__global__ void k_pm_mass_max(int64_t np, const float* __restrict__ mass, uint32_t* mmax)
{
  uint32_t m = 0u;
#pragma unroll 8
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
       p += (int64_t)gridDim.x * blockDim.x)
    m = max(m, __float_as_uint(fmaxf(mass[p], 0.0f)));  // non-negative floats order as integers
  m = __reduce_max_sync(0xffffffffu, m);
  // (most warps find the maximum there already: no queue at one address)
  if ((threadIdx.x & 31) == 0 && m > *reinterpret_cast<volatile uint32_t*>(mmax)) atomicMax(mmax, m);
}

__global__ void k_pm_deposit_fixed(Geom g, int64_t np, const int32_t* __restrict__ cell,
                                   const float* __restrict__ off3, const float* __restrict__ mass,
                                   const uint32_t* __restrict__ mmax, unsigned long long* __restrict__ acc)
{
  const float inv_m = mass ? 1.0f / __uint_as_float(*mmax) : 0.0f;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = cell[p];
    int x, y, z;
    cell_xyz(g, c, x, y, z);
    const int xs[2] = {x, x + 1 < g.n[0] ? x + 1 : 0};
    const int ys[2] = {y, y + 1 < g.n[1] ? y + 1 : 0};
    const int zs[2] = {z, z + 1 < g.n[2] ? z + 1 : 0};
    const uint32_t ux = weight_q(off3[3 * p]), uy = weight_q(off3[3 * p + 1]), uz = weight_q(off3[3 * p + 2]);
    const uint32_t qx[2] = {(1u << 31) - ux, ux}, qy[2] = {(1u << 31) - uy, uy}, qz[2] = {(1u << 31) - uz, uz};
    const uint64_t mq = mass ? (uint64_t)__float2uint_rn(fminf(__fmul_rn(mass[p], inv_m), 1.0f) * 16777216.0f) : 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int bx = (q >> 2) & 1, by = (q >> 1) & 1, bz = q & 1;
      uint64_t w = fixed_corner(qx[bx], qy[by], qz[bz]);
      if (mass) w = (w * mq + (1ull << 23)) >> 24;
      atomicAdd(&acc[site_index(g, xs[bx], ys[by], zs[bz])], (unsigned long long)w);
    }
  }
}

// Brick-tiled forms of the two deposits, for particles grouped by brick
// (brick_start[b] .. brick_start[b+1] hold the particles that were in brick
// b when the chain sorted its state; a particle that has since drifted out
// of the brick goes straight to the global sums).  A CTA adds its particles'
// corner weights into the brick's (BRICK+1)^3 vertex tile in shared memory,
// then the tile's non-zero sums go to the global field with one atomic each:
// 4913 global atomics per tile instead of 8 per particle.  Both keep integer
// sums, a low word whose carry goes to a high word: the fixed-point weights,
// or the FP32 products in a unit set by the largest (CompUnit; a
// floating-point shared atomic is a compare-and-swap loop), a small product's
// rest below the unit going straight to the field.  The CTA of a
// brick takes its first `part` particles; what a brick holds beyond those is
// shared out among CTAs by their slots, since each adds to the field on its
// own (one CTA took 1.4 ms for a brick of 131k particles at 256^3).
//
// Particles sorted by cell put whole warps into dense cells, whose lanes
// would add to the same words one after the other: a warp whose lanes lie in
// at most DENSE_RUNS runs of one cell sums each run with warp reductions
// first.
constexpr int DENSE_RUNS = 3;

__device__ __forceinline__ bool in_brick(int x, int y, int z, int x0, int y0, int z0)
{
  return (unsigned)(x - x0) < (unsigned)BRICK && (unsigned)(y - y0) < (unsigned)BRICK &&
         (unsigned)(z - z0) < (unsigned)BRICK;
}

// The group's range of brick b, clamped to the particle arrays.
__device__ __forceinline__ void group_range(const int64_t* brick_start, int64_t b, int64_t np,
                                            int64_t& p0, int64_t& p1)
{
  p0 = min(max(brick_start[b], (int64_t)0), np);
  p1 = min(max(brick_start[b + 1], p0), np);
}

// Vertex (x0 + i, y0 + j, z0 + k) of a brick tile, wrapped periodically.
__device__ __forceinline__ int64_t tile_site(const Geom& g, int t, int x0, int y0, int z0)
{
  int x = x0 + t % TILE, y = y0 + (t / TILE) % TILE, z = z0 + t / (TILE * TILE);
  x -= x >= g.n[0] ? g.n[0] : 0;
  y -= y >= g.n[1] ? g.n[1] : 0;
  z -= z >= g.n[2] ? g.n[2] : 0;
  return site_index(g, x, y, z);
}

// Brick of slot p: the last b with brick_start[b] <= p.
__device__ __forceinline__ int64_t brick_of_slot(const int64_t* brick_start, int64_t nb, int64_t p)
{
  int64_t lo = 0, hi = nb - 1;
  while (lo < hi) {
    const int64_t mid = lo + ((hi - lo + 1) >> 1);
    if (brick_start[mid] <= p) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Adds the integer w (below 2^33, or any signed 64-bit value) of every lane
// to the tile's words at t.
__device__ __forceinline__ void tile_add(uint32_t* lo, uint32_t* hi, int t, long long w)
{
  const uint32_t wl = (uint32_t)(unsigned long long)w;
  const uint32_t old = atomicAdd(&lo[t], wl);
  const int up = (int)(w >> 32) + ((uint32_t)(old + wl) < old ? 1 : 0);
  if (up) atomicAdd(reinterpret_cast<int*>(&hi[t]), up);
}

// FIXED: acc += integer weights (times the masses relative to *mmax);
// otherwise rho += FP32 products.  CTA u < nbricks: brick u's first `part`
// particles; CTA nbricks + r: what the slots [r part, (r + 1) part) hold of
// bricks beyond their first `part` particles (only the brick of the first slot
// can: one that starts later has no more than its first ones in the range).
template <bool FIXED>
__global__ void __launch_bounds__(256)
    k_pm_deposit_tile(Geom g, int64_t np, const int64_t* __restrict__ brick_start, int part,
                      const int32_t* __restrict__ cell, const float* __restrict__ off3,
                      const float* __restrict__ mass, const uint32_t* __restrict__ mmax, float gmass,
                      float inv_vol, unsigned long long* __restrict__ acc, float* __restrict__ rho)
{
  __shared__ uint32_t lo[TILE3], hi[TILE3];
  __shared__ unsigned s_max;
  const float inv_m = FIXED && mass ? 1.0f / __uint_as_float(*mmax) : 0.0f;
  const int lane = threadIdx.x & 31;
  int64_t b, p0, p1;
  if (blockIdx.x < g.nbricks) {
    b = blockIdx.x;
    group_range(brick_start, b, np, p0, p1);
    p1 = min(p1, p0 + part);
  } else {
    const int64_t r0 = ((int64_t)blockIdx.x - g.nbricks) * part, r1 = min(r0 + part, np);
    b = brick_of_slot(brick_start, g.nbricks, r0);
    group_range(brick_start, b, np, p0, p1);
    p0 = max(p0 + part, r0);
    p1 = min(p1, r1);
    if (p0 >= p1) return;
  }
  for (int t = threadIdx.x; t < TILE3; t += blockDim.x) lo[t] = hi[t] = 0u;
  CompUnit cu{1.0f, 1.0f, true};
  if (!FIXED)  // (slots may exceed 32 bits)
    cu = comp_unit<0>(mass ? mass + p0 : nullptr, inv_vol, gmass * inv_vol, nullptr, nullptr, nullptr,
                      0u, (int)(p1 - p0), &s_max);
  __syncthreads();
  int bx, by, bz;
  brick_coords(g, b, bx, by, bz);
  const int x0 = bx * BRICK, y0 = by * BRICK, z0 = bz * BRICK;
  // the next trip's particle is read while this one's is added
  int32_t c_next = 0;
  float f_next[3] = {0.f, 0.f, 0.f}, m_next = gmass;
  auto fetch = [&](int64_t p) {
    if (p >= p1) return;
    c_next = cell[p];
    f_next[0] = off3[3 * p], f_next[1] = off3[3 * p + 1], f_next[2] = off3[3 * p + 2];
    if (mass) m_next = mass[p];
  };
  fetch(p0 + threadIdx.x);
  for (int64_t q0 = p0; q0 < p1; q0 += blockDim.x) {
    const int64_t p = q0 + threadIdx.x;
    const bool on = p < p1;
    int x, y, z;
    cell_xyz(g, c_next, x, y, z);
    const float f[3] = {f_next[0], f_next[1], f_next[2]};
    float m = m_next;
    fetch(p + blockDim.x);
    uint32_t qx[2], qy[2], qz[2];
    uint64_t mq = 0;
    if (FIXED) {
      qx[1] = weight_q(f[0]), qy[1] = weight_q(f[1]), qz[1] = weight_q(f[2]);
      qx[0] = (1u << 31) - qx[1], qy[0] = (1u << 31) - qy[1], qz[0] = (1u << 31) - qz[1];
      if (mass) mq = (uint64_t)__float2uint_rn(fminf(__fmul_rn(m, inv_m), 1.0f) * 16777216.0f);
    } else {
      m *= inv_vol;
    }
    // corner q's integer contribution
    auto weight = [&](int q) -> long long {
      const int cx = (q >> 2) & 1, cy = (q >> 1) & 1, cz = q & 1;
      if (FIXED) {
        uint64_t w = fixed_corner(qx[cx], qy[cy], qz[cz]);
        if (mass) w = (w * mq + (1ull << 23)) >> 24;
        return (long long)w;
      }
      const float w = (cx ? f[0] : 1.0f - f[0]) * (cy ? f[1] : 1.0f - f[1]) * (cz ? f[2] : 1.0f - f[2]);
      const float term = w * m, v = __fmul_rn(term, cu.unit);  // |v| < 2^21, in units of 2^31 quanta
      const float h = __fadd_rn(v, 12582912.0f);
      const float r = __fsub_rn(v, __fsub_rn(h, 12582912.0f));
      return ((long long)(__float_as_int(h) - 0x4B400000) << 31) +
             (long long)__float2int_rn(__fmul_rn(r, 2147483648.0f));
    };
    const bool tiled = on && cu.ok && in_brick(x, y, z, x0, y0, z0);
    const int t0 = (x - x0) + TILE * ((y - y0) + TILE * (z - z0));
    if (!FIXED && tiled) {  // terms that are no whole number of quanta: their rests to the field
      const float least = fminf(f[0], 1.0f - f[0]) * fminf(f[1], 1.0f - f[1]) * fminf(f[2], 1.0f - f[2]) *
                          fabsf(m);
      if (may_have_rest(__fmul_rn(least, cu.unit))) {
#pragma unroll 1
        for (int q = 0; q < 8; q++) {
          const int cx = (q >> 2) & 1, cy = (q >> 1) & 1, cz = q & 1;
          const float w = (cx ? f[0] : 1.0f - f[0]) * (cy ? f[1] : 1.0f - f[1]) * (cz ? f[2] : 1.0f - f[2]);
          const float rest = comp_rest(w * m, cu.unit, cu.quantum);
          if (rest != 0.0f)
            atomicAdd(&rho[tile_site(g, t0 + cx + TILE * (cy + TILE * cz), x0, y0, z0)], rest);
        }
      }
    }
    // runs of lanes in one cell
    const int key = tiled ? t0 : -1 - lane;
    const int before = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || key != before);
    if (__popc(heads) <= DENSE_RUNS) {
      for (unsigned rest = heads; rest; rest &= rest - 1) {
        const int first = __ffs(rest) - 1, next = __ffs(rest & (rest - 1));
        const bool mine = lane >= first && (next == 0 || lane < next - 1);
        const int t = __shfl_sync(0xffffffffu, key, first);
        if (t < 0) continue;  // a lane that is not in the tile: below
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const long long w = mine ? weight(q) : 0ll;
          // 32 values below 2^52: the sums of 20-bit pieces stay below 2^31
          const long long sum =
              (long long)__reduce_add_sync(0xffffffffu, (unsigned)(w & 0xfffff)) +
              ((long long)__reduce_add_sync(0xffffffffu, (unsigned)((w >> 20) & 0xfffff)) << 20) +
              ((long long)__reduce_add_sync(0xffffffffu, (int)(w >> 40)) << 40);
          if (lane == q)
            tile_add(lo, hi, t + ((q >> 2) & 1) + TILE * (((q >> 1) & 1) + TILE * (q & 1)), sum);
        }
      }
    } else if (tiled) {
#pragma unroll
      for (int q = 0; q < 8; q++)
        tile_add(lo, hi, t0 + ((q >> 2) & 1) + TILE * (((q >> 1) & 1) + TILE * (q & 1)), weight(q));
    }
    if (on && !tiled) {  // drifted out of the brick since the sort, or no common unit
      const int xs[2] = {x, x + 1 < g.n[0] ? x + 1 : 0};
      const int ys[2] = {y, y + 1 < g.n[1] ? y + 1 : 0};
      const int zs[2] = {z, z + 1 < g.n[2] ? z + 1 : 0};
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int cx = (q >> 2) & 1, cy = (q >> 1) & 1, cz = q & 1;
        const int64_t site = site_index(g, xs[cx], ys[cy], zs[cz]);
        if (FIXED) {
          atomicAdd(&acc[site], (unsigned long long)weight(q));
        } else {
          const float w = (cx ? f[0] : 1.0f - f[0]) * (cy ? f[1] : 1.0f - f[1]) * (cz ? f[2] : 1.0f - f[2]);
          atomicAdd(&rho[site], w * m);
        }
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < TILE3; t += blockDim.x) {
    const unsigned long long v = ((unsigned long long)hi[t] << 32) | lo[t];
    if (!v) continue;
    if (FIXED)
      atomicAdd(&acc[tile_site(g, t, x0, y0, z0)], v);
    else
      atomicAdd(&rho[tile_site(g, t, x0, y0, z0)], __ll2float_rn((long long)v) * cu.quantum);
  }
}

__global__ void k_pm_fixed_to_rho(int64_t ns, unsigned long long* __restrict__ acc, const float* mass,
                                  const uint32_t* __restrict__ mmax, float gmass, float inv_vol,
                                  float* __restrict__ rho, uint32_t* flags)
{
  const float m = mass ? __uint_as_float(*mmax) : gmass;
  const float scale = ldexpf(__fmul_rn(m, inv_vol), -32);
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < ns;
       s += (int64_t)gridDim.x * blockDim.x) {
    const long long q = (long long)acc[s];
    if (q < 0) set_flag(flags, ERR_FIXED_OVERFLOW);
    rho[s] = __fadd_rn(rho[s], __fmul_rn(__ll2float_rn(q), scale));
    acc[s] = 0ull;  // clean for the next call
  }
}

__global__ void k_pm_gather(Geom g, int64_t np, const int32_t* __restrict__ cell,
                            const float* __restrict__ off3, const float4* __restrict__ F4,
                            float* __restrict__ out3)
{
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
       p += (int64_t)gridDim.x * blockDim.x) {
    Corners k;
    corners(g, cell[p], off3, p, k);
    float a[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float4 f = __ldg(F4 + k.site[q]);
      a[0] = fmaf(k.w[q], f.x, a[0]);
      a[1] = fmaf(k.w[q], f.y, a[1]);
      a[2] = fmaf(k.w[q], f.z, a[2]);
    }
    for (int c = 0; c < 3; c++) out3[3 * p + c] = a[c];
  }
}

// v += dt_kick * G; off += dtn * v with the carry into the cell (as the
// library's drift, LATfield2 move_particles_simple in cell units).
__global__ void k_pm_kick_drift(Geom g, int64_t np, int32_t* __restrict__ cell, float* __restrict__ off3,
                                float* __restrict__ vel3, const float* __restrict__ G3, float dtk,
                                float dtn, uint32_t* flags)
{
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = cell[p];
    int xyz[3];
    cell_xyz(g, c, xyz[0], xyz[1], xyz[2]);
    for (int d = 0; d < 3; d++) {
      float v = vel3[3 * p + d];
      if (G3) v = __fmaf_rn(dtk, G3[3 * p + d], v);
      vel3[3 * p + d] = v;
      float o = __fmaf_rn(dtn, v, off3[3 * p + d]);
      if (!isfinite(o)) {
        set_flag(flags, ERR_NONFINITE);
        continue;
      }
      const float fl = floorf(o);
      o = __fsub_rn(o, fl);
      int carry = (int)fl;
      if (o >= 1.0f) {
        o = 0.0f;
        carry += 1;
      }
      off3[3 * p + d] = o;
      xyz[d] = wrap_add(xyz[d], carry, g.n[d]);
    }
    cell[p] = (int32_t)site_index(g, xyz[0], xyz[1], xyz[2]);
  }
}

// The gather, the kick and the drift of one chain step in one pass, with
// the arithmetic of k_pm_gather and k_pm_kick_drift (the same results bit
// for bit) and no gathered field written in between.  The new state may go
// to other arrays, so that the old one stays as a checkpoint without a copy.
__global__ void k_pm_gather_kick_drift(Geom g, int64_t np, const int32_t* cell, const float* off3,
                                       const float* vel3, const float4* __restrict__ F4, float dtk,
                                       float dtn, int32_t* cell_out, float* off_out, float* vel_out,
                                       uint32_t* flags)
{
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = cell[p];
    const float o3[3] = {off3[3 * p], off3[3 * p + 1], off3[3 * p + 2]};
    const float v3[3] = {vel3[3 * p], vel3[3 * p + 1], vel3[3 * p + 2]};
    Corners k;
    corners(g, c, o3, 0, k);
    float a[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float4 f = __ldg(F4 + k.site[q]);
      a[0] = fmaf(k.w[q], f.x, a[0]);
      a[1] = fmaf(k.w[q], f.y, a[1]);
      a[2] = fmaf(k.w[q], f.z, a[2]);
    }
    int xyz[3];
    cell_xyz(g, c, xyz[0], xyz[1], xyz[2]);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float v = __fmaf_rn(dtk, a[d], v3[d]);
      vel_out[3 * p + d] = v;
      float o = __fmaf_rn(dtn, v, o3[d]);
      if (!isfinite(o)) {
        set_flag(flags, ERR_NONFINITE);
        off_out[3 * p + d] = o3[d];
        continue;
      }
      const float fl = floorf(o);
      o = __fsub_rn(o, fl);
      int carry = (int)fl;
      if (o >= 1.0f) {
        o = 0.0f;
        carry += 1;
      }
      off_out[3 * p + d] = o;
      xyz[d] = wrap_add(xyz[d], carry, g.n[d]);
    }
    cell_out[p] = (int32_t)site_index(g, xyz[0], xyz[1], xyz[2]);
  }
}

// FIRST: the adjoint of the loss, the first of a backward pass: g_rho is the
// loss weights, scaled by `scale`, and the gradients are written (g_vel3
// zero) instead of added to.
template <bool FIRST>
__global__ void k_pm_deposit_adj(Geom g, int64_t np, const int32_t* __restrict__ cell,
                                 const float* __restrict__ off3, const float* __restrict__ mass,
                                 float gmass, float inv_vol, const float* __restrict__ g_rho, float scale,
                                 float* __restrict__ g_off3, float* __restrict__ g_mass,
                                 float* __restrict__ g_vel3)
{
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
       p += (int64_t)gridDim.x * blockDim.x) {
    Corners k;
    corners(g, cell[p], off3, p, k);
    float s = 0.f, d[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 8; q++) {
      float gr = __ldg(g_rho + k.site[q]);
      if (FIRST) gr = __fmul_rn(gr, scale);
      s = fmaf(k.w[q], gr, s);
      for (int c = 0; c < 3; c++) d[c] = fmaf(k.dw[q][c], gr, d[c]);
    }
    const float m = (mass ? mass[p] : gmass) * inv_vol;
    if (g_mass) g_mass[p] = FIRST ? s * inv_vol : g_mass[p] + s * inv_vol;
    if (g_off3)
      for (int c = 0; c < 3; c++) g_off3[3 * p + c] = FIRST ? m * d[c] : g_off3[3 * p + c] + m * d[c];
    if (FIRST)
      for (int c = 0; c < 3; c++) g_vel3[3 * p + c] = 0.0f;
  }
}

// sum_i w[i] rho[i] in FP64, in a fixed order: a partial sum per CTA, then
// one CTA.
constexpr int LOSS_THREADS = 256;

__device__ __forceinline__ double block_sum(double v, double* sh)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += sh[w];
  return v;
}

__global__ void __launch_bounds__(LOSS_THREADS) k_pm_loss(int64_t n, const float* __restrict__ w,
                                                          const float* __restrict__ rho, double* partial)
{
  __shared__ double sh[LOSS_THREADS / 32];
  double v = 0.0;
#pragma unroll 4
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v = fma((double)__ldg(w + i), (double)__ldg(rho + i), v);
  v = block_sum(v, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

__global__ void __launch_bounds__(LOSS_THREADS) k_pm_loss_sum(int n, const double* __restrict__ partial,
                                                              double* loss)
{
  __shared__ double sh[LOSS_THREADS / 32];
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += LOSS_THREADS) v += partial[i];
  v = block_sum(v, sh);
  if (threadIdx.x == 0) *loss = v;
}

// Sum over the lanes of a warp of 24 values each: lane l < 24 returns the sum
// of value l (recursive halving: 31 exchanges for up to 32 values).
__device__ __forceinline__ float reduce24(float (&v)[32])
{
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) {
    const bool upper = lane & h;
#pragma unroll
    for (int i = 0; i < h; i++) {
      const float give = upper ? v[i] : v[i + h], keep = upper ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, h);
    }
  }
  return v[0];
}

// Gather adjoint.  STEP: with the adjoint of the drift and the kick before it
// (g_vel += dtn g_off, then the gradient of the gathered force is dtk g_vel),
// otherwise that gradient is given (gG3).  Bound by the vector atomics on the
// gradient field; the particles come sorted by cell, so a warp in a dense
// region adds to a few vertices only: where its lanes lie in at most
// DENSE_RUNS runs of one cell, each run's 24 sums are formed in the warp and
// added once (at one particle per cell the same costs more than the atomics
// it saves).
template <bool STEP>
__global__ void __launch_bounds__(PM_THREADS)
    k_pm_gather_adj(Geom g, int64_t np, const int32_t* __restrict__ cell, const float* __restrict__ off3,
                    const float4* __restrict__ F4, const float* __restrict__ gG3, float4* __restrict__ gF4,
                    float* __restrict__ g_off3, float* __restrict__ g_vel3, float dtk, float dtn)
{
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); p0 < np; p0 += stride) {
    const int64_t p = min(p0 + lane, np - 1);
    const bool on = p0 + lane < np;
    Corners k;
    const int32_t c = cell[p];
    corners(g, c, off3, p, k);
    float gg[3], go[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      if (STEP || g_off3) go[d] = g_off3[3 * p + d];
      if (STEP) {
        const float gv = __fadd_rn(g_vel3[3 * p + d], __fmul_rn(dtn, go[d]));
        if (on) g_vel3[3 * p + d] = gv;
        gg[d] = __fmul_rn(dtk, gv);
      } else {
        gg[d] = gG3[3 * p + d];
      }
    }
    if (gF4) {
      const int key = on ? c : -1;
      const int before = __shfl_up_sync(0xffffffffu, key, 1);
      const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || key != before);
      if (__popc(heads) <= DENSE_RUNS) {
        for (unsigned rest = heads; rest; rest &= rest - 1) {
          const int first = __ffs(rest) - 1, next = __ffs(rest & (rest - 1));
          const bool mine = on && lane >= first && (next == 0 || lane < next - 1);
          float v[32];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            v[q] = mine ? k.w[q] * gg[0] : 0.f;
            v[8 + q] = mine ? k.w[q] * gg[1] : 0.f;
            v[16 + q] = mine ? k.w[q] * gg[2] : 0.f;
            v[24 + q] = 0.f;
          }
          const float sum = reduce24(v);
          const float sy = __shfl_down_sync(0xffffffffu, sum, 8), sz = __shfl_down_sync(0xffffffffu, sum, 16);
          // the run's sites: corner q of its first lane
          int32_t site = 0;
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const int32_t s = __shfl_sync(0xffffffffu, k.site[q], first);
            if (lane == q) site = s;
          }
          if (lane < 8 && p0 + first < np)
            atomicAdd(&gF4[site], make_float4(sum, sy, sz, 0.f));
        }
      } else if (on) {
#pragma unroll
        for (int q = 0; q < 8; q++)
          atomicAdd(&gF4[k.site[q]], make_float4(k.w[q] * gg[0], k.w[q] * gg[1], k.w[q] * gg[2], 0.f));
      }
    }
    if (g_off3 && on) {
      float d[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const float4 f = __ldg(F4 + k.site[q]);
        const float dot = fmaf(gg[0], f.x, fmaf(gg[1], f.y, gg[2] * f.z));
#pragma unroll
        for (int i = 0; i < 3; i++) d[i] = fmaf(k.dw[q][i], dot, d[i]);
      }
#pragma unroll
      for (int i = 0; i < 3; i++) g_off3[3 * p + i] = go[i] + d[i];
    }
  }
}

// The three stencil kernels work on tiles of SX x SY x SZ sites, one CTA of
// SX x SY threads per tile; each thread walks one z-column of the tile.  The
// tile's input with a 1-site periodic halo is staged in shared memory, so
// every input value is read from global memory about 1.5 times.
constexpr int SX = 32, SY = 8, SZ = 8;
constexpr int HX = SX + 2, HY = SY + 2, HZ = SZ + 2;
constexpr int STENCIL_THREADS = SX * SY;

struct Tile {
  int x0, y0, z0, tx, ty;
};

__device__ inline Tile tile_of()
{
  return {(int)blockIdx.x * SX, (int)blockIdx.y * SY, (int)blockIdx.z * SZ, (int)threadIdx.x % SX,
          (int)threadIdx.x / SX};
}

// The tile's input with its halo, one warp per row of HX sites; `put` takes
// halo index and global site.  The wrapped coordinates are laid down once
// (`w`), and the loop over a warp's rows is unrolled, so that their loads are
// in flight together.
constexpr int HALO_WRAP = HX + HY + HZ;

template <typename Put>
__device__ __forceinline__ void halo_rows(const Geom& g, int x0, int y0, int z0, int32_t* w, Put put)
{
  const int t = threadIdx.x, lane = t & 31;
  if (t < HX) w[t] = wrap_add(x0, t - 1, g.n[0]);
  else if (t < HX + HY) w[t] = g.n[0] * wrap_add(y0, t - HX - 1, g.n[1]);
  else if (t < HALO_WRAP) w[t] = g.n[0] * g.n[1] * wrap_add(z0, t - HX - HY - 1, g.n[2]);
  __syncthreads();
  const int xa = w[lane], xb = w[32 + (lane < HX - 32 ? lane : 0)];
#pragma unroll
  for (int it = 0; it < (HY * HZ + STENCIL_THREADS / 32 - 1) / (STENCIL_THREADS / 32); it++) {
    const int row = (t >> 5) + it * (STENCIL_THREADS / 32);
    if (row < HY * HZ) {
      const int base = w[HX + row % HY] + w[HX + HY + row / HY];  // (fewer than 2^31 sites)
      put(row * HX + lane, base + xa);
      if (lane < HX - 32) put(row * HX + 32 + lane, base + xb);
    }
  }
}

// The three stencil kernels are bound by issue: 81 multiply-adds per site and
// the loads of their operands.  A thread keeps the 81 weights (or sums) in
// registers and walks its z column plane by plane: the 9 values of a plane
// serve the three sites whose stencils touch it, so that a site costs 9
// shared loads per input component instead of 27, and no weight is read again.

// The weights into registers, by way of shared memory.  (Volatile loads: an
// ordinary one would be repeated for every plane to save registers.)
__device__ __forceinline__ void weights_to_registers(const float* S, float* sh, float (&s)[81])
{
  if (threadIdx.x < 81) sh[threadIdx.x] = __ldg(S + threadIdx.x);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 81; q++) s[q] = reinterpret_cast<volatile float*>(sh)[q];
}

// F_c(g) = sum_o S[c][o] rho(g + o); o = (dz, dy, dx) in {-1,0,1}^3,
// S index c*27 + (dz+1)*9 + (dy+1)*3 + (dx+1), added in ascending o.
__global__ void __launch_bounds__(STENCIL_THREADS) k_stencil(Geom g, const float* __restrict__ rho,
                                                             const float* __restrict__ S,
                                                             float4* __restrict__ F4)
{
  __shared__ float r[HZ * HY * HX];
  __shared__ int32_t wrap[HALO_WRAP];
  const Tile T = tile_of();
  __shared__ float sh[81];
  float s[81];
  weights_to_registers(S, sh, s);
  halo_rows(g, T.x0, T.y0, T.z0, wrap, [&](int t, int site) { r[t] = __ldg(rho + site); });
  __syncthreads();
  const int x = T.x0 + T.tx, y = T.y0 + T.ty;
  if (x >= g.n[0] || y >= g.n[1]) return;
  // a[m]: the site one plane below (m = 0), at, or above the plane read
  float a[3][3] = {};
  const int64_t plane = (int64_t)g.n[0] * g.n[1];
  int64_t site = site_index(g, x, y, T.z0) - plane;
#pragma unroll
  for (int k = 0; k < HZ; k++) {
    float v[9];
#pragma unroll
    for (int o = 0; o < 9; o++) v[o] = r[(k * HY + T.ty + o / 3) * HX + T.tx + o % 3];
#pragma unroll
    for (int m = 0; m < 3; m++)  // the site's plane k sits at dz = 1 - m
#pragma unroll
      for (int o = 0; o < 9; o++)
#pragma unroll
        for (int c = 0; c < 3; c++) a[m][c] = fmaf(s[c * 27 + (2 - m) * 9 + o], v[o], a[m][c]);
    if (k >= 2 && T.z0 + k - 2 < g.n[2])
      F4[site] = make_float4(a[0][0], a[0][1], a[0][2], 0.f);
    if (k >= 1) site += plane;
#pragma unroll
    for (int c = 0; c < 3; c++) a[0][c] = a[1][c], a[1][c] = a[2][c], a[2][c] = 0.f;
  }
}

// gR(h) = sum_c sum_o S[c][o] gF_c(h - o), added in ascending o: the planes
// from the top of the column down.
__global__ void __launch_bounds__(STENCIL_THREADS) k_stencil_adj_rho(Geom g,
                                                                     const float4* __restrict__ gF4,
                                                                     const float* __restrict__ S,
                                                                     float* __restrict__ g_rho)
{
  __shared__ float f[3][HZ * HY * HX];
  __shared__ int32_t wrap[HALO_WRAP];
  const Tile T = tile_of();
  __shared__ float sh[81];
  float s[81];
  weights_to_registers(S, sh, s);
  halo_rows(g, T.x0, T.y0, T.z0, wrap, [&](int t, int site) {
    const float4 v = __ldg(gF4 + site);
    f[0][t] = v.x;
    f[1][t] = v.y;
    f[2][t] = v.z;
  });
  __syncthreads();
  const int x = T.x0 + T.tx, y = T.y0 + T.ty;
  if (x >= g.n[0] || y >= g.n[1]) return;
  float a[3] = {};  // the site above, at, or below the plane read
  const int64_t plane = (int64_t)g.n[0] * g.n[1];
#pragma unroll
  for (int k = HZ - 1; k >= 0; k--) {
#pragma unroll
    for (int o = 0; o < 9; o++) {
      // h - o: halo offset (1 - d) per axis
      const int t = (k * HY + T.ty + 2 - o / 3) * HX + T.tx + 2 - o % 3;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const float v = f[c][t];
        // plane k is h - dz with dz = -1 for the site below it, 0, 1
        a[2] = fmaf(s[c * 27 + o], v, a[2]);
        a[1] = fmaf(s[c * 27 + 9 + o], v, a[1]);
        a[0] = fmaf(s[c * 27 + 18 + o], v, a[0]);
      }
    }
    const int z = T.z0 + k;  // the site above plane k is complete
    if (k < SZ && z < g.n[2]) g_rho[site_index(g, x, y, T.z0) + plane * k] += a[0];
    a[0] = a[1], a[1] = a[2], a[2] = 0.f;
  }
}

// gS[c][o] = sum_g gF_c(g) rho(g + o).  A CTA takes one component c
// (blockIdx.y); every thread keeps its 27 sums in registers over the z-columns
// of the CTA's tiles (three CTAs per SM); the warps then reduce them with
// shuffles, the CTA adds its 8 warps in order and writes its third of a row
// of `partial`; k_stencil_adj_S_sum adds the rows in a fixed order.  The next
// tile's input is copied to shared memory (cp.async) while a tile is summed
// (128^3: 58 us, 37 with the copies).
__device__ __forceinline__ void copy_async(float* dst, const float* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

__global__ void __launch_bounds__(STENCIL_THREADS, 3) k_stencil_adj_S(Geom g, int ntx, int nty, int ntiles,
                                                                      const float4* __restrict__ gF4,
                                                                      const float* __restrict__ rho,
                                                                      float* __restrict__ partial)
{
  __shared__ float r[2][HZ * HY * HX];
  __shared__ int32_t wrap[HALO_WRAP];
  __shared__ float red[STENCIL_THREADS / 32][27];
  const int tx = threadIdx.x % SX, ty = threadIdx.x / SX;
  const float* gF = reinterpret_cast<const float*>(gF4) + blockIdx.y;
  const int64_t plane = (int64_t)g.n[0] * g.n[1];
  float acc[27], q[SZ], q_next[SZ];
#pragma unroll
  for (int k = 0; k < 27; k++) acc[k] = 0.f;
  // the input of a tile: its halo to shared memory, the thread's column of gF
  auto fetch = [&](int tile, float* buf) {
    const int x0 = (tile % ntx) * SX, y0 = (tile / ntx % nty) * SY, z0 = tile / (ntx * nty) * SZ;
    halo_rows(g, x0, y0, z0, wrap, [&](int t, int site) { copy_async(buf + t, rho + site); });
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int x = x0 + tx, y = y0 + ty;
    const bool on = x < g.n[0] && y < g.n[1];
    const int64_t site = on ? site_index(g, x, y, z0) : 0;
#pragma unroll
    for (int k = 0; k < SZ; k++)
      q_next[k] = on && z0 + k < g.n[2] ? __ldg(gF + 4 * (site + plane * k)) : 0.f;
  };
  if ((int)blockIdx.x < ntiles) fetch(blockIdx.x, r[0]);
  int cur = 0;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, cur ^= 1) {
#pragma unroll
    for (int k = 0; k < SZ; k++) q[k] = q_next[k];
    __syncthreads();  // the other buffer and `wrap` are read
    const bool more = tile + (int)gridDim.x < ntiles;
    if (more) {
      fetch(tile + gridDim.x, r[cur ^ 1]);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();  // every thread's copies of this tile have landed
    // plane k of the halo lies above site k - 2, at site k - 1 and below site k
    const float* buf = r[cur];
#pragma unroll
    for (int k = 0; k < HZ; k++) {
#pragma unroll
      for (int o = 0; o < 9; o++) {
        const float v = buf[(k * HY + ty + o / 3) * HX + tx + o % 3];
#pragma unroll
        for (int m = 0; m < 3; m++)
          if (k - m >= 0 && k - m < SZ) acc[9 * m + o] = fmaf(q[k - m], v, acc[9 * m + o]);
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 27; k++) {
    float v = acc[k];
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    if (lane == 0) red[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < 27) {
    float v = 0.f;
    for (int w = 0; w < STENCIL_THREADS / 32; w++) v += red[w][threadIdx.x];
    partial[(size_t)blockIdx.x * 81 + blockIdx.y * 27 + threadIdx.x] = v;
  }
}

__global__ void k_stencil_adj_S_sum(int ntiles, const float* __restrict__ partial, float* gS)
{
  __shared__ float red[4][81];
  // 4 x 81 threads: each sums a quarter of the tiles, then the quarters
  const int out = threadIdx.x % 81, q = threadIdx.x / 81;
  if (threadIdx.x < 324) {
    float v = 0.f;
    for (int t = q; t < ntiles; t += 4) v += partial[(size_t)t * 81 + out];
    red[q][out] = v;
  }
  __syncthreads();
  if (threadIdx.x < 81) gS[threadIdx.x] += (red[0][threadIdx.x] + red[1][threadIdx.x]) +
                                           (red[2][threadIdx.x] + red[3][threadIdx.x]);
}

// ------------------------------------------------------ chain state
// Cell and FP32 in-cell offset of a box-unit FP64 position: u = pos * inv_res
// (the product by the reciprocal, as a division by a scalar runs on the GPU
// in torch), floor, the offset u - floor(u) rounded to FP32 with the carry of
// an offset that rounds up to 1, then the periodic wrap.
__device__ __forceinline__ int32_t pos_state(const Geom& g, const double* p, double inv_res,
                                             float o[3])
{
  long long ci[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double u = __dmul_rn(p[d], inv_res);
    double fl = floor(u);
    float od = __double2float_rn(__dsub_rn(u, fl));
    if (od >= 1.0f) {
      od = 0.0f;
      fl = __dadd_rn(fl, 1.0);
    }
    long long c = (long long)fl % (long long)g.n[d];
    if (c < 0) c += g.n[d];
    ci[d] = c;
    o[d] = od;
  }
  return (int32_t)(ci[0] + (long long)g.n[0] * (ci[1] + (long long)g.n[1] * ci[2]));
}

// Sort key of a cell: its brick, then its place in the brick (x fastest),
// so that sorted particles come grouped by brick and by cell inside it.
__device__ __forceinline__ int32_t brick_key(const Geom& g, int32_t c)
{
  int x, y, z;
  cell_xyz(g, c, x, y, z);
  const int64_t b = brick_of(g, x, y, z);
  return (int32_t)(b * (BRICK * BRICK * BRICK) + (x % BRICK) + BRICK * ((y % BRICK) + BRICK * (z % BRICK)));
}

// A particle's 32-byte record: one 32-byte access where the array starts on
// such a boundary (WIDE), so that the permutations' random accesses touch
// their sector once; two of 16 bytes otherwise.
struct Record {
  uint32_t w[8];
};

template <bool WIDE>
__device__ __forceinline__ Record load_record(const uint4* rec, int64_t i)
{
  Record r;
  const uint4* p = rec + 2 * i;
  if (WIDE) {
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]),
                   "=r"(r.w[6]), "=r"(r.w[7])
                 : "l"(p));
  } else {
    const uint4 a = p[0], b = p[1];
    r.w[0] = a.x, r.w[1] = a.y, r.w[2] = a.z, r.w[3] = a.w;
    r.w[4] = b.x, r.w[5] = b.y, r.w[6] = b.z, r.w[7] = b.w;
  }
  return r;
}

template <bool WIDE>
__device__ __forceinline__ void store_record(uint4* rec, int64_t i, const Record& r)
{
  uint4* p = rec + 2 * i;
  if (WIDE) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r.w[0]), "r"(r.w[1]),
                 "r"(r.w[2]), "r"(r.w[3]), "r"(r.w[4]), "r"(r.w[5]), "r"(r.w[6]), "r"(r.w[7])
                 : "memory");
  } else {
    p[0] = make_uint4(r.w[0], r.w[1], r.w[2], r.w[3]);
    p[1] = make_uint4(r.w[4], r.w[5], r.w[6], r.w[7]);
  }
}

inline bool wide_records(const void* rec) { return (reinterpret_cast<uintptr_t>(rec) & 31) == 0; }

// Caller order, coalesced: the sort key of every particle (brick_key) and
// its 32-byte record (cell, offsets, FP32 velocity, FP32 mass), so that the
// permutation reads one full sector per particle.
template <bool WIDE>
__global__ void k_pm_pack(Geom g, int64_t np, const double* __restrict__ pos,
                          const double* __restrict__ vel, const double* __restrict__ mass,
                          double inv_res, int32_t* __restrict__ key, uint4* __restrict__ rec)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np;
       i += (int64_t)gridDim.x * blockDim.x) {
    float o[3];
    const int32_t c = pos_state(g, pos + 3 * i, inv_res, o);
    key[i] = brick_key(g, c);
    const float m = mass ? __double2float_rn(mass[i]) : 0.0f;
    const Record r{{(uint32_t)c, __float_as_uint(o[0]), __float_as_uint(o[1]), __float_as_uint(o[2]),
                    __float_as_uint(__double2float_rn(vel[3 * i])),
                    __float_as_uint(__double2float_rn(vel[3 * i + 1])),
                    __float_as_uint(__double2float_rn(vel[3 * i + 2])), __float_as_uint(m)}};
    store_record<WIDE>(rec, i, r);
  }
}

// Slot i takes the record of particle order[i].
template <bool WIDE>
__global__ void k_pm_unpack(int64_t np, const int64_t* __restrict__ order, const uint4* __restrict__ rec,
                            int32_t* __restrict__ cell, float* __restrict__ off3,
                            float* __restrict__ vel3, float* __restrict__ m)
{
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int U = 4;  // records in flight per thread
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < np; i0 += U * stride) {
    Record r[U];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i0 + u * stride < np) r[u] = load_record<WIDE>(rec, order[i0 + u * stride]);
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t i = i0 + u * stride;
      if (i >= np) continue;
      cell[i] = (int32_t)r[u].w[0];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        off3[3 * i + k] = __uint_as_float(r[u].w[1 + k]);
        vel3[3 * i + k] = __uint_as_float(r[u].w[4 + k]);
      }
      if (m) m[i] = __uint_as_float(r[u].w[7]);
    }
  }
}

// First slot of every brick among cells sorted by brick_key (bricks without
// particles start where the next one does; brick_start[nb] = np): one thread
// per brick, a binary search over the sorted slots.
__global__ void k_pm_brick_start(Geom g, int64_t np, const int32_t* __restrict__ cell,
                                 int64_t* __restrict__ brick_start)
{
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b <= g.nbricks;
       b += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = np;  // first slot whose brick is b or later
    while (lo < hi) {
      const int64_t mid = lo + ((hi - lo) >> 1);
      const int32_t c = cell[mid];
      int x, y, z;
      cell_xyz(g, c, x, y, z);
      if (brick_of(g, x, y, z) < b) lo = mid + 1;
      else hi = mid;
    }
    brick_start[b] = lo;
  }
}

// The gradients of slot i as the 32-byte record of particle order[i] (one
// full sector written per particle; no partial-sector writes).
template <bool WIDE>
__global__ void k_pm_grads_scatter(int64_t np, const int64_t* __restrict__ order,
                                   const float* __restrict__ g_off3, const float* __restrict__ g_vel3,
                                   const float* __restrict__ g_m, uint4* __restrict__ rec)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Record r{{__float_as_uint(g_off3[3 * i]), __float_as_uint(g_off3[3 * i + 1]),
                    __float_as_uint(g_off3[3 * i + 2]), __float_as_uint(g_m[i]),
                    __float_as_uint(g_vel3[3 * i]), __float_as_uint(g_vel3[3 * i + 1]),
                    __float_as_uint(g_vel3[3 * i + 2]), 0u}};
    store_record<WIDE>(rec, order[i], r);
  }
}

// Caller order, coalesced: the records into FP64 gradients (the offset
// gradient times inv_res: per box unit).
template <bool WIDE>
__global__ void k_pm_grads_unpack(int64_t np, const uint4* __restrict__ rec, double inv_res,
                                  double* __restrict__ g_pos, double* __restrict__ g_vel,
                                  double* __restrict__ g_mass)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Record r = load_record<WIDE>(rec, i);
    g_mass[i] = (double)__uint_as_float(r.w[3]);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      g_pos[3 * i + k] = __dmul_rn((double)__uint_as_float(r.w[k]), inv_res);
      g_vel[3 * i + k] = (double)__uint_as_float(r.w[4 + k]);
    }
  }
}

}  // namespace

inline dim3 stencil_grid(const Geom& g)
{
  return dim3((g.n[0] + SX - 1) / SX, (g.n[1] + SY - 1) / SY, (g.n[2] + SZ - 1) / SZ);
}

inline int64_t stencil_tiles(const Geom& g)
{
  const dim3 d = stencil_grid(g);
  return (int64_t)d.x * d.y * d.z;
}

// Rows of partial sums of the weight gradient: three CTAs per SM, three to a row.
inline int stencil_rows(const lf2_ctx* c) { return c->num_sms; }

// The chain's deposit into rho (+=): per particle, or brick-tiled when
// brick_start is given (particles grouped by brick, nbricks + 1 entries).
cudaError_t launch_pm_deposit(lf2_ctx* c, int64_t np, const int64_t* brick_start, const int32_t* cell,
                              const float* off3, const float* mass, float gmass, float* rho)
{
  const double vol = c->res * c->res * c->res;
  const float inv_vol = (float)(1.0 / vol);
  const Geom g = c->g;
  const unsigned nb = (unsigned)g.nbricks;
  // particles of one CTA: twice a brick's at one per cell, fewer where that
  // would leave SMs without two CTAs
  const int part = (int)std::max<int64_t>(1024, std::min<int64_t>(2 * BRICK * BRICK * BRICK,
                                                                  np / (2 * c->num_sms)));
  const unsigned extra = (unsigned)((np + part - 1) / part);
  if (c->mode == LF2_DEPOSIT_FIXED64) {
    // integer sums in the context's scratch (zero between calls)
    if (!c->pm_acc) {
      cudaError_t e = cudaMalloc(&c->pm_acc, sizeof(unsigned long long) * (size_t)g.nsites + 256);
      if (e != cudaSuccess) return e;
      e = cudaMemsetAsync(c->pm_acc, 0, sizeof(unsigned long long) * (size_t)g.nsites + 256, c->stream);
      if (e != cudaSuccess) return e;
    }
    uint32_t* mmax = reinterpret_cast<uint32_t*>(c->pm_acc + g.nsites);
    if (mass) {
      cudaError_t e = cudaMemsetAsync(mmax, 0, sizeof(uint32_t), c->stream);
      if (e != cudaSuccess) return e;
      c->launches += 1;
      k_pm_mass_max<<<grid_for((np + 7) / 8, PM_THREADS), PM_THREADS, 0, c->stream>>>(np, mass, mmax);
    }
    c->launches += 2;
    if (brick_start)
      k_pm_deposit_tile<true><<<nb + extra, 256, 0, c->stream>>>(g, np, brick_start, part, cell,
                                                                off3, mass, mmax, gmass, inv_vol, c->pm_acc,
                                                                nullptr);
    else
      k_pm_deposit_fixed<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(g, np, cell, off3,
                                                                                mass, mmax, c->pm_acc);
    k_pm_fixed_to_rho<<<grid_for(g.nsites, PM_THREADS), PM_THREADS, 0, c->stream>>>(
        g.nsites, c->pm_acc, mass, mmax, gmass, inv_vol, rho, c->flags);
    return cudaGetLastError();
  }
  c->launches += 1;
  if (brick_start)
    k_pm_deposit_tile<false><<<nb + extra, 256, 0, c->stream>>>(g, np, brick_start, part, cell,
                                                               off3, mass, nullptr, gmass, inv_vol,
                                                               nullptr, rho);
  else
    k_pm_deposit<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(g, np, cell, off3, mass,
                                                                          gmass, inv_vol, rho);
  return cudaGetLastError();
}

cudaError_t launch_pm(lf2_ctx* c, int op, int64_t np, const int32_t* cell, const float* off3,
                      const float* mass, float gmass, const float* in_a, const float* in_b,
                      float* out_a, float* out_b, float dta, float dtb, int32_t* cell_rw,
                      float* off_rw, float* vel_rw)
{
  const double vol = c->res * c->res * c->res;
  const float inv_vol = (float)(1.0 / vol);
  const Geom g = c->g;
  switch (op) {
    case 0:  // deposit into out_a
      return launch_pm_deposit(c, np, nullptr, cell, off3, mass, gmass, out_a);
    case 1:  // gather in_a (F4) -> out_a (np x 3)
      c->launches += 1;
      k_pm_gather<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
          g, np, cell, off3, reinterpret_cast<const float4*>(in_a), out_a);
      break;
    case 2:  // kick (in_a = G, may be NULL) + drift
      c->launches += 1;
      k_pm_kick_drift<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
          g, np, cell_rw, off_rw, vel_rw, in_a, dta, dtb, c->flags);
      break;
    case 3:  // deposit adjoint: in_a = g_rho; out_a = g_off (+=), out_b = g_mass (+=)
      c->launches += 1;
      k_pm_deposit_adj<false><<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
          g, np, cell, off3, mass, gmass, inv_vol, in_a, 1.0f, out_a, out_b, nullptr);
      break;
    case 4:  // gather adjoint: in_a = F4, in_b = gG; out_a = gF4 (+=), out_b = g_off (+=)
      c->launches += 1;
      k_pm_gather_adj<false><<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
          g, np, cell, off3, reinterpret_cast<const float4*>(in_a), in_b,
          reinterpret_cast<float4*>(out_a), out_b, nullptr, 0.0f, 0.0f);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_stencil(lf2_ctx* c, int op, const float* a, const float* S, float* out,
                           float* partial)
{
  const Geom g = c->g;
  const dim3 grid = stencil_grid(g);
  if (op == 0) {  // a = rho -> out = F4
    c->launches += 1;
    k_stencil<<<grid, STENCIL_THREADS, 0, c->stream>>>(g, a, S, reinterpret_cast<float4*>(out));
  } else if (op == 1) {  // a = gF4 -> out = g_rho (+=)
    c->launches += 1;
    k_stencil_adj_rho<<<grid, STENCIL_THREADS, 0, c->stream>>>(
        g, reinterpret_cast<const float4*>(a), S, out);
  } else {  // a = gF4, S = rho -> out = gS (+=)
    c->launches += 2;
    const int ntiles = (int)stencil_tiles(g), ctas = std::min(ntiles, stencil_rows(c));
    k_stencil_adj_S<<<dim3(ctas, 3), STENCIL_THREADS, 0, c->stream>>>(
        g, (int)grid.x, (int)grid.y, ntiles, reinterpret_cast<const float4*>(a), S, partial);
    k_stencil_adj_S_sum<<<1, 352, 0, c->stream>>>(ctas, partial, out);
  }
  return cudaGetLastError();
}

size_t stencil_partial_floats(const lf2_ctx* c)
{
  return (size_t)std::min<int64_t>(stencil_tiles(c->g), stencil_rows(c)) * 81;
}

cudaError_t launch_pm_step(lf2_ctx* c, int64_t np, const int32_t* cell, const float* off3,
                           const float* vel3, const float* F4, float dtk, float dtn, int32_t* cell_out,
                           float* off_out, float* vel_out)
{
  if (np == 0) return cudaSuccess;
  c->launches += 1;
  k_pm_gather_kick_drift<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      c->g, np, cell, off3, vel3, reinterpret_cast<const float4*>(F4), dtk, dtn, cell_out, off_out,
      vel_out, c->flags);
  return cudaGetLastError();
}

cudaError_t launch_pm_step_adjoint(lf2_ctx* c, int64_t np, const int32_t* cell, const float* off3,
                                   const float* F4, float* g_vel3, float* g_off3, float* gF4, float dtk,
                                   float dtn)
{
  if (np == 0) return cudaSuccess;
  c->launches += 1;
  k_pm_gather_adj<true><<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      c->g, np, cell, off3, reinterpret_cast<const float4*>(F4), nullptr, reinterpret_cast<float4*>(gF4),
      g_off3, g_vel3, dtk, dtn);
  return cudaGetLastError();
}

cudaError_t launch_pm_loss_adjoint(lf2_ctx* c, int64_t np, const int32_t* cell, const float* off3,
                                   const float* mass, const float* w, float scale, float* g_off3,
                                   float* g_mass, float* g_vel3)
{
  if (np == 0) return cudaSuccess;
  c->launches += 1;
  k_pm_deposit_adj<true><<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      c->g, np, cell, off3, mass, 0.0f, (float)(1.0 / (c->res * c->res * c->res)), w, scale, g_off3, g_mass,
      g_vel3);
  return cudaGetLastError();
}

// Partial sums of the loss (c->loss_part): four CTAs per SM.
int loss_ctas(const lf2_ctx* c) { return 4 * c->num_sms; }

cudaError_t launch_pm_loss(lf2_ctx* c, const float* w, const float* rho, double* loss)
{
  c->launches += 2;
  k_pm_loss<<<loss_ctas(c), LOSS_THREADS, 0, c->stream>>>(c->g.nsites, w, rho, c->loss_part);
  k_pm_loss_sum<<<1, LOSS_THREADS, 0, c->stream>>>(loss_ctas(c), c->loss_part, loss);
  return cudaGetLastError();
}

cudaError_t launch_pm_pack(lf2_ctx* c, int64_t np, const double* pos, const double* vel,
                           const double* mass, double inv_res, int32_t* key, void* rec)
{
  if (np == 0) return cudaSuccess;
  c->launches += 1;
  const auto kern = wide_records(rec) ? k_pm_pack<true> : k_pm_pack<false>;
  kern<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      c->g, np, pos, vel, mass, inv_res, key, reinterpret_cast<uint4*>(rec));
  return cudaGetLastError();
}

cudaError_t launch_pm_unpack(lf2_ctx* c, int64_t np, const int64_t* order, const void* rec,
                             int32_t* cell, float* off3, float* vel3, float* m)
{
  if (np == 0) return cudaSuccess;
  c->launches += 1;
  const auto kern = wide_records(rec) ? k_pm_unpack<true> : k_pm_unpack<false>;
  kern<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      np, order, reinterpret_cast<const uint4*>(rec), cell, off3, vel3, m);
  return cudaGetLastError();
}

cudaError_t launch_pm_brick_start(lf2_ctx* c, int64_t np, const int32_t* cell, int64_t* brick_start)
{
  c->launches += 1;
  k_pm_brick_start<<<grid_for(c->g.nbricks + 1, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      c->g, np, cell, brick_start);
  return cudaGetLastError();
}

cudaError_t launch_pm_grads_back(lf2_ctx* c, int64_t np, const int64_t* order, const float* g_off3,
                                 const float* g_vel3, const float* g_m, double inv_res, void* rec,
                                 double* g_pos, double* g_vel, double* g_mass)
{
  if (np == 0) return cudaSuccess;
  c->launches += 2;
  const bool wide = wide_records(rec);
  const auto scatter = wide ? k_pm_grads_scatter<true> : k_pm_grads_scatter<false>;
  const auto unpack = wide ? k_pm_grads_unpack<true> : k_pm_grads_unpack<false>;
  scatter<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      np, order, g_off3, g_vel3, g_m, reinterpret_cast<uint4*>(rec));
  unpack<<<grid_for(np, PM_THREADS), PM_THREADS, 0, c->stream>>>(
      np, reinterpret_cast<const uint4*>(rec), inv_res, g_pos, g_vel, g_mass);
  return cudaGetLastError();
}

}  // namespace lf2
