// lf2_deposit.cu -- CIC deposits of the brick-binned particles.
//
//   kind 0  scalar CIC        scalarProjectionCIC_project/_comm
//                             (projections.hpp:75-300)
//   kind 1  vector CIC-NGP    vectorProjectionCICNGP_project/_comm (:421-681)
//   kind 2  symtensor CIC-NGP symtensorProjectionCICNGP_project/_comm (:708-976)
//
// One CTA per brick accumulates its particles into a shared-memory tile of the
// (BRICK+1)^3 vertices they touch, then writes the tile once:
//   - vertices with every coordinate in [1, e-1] receive contributions from
//     this brick only, so their final value goes straight to the field;
//   - the other tile vertices (the "shell": a coordinate equal to 0 or to the
//     brick extent e) are written to a per-brick shell store.
// k_fixup then finishes every owned vertex with a zero coordinate by summing
// the shell values of the up to 8 bricks that touch it, in a fixed order.
// The periodic upper-halo fold of the reference's *_comm functions is thus
// part of the deposit, every vertex is written exactly once and no global
// atomics are used.
//
// Three accumulation modes (the context's deposit mode):
//   LF2_DEPOSIT_FP32        the reference's FP32 terms, their sum compensated:
//                           integers in a unit set by the part's largest term
//                           (add_comp_int) with what small terms leave below
//                           it (add_rest), or, where that range does not hold,
//                           FP32 atomics that return the value they replaced,
//                           the rounding error of each recovered exactly
//                           (TwoSum) and accumulated in a second FP32 word.
//                           hi + lo is the sum to within the rounding of the
//                           terms (about 1e-7 of the sum of their magnitudes),
//                           whatever the order and whatever else the brick
//                           holds.
//   LF2_DEPOSIT_FIXED64     int64 fixed point: every contribution is rounded
//                           once, deterministically, to an integer quantum;
//                           the integer sums do not depend on the order, so
//                           the result is bit-exact run to run.  Scalar: 2^-32
//                           of a unit mass.  Momentum and stress are signed:
//                           2^-48 of a unit mass times V (momentum) or V^2
//                           (stress), V the smallest power of two above every
//                           |v_i| of the particles (found on the device before
//                           the deposit, k_vmax).
//   LF2_DEPOSIT_FP32_PLAIN  FP32 shared atomics without compensation: the
//                           speed reference; its sums in dense vertices carry
//                           the rounding of unordered FP32 additions.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "lf2_deposit_common.cuh"
#include "lf2_internal.h"

namespace lf2 {

namespace {

// Threads of a tile pass, and of one whose tile leaves room for one CTA per SM.
// (512 for stores with few particles per brick won 3% in fixed point and lost as
// much with the FP32 sums: 128^3 at 0.02 per site, six components.)
constexpr int DEP_THREADS = 256, DEP_BIG_THREADS = 1024;

// Fewest particles of a part of a split brick, and of any item (a brick below
// that ends soon wherever it starts: four trips of a CTA's threads at most).
constexpr int64_t PART_MIN = 4096, ITEM_MIN = 1024;

// Components of the field of a kind.
template <int KIND>
struct Comps { static constexpr int value = KIND == 0 ? 1 : KIND == 1 ? 3 : 6; };

// A tile pass accumulates NC components of the field.  The plain mode keeps
// one 32-bit word per vertex and component and does every kind in one pass
// (the tensor's six components in a 118 KB tile); the compensated and the
// fixed-point modes keep two words, so the tensor takes two passes of three
// components (T_00, T_11, T_22 at the vertices, then T_01, T_02, T_12 on the
// plaquettes), each with a 118 KB tile.
template <int KIND, int PASS, int ACC>
struct Pass {
  static constexpr int NC = KIND == 0 ? 1 : KIND == 1 ? 3 : (ACC == ACC_PLAIN ? 6 : 3);
  static constexpr int WORDS = ACC == ACC_PLAIN ? 1 : 2;
  // field component of pass-local component j
  __host__ __device__ static constexpr int comp(int j)
  {
    return KIND != 2 || ACC == ACC_PLAIN ? j
           : PASS == 0                   ? (j == 0 ? 0 : j == 1 ? 3 : 5)
                                         : (j == 0 ? 1 : j == 1 ? 2 : 4);
  }
  static constexpr size_t smem() { return (size_t)NC * WORDS * TILE3 * 4; }
  // after the tile, the compensated mode's rests of small terms (Rests): room for
  // what five CTAs per SM leave, or for 64 KB
  static constexpr int RESTS = ACC != ACC_COMP ? 0 : smem() > 100 * 1024 ? 8192 : 512;
  static constexpr size_t dyn() { return smem() + RESTS * sizeof(uint2); }
  // a tile above 100 KB leaves room for one CTA per SM
  static constexpr int THREADS = smem() > 100 * 1024 ? DEP_BIG_THREADS : DEP_THREADS;
  static constexpr int ITEMS = smem() > 100 * 1024 ? 2 : 4;  // particles in flight per thread
  // CTAs per SM that the registers leave room for: those whose tiles fit
  static constexpr int CTAS = smem() > 100 * 1024 ? 1 : smem() > 50 * 1024 ? 3 : 5;
};

__device__ __forceinline__ float sel(int b, float up, float dn) { return b ? up : dn; }

// ------------------------------------------------------------- tile pass
// HM: per-particle masses, or a global one (a kernel each: 1332 us against
// 1353 for both in one at 512^3).
template <int KIND, int PASS, int ACC, bool HM>
__global__ void __launch_bounds__(Pass<KIND, PASS, ACC>::THREADS, Pass<KIND, PASS, ACC>::CTAS)
    k_deposit(StoreView v, DepositParams dp, float* __restrict__ out, uint64_t* __restrict__ spill,
              const uint32_t* __restrict__ vmax_bits, uint32_t* flags, const uint32_t* gate,
              PartView pv)
{
  // gate: run only when the word is set (the redo of a fused deposit)
  if (gate && *gate == 0u) return;
  using P = Pass<KIND, PASS, ACC>;
  constexpr int NC = P::NC;
  constexpr int C = Comps<KIND>::value;
  constexpr bool FIXED = ACC == ACC_FIXED;
  constexpr bool SIGNED = KIND != 0;
  constexpr int T = P::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];

  __shared__ unsigned s_max;
  __shared__ int s_tile;  // (not a register of the particle loop)
  __shared__ int s_rests, s_any;
  __shared__ uint32_t s_marks[ACC == ACC_COMP ? (NC * TILE3 + 31) / 32 : 1];
  __shared__ float s_quantum;

  const Geom& g = v.g;
  Part part;
  if (!part_take(pv, g.nbricks, v.count, v.cap, v.seg_start, part)) return;
  if (threadIdx.x == 0) s_tile = part.tile;
  const int64_t b = part.b;
  int bx, by, bz;
  brick_coords(g, b, bx, by, bz);
  const int ex = brick_extent(g.n[0], bx), ey = brick_extent(g.n[1], by),
            ez = brick_extent(g.n[2], bz);
  const int x0 = bx * BRICK, y0 = by * BRICK, z0 = bz * BRICK;
  const uint32_t base = (uint32_t)(part.start + part.first);  // slots fit in 32 bits
  const int cnt = part.cnt;
  const int mass_bound = FIXED && HM ? part_mass_bound(v.a.mass, base, cnt, dp.inv_unit, &s_max) : 1;
  CompUnit cu{1.0f, 1.0f, false};
  if (ACC == ACC_COMP)
    cu = comp_unit<KIND>(HM ? v.a.mass : nullptr, dp.inv_vol, dp.mf, v.a.vx, v.a.vy, v.a.vz,
                         base, cnt, &s_max);
  // two integer words per vertex, or the sums that hold anything
  const bool ints = FIXED ? cnt <= split_max<SIGNED>(mass_bound) : cu.ok;
  TileRef<TILE3> tr{smem_raw, ints, nullptr};
  // fixed point: velocity quantum and conversion scale for this field
  int vexp = 0;
  if (FIXED && KIND != 0) vexp = vexp_of(*vmax_bits);
  const float vscale = vel_scale(vexp);
  const float conv =
      FIXED ? ldexpf(dp.fixed_scale, (KIND == 1 ? vexp : 2 * vexp) - (KIND != 0 ? 16 : 0)) : 0.0f;
  if (FIXED && threadIdx.x == 0 && b == 0 && !(conv > 0.0f && conv <= 3.402823466e38f))
    set_flag(flags, ERR_FIXED_OVERFLOW);  // V^p / res^3 outside the FP32 range

  {
    uint32_t* z = reinterpret_cast<uint32_t*>(smem_raw);
    constexpr int words = NC * P::WORDS * TILE3;
    for (int t = threadIdx.x; t < words; t += blockDim.x) z[t] = 0u;
    if (ACC == ACC_COMP)
      for (int t = threadIdx.x; t < (NC * TILE3 + 31) / 32; t += blockDim.x) s_marks[t] = 0u;
    if (threadIdx.x == 0) s_rests = 0, s_any = 0, s_quantum = cu.quantum;
  }
  __syncthreads();
  const Rests rs{reinterpret_cast<uint2*>(smem_raw + P::smem()), &s_rests, P::RESTS, s_marks, &s_any, &s_quantum};

  // The particle loop, instantiated for the tile of two integer words per
  // vertex or the other one, chosen once per CTA.
  constexpr int ITEMS = P::ITEMS;
  auto particles = [&](auto split_c) {
    constexpr bool SPLIT = decltype(split_c)::value;
    for (int c0 = 0; c0 < cnt; c0 += ITEMS * T) {
      uint32_t key[ITEMS];
      float fx[ITEMS], fy[ITEMS], fz[ITEMS], m[ITEMS];
      float vx[ITEMS], vy[ITEMS], vz[ITEMS];
  #pragma unroll
      for (int j = 0; j < ITEMS; j++) {
        const int i = c0 + j * T + threadIdx.x;
        if (i < cnt) {
          const uint32_t p = base + (uint32_t)i;
          key[j] = v.a.key[p];
          fx[j] = v.a.ox[p];
          fy[j] = v.a.oy[p];
          fz[j] = v.a.oz[p];
          m[j] = HM ? v.a.mass[p] : 0.0f;
          if (KIND != 0) {
            vx[j] = v.a.vx[p];
            vy[j] = v.a.vy[p];
            vz[j] = v.a.vz[p];
          }
        }
      }
  #pragma unroll
      for (int j = 0; j < ITEMS; j++) {
        const int i = c0 + j * T + threadIdx.x;
        if (i >= cnt) continue;
        int x, y, z;
        unpack_key(g, key[j], x, y, z);
        const int t0 = (x - x0) + TILE * ((y - y0) + TILE * (z - z0));
        constexpr int TY = TILE, TZ = TILE * TILE;
        if (FIXED) {
          uint64_t mq = 0;
          if (HM) mq = mass_q(m[j], dp.inv_unit, flags);
          // 1-D weights in units of 2^-31 (lf2o_fixed_weight in the oracle)
          const uint32_t ux = weight_q(fx[j]), uy = weight_q(fy[j]), uz = weight_q(fz[j]);
          const uint32_t qx[2] = {(1u << 31) - ux, ux};
          const uint32_t qy[2] = {(1u << 31) - uy, uy};
          const uint32_t qz[2] = {(1u << 31) - uz, uz};
          if (KIND == 0) {
            const uint64_t pxy[4] = {(uint64_t)qx[0] * qy[0], (uint64_t)qx[0] * qy[1],
                                     (uint64_t)qx[1] * qy[0], (uint64_t)qx[1] * qy[1]};
  #pragma unroll
            for (int k = 0; k < 8; k++) {
              const int cx = (k >> 2) & 1, cy = (k >> 1) & 1, cz = k & 1;
              const int t = t0 + cx + cy * TY + cz * TZ;
              if (SPLIT && !HM) {
                add_corner_split<TILE3>(reinterpret_cast<uint32_t*>(smem_raw), t, pxy[cx * 2 + cy], qz[cz]);
              } else {
                const uint64_t q = fixed_corner(qx[cx], qy[cy], qz[cz]);
                add_fixed_t<SPLIT, TILE3>(smem_raw, 0, t, mass_sign_t<HM>(q, mq, false));
              }
            }
          } else if (KIND == 1) {
            // projections.hpp:501-544: component i is NGP along i, CIC across
            const float vv[3] = {vx[j], vy[j], vz[j]};
  #pragma unroll
            for (int c = 0; c < 3; c++) {
              const uint32_t vq = vel_q(vv[c], vscale);
              const bool neg = vv[c] < 0.0f;
  #pragma unroll
              for (int k = 0; k < 4; k++) {
                const int a = (k >> 1) & 1, bb = k & 1;
                uint64_t w;
                int t;
                if (c == 0) w = fixed_edge(qy[a], qz[bb]), t = t0 + a * TY + bb * TZ;
                else if (c == 1) w = fixed_edge(qx[a], qz[bb]), t = t0 + a + bb * TZ;
                else w = fixed_edge(qx[a], qy[bb]), t = t0 + a + bb * TY;
                add_fixed48_t<SPLIT, TILE3>(smem_raw, c, t, mass_sign48_t<HM>(mul_wv48(w, vq), mq, neg));
              }
            }
          } else if (PASS == 0) {
            // projections.hpp:788-807: T_ii = m v_i^2 at the 8 vertices
            const float vv[3] = {vx[j], vy[j], vz[j]};
            double f2[3];  // v_d^2 2^-46 (times the relative mass), FP64
  #pragma unroll
            for (int d = 0; d < 3; d++) {
              const uint32_t q = vel_q(vv[d], vscale);
              f2[d] = stress_factor<HM>(q, q, 0x1p-46, mq);  // 2^-46
            }
  #pragma unroll
            for (int k = 0; k < 8; k++) {
              const int cx = (k >> 2) & 1, cy = (k >> 1) & 1, cz = k & 1;
              const uint64_t w = fixed_corner(qx[cx], qy[cy], qz[cz]);
              const int t = t0 + cx + cy * TY + cz * TZ;
  #pragma unroll
              for (int d = 0; d < 3; d++) add_fixed48_t<SPLIT, TILE3>(smem_raw, d, t, stress_q(w, f2[d], false));
            }
          } else {
            // projections.hpp:809-821: T_ij on the (i,j) plaquette, CIC along
            // the third dim
            const float vv[3] = {vx[j], vy[j], vz[j]};
            const uint32_t q0 = vel_q(vv[0], vscale), q1 = vel_q(vv[1], vscale), q2 = vel_q(vv[2], vscale);
            // velocity products times 2^-45 (FP64): a 1-D weight in 2^-31
            // units times one of them is in 2^-48 V^2 units
            const double v01 = stress_factor<HM>(q0, q1, 0x1p-45, mq),
                         v02 = stress_factor<HM>(q0, q2, 0x1p-45, mq),
                         v12 = stress_factor<HM>(q1, q2, 0x1p-45, mq);
            const bool n01 = (vv[0] < 0.0f) != (vv[1] < 0.0f), n02 = (vv[0] < 0.0f) != (vv[2] < 0.0f),
                       n12 = (vv[1] < 0.0f) != (vv[2] < 0.0f);
            add_fixed48_t<SPLIT, TILE3>(smem_raw, 0, t0, stress_q(qz[0], v01, n01));
            add_fixed48_t<SPLIT, TILE3>(smem_raw, 0, t0 + TZ, stress_q(qz[1], v01, n01));
            add_fixed48_t<SPLIT, TILE3>(smem_raw, 1, t0, stress_q(qy[0], v02, n02));
            add_fixed48_t<SPLIT, TILE3>(smem_raw, 1, t0 + TY, stress_q(qy[1], v02, n02));
            add_fixed48_t<SPLIT, TILE3>(smem_raw, 2, t0, stress_q(qx[0], v12, n12));
            add_fixed48_t<SPLIT, TILE3>(smem_raw, 2, t0 + 1, stress_q(qx[1], v12, n12));
          }
          continue;
        }
        // FP32 modes: the arithmetic of the reference's projections in FP32
        const float gx = __fsub_rn(1.0f, fx[j]), gy = __fsub_rn(1.0f, fy[j]),
                    gz = __fsub_rn(1.0f, fz[j]);
        const float ox = fx[j], oy = fy[j], oz = fz[j];
        const float mf = HM ? __fmul_rn(m[j], dp.inv_vol) : dp.mf;
        if (KIND == 0) {
  #pragma unroll
          for (int k = 0; k < 8; k++) {
            const int cx = (k >> 2) & 1, cy = (k >> 1) & 1, cz = k & 1;
            const float w = __fmul_rn(
                __fmul_rn(__fmul_rn(sel(cx, ox, gx), sel(cy, oy, gy)), sel(cz, oz, gz)), mf);
            add_float<ACC, SPLIT, false, TILE3>(smem_raw, 0, t0 + cx + cy * TY + cz * TZ, w, cu.unit, rs);
          }
          // the rests, for a particle in a thousand (asked of every term: 269 us
          // against 261 at 256^3), from its arrays again, so that the loop keeps
          // no registers for them
          if (ACC == ACC_COMP && SPLIT &&
              may_have_rest(__fmul_rn(
                  __fmul_rn(__fmul_rn(__fmul_rn(fminf(ox, gx), fminf(oy, gy)), fminf(oz, gz)), fabsf(mf)),
                  cu.unit))) {
            const uint32_t p = base + (uint32_t)i;
            const float mass = HM ? __fmul_rn(v.a.mass[p], dp.inv_vol) : dp.mf;
  #pragma unroll 1
            for (int k = 0; k < 8; k++) {
              const int cx = (k >> 2) & 1, cy = (k >> 1) & 1, cz = k & 1;
              const float wx = cx ? v.a.ox[p] : __fsub_rn(1.0f, v.a.ox[p]);
              const float wy = cy ? v.a.oy[p] : __fsub_rn(1.0f, v.a.oy[p]);
              const float wz = cz ? v.a.oz[p] : __fsub_rn(1.0f, v.a.oz[p]);
              const float rest = comp_rest(__fmul_rn(__fmul_rn(__fmul_rn(wx, wy), wz), mass), cu.unit, s_quantum);
              if (rest != 0.0f) note_rest(rs, t0 + cx + cy * TY + cz * TZ, rest);
            }
          }
        } else if (KIND == 1) {
          // projections.hpp:501-544: component i is NGP along i, CIC across.
          const float vxm = __fmul_rn(mf, vx[j]);
          const float vym = __fmul_rn(mf, vy[j]);
          const float vzm = __fmul_rn(mf, vz[j]);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 0, t0, __fmul_rn(__fmul_rn(vxm, gy), gz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 0, t0 + TY, __fmul_rn(__fmul_rn(vxm, oy), gz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 0, t0 + TZ, __fmul_rn(__fmul_rn(vxm, gy), oz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 0, t0 + TY + TZ, __fmul_rn(__fmul_rn(vxm, oy), oz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 1, t0, __fmul_rn(__fmul_rn(vym, gx), gz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 1, t0 + 1, __fmul_rn(__fmul_rn(vym, ox), gz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 1, t0 + TZ, __fmul_rn(__fmul_rn(vym, gx), oz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 1, t0 + 1 + TZ, __fmul_rn(__fmul_rn(vym, ox), oz), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 2, t0, __fmul_rn(__fmul_rn(vzm, gx), gy), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 2, t0 + 1, __fmul_rn(__fmul_rn(vzm, ox), gy), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 2, t0 + TY, __fmul_rn(__fmul_rn(vzm, gx), oy), cu.unit, rs);
          add_float<ACC, SPLIT, true, TILE3>(smem_raw, 2, t0 + 1 + TY, __fmul_rn(__fmul_rn(vzm, ox), oy), cu.unit, rs);
        } else {
          // projections.hpp:786-843: T_ii at the 8 vertices, T_ij on plaquettes.
          const float vv[3] = {vx[j], vy[j], vz[j]};
          constexpr bool DIAG = ACC == ACC_PLAIN || PASS == 0;
          constexpr bool OFF = ACC == ACC_PLAIN || PASS == 1;
          if (DIAG) {
  #pragma unroll
            for (int d = 0; d < 3; d++) {
              // pass-local component of T_dd: 0, 3, 5 in the six-component
              // plain tile, 0, 1, 2 in the diagonal pass
              const int jd = ACC == ACC_PLAIN ? (d == 0 ? 0 : d == 1 ? 3 : 5) : d;
              const float mv2 = __fmul_rn(__fmul_rn(mf, vv[d]), vv[d]);
  #pragma unroll
              for (int k = 0; k < 8; k++) {
                const int cx = (k >> 2) & 1, cy = (k >> 1) & 1, cz = k & 1;
                const float w = __fmul_rn(
                    __fmul_rn(__fmul_rn(mv2, sel(cx, ox, gx)), sel(cy, oy, gy)), sel(cz, oz, gz));
                add_float<ACC, SPLIT, true, TILE3>(smem_raw, jd, t0 + cx + cy * TY + cz * TZ, w, cu.unit, rs);
              }
            }
          }
          if (OFF) {
            const int j01 = ACC == ACC_PLAIN ? 1 : 0, j02 = ACC == ACC_PLAIN ? 2 : 1,
                      j12 = ACC == ACC_PLAIN ? 4 : 2;
            const float m01 = __fmul_rn(__fmul_rn(mf, vv[0]), vv[1]);
            const float m02 = __fmul_rn(__fmul_rn(mf, vv[0]), vv[2]);
            const float m12 = __fmul_rn(__fmul_rn(mf, vv[1]), vv[2]);
            add_float<ACC, SPLIT, true, TILE3>(smem_raw, j01, t0, __fmul_rn(m01, gz), cu.unit, rs);
            add_float<ACC, SPLIT, true, TILE3>(smem_raw, j01, t0 + TZ, __fmul_rn(m01, oz), cu.unit, rs);
            add_float<ACC, SPLIT, true, TILE3>(smem_raw, j02, t0, __fmul_rn(m02, gy), cu.unit, rs);
            add_float<ACC, SPLIT, true, TILE3>(smem_raw, j02, t0 + TY, __fmul_rn(m02, oy), cu.unit, rs);
            add_float<ACC, SPLIT, true, TILE3>(smem_raw, j12, t0, __fmul_rn(m12, gx), cu.unit, rs);
            add_float<ACC, SPLIT, true, TILE3>(smem_raw, j12, t0 + 1, __fmul_rn(m12, ox), cu.unit, rs);
          }
        }
      }
    }
  };
  
  bool split = ACC != ACC_PLAIN && tr.split;
  if constexpr (ACC != ACC_PLAIN) {
    if (split) particles(std::true_type{});
  }
  if constexpr (ACC == ACC_COMP) {
    __syncthreads();
    if (split) split = take_rests(tr, NC, rs);
  }
  if (!split) particles(std::false_type{});
  __syncthreads();
  if (s_tile >= 0) {  // k_part_finish writes the vertices
    part_store<ACC, SIGNED, NC, TILE3>(scratch_tile(pv, s_tile, NC * TILE3), tr, s_quantum);
    return;
  }

  // Flush: interior vertices to the field, shell vertices to the shell store
  // (8-byte slots: the integer sum, hi and lo, or the plain float).  Two
  // loops with constant divisors: the interior [1, e-1]^3 (walked as 15^3,
  // skipping what lies beyond the extents), and the shell slots in their
  // storage order (shell_index), so that those writes are contiguous.
  uint64_t* sp = spill + (size_t)b * C * SHELL;
  const float* facc = reinterpret_cast<const float*>(smem_raw);
  const int64_t site0 = site_index(g, x0, y0, z0);
  const int64_t sy = g.n[0], sz = (int64_t)g.n[0] * g.n[1];
  constexpr int I = BRICK - 1;
  for (int u = threadIdx.x; u < I * I * I; u += blockDim.x) {
    const int i = 1 + u % I, jj = 1 + (u / I) % I, k = 1 + u / (I * I);
    if (i >= ex || jj >= ey || k >= ez) continue;
    const int t = i + TILE * (jj + TILE * k);
    const int64_t s = site0 + i + sy * jj + sz * k;
#pragma unroll
    for (int j = 0; j < NC; j++) {
      const int c = P::comp(j);
      if (FIXED) {
        const long long q = tile_fixed<SIGNED>(tr, j, t);
        if (!SIGNED && q < 0) set_flag(flags, ERR_FIXED_OVERFLOW);
        out[(size_t)c * g.nsites + s] = __fmul_rn(__ll2float_rn(q), conv);
      } else if (ACC == ACC_COMP) {
        const float2 p = comp_pair(tr, j, t, s_quantum);
        out[(size_t)c * g.nsites + s] = __fadd_rn(p.x, p.y);
      } else {
        out[(size_t)c * g.nsites + s] = facc[(size_t)j * TILE3 + t];
      }
    }
  }
  // canonical shell coordinate (0, 1..BRICK-1 or BRICK) -> tile coordinate,
  // or -1 where the brick's extent e leaves it out
  auto tile_of = [](int cc, int e) { return cc == BRICK ? e : (cc == 0 || cc < e ? cc : -1); };
  for (int f = threadIdx.x; f < SHELL; f += blockDim.x) {
    int ci, cj, ck;
    if (f < 2 * TILE * TILE) {  // x faces: slot (i == BRICK) TILE^2 + k TILE + j
      ci = f < TILE * TILE ? 0 : BRICK;
      const int r = f % (TILE * TILE);
      ck = r / TILE, cj = r % TILE;
    } else if (f < 2 * TILE * TILE + 2 * I * TILE) {  // y faces: + (j == BRICK) I TILE + k I + i - 1
      const int r = f - 2 * TILE * TILE;
      cj = r < I * TILE ? 0 : BRICK;
      const int r2 = r % (I * TILE);
      ck = r2 / I, ci = 1 + r2 % I;
    } else {  // z faces: + (k == BRICK) I^2 + (j - 1) I + i - 1
      const int r = f - 2 * TILE * TILE - 2 * I * TILE;
      ck = r < I * I ? 0 : BRICK;
      const int r2 = r % (I * I);
      cj = 1 + r2 / I, ci = 1 + r2 % I;
    }
    const int i = tile_of(ci, ex), jj = tile_of(cj, ey), k = tile_of(ck, ez);
    if (i < 0 || jj < 0 || k < 0) continue;
    const int t = i + TILE * (jj + TILE * k);
#pragma unroll
    for (int j = 0; j < NC; j++) {
      const int c = P::comp(j);
      if (FIXED) {
        sp[(size_t)c * SHELL + f] = (uint64_t)tile_fixed<SIGNED>(tr, j, t);
      } else if (ACC == ACC_COMP) {
        reinterpret_cast<float2*>(sp)[(size_t)c * SHELL + f] = comp_pair(tr, j, t, s_quantum);
      } else {
        reinterpret_cast<float*>(sp)[(size_t)c * SHELL + f] = facc[(size_t)j * TILE3 + t];
      }
    }
  }
}

// The vertices of the split bricks, from the sums of their parts: to the
// field and the shell store as the tile pass writes them.
constexpr int FINISH_CHUNK = 512;  // vertices per unit of work

template <int KIND, int PASS, int ACC>
__global__ void __launch_bounds__(FINISH_CHUNK) k_part_finish(Geom g, PartView pv, float fixed_scale,
                                                     float* __restrict__ out,
                                                     uint64_t* __restrict__ spill,
                                                     const uint32_t* __restrict__ vmax_bits,
                                                     uint32_t* flags, const uint32_t* gate)
{
  if (gate && *gate == 0u) return;
  using P = Pass<KIND, PASS, ACC>;
  constexpr int C = Comps<KIND>::value;
  constexpr int CHUNKS = (TILE3 + FINISH_CHUNK - 1) / FINISH_CHUNK;
  const int units = pv.head->splits * CHUNKS;
  if ((int)blockIdx.x >= units) return;
  const int vexp = ACC == ACC_FIXED && KIND != 0 ? vexp_of(*vmax_bits) : 0;
  const float conv = ldexpf(fixed_scale, (KIND == 1 ? vexp : 2 * vexp) - (KIND != 0 ? 16 : 0));
  for (int w = blockIdx.x; w < units; w += gridDim.x) {
    const int4 sp = pv.split[w / CHUNKS];
    const int t = (w % CHUNKS) * FINISH_CHUNK + threadIdx.x;
    int bx, by, bz;
    brick_coords(g, sp.x, bx, by, bz);
    const int ex = brick_extent(g.n[0], bx), ey = brick_extent(g.n[1], by),
              ez = brick_extent(g.n[2], bz);
    const int i = t % TILE, j = (t / TILE) % TILE, k = t / (TILE * TILE);
    if (t >= TILE3 || i > ex || j > ey || k > ez) continue;
    const bool inner = i >= 1 && i < ex && j >= 1 && j < ey && k >= 1 && k < ez;
    const int64_t site = inner ? site_index(g, bx * BRICK + i, by * BRICK + j, bz * BRICK + k) : 0;
    const int si = inner ? 0
                         : shell_index(i == ex ? BRICK : i, j == ey ? BRICK : j, k == ez ? BRICK : k);
    uint64_t* shell = spill + (size_t)sp.x * C * SHELL;
#pragma unroll
    for (int jc = 0; jc < P::NC; jc++) {
      const int c = P::comp(jc);
      const PartSum s = part_sum<ACC>(pv, sp, P::NC * TILE3, jc * TILE3 + t);
      if (inner) {
        if (KIND == 0 && s.q < 0) set_flag(flags, ERR_FIXED_OVERFLOW);
        out[(size_t)c * g.nsites + site] =
            ACC == ACC_FIXED ? __fmul_rn(__ll2float_rn(s.q), conv) : __fadd_rn(s.hi, s.lo);
      } else if (ACC == ACC_FIXED) {
        shell[(size_t)c * SHELL + si] = (uint64_t)s.q;
      } else if (ACC == ACC_COMP) {
        reinterpret_cast<float2*>(shell)[(size_t)c * SHELL + si] = make_float2(s.hi, s.lo);
      } else {
        reinterpret_cast<float*>(shell)[(size_t)c * SHELL + si] = s.hi;
      }
    }
  }
}

// One CTA per brick: every owned vertex with a zero coordinate sums the shell
// values of the bricks that touch it: its own tile (subset 0) and, for every
// non-empty subset S of the dims where its coordinate is 0, the lower
// neighbour brick across S at tile coordinate BRICK in those dims.  The sum
// runs in that fixed order: exact integers (fixed point), a compensated FP32
// sum of the hi and lo words, or plain FP32 additions.
//
// The pass is bound by its scattered reads and the partial sectors it writes:
// at 512^3 about 1.1 GB of traffic (160 us) in 252 us (263 with two vertices
// of any kind per thread), at 256^3 33 us (41).  675 of the 721
// vertices lie inside one of the three faces and have one neighbour: thread
// t < 225 takes vertex t of each face, so that all its reads (two per face
// and component, at fixed offsets from one another) are in flight together;
// the other threads take one edge vertex each (3 neighbours) or the corner
// (7), so that no thread waits for memory twice.
template <int ACC>
struct ShellSum {
  long long q = 0;
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(uint64_t v)
  {
    if (ACC == ACC_FIXED)
      q += (long long)v;
    else if (ACC == ACC_COMP)
      comp_acc(s, c, __uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
    else
      s = __fadd_rn(s, __uint_as_float((uint32_t)v));
  }
  __device__ __forceinline__ float value(float conv) const
  {
    return ACC == ACC_FIXED ? __fmul_rn(__ll2float_rn(q), conv) : ACC == ACC_COMP ? __fadd_rn(s, c) : s;
  }
};

constexpr int FIX_FACE = (BRICK - 1) * (BRICK - 1), FIX_EDGE = 3 * (BRICK - 1);
// CTAs per SM: with more of them (their registers cut to 32) the scalar pass is
// faster where the L2 holds the shell store (256^3: 30 us against 33) and
// slower where it does not (512^3: 278 us against 252).
constexpr int FIX_CTAS = 4;
constexpr int FIX_VERTICES = FIX_FACE + FIX_EDGE + 1, FIX_THREADS = (FIX_VERTICES + 31) & ~31;

// THIN: fewer threads than vertices (fix_threads).  (As a loop for every lattice,
// with 38 registers the scalar pass took 269 us at 512^3, against 252 with 56.)
template <int KIND, int ACC, bool THIN>
__global__ void __launch_bounds__(FIX_THREADS, KIND == 0 ? FIX_CTAS : 1)
    k_fixup(Geom g, const uint64_t* __restrict__ spill, float fixed_scale,
            const uint32_t* __restrict__ vmax_bits, float* __restrict__ out, uint32_t* flags,
            const uint32_t* gate)
{
  if (gate && *gate == 0u) return;
  constexpr int CT = Comps<KIND>::value, C = CT < 3 ? CT : 3;  // of the field, of this CTA
  const int c0 = C * blockIdx.y;
  // the bricks in descending order: the L2 still holds what the tile pass wrote last
  const int64_t b = gridDim.x - 1 - blockIdx.x;
  int bx, by, bz;
  brick_coords(g, b, bx, by, bz);
  const int e[3] = {brick_extent(g.n[0], bx), brick_extent(g.n[1], by), brick_extent(g.n[2], bz)};
  // index of the lower neighbour across a dim, minus the brick's own
  const int64_t nb0 = g.nb[0], nb01 = nb0 * g.nb[1];
  const int64_t lower[3] = {bx ? -1 : nb0 - 1, by ? -nb0 : nb01 - nb0,
                            bz ? -nb01 : (int64_t)g.nbricks - nb01};
  float conv = 0.0f;
  if (ACC == ACC_FIXED) {
    const int vexp = KIND != 0 ? vexp_of(*vmax_bits) : 0;
    conv = ldexpf(fixed_scale, KIND == 0 ? 0 : (KIND == 1 ? vexp : 2 * vexp) - 16);
  }
  const int64_t site0 = site_index(g, bx * BRICK, by * BRICK, bz * BRICK);
  const int64_t step[3] = {1, g.n[0], (int64_t)g.n[0] * g.n[1]};
  // shell value `si` of component c0 + c of brick nb (a brick's region is
  // SHELL 8-byte slots per component; the plain mode fills the first CT *
  // SHELL floats)
  auto read = [&](int64_t nb, int c, int si) -> uint64_t {
    const uint64_t* sp = spill + (size_t)nb * (CT * SHELL);
    const int at = (c0 + c) * SHELL + si;
    return ACC == ACC_PLAIN ? (uint64_t)__float_as_uint(__ldg(reinterpret_cast<const float*>(sp) + at))
                            : __ldg(sp + at);
  };
  auto put = [&](int64_t site, int c, const ShellSum<ACC>& r) {
    if (ACC == ACC_FIXED && KIND == 0 && r.q < 0) set_flag(flags, ERR_FIXED_OVERFLOW);
    out[(c0 + c) * g.nsites + site] = r.value(conv);
  };
  auto vertex = [&](unsigned v) {
    if (v < FIX_FACE) {
      constexpr int I = BRICK - 1;
      const int u = 1 + v % I, w = 1 + v / I;
      // face d: coordinate 0 in dim d, (u, w) in the others; its own shell slot
      // and the lower neighbour's (shell_index at 0 and at BRICK)
      const int own[3] = {w * TILE + u, 2 * TILE * TILE + w * I + (u - 1),
                          2 * TILE * TILE + 2 * I * TILE + (w - 1) * I + (u - 1)};
      constexpr int up[3] = {TILE * TILE, I * TILE, I * I};
      constexpr int du[3] = {1, 0, 0}, dw[3] = {2, 2, 1};
      uint64_t r[3][C][2];
      bool on[3];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        on[d] = u < e[du[d]] && w < e[dw[d]];
#pragma unroll
        for (int c = 0; c < C; c++) {
          r[d][c][0] = on[d] ? read(b, c, own[d]) : 0;
          r[d][c][1] = on[d] ? read(b + lower[d], c, own[d] + up[d]) : 0;
        }
      }
#pragma unroll
      for (int d = 0; d < 3; d++) {
        if (!on[d]) continue;
        const int64_t site = site0 + u * step[du[d]] + w * step[dw[d]];
#pragma unroll
        for (int c = 0; c < C; c++) {
          ShellSum<ACC> s;
          s.add(r[d][c][0]);
          s.add(r[d][c][1]);
          put(site, c, s);
        }
      }
    }
    // edges: coordinate m > 0 along one dim, 0 in the others; then the corner
    const int f = (int)v - FIX_FACE;
    if (f >= 0 && f <= FIX_EDGE) {
      const int d = f == FIX_EDGE ? 3 : f / (BRICK - 1), m = 1 + f % (BRICK - 1);
      if (d < 3 && m >= e[d]) return;
      const int i = d == 0 ? m : 0, j = d == 1 ? m : 0, k = d == 2 ? m : 0;
      const int zmask = 7 & ~(d < 3 ? 1 << d : 0);
      ShellSum<ACC> r[C];
#pragma unroll
      for (int s = 0; s < 8; s++) {  // the subsets of zmask in ascending order
        if ((s & zmask) != s) continue;
        const int64_t nb = b + ((s & 1) ? lower[0] : 0) + ((s & 2) ? lower[1] : 0) + ((s & 4) ? lower[2] : 0);
        const int si = shell_index((s & 1) ? BRICK : i, (s & 2) ? BRICK : j, (s & 4) ? BRICK : k);
#pragma unroll
        for (int c = 0; c < C; c++) r[c].add(read(nb, c, si));
      }
      const int64_t site = site0 + i * step[0] + j * step[1] + k * step[2];
#pragma unroll
      for (int c = 0; c < C; c++) put(site, c, r[c]);
    }
  };
  if (!THIN) vertex(threadIdx.x);
  else
    for (unsigned v = threadIdx.x; v < FIX_VERTICES; v += blockDim.x) vertex(v);
}

// Largest |v_i| of the stored particles, as the bits of a non-negative float
// (they order as unsigned integers); a non-finite velocity raises the flag.
__global__ void __launch_bounds__(256) k_vmax(StoreView v, uint32_t* vmax_bits, uint32_t* flags, PartView pv)
{
  Part part;  // the tile passes' units, so that no CTA reads a heavy brick alone
  if (!part_take(pv, v.g.nbricks, v.count, v.cap, v.seg_start, part)) return;
  // four slots per load: segments and parts start on multiples of four
  const int64_t base = part.start + part.first;
  const float* const comp[3] = {v.a.vx + base, v.a.vy + base, v.a.vz + base};
  uint32_t m = 0u;
#pragma unroll 4
  for (int i = 4 * threadIdx.x; i < part.cnt; i += 4 * blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(comp[d] + i));
      m = max(m, q.x & 0x7fffffffu);
      if (i + 1 < part.cnt) m = max(m, q.y & 0x7fffffffu);
      if (i + 2 < part.cnt) m = max(m, q.z & 0x7fffffffu);
      if (i + 3 < part.cnt) m = max(m, q.w & 0x7fffffffu);
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) != 0) return;
  if (m >= 0x7f800000u) set_flag(flags, ERR_NONFINITE);
  if (m > *reinterpret_cast<volatile uint32_t*>(vmax_bits)) atomicMax(vmax_bits, m);
}

// The plan, where no rebin has made it.  One CTA (which clears the counters),
// or several after they have been cleared.
__global__ void __launch_bounds__(1024) k_part_plan(int nb, const int32_t* __restrict__ count,
                                                    const int32_t* __restrict__ cap, PartPlan pl)
{
  if (gridDim.x == 1) {
    if (threadIdx.x == 0) pl.head->items = pl.head->splits = pl.head->tiles = 0;
    __syncthreads();
  }
  constexpr int U = 4;  // bricks in flight per thread
  for (int b0 = blockIdx.x * blockDim.x + threadIdx.x; b0 < nb; b0 += U * gridDim.x * blockDim.x) {
    int c[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int b = b0 + u * gridDim.x * blockDim.x;
      c[u] = b < nb ? min(count[b], cap[b]) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int b = b0 + u * gridDim.x * blockDim.x;
      if (b < nb) part_plan_brick(pl, b, c[u]);
    }
  }
}

template <int KIND, int PASS, int ACC>
cudaError_t tile_pass(lf2_ctx* c, float* out, const DepositParams& dp, const uint32_t* gate,
                      const PartView& pv)
{
  using P = Pass<KIND, PASS, ACC>;
  const size_t smem = P::dyn();
  const auto kern = dp.has_mass ? k_deposit<KIND, PASS, ACC, true> : k_deposit<KIND, PASS, ACC, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  c->launches += 1;
  kern<<<(unsigned)(c->g.nbricks + pv.max_items), P::THREADS, smem, c->stream>>>(
      view(c), dp, out, c->spill, c->vmax_bits, c->flags, gate, pv);
  if (!pv.max_items) return cudaGetLastError();
  c->launches += 1;
  k_part_finish<KIND, PASS, ACC><<<4 * c->num_sms, FINISH_CHUNK, 0, c->stream>>>(
      c->g, pv, dp.fixed_scale, out, c->spill, c->vmax_bits, c->flags, gate);
  return cudaGetLastError();
}

template <int KIND, int ACC>
PartPlan tile_plan(lf2_ctx* c)
{
  using P = Pass<KIND, 0, ACC>;
  return part_plan(c, P::dyn(), P::THREADS, (size_t)P::NC * TILE3,
                   ACC == ACC_FIXED  ? split_max<KIND != 0>(c->has_mass ? 2 : 1)
                   : ACC == ACC_COMP ? split_max<true>(1)
                                     : 0);
}

template <int KIND, int ACC>
cudaError_t run(lf2_ctx* c, float* out, const DepositParams& dp, int stage, const uint32_t* gate,
                bool planned)
{
  const unsigned nb = (unsigned)c->g.nbricks;
  if (stage == 0) {
    const PartPlan pl = tile_plan<KIND, ACC>(c);
    const PartView pv = part_view(c, pl, (size_t)Pass<KIND, 0, ACC>::NC * TILE3);
    if (!planned) {
      const cudaError_t ep = launch_part_plan(c, pl);
      if (ep != cudaSuccess) return ep;
    }
    if (ACC == ACC_FIXED && KIND != 0) {
      cudaError_t e = launch_vmax(c, pv);
      if (e != cudaSuccess) return e;
    }
    cudaError_t e = tile_pass<KIND, 0, ACC>(c, out, dp, gate, pv);
    if constexpr (KIND == 2 && ACC != ACC_PLAIN) {
      if (e == cudaSuccess) e = tile_pass<KIND, 1, ACC>(c, out, dp, gate, pv);
    }
    return e;
  }
  c->launches += 1;
  const int threads = fix_threads(c, FIX_THREADS);
  const auto kern = threads < FIX_THREADS ? k_fixup<KIND, ACC, true> : k_fixup<KIND, ACC, false>;
  kern<<<dim3(nb, KIND == 2 ? 2 : 1), threads, 0, c->stream>>>(c->g, c->spill, dp.fixed_scale, c->vmax_bits,
                                                               out, c->flags, gate);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t run_mode(lf2_ctx* c, float* out, const DepositParams& dp, int stage, const uint32_t* gate,
                     bool planned)
{
  if (c->mode == LF2_DEPOSIT_FIXED64) return run<KIND, ACC_FIXED>(c, out, dp, stage, gate, planned);
  if (c->mode == LF2_DEPOSIT_FP32_PLAIN) return run<KIND, ACC_PLAIN>(c, out, dp, stage, gate, planned);
  return run<KIND, ACC_COMP>(c, out, dp, stage, gate, planned);
}

}  // namespace

// Whether the plan can be left out, with its launch and that of every pass's
// finishing kernel (5 us each: an even 64^3 in fixed point, density 28 us against
// 22): no brick can be split, or the host knows the store to be even, its largest
// brick a quarter below an item and read a few rebins ago.  A captured call is
// replayed on stores that the host has not seen.
static bool no_heavy_brick(const lf2_ctx* c, int64_t split, int64_t first)
{
  if (c->np <= split) return true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  return c->most_age <= 32 && c->most + c->most / 4 <= first &&
         cudaStreamIsCapturing(c->stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
}

// What is heavy depends on the chip's share of the particles per CTA that runs
// at once (`share`).  A brick is an item, taken first, above a quarter of the
// share (a brick that starts last then ends with the others), three times
// the mean count (an even distribution has no items) and ITEM_MIN (the others
// are 0 for stores with fewer particles than bricks and CTAs).  It is split
// above 3/2 P with P half the share, so that no CTA is left with more than
// that, but parts hold at least PART_MIN particles: each clears and writes its
// tile (parts of 1024 took 41 us for 64 uniform bricks of 4096 against 35
// unsplit).
// `cap` bounds what a split fixed-point tile sums.  The scratch tiles lie in
// the repack scratch (c->alt), which nothing uses between the rebins.
PartPlan part_plan(lf2_ctx* c, size_t smem, int threads, size_t tile_slots, int cap)
{
  PartPlan pl{};
  pl.item = c->part_item;
  pl.split_list = c->part_item + PART_ITEMS;
  pl.mark = c->part_mark;
  pl.head = c->head;
  if (c->np == 0) return pl;
  const int per_sm = std::max(1, std::min((int)(227 * 1024 / (smem + 1024)), 2048 / threads));
  const int64_t share = c->np / ((int64_t)c->num_sms * per_sm);
  if (cap <= 0) cap = 1 << 28;
  const int64_t P = std::min<int64_t>(std::max<int64_t>(share / 2, PART_MIN), cap - cap / 16);
  const int64_t split = std::min<int64_t>(P + P / 2, cap);
  const int64_t first =
      std::min(split, std::max({ITEM_MIN, share / 4, 3 * (c->np / c->g.nbricks)}));
  pl.P = (int)P, pl.split = (int)split, pl.first = (int)first;
  if (no_heavy_brick(c, split, first)) return pl;
  // np particles make at most 3/2 np / P parts and np / first items
  pl.max_items = (int)std::min<int64_t>(PART_ITEMS, c->np * 3 / (2 * P) + c->np / first);
  pl.max_tiles = (int)std::min<int64_t>(7 * (c->capacity / 2 / (int64_t)tile_slots), PART_TILES);
  return pl;
}

PartView part_view(const lf2_ctx* c, const PartPlan& pl, size_t tile_slots)
{
  PartView pv{};
  pv.item = pl.item, pv.split = pl.split_list, pv.mark = pl.mark, pv.head = pl.head;
  float* const banks[7] = {reinterpret_cast<float*>(c->alt.key), c->alt.ox, c->alt.oy, c->alt.oz,
                           c->alt.vx, c->alt.vy, c->alt.vz};
  for (int i = 0; i < 7; i++) pv.bank[i] = reinterpret_cast<uint64_t*>(banks[i]);
  pv.bank_tiles = (int)std::min<int64_t>(c->capacity / 2 / (int64_t)tile_slots, PART_TILES);
  pv.max_items = pl.max_items;
  return pv;
}

cudaError_t launch_part_plan(lf2_ctx* c, const PartPlan& pl)
{
  if (!pl.max_items) return cudaSuccess;
  const int nb = (int)c->g.nbricks, ctas = (nb + 4095) / 4096;
  if (ctas > 1) {
    const cudaError_t e = cudaMemsetAsync(&c->head->items, 0, 3 * sizeof(int32_t), c->stream);
    if (e != cudaSuccess) return e;
  }
  c->launches += 1;
  k_part_plan<<<ctas, 1024, 0, c->stream>>>(nb, c->count, c->cap, pl);
  return cudaGetLastError();
}

// Threads of a fix-up: one to a vertex of a whole brick's faces, fewer where the
// lattice is thinner than half a brick and most would have none but take their
// registers (2 x 2 x 100,000 in fixed point, momentum 76 us to 50, stress 146 to
// 90, full-CIC momentum 104 to 60 and stress 197 to 103).
int fix_threads(const lf2_ctx* c, int whole)
{
  return c->g.n[0] < BRICK / 2 || c->g.n[1] < BRICK / 2 || c->g.n[2] < BRICK / 2 ? 96 : whole;
}

// The plan of the scalar deposit that follows a rebin.
PartPlan scalar_plan(lf2_ctx* c)
{
  if (c->mode == LF2_DEPOSIT_FIXED64) return tile_plan<0, ACC_FIXED>(c);
  if (c->mode == LF2_DEPOSIT_FP32_PLAIN) return tile_plan<0, ACC_PLAIN>(c);
  return tile_plan<0, ACC_COMP>(c);
}

// Shell-store slots (8 bytes each) a deposit of `comps` components needs.
size_t deposit_spill_slots(const lf2_ctx* c, int comps)
{
  return (size_t)c->g.nbricks * (size_t)comps * SHELL;
}

cudaError_t launch_vmax(lf2_ctx* c, const PartView& pv)
{
  cudaError_t e = cudaMemsetAsync(c->vmax_bits, 0, sizeof(uint32_t), c->stream);
  if (e != cudaSuccess) return e;
  c->launches += 1;
  k_vmax<<<(unsigned)(c->g.nbricks + pv.max_items), 256, 0, c->stream>>>(view(c), c->vmax_bits, c->flags,
                                                                         pv);
  return cudaGetLastError();
}

DepositParams deposit_params(const lf2_ctx* c)
{
  DepositParams dp;
  const double vol = c->res * c->res * c->res;
  dp.inv_vol = (float)(1.0 / vol);
  dp.mf = (float)(c->gmass / vol);
  dp.fixed_scale = (float)(std::ldexp(1.0, -32) * c->m_unit / vol);
  dp.inv_unit = (float)(1.0 / c->m_unit);
  dp.has_mass = c->has_mass ? 1 : 0;
  return dp;
}

cudaError_t launch_deposit(lf2_ctx* c, int kind, float* out, int stage, const uint32_t* gate, bool planned)
{
  const DepositParams dp = deposit_params(c);
  if (kind == 0) return run_mode<0>(c, out, dp, stage, gate, planned);
  if (kind == 1) return run_mode<1>(c, out, dp, stage, gate, false);
  return run_mode<2>(c, out, dp, stage, gate, false);
}

}  // namespace lf2
