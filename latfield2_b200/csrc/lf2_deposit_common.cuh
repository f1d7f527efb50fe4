// lf2_deposit_common.cuh -- accumulation helpers shared by the deposit tile
// passes of lf2_deposit.cu (CIC and CIC-NGP projections) and
// lf2_deposit_full.cu (full-CIC projections): the compensated FP32 add, the
// split fixed-point accumulation and the deterministic integer weights of the
// fixed-point mode.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "lf2_common.cuh"
#include "lf2gpu.h"

namespace lf2 {

enum : int {
  ACC_COMP = LF2_DEPOSIT_FP32,
  ACC_FIXED = LF2_DEPOSIT_FIXED64,
  ACC_PLAIN = LF2_DEPOSIT_FP32_PLAIN
};

// ------------------------------------------------------------ accumulation
// Fixed point: each 64-bit vertex sum is kept as two 32-bit partial sums,
// lo = sum(q & 0xffff) and hi = sum(q >> 16) (arithmetic shift), so that every
// update is a native 32-bit shared-memory reduction; the sum is
// lo + hi * 2^16, hi read as unsigned (scalar, q >= 0) or as signed (momentum
// and stress).  Neither partial sum may wrap: per particle and vertex
// |q| <= 2^32 * M with M = 1 for a global mass and otherwise the largest
// relative mass of the particles summed, rounded up (mass_q keeps it below
// 64), so the split is exact for up to split_max(M) particles; more use
// 64-bit shared atomics, which compile to compare-and-swap loops.
template <bool SIGNED>
__host__ __device__ inline int split_max(int mass_bound)
{
  return (SIGNED ? 32767 : 65535) / mass_bound;
}

// A tile of N vertices per component in shared memory: component j occupies
// words [2 j N, 2 (j + 1) N) (two 32-bit words per vertex), or [j N, (j+1) N)
// in the plain mode.
// marks: a bit per component and vertex (j N + t) whose words are the FP32 pair
// although the tile is split (compensated mode), or null.
template <int N>
struct TileRef {
  unsigned char* smem;
  bool split;
  const uint32_t* marks;
  __device__ __forceinline__ bool pair(int i) const
  {
    return !split || (marks && (marks[i >> 5] >> (i & 31) & 1u));
  }
};

template <int N>
__device__ __forceinline__ void add_fixed(TileRef<N> tr, int j, int t, long long q)
{
  if (tr.split) {
    uint32_t* w = reinterpret_cast<uint32_t*>(tr.smem) + (size_t)j * 2 * N;
    atomicAdd(&w[t], (uint32_t)((unsigned long long)q & 0xffffu));
    atomicAdd(&w[N + t], (uint32_t)(q >> 16));
  } else {
    atomicAdd(reinterpret_cast<unsigned long long*>(tr.smem) + (size_t)j * N + t,
              (unsigned long long)q);
  }
}

// The same with the split decided at compile time (the tile passes
// instantiate their particle loop once per choice, per CTA).
template <bool SPLIT, int N>
__device__ __forceinline__ void add_fixed_t(unsigned char* smem, int j, int t, long long q)
{
  if (SPLIT) {
    uint32_t* w = reinterpret_cast<uint32_t*>(smem) + (size_t)j * 2 * N;
    atomicAdd(&w[t], (uint32_t)((unsigned long long)q & 0xffffu));
    atomicAdd(&w[N + t], (uint32_t)(q >> 16));
  } else {
    atomicAdd(reinterpret_cast<unsigned long long*>(smem) + (size_t)j * N + t, (unsigned long long)q);
  }
}

// Compensated FP32 add: the atomic returns the value it replaced, so the
// rounding error of the stored sum fl(old + w) is recovered exactly by
// Knuth's TwoSum and added to the second word.
__device__ __forceinline__ void add_comp(float* hi, float* lo, float w)
{
  const float old = atomicAdd(hi, w);
  const float s = __fadd_rn(old, w);
  const float bb = __fsub_rn(s, old);
  const float err = __fadd_rn(__fsub_rn(old, __fsub_rn(s, bb)), __fsub_rn(w, bb));
  atomicAdd(lo, err);
}

// (s, c) += (h, l): TwoSum of s and h, the error and l carried in c.
__device__ __forceinline__ void comp_acc(float& s, float& c, float h, float l)
{
  const float t = __fadd_rn(s, h);
  const float bb = __fsub_rn(t, s);
  const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bb)), __fsub_rn(h, bb));
  s = t;
  c = __fadd_rn(c, __fadd_rn(err, l));
}


// Signed kinds (momentum and stress): contributions are in units of 2^-48
// of a unit mass times V or V^2, |q| <= 2^48 for a global mass and 2^54 with
// per-particle masses.  The split keeps lo = the low 32 bits of the sum
// (every carry out of the 32-bit add, seen in the value the atomic returns,
// goes to hi) and hi = the sum of (q >> 32) plus those carries, so the
// vertex sum is hi 2^32 + lo exactly while hi stays within int32: bricks of
// at most split_max<true> particles.
template <bool SPLIT, int N>
__device__ __forceinline__ void add_fixed48_t(unsigned char* smem, int j, int t, long long q)
{
  if (SPLIT) {
    uint32_t* w = reinterpret_cast<uint32_t*>(smem) + (size_t)j * 2 * N;
    const uint32_t lo = (uint32_t)(unsigned long long)q;
    const uint32_t old = atomicAdd(&w[t], lo);
    const int carry = (uint32_t)(old + lo) < old ? 1 : 0;
    atomicAdd(reinterpret_cast<int*>(&w[N + t]), (int)(q >> 32) + carry);
  } else {
    atomicAdd(reinterpret_cast<unsigned long long*>(smem) + (size_t)j * N + t, (unsigned long long)q);
  }
}

// Compensated FP32 mode.  The terms are the FP32 products of the reference's
// arithmetic; their sum is kept, as in the signed fixed-point kinds, as a
// 64-bit integer in two 32-bit words, in units of a quantum set by the largest
// term of the CTA's particles (CompUnit).  A term at or above 2^23 quanta is a
// whole number of them.  What a smaller one (one in 10^5 of the density's, 0.3%
// of the diagonal stress's for Gaussian velocities) leaves below the quantum is
// noted, and joins its vertex at the end where that can tell it from its
// rounding (take_rests), so that every term counts in full whatever stands
// beside it.  (An FP32 shared atomic compiles to a compare-and-swap loop: the
// TwoSum pair of add_comp takes 3.4 times the shared wavefronts of the two
// integer words.)  add_comp stays for what the integers cannot hold: terms that
// are not finite or out of range, more than split_max particles, and more rests
// than there is room for.  The tile passes of the two full-CIC calls at 256^3 in
// clumps take 2.54 ms, as they did with the rests dropped and ldexpf for the
// powers of two (a list of particles that may have one, looked through after
// the loop: 2.74).
struct Rests {
  uint2* note;      // word of the vertex in the tile, bits of the rest
  int* count;       // how many were to be noted
  int room;
  uint32_t* marks;  // TileRef
  int* any;         // set with the first mark
  const float* quantum;  // (in shared memory: the particle loop keeps no register for it)
};

// What a term w leaves below the quantum (0: a whole number of them).
__device__ __forceinline__ float comp_rest(float w, float unit, float quantum)
{
  const float x = __fmul_rn(w, unit);
  if (!(fabsf(x) < 0x1p-8f)) return 0.0f;
  return __fmaf_rn(-__int2float_rn(__float2int_rn(__fmul_rn(x, 2147483648.0f))), quantum, w);  // exact
}

// For a particle's smallest term in units of 2^31 quanta (a factor of two for
// the rounding of its product).
__device__ __forceinline__ bool may_have_rest(float least) { return least < 0x1p-7f; }

__device__ __forceinline__ void note_rest(const Rests& rs, int word, float rest)
{
  const int k = atomicAdd(rs.count, 1);
  if (k < rs.room) rs.note[k] = make_uint2((uint32_t)word, __float_as_uint(rest));
}

// w: the term; x = w in units of 2^31 quanta, |x| < 2^21.  x = hi + lo 2^-31
// with hi the nearest integer (the sum with 1.5 * 2^23 rounds there) and lo
// the nearest integer to the remainder, |lo| <= 2^30.  The words hold
// hi 2^31 + lo: a carry or borrow of the low word is worth 2 of the high one.
template <int N, bool NOTE>
__device__ __forceinline__ void add_comp_int(unsigned char* smem, int j, int t, float w, float unit,
                                             const Rests& rs)
{
  uint32_t* words = reinterpret_cast<uint32_t*>(smem) + (size_t)j * 2 * N;
  const float x = __fmul_rn(w, unit);
  const float h = __fadd_rn(x, 12582912.0f);
  const int hi = __float_as_int(h) - 0x4B400000;
  const float r = __fsub_rn(x, __fsub_rn(h, 12582912.0f));  // exact, |r| <= 1/2
  const int lo = __float2int_rn(__fmul_rn(r, 2147483648.0f));
  const uint32_t old = atomicAdd(&words[t], (uint32_t)lo);
  const int carry = old + (uint32_t)lo < old ? 1 : 0;
  atomicAdd(reinterpret_cast<int*>(&words[N + t]), hi + 2 * ((lo >> 31) + carry));
  if (NOTE && fabsf(x) < 0x1p-8f) {
    const float rest = __fmaf_rn(-__int2float_rn(lo), *rs.quantum, w);  // as comp_rest: here hi = 0
    if (rest != 0.0f) note_rest(rs, j * 2 * N + t, rest);
  }
}

// One FP32 term of either mode; SPLIT: the integer sums of the compensated one
// (NOTE: with their rests).
template <int ACC, bool SPLIT, bool NOTE, int N>
__device__ __forceinline__ void add_float(unsigned char* smem, int j, int t, float w, float unit,
                                          const Rests& rs)
{
  float* f = reinterpret_cast<float*>(smem);
  if (ACC == ACC_PLAIN)
    atomicAdd(&f[(size_t)j * N + t], w);
  else if (SPLIT)
    add_comp_int<N, NOTE>(smem, j, t, w, unit, rs);
  else
    add_comp(&f[(size_t)j * 2 * N + t], &f[(size_t)j * 2 * N + N + t], w);
}

// The unit of a CTA's terms, from the largest bound M of any of its particles:
// 2^q is the quantum of the integer sums, `unit` = 2^(-32 - q).  With M < 2^e
// and fewer than 2^k particles the high words stay within int32 for
// |x| <= 2^(31 - k).  ok: both powers and every whole number of quanta are
// normal FP32 numbers, and the particles are few enough for 16 bits of x.
struct CompUnit {
  float quantum, unit;
  bool ok;
};

__device__ __forceinline__ CompUnit comp_unit_of(unsigned bits, int cnt)
{
  const int e = (int)(bits >> 23) - 126;  // M < 2^e for a normal number
  const int s = min(21, __clz(cnt) - 1);
  CompUnit r;
  r.ok = e >= -70 && e <= 127 && cnt <= split_max<true>(1);
  r.unit = r.ok ? ldexpf(1.0f, s - e) : 1.0f;
  r.quantum = r.ok ? ldexpf(1.0f, e - s - 31) : 1.0f;
  return r;
}

// M: the product of |mass / volume| (mf for a global mass) and P times the
// largest |v_i| of a particle, rounded as the terms' products are: rounding is
// monotonic and the weights are at most 1, so no |term| is above it, and a
// particle whose product leaves the FP32 range shows in it (infinity, or NaN,
// whose bits order above it).
template <int P>
__device__ __forceinline__ CompUnit comp_unit(const float* mass, float inv_vol, float mf,
                                              const float* vx, const float* vy, const float* vz,
                                              uint32_t p0, int cnt, unsigned* s_max)
{
  if (!mass && P == 0) return comp_unit_of(__float_as_uint(mf) & 0x7fffffffu, cnt);
  if (threadIdx.x == 0) *s_max = 0u;
  __syncthreads();
  unsigned m = 0u;
  for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
    const uint32_t p = p0 + (uint32_t)i;
    float f = mass ? __fmul_rn(mass[p], inv_vol) : mf;
    if (P > 0) {
      const float v = __uint_as_float(max(max(__float_as_uint(vx[p]) & 0x7fffffffu,
                                              __float_as_uint(vy[p]) & 0x7fffffffu),
                                          __float_as_uint(vz[p]) & 0x7fffffffu));
      f = __fmul_rn(f, v);
      if (P > 1) f = __fmul_rn(f, v);
    }
    m = max(m, __float_as_uint(f) & 0x7fffffffu);
  }
  m = __reduce_max_sync(0xffffffffu, m);  // bits of |x| order as integers
  if ((threadIdx.x & 31) == 0) atomicMax(s_max, m);
  __syncthreads();
  return comp_unit_of(*s_max, cnt);
}

// hi/lo pair of a compensated vertex sum, from the integers or the floats.
template <int N>
__device__ __forceinline__ float2 comp_pair(const TileRef<N>& tr, int j, int t, float quantum)
{
  const uint32_t* w = reinterpret_cast<const uint32_t*>(tr.smem) + (size_t)j * 2 * N;
  if (tr.pair(j * N + t)) return make_float2(__uint_as_float(w[t]), __uint_as_float(w[N + t]));
  const long long s = (long long)(int32_t)w[N + t] * 2147483648ll + (long long)w[t];
  const float hi = __ll2float_rn(s), lo = __ll2float_rn(s - (long long)hi);
  return make_float2(__fmul_rn(hi, quantum), __fmul_rn(lo, quantum));
}

// After the particles, by the whole CTA: the noted rests into the sums.  Half a
// quantum each of n rests is under 2^-28 of a vertex sum of 2^27 n quanta, a
// sixteenth of the last rounding; a smaller sum with a rest is marked, becomes
// an FP32 pair and takes its rests.  (All sums as pairs in every CTA with a rest
// cost the full-CIC passes 15%.)  False, with the tile cleared for a run with
// pairs, where there were more rests than room.
template <int N>
__device__ __forceinline__ bool take_rests(TileRef<N>& tr, int comps, const Rests& rs)
{
  uint32_t* w = reinterpret_cast<uint32_t*>(tr.smem);
  float* f = reinterpret_cast<float*>(tr.smem);
  const int n = *rs.count;
  if (n == 0) return true;
  if (n > rs.room) {
    for (int t = threadIdx.x; t < comps * 2 * N; t += blockDim.x) w[t] = 0u;
    tr.split = false;
    __syncthreads();
    return false;
  }
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const int at = (int)rs.note[k].x, i = at - at / (2 * N) * N;
    if (abs((int)w[at + N]) < n / 16 + 3) {  // (high word: units of 2^31 quanta, at least |h| - 2 of them)
      atomicOr(&rs.marks[i >> 5], 1u << (i & 31));
      *rs.any = 1;
    } else {
      rs.note[k].y = 0u;
    }
  }
  __syncthreads();
  if (!*rs.any) return true;
  for (int k = threadIdx.x; k < (comps * N + 31) / 32; k += blockDim.x) {
    for (uint32_t m = rs.marks[k]; m; m &= m - 1) {
      const int i = 32 * k + __ffs(m) - 1, j = i / N, t = i % N, at = j * 2 * N + t;
      const float2 p = comp_pair(tr, j, t, *rs.quantum);
      w[at] = __float_as_uint(p.x);
      w[at + N] = __float_as_uint(p.y);
    }
  }
  tr.marks = rs.marks;
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x)
    if (rs.note[k].y) add_comp(&f[rs.note[k].x], &f[rs.note[k].x + N], __uint_as_float(rs.note[k].y));
  return true;
}

// Integer vertex sum of component j: the scalar's split (lo + hi 2^16) or
// the signed kinds' split (hi 2^32 + lo, add_fixed48_t).
template <bool SIGNED, int N>
__device__ __forceinline__ long long tile_fixed(const TileRef<N>& tr, int j, int t)
{
  if (tr.split) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(tr.smem) + (size_t)j * 2 * N;
    if (SIGNED) return (long long)(int32_t)w[N + t] * 4294967296ll + (long long)w[t];
    return (long long)w[t] + (long long)w[N + t] * 65536ll;
  }
  return (long long)reinterpret_cast<const unsigned long long*>(tr.smem)[(size_t)j * N + t];
}

// ----------------------------------------------------- fixed-point weights
// 1-D weight in units of 2^-31 (lf2o_fixed_weight in the oracle).
__device__ __forceinline__ uint32_t weight_q(float w) { return __float2uint_rn(w * 2147483648.0f); }

// Velocity in units of 2^-31 V (V = 2^e > |v|): |v| 2^(31-e) is exact in FP32
// and below 2^31; rounded to the nearest integer.
__device__ __forceinline__ uint32_t vel_q(float v, float vscale)
{
  return __float2uint_rn(fabsf(v) * vscale);
}

// fixed_corner with one weight equal to 1 (2^31): (qa qb 2^31 + 2^60) >> 61.
__device__ __forceinline__ uint64_t fixed_edge(uint32_t qa, uint32_t qb)
{
  return ((uint64_t)qa * qb + (1ull << 29)) >> 30;
}

// Product of two such velocities in units of 2^-31 V^2, rounded.
__device__ __forceinline__ uint64_t vel2_q(uint32_t a, uint32_t b)
{
  return ((uint64_t)a * (uint64_t)b + (1ull << 30)) >> 31;
}

// w (2^-32 units) times a factor in 2^-31 units, rounded to 2^-32 units.
__device__ __forceinline__ uint64_t mul31(uint64_t w, uint64_t f) { return (w * f + (1ull << 30)) >> 31; }

// Momentum: w (2^-32 units, <= 2^32) times a velocity (2^-31 V units,
// < 2^31), rounded to 2^-48 V units.
__device__ __forceinline__ uint64_t mul_wv48(uint64_t w, uint64_t f) { return (w * f + (1ull << 14)) >> 15; }

// round(a * b / 2^s) for a product of up to 128 bits (32 <= s < 64), from
// its two 64-bit halves.
template <int S>
__device__ __forceinline__ uint64_t mul_round(uint64_t a, uint64_t b)
{
  const uint64_t lo = a * b, hi = __umul64hi(a, b);
  return ((lo >> S) | (hi << (64 - S))) + ((lo >> (S - 1)) & 1ull);
}

// Stress: w (2^-32 units) times the exact product of two velocities (2^-62
// V^2 units, < 2^62), rounded to 2^-48 V^2 units; a 1-D weight (2^-31 units)
// times that product likewise.
__device__ __forceinline__ uint64_t mul_wvv48(uint64_t w, uint64_t vv) { return mul_round<46>(w, vv); }
__device__ __forceinline__ uint64_t mul_avv48(uint64_t a, uint64_t vv) { return mul_round<45>(a, vv); }

// Stress contributions in FP64: the weight w (an integer below 2^52, exact
// in double) times a per-particle factor f = v_a v_b 2^-s (times the
// relative mass), both products rounded by IEEE double multiplication, then
// rounded to the nearest integer (half to even): units of 2^-48 V^2.  The
// sequence is deterministic and restated in the oracle operation by
// operation.
__device__ __forceinline__ double u2d_exact(uint64_t w)  // w < 2^52
{
  return __dadd_rn(__longlong_as_double((long long)(0x4330000000000000ull | w)), -4503599627370496.0);
}
__device__ __forceinline__ uint64_t d2u_rn(double x)  // 0 <= x < 2^51
{
  const double y = __dadd_rn(x, 6755399441055744.0);  // 1.5 * 2^52: integer part in the low bits
  return ((uint64_t)__double_as_longlong(y) & 0xFFFFFFFFFFFFFull) - (1ull << 51);
}
// f = (v_a v_b) 2^-s, times m / m_unit when HM (mq: the relative mass in
// 2^-24 units)
template <bool HM>
__device__ __forceinline__ double stress_factor(uint32_t va, uint32_t vb, double scale, uint64_t mq)
{
  double f = __dmul_rn(__dmul_rn(u2d_exact(va), u2d_exact(vb)), scale);
  if (HM) f = __dmul_rn(f, __dmul_rn(u2d_exact(mq), 0x1p-24));  // 2^-24
  return f;
}
__device__ __forceinline__ long long stress_q(uint64_t w, double f, bool neg)
{
  const long long q = (long long)d2u_rn(__dmul_rn(u2d_exact(w), f));
  return neg ? -q : q;
}

// Per-particle relative mass (2^-24 units) applied to a signed-kind
// contribution (|q| <= 2^48, so the product needs 128 bits), then the sign.
template <bool HM>
__device__ __forceinline__ long long mass_sign48_t(uint64_t q, uint64_t mq, bool neg)
{
  if (HM) q = mul_round<24>(q, mq);
  return neg ? -(long long)q : (long long)q;
}

// Per-particle relative mass m / m_unit in units of 2^-24 (range-checked).
__device__ __forceinline__ uint64_t mass_q(float m, float inv_unit, uint32_t* flags)
{
  const float mr = __fmul_rn(m, inv_unit);
  if (!(mr >= 0.0f && mr < 64.0f)) set_flag(flags, ERR_MASS_RANGE);
  return (uint64_t)__float2uint_rn(fminf(fmaxf(mr, 0.0f), 63.0f) * 16777216.0f);
}

__device__ __forceinline__ long long apply_mass_sign(uint64_t q, bool has_mass, uint64_t mq, bool neg)
{
  if (has_mass) q = (q * mq + (1ull << 23)) >> 24;
  return neg ? -(long long)q : (long long)q;
}

template <bool HM>
__device__ __forceinline__ long long mass_sign_t(uint64_t q, uint64_t mq, bool neg)
{
  if (HM) q = (q * mq + (1ull << 23)) >> 24;
  return neg ? -(long long)q : (long long)q;
}

// Scalar corner weight of a global-mass particle straight into the split
// tile: q = fixed_corner(qx, qy, qz) with p = qx qy given, so that
// q & 0xffff = bits [29, 45) and q >> 16 = bits [45, 64) of
// h = ph qz + umulhi(pl, qz) + 2^28.
template <int N>
__device__ __forceinline__ void add_corner_split(uint32_t* tile, int t, uint64_t p, uint32_t qz)
{
  const uint64_t h = (uint64_t)(uint32_t)(p >> 32) * qz + __umulhi((uint32_t)p, qz) + (1ull << 28);
  const uint32_t hl = (uint32_t)h, hh = (uint32_t)(h >> 32);
  atomicAdd(&tile[t], __funnelshift_r(hl, hh, 29) & 0xffffu);
  atomicAdd(&tile[N + t], hh >> 13);
}

// Scale 2^(31-e) as an FP32 (e within [-96, 128]).
__device__ __forceinline__ float vel_scale(int e) { return ldexpf(1.0f, 31 - e); }

// Exponent e of V = 2^e, the smallest power of two above the largest |v_i|
// (bits of a non-negative float; 0 when every velocity is 0), at least
// 2^-96 so that 2^(31-e) stays a finite FP32.
__host__ __device__ inline int vexp_of(uint32_t bits)
{
  if (bits == 0u) return 0;
  const int e = (int)((bits >> 23) & 0xffu) - 126;
  return e < -96 ? -96 : e;
}

// --------------------------------------------------- parts of heavy bricks
// A brick that holds far more particles than the others would keep one CTA
// busy long after the rest of the chip is done.  A plan (PartPlan) lists the
// heavy bricks as items that the first CTAs of a tile pass take, the heaviest
// of them split into parts of equal particle counts.  A part's CTA writes its
// whole tile to the scratch; a finishing kernel sums the parts of each split
// brick in part order and writes the brick's vertices as the tile pass does
// for a brick in one part.  (Finishing in the CTA of the last part cost the
// particle loops registers: 1591 us against 1364 at 512^3.)
struct PartView {
  const int4* item;       // brick (-1: none), part, parts of the brick, tile of part 0
  const int4* split;      // brick, parts, tile of part 0
  const uint8_t* mark;    // per brick: 1 when it is an item
  const PassHead* head;
  uint64_t* bank[7];      // scratch tiles, NC * N 8-byte slots each,
  int bank_tiles;         // so many to a bank
  int max_items;          // what the plan may list
};

__device__ __forceinline__ uint64_t* scratch_tile(const PartView& pv, int i, int slots)
{
  uint64_t* p = pv.bank[0];  // (selected, so that the view stays in parameter space)
#pragma unroll
  for (int k = 1; k < 7; k++)
    if (i >= k * pv.bank_tiles) p = pv.bank[k];
  return p + (size_t)(i % pv.bank_tiles) * slots;
}

__device__ __forceinline__ int part_items(const PartView& pv)
{
  return pv.max_items ? min(pv.head->items, pv.max_items) : 0;
}

// One unit of work of a tile pass: particles [first, first + cnt) of a brick.
struct Part {
  int64_t b, start;  // the brick, and its first slot
  int first, cnt;
  int tile;  // scratch tile of a part of a split brick, or -1
};

// The unit of this CTA in a grid of nbricks + max_items: the items, then the
// bricks in their order; false where there is none or the brick is an item.
// The brick's counts and first slot are read with the number of items, as if
// there were none, so that a plan without items (the ordinary one) costs a CTA
// one trip to memory and not three.
__device__ __forceinline__ bool part_take(const PartView& pv, int64_t nbricks, const int32_t* count,
                                          const int32_t* cap, const int64_t* seg_start, Part& p)
{
  const int i = (int)blockIdx.x;
  p.first = 0, p.tile = -1;
  p.cnt = i < nbricks ? min(count[i], cap[i]) : 0;
  p.start = i < nbricks ? seg_start[i] : 0;
  const int items = part_items(pv);
  p.b = i - items;
  if (i >= items) {
    if (p.b >= nbricks) return false;
    if (items) {
      if (pv.mark[p.b]) return false;
      p.cnt = min(count[p.b], cap[p.b]);
      p.start = seg_start[p.b];
    }
    return true;
  }
  const int4 w = pv.item[i];
  p.b = w.x;
  if (w.x < 0) return false;
  const int64_t n = min(count[p.b], cap[p.b]);
  p.start = seg_start[p.b];
  const int k = w.y;
  p.first = (int)(n * k / w.z) & ~3;  // parts start on 16-byte boundaries
  p.cnt = (k + 1 == w.z ? (int)n : (int)(n * (k + 1) / w.z) & ~3) - p.first;
  if (w.z > 1) p.tile = w.w + k;
  return true;
}

// A part's tile to the scratch: 8-byte values, component j of vertex t at
// j * N + t (the integer sum, the hi/lo pair or the float); quantum: CompUnit.
template <int ACC, bool SIGNED, int NC, int N>
__device__ __forceinline__ void part_store(uint64_t* dst, const TileRef<N>& tr, float quantum)
{
  const uint32_t* w = reinterpret_cast<const uint32_t*>(tr.smem);
  for (int t = threadIdx.x; t < N; t += blockDim.x) {
#pragma unroll
    for (int j = 0; j < NC; j++) {
      uint64_t q;
      if (ACC == ACC_FIXED) {
        q = (uint64_t)tile_fixed<SIGNED>(tr, j, t);
      } else if (ACC == ACC_COMP) {
        const float2 v = comp_pair(tr, j, t, quantum);
        q = (uint64_t)__float_as_uint(v.x) | ((uint64_t)__float_as_uint(v.y) << 32);
      } else {
        q = w[(size_t)j * N + t];
      }
      dst[(size_t)j * N + t] = q;
    }
  }
}

// Vertex sum over a split brick's parts, in part order: the integer, or the
// hi and lo words (lo 0 in the plain mode).
struct PartSum {
  long long q;
  float hi, lo;
};

template <int ACC>
__device__ __forceinline__ PartSum part_sum(const PartView& pv, const int4& sp, int slots, int at)
{
  PartSum r{0, 0.0f, 0.0f};
#pragma unroll 4
  for (int k = 0; k < sp.y; k++) {
    const uint64_t v = __ldg(scratch_tile(pv, sp.z + k, slots) + at);
    if (ACC == ACC_FIXED)
      r.q += (long long)v;
    else if (ACC == ACC_COMP)
      comp_acc(r.hi, r.lo, __uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
    else
      r.hi = __fadd_rn(r.hi, __uint_as_float((uint32_t)v));
  }
  return r;
}

// Largest relative mass of the part's particles, clamped as mass_q clamps it
// and rounded up to a whole number (at least 1): the factor by which a
// contribution can exceed a global-mass particle's.
__device__ __forceinline__ int part_mass_bound(const float* mass, uint32_t p0, int cnt,
                                               float inv_unit, unsigned* s_max)
{
  if (threadIdx.x == 0) *s_max = 0u;
  __syncthreads();
  float m = 0.0f;
  for (int i = threadIdx.x; i < cnt; i += blockDim.x)
    m = fmaxf(m, fminf(fmaxf(__fmul_rn(mass[p0 + (uint32_t)i], inv_unit), 0.0f), 63.0f));
  const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));  // non-negative floats
  if ((threadIdx.x & 31) == 0 && w) atomicMax(s_max, w);
  __syncthreads();
  return max(1, (int)ceilf(__uint_as_float(*s_max)));
}

}  // namespace lf2
