// lf2_store.cu -- device particle store: bulk load (counting sort into brick
// segments), download, per-cell counts and the repack that runs when a brick
// runs out of free slots.
//
// Replaces the per-cell std::forward_list storage of the reference
// (LATfield2_Particles.hpp:97-103, :333, :370-373) and addParticle_global
// (:500-540).  Loading is a counting sort over bricks: histogram, capacity
// (count + slack) and exclusive scan, then a scatter into the segments.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "lf2_internal.h"

namespace lf2 {

namespace {

constexpr int SLACK_MIN = 32;
__host__ __device__ inline int32_t slack_of(int32_t count)
{
  const int32_t s = count >> 3;
  return s > SLACK_MIN ? s : SLACK_MIN;
}

// Slots of a brick segment: the particles plus slack, rounded up to a
// multiple of 4 so that every segment starts on a 16-byte boundary.
__host__ __device__ inline int32_t cap_of(int32_t count)
{
  return (count + slack_of(count) + 3) & ~3;
}

__device__ inline bool decode_cell(const Geom& g, int32_t c, int& x, int& y, int& z)
{
  if (c < 0 || (int64_t)c >= g.nsites) return false;
  cell_xyz(g, c, x, y, z);
  return true;
}

__device__ inline bool valid_off(float o) { return o >= 0.0f && o < 1.0f; }

__global__ void k_load_count(Geom g, int64_t n, const int32_t* __restrict__ cell,
                             const float* __restrict__ off3, int32_t* count, uint32_t* flags)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, z;
    const bool ok = decode_cell(g, cell[i], x, y, z) && valid_off(off3[3 * i]) &&
                    valid_off(off3[3 * i + 1]) && valid_off(off3[3 * i + 2]);
    if (!ok) {
      set_flag(flags, ERR_BAD_CELL);
      continue;
    }
    atomicAdd(&count[brick_of(g, x, y, z)], 1);
  }
}

// The same for lattices whose brick counters fit a CTA's shared memory: a CTA
// counts its share of the particles there and adds each brick once, so that
// the bricks of a clump (millions of additions to one counter) do not
// serialise on their counter's address.  At 256^3 with half of 16.8M particles
// in 64 clumps: 78 us against 631 with the global counters.  (The scatter below
// keeps them: it is bound by its 4-byte writes to nine arrays, and ranks formed
// in shared memory took 1456 us against 1321 there.)
constexpr int LOAD_THREADS = 1024;

__device__ __forceinline__ void load_share(int64_t n, int64_t& i0, int64_t& i1)
{
  i0 = n * blockIdx.x / gridDim.x;
  i1 = n * (blockIdx.x + 1) / gridDim.x;
}

__global__ void __launch_bounds__(LOAD_THREADS) k_load_count_sh(Geom g, int64_t n,
                                                                const int32_t* __restrict__ cell,
                                                                const float* __restrict__ off3,
                                                                int32_t* count, uint32_t* flags)
{
  extern __shared__ int32_t h[];
  for (int b = threadIdx.x; b < g.nbricks; b += blockDim.x) h[b] = 0;
  __syncthreads();
  int64_t i0, i1;
  load_share(n, i0, i1);
  bool bad = false;
#pragma unroll 4
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    int x, y, z;
    const bool ok = decode_cell(g, cell[i], x, y, z);
    bad |= !ok || !valid_off(off3[3 * i]) || !valid_off(off3[3 * i + 1]) || !valid_off(off3[3 * i + 2]);
    if (ok) atomicAdd(&h[brick_of(g, x, y, z)], 1);
  }
  if (bad) set_flag(flags, ERR_BAD_CELL);  // the load is refused
  __syncthreads();
  for (int b = threadIdx.x; b < g.nbricks; b += blockDim.x)
    if (h[b]) atomicAdd(&count[b], h[b]);
}

// One CTA: cap[b] = count[b] + slack (when caps != nullptr), starts = exclusive
// scan of caps (or of counts), starts[nb] = total.
__global__ void __launch_bounds__(1024) k_caps_scan(int64_t nb, const int32_t* __restrict__ counts,
                                                    int32_t* caps, int64_t* starts, double* most)
{
  __shared__ int64_t sh[1024];
  __shared__ int s_most;
  const int t = threadIdx.x;
  const int64_t per = (nb + blockDim.x - 1) / blockDim.x;
  const int64_t lo = t * per, hi = min(nb, lo + per);
  int64_t s = 0;
  int m = 0;
  for (int64_t b = lo; b < hi; b++) {
    const int32_t c = counts[b], v = caps ? cap_of(c) : c;
    if (caps) caps[b] = v;
    s += v;
    m = max(m, c);
  }
  if (t == 0) s_most = 0;
  sh[t] = s;
  __syncthreads();
  m = __reduce_max_sync(0xffffffffu, m);
  if ((t & 31) == 0) atomicMax(&s_most, m);
  for (int o = 1; o < (int)blockDim.x; o <<= 1) {
    const int64_t add = t >= o ? sh[t - o] : 0;
    __syncthreads();
    sh[t] += add;
    __syncthreads();
  }
  int64_t run = sh[t] - s;
  for (int64_t b = lo; b < hi; b++) {
    starts[b] = run;
    run += caps ? caps[b] : counts[b];
  }
  if (t == blockDim.x - 1) starts[nb] = sh[t];
  if (t == 0 && most) *most = (double)s_most;
}

__global__ void k_load_scatter(Geom g, int64_t n, const int32_t* __restrict__ cell,
                               const float* __restrict__ off3, const float* __restrict__ vel3,
                               const float* __restrict__ mass, const int64_t* __restrict__ id,
                               const int64_t* __restrict__ seg_start, int32_t* fill, PartArrays a)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, z;
    const bool ok = decode_cell(g, cell[i], x, y, z) && valid_off(off3[3 * i]) &&
                    valid_off(off3[3 * i + 1]) && valid_off(off3[3 * i + 2]);
    if (!ok) continue;
    const int64_t b = brick_of(g, x, y, z);
    const int64_t p = seg_start[b] + atomicAdd(&fill[b], 1);
    a.key[p] = pack_key(g, x, y, z);
    a.ox[p] = off3[3 * i];
    a.oy[p] = off3[3 * i + 1];
    a.oz[p] = off3[3 * i + 2];
    a.vx[p] = vel3[3 * i];
    a.vy[p] = vel3[3 * i + 1];
    a.vz[p] = vel3[3 * i + 2];
    if (a.mass) a.mass[p] = mass[i];
    if (a.id) a.id[p] = id[i];
  }
}

// Position in box units -> (cell, offset): u = pos / res, cell = floor(u) mod n
// (getPartCoord, LATfield2_Particles.hpp:463-467), offset = u - floor(u) in FP32.
template <typename T>
__global__ void k_pos_to_state(Geom g, double inv_res, int64_t n, const T* __restrict__ pos3,
                               int32_t* cell, float* off3)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int c[3];
    for (int d = 0; d < 3; d++) {
      const double u = (double)pos3[3 * i + d] * inv_res;
      double fl = floor(u);
      float o = (float)(u - fl);
      if (o >= 1.0f) {
        o = 0.0f;
        fl += 1.0;
      }
      long long ci = (long long)fl % g.n[d];
      if (ci < 0) ci += g.n[d];
      c[d] = (int)ci;
      off3[3 * i + d] = isfinite(u) ? o : -1.0f;  // -1 is rejected by the load
    }
    cell[i] = (int32_t)site_index(g, c[0], c[1], c[2]);
  }
}

template <typename T>
__global__ void k_state_to_pos(Geom g, double res, int64_t n, const int32_t* __restrict__ cell,
                               const float* __restrict__ off3, T* pos3)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = cell[i];
    int x, y, z;
    cell_xyz(g, c, x, y, z);
    pos3[3 * i + 0] = (T)(((double)x + (double)off3[3 * i + 0]) * res);
    pos3[3 * i + 1] = (T)(((double)y + (double)off3[3 * i + 1]) * res);
    pos3[3 * i + 2] = (T)(((double)z + (double)off3[3 * i + 2]) * res);
  }
}

// One CTA per brick: copy the brick's particles to a dense output.
__global__ void k_get(StoreView v, const int64_t* __restrict__ out_start, int32_t* cell,
                      float* off3, float* vel3, float* mass, int64_t* id)
{
  const int64_t b = blockIdx.x;
  const int64_t base = v.seg_start[b], o0 = out_start[b];
  const int cnt = LF2_BRICK_COUNT(v, b);
  for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
    const int64_t p = base + i, o = o0 + i;
    int x, y, z;
    unpack_key(v.g, v.a.key[p], x, y, z);
    if (cell) cell[o] = (int32_t)site_index(v.g, x, y, z);
    if (off3) {
      off3[3 * o] = v.a.ox[p];
      off3[3 * o + 1] = v.a.oy[p];
      off3[3 * o + 2] = v.a.oz[p];
    }
    if (vel3) {
      vel3[3 * o] = v.a.vx[p];
      vel3[3 * o + 1] = v.a.vy[p];
      vel3[3 * o + 2] = v.a.vz[p];
    }
    if (mass && v.a.mass) mass[o] = v.a.mass[p];
    if (id && v.a.id) id[o] = v.a.id[p];
  }
}

__global__ void k_cell_counts(StoreView v, int32_t* counts)
{
  const int64_t b = blockIdx.x;
  const int64_t base = v.seg_start[b];
  const int cnt = LF2_BRICK_COUNT(v, b);
  for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
    int x, y, z;
    unpack_key(v.g, v.a.key[base + i], x, y, z);
    atomicAdd(&counts[site_index(v.g, x, y, z)], 1);
  }
}

// ------------------------------------------------- relocation and repack
// After k_insert.  A brick that ran out of free slots there is moved on its
// own to a fresh, larger segment carved from the relocation region (bump
// allocation past the contiguous segments); its old slots are abandoned until
// the next full repack.  Only when the region is exhausted is the whole store
// repacked.  One cooperative kernel: in most steps no brick ran out and it
// returns at once (nine kernels that each found nothing to do took 20 us of
// a step, 25% of the smallest); otherwise its phases are separated by grid
// barriers, without a host round trip.

// One particle's arrays, read before any is written (source and destination
// may be the same arrays, so interleaved loads and stores would wait for
// each other).
struct PartVal {
  uint32_t key;
  float ox, oy, oz, vx, vy, vz, m;
  int64_t id;
};

__device__ inline PartVal load_particle(const PartArrays& s, int64_t ps)
{
  PartVal p;
  p.key = s.key[ps];
  p.ox = s.ox[ps];
  p.oy = s.oy[ps];
  p.oz = s.oz[ps];
  p.vx = s.vx[ps];
  p.vy = s.vy[ps];
  p.vz = s.vz[ps];
  p.m = s.mass ? s.mass[ps] : 0.0f;
  p.id = s.id ? s.id[ps] : 0;
  return p;
}

__device__ inline void store_particle(const PartArrays& d, int64_t pd, const PartVal& p)
{
  d.key[pd] = p.key;
  d.ox[pd] = p.ox;
  d.oy[pd] = p.oy;
  d.oz[pd] = p.oz;
  d.vx[pd] = p.vx;
  d.vy[pd] = p.vy;
  d.vz[pd] = p.vz;
  if (d.mass) d.mass[pd] = p.m;
  if (d.id) d.id[pd] = p.id;
}

__device__ inline void copy_particle(const PartArrays& s, int64_t ps, const PartArrays& d, int64_t pd)
{
  store_particle(d, pd, load_particle(s, ps));
}

// Copies n consecutive particles, four per thread in flight.
__device__ inline void copy_run(const PartArrays& s, int64_t s0, const PartArrays& d, int64_t d0, int n)
{
  for (int i = threadIdx.x; i < n; i += 4 * blockDim.x) {
    PartVal v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = i + u * (int)blockDim.x;
      if (k < n) v[u] = load_particle(s, s0 + k);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = i + u * (int)blockDim.x;
      if (k < n) store_particle(d, d0 + k, v[u]);
    }
  }
}

struct RebinTail {
  StoreView v;
  PartArrays alt, mov;
  int64_t* seg_start;
  int32_t* cap;
  int64_t* start_alt;
  int32_t* cap_alt;
  int32_t* fill;
  int32_t* placed;
  const unsigned long long* mov_count;
  const int32_t* list;  // bricks that ran out of slots
  int32_t* nlist;
  int32_t* state;       // 1 listed, 2 relocated
  unsigned long long* heap_top;
  int64_t capacity;
  int32_t* repack;
  uint32_t* flags;
  unsigned long long* diag;
  PartPlan plan;        // of the deposit that follows (0 items: none)
};

constexpr int TAIL_THREADS = 1024;

// Capacities and starts of a full repack (one CTA).
__device__ void repack_caps(const RebinTail& t, int64_t* sh)
{
  const int64_t nb = t.v.g.nbricks, per = (nb + blockDim.x - 1) / blockDim.x;
  const int64_t lo = threadIdx.x * per, hi = min(nb, lo + per);
  int64_t s = 0;
  for (int64_t b = lo; b < hi; b++) s += t.cap_alt[b] = cap_of(t.v.count[b]);
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < (int)blockDim.x; o <<= 1) {
    const int64_t add = (int)threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
    __syncthreads();
    sh[threadIdx.x] += add;
    __syncthreads();
  }
  int64_t run = sh[threadIdx.x] - s;
  for (int64_t b = lo; b < hi; b++) {
    t.start_alt[b] = run;
    run += t.cap_alt[b];
  }
  if (threadIdx.x == blockDim.x - 1) {
    t.start_alt[nb] = sh[threadIdx.x];
    if (sh[threadIdx.x] > t.capacity) {
      set_flag(t.flags, ERR_CAPACITY);
      *t.repack = 0;  // cannot repack: leave the store as it is
    }
  }
}

__global__ void __launch_bounds__(TAIL_THREADS, 1) k_rebin_tail(RebinTail t)
{
  __shared__ int64_t sh[TAIL_THREADS];
  __shared__ long long s_new;
  const int n = *t.nlist;
  const Geom& g = t.v.g;
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  auto plan = [&]() {
    if (t.plan.max_items)
      for (int64_t b = i0; b < g.nbricks; b += stride)
        part_plan_brick(t.plan, (int)b, min(t.v.count[b], t.cap[b]));
  };
  if (n == 0) {
    plan();
    if (blockIdx.x == 0 && threadIdx.x == 0) t.diag[1] = *t.mov_count;
    return;
  }
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const int64_t nm = (int64_t)*t.mov_count;

  // full bricks into new segments
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t b = t.list[i];
    const int32_t need = t.v.count[b];  // stays + every arrival that tried
    const int32_t placed = min(need, t.cap[b]);
    const int32_t ncap = cap_of(need);
    if (threadIdx.x == 0) {
      const unsigned long long s0 = atomicAdd(t.heap_top, (unsigned long long)ncap);
      s_new = (s0 + (unsigned long long)ncap <= (unsigned long long)t.capacity) ? (long long)s0 : -1;
      if (s_new < 0) *t.repack = 1;  // region exhausted: repack everything
    }
    __syncthreads();
    const long long d0 = s_new;
    if (d0 >= 0) {
      const int64_t s0 = t.seg_start[b];
      copy_run(t.v.a, s0, t.v.a, d0, placed);
      __syncthreads();
      if (threadIdx.x == 0) {
        t.seg_start[b] = d0;
        t.cap[b] = ncap;
        t.fill[b] = placed;
        t.state[b] = 2;
        atomicAdd(&t.diag[2], 1ull);
      }
    }
    __syncthreads();
  }
  grid.sync();
  // their movers that found no slot
  for (int64_t m = i0; m < nm; m += stride) {
    if (t.placed[m]) continue;
    int x, y, z;
    unpack_key(g, t.mov.key[m], x, y, z);
    const int64_t b = brick_of(g, x, y, z);
    if (t.state[b] != 2) continue;  // not relocated: left to the full repack
    copy_particle(t.mov, m, t.v.a, t.seg_start[b] + atomicAdd(&t.fill[b], 1));
    t.placed[m] = 1;
  }
  if (*t.repack) {  // set before the barrier
    grid.sync();
    if (blockIdx.x == 0) repack_caps(t, sh);
    grid.sync();
    if (*t.repack) {
      for (int64_t b = blockIdx.x; b < g.nbricks; b += gridDim.x) {
        const int placed = min(t.v.count[b], t.cap[b]);
        copy_run(t.v.a, t.seg_start[b], t.alt, t.start_alt[b], placed);
        if (threadIdx.x == 0) t.fill[b] = placed;
      }
      grid.sync();
      for (int64_t m = i0; m < nm; m += stride) {
        if (t.placed[m]) continue;
        int x, y, z;
        unpack_key(g, t.mov.key[m], x, y, z);
        const int64_t b = brick_of(g, x, y, z);
        copy_particle(t.mov, m, t.alt, t.start_alt[b] + atomicAdd(&t.fill[b], 1));
      }
      grid.sync();
      for (int64_t b = blockIdx.x; b < g.nbricks; b += gridDim.x) {
        copy_run(t.alt, t.start_alt[b], t.v.a, t.start_alt[b], t.fill[b]);
        if (threadIdx.x == 0) {
          t.v.count[b] = t.fill[b];
          t.seg_start[b] = t.start_alt[b];
          t.cap[b] = t.cap_alt[b];
        }
      }
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        t.seg_start[g.nbricks] = t.start_alt[g.nbricks];
        // the relocation region starts after the segments
        *t.heap_top = (unsigned long long)t.start_alt[g.nbricks];
      }
    }
  }
  grid.sync();
  plan();
  if (blockIdx.x != 0) return;
  for (int i = threadIdx.x; i < n; i += blockDim.x) t.state[t.list[i]] = 0;
  if (threadIdx.x == 0) {
    if (*t.repack) {
      set_flag(t.flags, ERR_REPACK);
      t.diag[0] += 1;
      *t.repack = 0;
    }
    t.diag[1] = *t.mov_count;
    *t.nlist = 0;
  }
}

inline int grid_for(int64_t n, int threads)
{
  int64_t g = (n + threads - 1) / threads;
  if (g > 148 * 32) g = 148 * 32;
  return (int)(g > 0 ? g : 1);
}

}  // namespace

// Brick counters of a load in a CTA's shared memory: bytes, or 0 where they
// do not fit (above 51,200 bricks, lattices beyond 590^3).
constexpr size_t LOAD_COUNTERS_MAX = 200 * 1024;

static size_t load_counters(const lf2_ctx* c)
{
  const size_t bytes = sizeof(int32_t) * (size_t)c->g.nbricks;
  return bytes <= LOAD_COUNTERS_MAX ? bytes : 0;
}

// CTAs of a load: those that run at once, fewer when they would hold under 4096
// particles.
static unsigned load_ctas(const lf2_ctx* c, int64_t n)
{
  const int64_t most = (n + 4095) / 4096;
  const int64_t all = (int64_t)c->num_sms * (load_counters(c) <= 100 * 1024 ? 2 : 1);
  return (unsigned)(most < 1 ? 1 : most < all ? most : all);
}

cudaError_t launch_load_count(lf2_ctx* c, int64_t n, const int32_t* cell, const float* off3)
{
  c->launches += 1;
  if (const size_t sh = load_counters(c)) {
    // (the setting is the kernel's, not the call's: one value for all, since
    // contexts of other sizes may load from other threads)
    const cudaError_t e = cudaFuncSetAttribute(k_load_count_sh, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)LOAD_COUNTERS_MAX);
    if (e != cudaSuccess) return e;
    k_load_count_sh<<<load_ctas(c, n), LOAD_THREADS, sh, c->stream>>>(c->g, n, cell, off3, c->count, c->flags);
    return cudaGetLastError();
  }
  k_load_count<<<grid_for(n, 256), 256, 0, c->stream>>>(c->g, n, cell, off3, c->count, c->flags);
  return cudaGetLastError();
}

cudaError_t launch_caps_and_scan(lf2_ctx* c, const int32_t* counts, int32_t* caps, int64_t* starts,
                                 int64_t*)
{
  c->launches += 1;
  k_caps_scan<<<1, 1024, 0, c->stream>>>(c->g.nbricks, counts, caps, starts, c->stats + 1);
  return cudaGetLastError();
}

cudaError_t launch_scan_counts(lf2_ctx* c, int64_t* out_start)
{
  c->launches += 1;
  k_caps_scan<<<1, 1024, 0, c->stream>>>(c->g.nbricks, c->count, nullptr, out_start, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_load_scatter(lf2_ctx* c, int64_t n, const int32_t* cell, const float* off3,
                                const float* vel3, const float* mass, const int64_t* id)
{
  c->launches += 1;
  k_load_scatter<<<grid_for(n, 256), 256, 0, c->stream>>>(c->g, n, cell, off3, vel3, mass, id,
                                                           c->seg_start, c->fill, c->cur);
  return cudaGetLastError();
}

cudaError_t launch_pos_to_state(lf2_ctx* c, int64_t n, const void* pos3, int real_bytes,
                                int32_t* cell, float* off3)
{
  c->launches += 1;
  const double inv_res = 1.0 / c->res;
  if (real_bytes == 8)
    k_pos_to_state<double><<<grid_for(n, 256), 256, 0, c->stream>>>(
        c->g, inv_res, n, (const double*)pos3, cell, off3);
  else
    k_pos_to_state<float><<<grid_for(n, 256), 256, 0, c->stream>>>(
        c->g, inv_res, n, (const float*)pos3, cell, off3);
  return cudaGetLastError();
}

cudaError_t launch_state_to_pos(lf2_ctx* c, int64_t n, const int32_t* cell, const float* off3,
                                void* pos3, int real_bytes)
{
  c->launches += 1;
  if (real_bytes == 8)
    k_state_to_pos<double><<<grid_for(n, 256), 256, 0, c->stream>>>(c->g, c->res, n, cell, off3,
                                                                     (double*)pos3);
  else
    k_state_to_pos<float><<<grid_for(n, 256), 256, 0, c->stream>>>(c->g, c->res, n, cell, off3,
                                                                    (float*)pos3);
  return cudaGetLastError();
}

cudaError_t launch_get(lf2_ctx* c, int64_t* out_start, int32_t* cell, float* off3, float* vel3,
                       float* mass, int64_t* id)
{
  c->launches += 1;
  k_get<<<(unsigned)c->g.nbricks, 256, 0, c->stream>>>(view(c), out_start, cell, off3, vel3, mass,
                                                       id);
  return cudaGetLastError();
}

cudaError_t launch_cell_counts(lf2_ctx* c, int32_t* counts)
{
  c->launches += 1;
  cudaError_t e = cudaMemsetAsync(counts, 0, sizeof(int32_t) * c->g.nsites, c->stream);
  if (e != cudaSuccess) return e;
  k_cell_counts<<<(unsigned)c->g.nbricks, 256, 0, c->stream>>>(view(c), counts);
  return cudaGetLastError();
}

cudaError_t launch_heap_reset(lf2_ctx* c)
{
  return cudaMemcpyAsync(c->heap_top, c->seg_start + c->g.nbricks, sizeof(unsigned long long),
                         cudaMemcpyDeviceToDevice, c->stream);
}

cudaError_t launch_repack(lf2_ctx* c, const PartPlan* plan)
{
  RebinTail t;
  t.plan = plan ? *plan : PartPlan{};
  t.v = view(c);
  t.alt = c->alt, t.mov = c->mov;
  t.seg_start = c->seg_start, t.cap = c->cap;
  t.start_alt = c->seg_start_alt, t.cap_alt = c->cap_alt, t.fill = c->fill;
  t.placed = c->mov_placed, t.mov_count = c->mov_count;
  t.list = c->ovf_list, t.nlist = c->ovf_count, t.state = c->ovf_state;
  t.heap_top = c->heap_top, t.capacity = c->capacity;
  t.repack = c->repack, t.flags = c->flags, t.diag = c->diag;
  void* args[] = {&t};
  c->launches += 1;
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&k_rebin_tail), dim3(c->num_sms),
                                     dim3(TAIL_THREADS), args, 0, c->stream);
}

}  // namespace lf2
