// lf2_field.cu -- field layout conversion, periodic halo fill and the FP64
// conservation reductions.
//
// Internal field layout: FP32, component-major, no halo, periodic.  The
// reference layout (LATfield2_Field_decl.hpp:760-788, LATfield2_Lattice.hpp:
// 110-113) is halo'd with interleaved components: data[idx * C + c] with
// idx = (x+h) + G0 * ((y+h) + G1 * (z+h)), Gi = ni + 2h.
#include <cuda_runtime.h>

#include <type_traits>

#include "lf2_internal.h"

namespace lf2 {

namespace {

inline int grid_for(int64_t n, int threads)
{
  int64_t g = (n + threads - 1) / threads;
  if (g > 148 * 64) g = 148 * 64;
  return (int)(g > 0 ? g : 1);
}

__device__ inline int wrap_coord(int v, int n)
{
  v %= n;
  return v < 0 ? v + n : v;
}

// Layout conversion, a warp per row of sites along x, or per chunk of a long
// row: the row's y and z are divided out and wrapped once, and a lane takes
// elements e = x * comps + c of the reference's row, so that its accesses are
// contiguous.  Rows under ROW_MIN sites leave lanes idle and pay the divisions
// for few of them: those go by sites.  In us, by sites / by rows: 256^3 to double
// with a halo 138 / 52, its 3-component import 101 / 74; 33 x 200 x 200, 3
// components 17 / 21; 20 x 20 x 20,000, 3 components to double 96 / 156; 7 x 9 x
// 100,000, 3 components 62 / 172; 10^6 x 1 x 1 13 / 17 (6400 without chunks).
constexpr int ROW_MIN = 48;

struct RowUnits {
  int64_t units;  // chunks of all rows
  int chunks;     // of a row
  int span;       // elements of a chunk
};

inline RowUnits row_units(int64_t rows, int64_t row_elements, int lane_elements)
{
  RowUnits u;
  u.span = 32 * lane_elements;
  u.chunks = (int)((row_elements + u.span - 1) / u.span);
  u.units = rows * u.chunks;
  return u;
}

// fn(row, first element of the lane, end) for the chunks of this warp.
// I: an integer that holds the elements of a row and 32 more.
template <typename I, typename Fn>
__device__ __forceinline__ void for_rows(const RowUnits& ru, I row_elements, Fn fn)
{
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t u = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); u < ru.units; u += warps) {
    int64_t row = u;
    I e0 = lane, end = row_elements;
    if (ru.chunks > 1) {
      row = u / ru.chunks;
      const I first = (I)(u - row * ru.chunks) * ru.span, left = row_elements - first;
      e0 += first;
      end = first + (left < ru.span ? left : ru.span);
    }
    fn(row, e0, end);
  }
}

// COMPS 0: any number of components.
template <int COMPS, typename I>
__device__ __forceinline__ void element(I e, int comps, int& x, int& c)
{
  if (COMPS == 1) {
    x = (int)e, c = 0;
  } else {
    const I n = COMPS ? COMPS : comps;
    x = (int)(e / n);
    c = (int)(e - x * n);
  }
}

// Every gross site of the reference layout; halo sites either copy their
// periodic image (Field::updateHalo, LATfield2_Field_decl.hpp:889-935) or are 0.
template <typename T, int COMPS, typename I>
__global__ void __launch_bounds__(256) k_export(Geom g, RowUnits ru, int comps, const float* __restrict__ src,
                                                T* __restrict__ dst, int halo, int fill_halo)
{
  const int G0 = g.n[0] + 2 * halo, G1 = g.n[1] + 2 * halo;
  const int nc = COMPS ? COMPS : comps;
  for_rows<I>(ru, (I)G0 * nc, [&](int64_t row, I e0, I end) {
    int y = (int)(row % G1) - halo, z = (int)(row / G1) - halo;
    const bool inside = y >= 0 && y < g.n[1] && z >= 0 && z < g.n[2];
    y = wrap_coord(y, g.n[1]);
    z = wrap_coord(z, g.n[2]);
    const float* s = src + site_index(g, 0, y, z);
    T* d = dst + row * G0 * nc;
#pragma unroll 4
    for (I e = e0; e < end; e += 32) {
      int x, c;
      element<COMPS, I>(e, comps, x, c);
      x -= halo;
      const bool in = inside && x >= 0 && x < g.n[0];
      if (x < 0 || x >= g.n[0]) x = wrap_coord(x, g.n[0]);
      d[e] = in || fill_halo ? (T)__ldg(s + c * g.nsites + x) : (T)0;
    }
  });
}

// By elements up to 3 components, by sites above: there the writes of one
// component would be short runs (6 components at 256^3 by elements: 198 us).
constexpr bool by_sites(int comps) { return comps == 0 || comps > 3; }

template <typename T, int COMPS, typename I>
__global__ void __launch_bounds__(256) k_import(Geom g, RowUnits ru, int comps, float* __restrict__ dst,
                                                const T* __restrict__ src, int halo)
{
  const int64_t G0 = g.n[0] + 2 * halo, G1 = g.n[1] + 2 * halo;
  const int nc = COMPS ? COMPS : comps;
  constexpr bool SITES = by_sites(COMPS);
  for_rows<I>(ru, (I)g.n[0] * (SITES ? 1 : nc), [&](int64_t row, I e0, I end) {
    const int y = (int)(row % g.n[1]), z = (int)(row / g.n[1]);
    const T* s = src + (halo + G0 * (y + halo + G1 * (z + halo))) * nc;
    float* d = dst + row * g.n[0];
    if constexpr (SITES) {
      for (I e = e0; e < end; e += 32) {
#pragma unroll(COMPS ? COMPS : 4)
        for (int c = 0; c < nc; c++) d[c * g.nsites + e] = (float)__ldg(s + (int64_t)e * nc + c);
      }
    } else {
#pragma unroll 4
      for (I e = e0; e < end; e += 32) {
        int x, c;
        element<COMPS, I>(e, comps, x, c);
        d[c * g.nsites + x] = (float)__ldg(s + e);
      }
    }
  });
}

// The same by sites, for short rows.
template <typename T>
__global__ void __launch_bounds__(256) k_export_sites(Geom g, int comps, const float* __restrict__ src,
                                                      T* __restrict__ dst, int halo, int fill_halo)
{
  const int64_t G0 = g.n[0] + 2 * halo, G1 = g.n[1] + 2 * halo, total = G0 * G1 * (g.n[2] + 2 * halo);
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = idx / G0;
    int x = (int)(idx - row * G0) - halo, y = (int)(row % G1) - halo, z = (int)(row / G1) - halo;
    const bool inside = x >= 0 && x < g.n[0] && y >= 0 && y < g.n[1] && z >= 0 && z < g.n[2];
    x = wrap_coord(x, g.n[0]);
    y = wrap_coord(y, g.n[1]);
    z = wrap_coord(z, g.n[2]);
    const int64_t s = site_index(g, x, y, z);
    for (int c = 0; c < comps; c++)
      dst[idx * comps + c] = inside || fill_halo ? (T)src[c * g.nsites + s] : (T)0;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_import_sites(Geom g, int comps, float* __restrict__ dst,
                                                      const T* __restrict__ src, int halo)
{
  const int64_t G0 = g.n[0] + 2 * halo, G1 = g.n[1] + 2 * halo;
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < g.nsites;
       s += (int64_t)gridDim.x * blockDim.x) {
    int x, y, z;
    cell_xyz(g, (int32_t)s, x, y, z);
    const int64_t idx = (x + halo) + G0 * ((y + halo) + G1 * (int64_t)(z + halo));
    for (int c = 0; c < comps; c++) dst[c * g.nsites + s] = (float)src[idx * comps + c];
  }
}

// In-place halo fill of a device array in the reference layout.
template <typename T>
__global__ void k_halo_fill(Geom g, int comps, T* __restrict__ data, int halo)
{
  const int64_t G0 = g.n[0] + 2 * halo, G1 = g.n[1] + 2 * halo, G2 = g.n[2] + 2 * halo;
  const int64_t total = G0 * G1 * G2;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(idx % G0) - halo;
    const int y = (int)((idx / G0) % G1) - halo;
    const int z = (int)(idx / (G0 * G1)) - halo;
    if (x >= 0 && x < g.n[0] && y >= 0 && y < g.n[1] && z >= 0 && z < g.n[2]) continue;
    const int64_t from = (wrap_coord(x, g.n[0]) + halo) +
                         G0 * ((wrap_coord(y, g.n[1]) + halo) + G1 * (int64_t)(wrap_coord(z, g.n[2]) + halo));
    for (int c = 0; c < comps; c++) data[idx * comps + c] = data[from * comps + c];
  }
}

// FP64 sums per brick: mass, m*vx, m*vy, m*vz and max |v|^2, then a fixed-order
// reduction over bricks (one CTA) so the totals are reproducible.
// Per brick, in a fixed order: mass, momentum (3), max |v|^2, sum |v|^2,
// min |v|^2 (FP64; |v|^2 in double from the FP32 components, as the
// reference's callbacks compute it).
constexpr int NSUM = 7;

__global__ void __launch_bounds__(256) k_brick_sums(StoreView v, double gmass, double* out)
{
  __shared__ double sh[NSUM][256];
  const int64_t b = blockIdx.x;
  const int64_t base = v.seg_start[b];
  const int cnt = LF2_BRICK_COUNT(v, b);
  double s[NSUM] = {0, 0, 0, 0, 0, 0, INFINITY};
  for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
    const int64_t p = base + i;
    const double m = v.a.mass ? (double)v.a.mass[p] : gmass;
    const double vx = v.a.vx[p], vy = v.a.vy[p], vz = v.a.vz[p];
    const double v2 = vx * vx + vy * vy + vz * vz;
    s[0] += m;
    s[1] += m * vx;
    s[2] += m * vy;
    s[3] += m * vz;
    s[4] = fmax(s[4], v2);
    s[5] += v2;
    s[6] = fmin(s[6], v2);
  }
  for (int k = 0; k < NSUM; k++) sh[k][threadIdx.x] = s[k];
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      for (int k = 0; k < 4; k++) sh[k][threadIdx.x] += sh[k][threadIdx.x + o];
      sh[4][threadIdx.x] = fmax(sh[4][threadIdx.x], sh[4][threadIdx.x + o]);
      sh[5][threadIdx.x] += sh[5][threadIdx.x + o];
      sh[6][threadIdx.x] = fmin(sh[6][threadIdx.x], sh[6][threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x < NSUM) out[b * NSUM + threadIdx.x] = sh[threadIdx.x][0];
}

__global__ void __launch_bounds__(512) k_sum_bricks(int64_t nb, const double* __restrict__ in,
                                                    double* stats)
{
  __shared__ double sh[NSUM][512];
  const int t = threadIdx.x;
  const int64_t per = (nb + blockDim.x - 1) / blockDim.x;
  const int64_t lo = t * per, hi = min(nb, lo + per);
  double s[NSUM] = {0, 0, 0, 0, 0, 0, INFINITY};
  for (int64_t b = lo; b < hi; b++) {
    for (int k = 0; k < 4; k++) s[k] += in[b * NSUM + k];
    s[4] = fmax(s[4], in[b * NSUM + 4]);
    s[5] += in[b * NSUM + 5];
    s[6] = fmin(s[6], in[b * NSUM + 6]);
  }
  for (int k = 0; k < NSUM; k++) sh[k][t] = s[k];
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (t < o) {
      for (int k = 0; k < 4; k++) sh[k][t] += sh[k][t + o];
      sh[4][t] = fmax(sh[4][t], sh[4][t + o]);
      sh[5][t] += sh[5][t + o];
      sh[6][t] = fmin(sh[6][t], sh[6][t + o]);
    }
    __syncthreads();
  }
  if (t < NSUM) stats[1 + t] = sh[t][0];
}

}  // namespace

// The conversion kernel of a component count, by type: fn(comps constant,
// row index type).
template <typename Fn>
static void by_comps(int comps, int64_t row_elements, Fn fn)
{
  using std::integral_constant;
  if (row_elements > INT32_MAX - 64) fn(integral_constant<int, 0>{}, int64_t{});
  else if (comps == 1) fn(integral_constant<int, 1>{}, int{});
  else if (comps == 3) fn(integral_constant<int, 3>{}, int{});
  else if (comps == 6) fn(integral_constant<int, 6>{}, int{});
  else fn(integral_constant<int, 0>{}, int{});
}

cudaError_t launch_export(lf2_ctx* c, int comps, const float* src, void* dst, int halo,
                          int real_bytes, int fill_halo)
{
  c->launches += 1;
  const int64_t G0 = (int64_t)c->g.n[0] + 2 * halo;
  if (G0 < ROW_MIN) {
    const int sites = grid_for(G0 * (c->g.n[1] + 2 * halo) * (c->g.n[2] + 2 * halo), 256);
    if (real_bytes == 8)
      k_export_sites<double><<<sites, 256, 0, c->stream>>>(c->g, comps, src, (double*)dst, halo, fill_halo);
    else
      k_export_sites<float><<<sites, 256, 0, c->stream>>>(c->g, comps, src, (float*)dst, halo, fill_halo);
    return cudaGetLastError();
  }
  const RowUnits ru = row_units((int64_t)(c->g.n[1] + 2 * halo) * (c->g.n[2] + 2 * halo), G0 * comps, 64);
  const int grid = grid_for(ru.units * 32, 256);
  by_comps(comps, G0 * comps, [&](auto k, auto i) {
    constexpr int K = decltype(k)::value;
    using I = decltype(i);
    if (real_bytes == 8)
      k_export<double, K, I><<<grid, 256, 0, c->stream>>>(c->g, ru, comps, src, (double*)dst, halo, fill_halo);
    else
      k_export<float, K, I><<<grid, 256, 0, c->stream>>>(c->g, ru, comps, src, (float*)dst, halo, fill_halo);
  });
  return cudaGetLastError();
}

cudaError_t launch_import(lf2_ctx* c, int comps, float* dst, const void* src, int halo,
                          int real_bytes)
{
  c->launches += 1;
  if (c->g.n[0] < ROW_MIN) {
    const int sites = grid_for(c->g.nsites, 256);
    if (real_bytes == 8)
      k_import_sites<double><<<sites, 256, 0, c->stream>>>(c->g, comps, dst, (const double*)src, halo);
    else
      k_import_sites<float><<<sites, 256, 0, c->stream>>>(c->g, comps, dst, (const float*)src, halo);
    return cudaGetLastError();
  }
  by_comps(comps, (int64_t)c->g.n[0] * comps, [&](auto k, auto i) {
    constexpr int K = decltype(k)::value;
    using I = decltype(i);
    const RowUnits ru =
        row_units((int64_t)c->g.n[1] * c->g.n[2], (int64_t)c->g.n[0] * (by_sites(K) ? 1 : comps),
                  by_sites(K) ? 16 : 64);
    const int grid = grid_for(ru.units * 32, 256);
    if (real_bytes == 8)
      k_import<double, K, I><<<grid, 256, 0, c->stream>>>(c->g, ru, comps, dst, (const double*)src, halo);
    else
      k_import<float, K, I><<<grid, 256, 0, c->stream>>>(c->g, ru, comps, dst, (const float*)src, halo);
  });
  return cudaGetLastError();
}

cudaError_t launch_halo_fill(lf2_ctx* c, void* data, int comps, int halo, int real_bytes)
{
  c->launches += 1;
  const int64_t total =
      (int64_t)(c->g.n[0] + 2 * halo) * (c->g.n[1] + 2 * halo) * (c->g.n[2] + 2 * halo);
  if (real_bytes == 8)
    k_halo_fill<double><<<grid_for(total, 256), 256, 0, c->stream>>>(c->g, comps, (double*)data,
                                                                     halo);
  else
    k_halo_fill<float><<<grid_for(total, 256), 256, 0, c->stream>>>(c->g, comps, (float*)data,
                                                                    halo);
  return cudaGetLastError();
}

cudaError_t launch_conservation(lf2_ctx* c)
{
  c->launches += 2;
  k_brick_sums<<<(unsigned)c->g.nbricks, 256, 0, c->stream>>>(view(c), c->gmass, c->brick_sums);
  k_sum_bricks<<<1, 512, 0, c->stream>>>(c->g.nbricks, c->brick_sums, c->stats);
  return cudaGetLastError();
}

}  // namespace lf2
