// mf_cells.cu -- uniform-grid cell lists and the near-field correction pass.
//
// The packed all-pairs loop (FieldF2Body / ForceF2Body) evaluates every pair
// with the far-field form at max(r^2, r_near^2), which is exact beyond the
// near radius (2h for the field, 4h for the force) and merely finite inside
// it.  This pass visits, for each target, only the sources inside that radius
// (through a cell list with cells of edge >= 2h) and adds
//     exact pair term (SPH weights / fitted curves) - clamped far term,
// so the sum of both launches is the reference's kernel over all pairs.
// Near pairs are about 0.4 % (field) and 3 % (force) of all pairs at the
// benchmark densities.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "mf_internal.h"
#include "mf_sym.cuh"

namespace mfgb {
namespace {

__device__ __forceinline__ int32_t f2ord(float f) {
  const int32_t b = __float_as_int(f);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__host__ __device__ __forceinline__ float ord2f(int32_t b) {
#ifdef __CUDA_ARCH__
  return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff);
#else
  int32_t v = b >= 0 ? b : b ^ 0x7fffffff;
  float f;
  memcpy(&f, &v, 4);
  return f;
#endif
}

__global__ void k_bbox_init(int32_t* bbox, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 6 * n) bbox[i] = (i % 6) < 3 ? 0x7fffffff : int32_t(0x80000000);
}

// blockIdx.y = scene; blocks stride over its particles.
__global__ void k_bbox(const float4* __restrict__ pos, const int64_t* __restrict__ ranges, int32_t* bbox) {
  const int s = blockIdx.y;
  const int64_t off = ranges[2 * s], n = ranges[2 * s + 1];
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x) {
    const float4 p = pos[off + k];
    lo[0] = fminf(lo[0], p.x);
    lo[1] = fminf(lo[1], p.y);
    lo[2] = fminf(lo[2], p.z);
    hi[0] = fmaxf(hi[0], p.x);
    hi[1] = fmaxf(hi[1], p.y);
    hi[2] = fmaxf(hi[2], p.z);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      lo[c] = fminf(lo[c], __shfl_down_sync(0xffffffffu, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_down_sync(0xffffffffu, hi[c], o));
    }
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < 3; ++c) {
      atomicMin(&bbox[6 * s + c], f2ord(lo[c]));
      atomicMax(&bbox[6 * s + 3 + c], f2ord(hi[c]));
    }
}

__device__ __forceinline__ void cell_coords(const CellGrid& g, float x, float y, float z, int& ix, int& iy,
                                            int& iz) {
  ix = min(max(int((x - g.ox) * g.inv_cs), 0), g.nx - 1);
  iy = min(max(int((y - g.oy) * g.inv_cs), 0), g.ny - 1);
  iz = min(max(int((z - g.oz) * g.inv_cs), 0), g.nz - 1);
}

__global__ void k_count(const float4* __restrict__ pos, const CellGrid* __restrict__ grids, int n_scenes,
                        int64_t n_total, int32_t* __restrict__ counts, int32_t* __restrict__ cell_of) {
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < n_total;
       k += int64_t(gridDim.x) * blockDim.x) {
    // k enumerates the scenes' particles back to back; map it to a particle index.
    int lo = 0, hi = n_scenes - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (grids[mid].k_off <= k) lo = mid;
      else hi = mid - 1;
    }
    const CellGrid& g = grids[lo];
    const int64_t i = g.p_off + (k - g.k_off);
    const float4 p = pos[i];
    int ix, iy, iz;
    cell_coords(g, p.x, p.y, p.z, ix, iy, iz);
    const int64_t c = g.cell_off + (int64_t(iz) * g.ny + iy) * g.nx + ix;
    cell_of[k] = int32_t(c);
    atomicAdd(&counts[c], 1);
  }
}

// Exclusive scan of counts[0..n) into start[0..n], in three launches:
// per-tile sums, a scan of the tile sums, and each tile's scan plus its
// offset.  Tiles are kScanTile consecutive counts; integer sums, so the
// result does not depend on the split.
constexpr int kScanThreads = 256, kScanPer = 16, kScanTile = kScanThreads * kScanPer;

// Exclusive prefix of v over the block (blockDim.x == kScanThreads); *total
// gets the block's sum.  Uses `ws` (kScanThreads / 32 ints of shared memory).
__device__ __forceinline__ int32_t block_exclusive_scan(int32_t v, int32_t* ws, int32_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int kW = kScanThreads / 32;
  int32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();  // ws is free (an earlier call may still read it)
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  if (w == 0) {
    const int32_t x = lane < kW ? ws[lane] : 0;
    int32_t xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, xi, o);
      if (lane >= o) xi += t;
    }
    if (lane < kW) ws[lane] = xi - x;
    if (lane == kW - 1) ws[kW] = xi;
  }
  __syncthreads();
  *total = ws[kW];
  return inc - v + ws[w];
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const int32_t* __restrict__ counts, int64_t n,
                                                             int32_t* __restrict__ tile_sum) {
  __shared__ int32_t ws[kScanThreads / 32 + 1];
  const int64_t base = int64_t(blockIdx.x) * kScanTile;
  int32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t i = base + int64_t(k) * kScanThreads + threadIdx.x;
    if (i < n) s += counts[i];
  }
  int32_t total;
  block_exclusive_scan(s, ws, &total);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}

// One block: tile sums -> exclusive tile offsets (in place); start[n] = total.
__global__ void __launch_bounds__(kScanThreads) k_scan_tile_sums(int32_t* __restrict__ tile_sum, int64_t n_tiles,
                                                                 int32_t* __restrict__ start, int64_t n) {
  __shared__ int32_t ws[kScanThreads / 32 + 1];
  int32_t run = 0;
  for (int64_t b0 = 0; b0 < n_tiles; b0 += kScanThreads) {
    const int64_t b = b0 + threadIdx.x;
    const int32_t v = b < n_tiles ? tile_sum[b] : 0;
    int32_t total;
    const int32_t ex = block_exclusive_scan(v, ws, &total);
    if (b < n_tiles) tile_sum[b] = run + ex;
    run += total;
  }
  if (threadIdx.x == 0) start[n] = run;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const int32_t* __restrict__ counts, int64_t n,
                                                             const int32_t* __restrict__ tile_off,
                                                             int32_t* __restrict__ start) {
  __shared__ int32_t ws[kScanThreads / 32 + 1];
  const int64_t base = int64_t(blockIdx.x) * kScanTile + int64_t(threadIdx.x) * kScanPer;
  int32_t c[kScanPer];
  int32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    c[k] = base + k < n ? counts[base + k] : 0;
    s += c[k];
  }
  int32_t total;
  int32_t run = tile_off[blockIdx.x] + block_exclusive_scan(s, ws, &total);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    if (base + k < n) start[base + k] = run;
    run += c[k];
  }
}

__global__ void k_scatter(const CellGrid* __restrict__ grids, int n_scenes, int64_t n_total,
                          const int32_t* __restrict__ cell_of, int32_t* __restrict__ cursor,
                          int32_t* __restrict__ perm) {
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < n_total;
       k += int64_t(gridDim.x) * blockDim.x) {
    int lo = 0, hi = n_scenes - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (grids[mid].k_off <= k) lo = mid;
      else hi = mid - 1;
    }
    const int64_t i = grids[lo].p_off + (k - grids[lo].k_off);
    const int32_t slot = atomicAdd(&cursor[cell_of[k]], 1);
    perm[slot] = int32_t(i);
  }
}

// Each cell's list in increasing particle index: one warp per cell places
// every entry at its rank (entries are distinct), from the scattered list
// `in` into `out`.
__global__ void k_sort_cells(const int32_t* __restrict__ start, int64_t n_cells, const int32_t* __restrict__ in,
                             int32_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t c = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); c < n_cells; c += warps) {
    const int32_t b = start[c], m = start[c + 1] - b;
    for (int32_t k = lane; k < m; k += 32) {
      const int32_t v = in[b + k];
      int32_t rank = 0;
      for (int32_t l = 0; l < m; ++l) rank += in[b + l] < v;
      out[b + rank] = v;
    }
  }
}

// Records 2 p and 2 p + 1 of src[0..n) in pair layout (a missing partner as zeros).
__device__ __forceinline__ void pair_records(const float4* __restrict__ src, float4* __restrict__ dst, int64_t n,
                                             int64_t p) {
  const float4 a = src[2 * p];
  const float4 b = (2 * p + 1 < n) ? src[2 * p + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
  dst[2 * p] = make_float4(a.x, b.x, a.y, b.y);
  dst[2 * p + 1] = make_float4(a.z, b.z, 0.f, 0.f);
}

__constant__ ForceTable c_fit_tbl = make_force_table();

// The binned particles in cell order (positions and the product's dipoles),
// so the correction reads each row of cells as one contiguous range.  mom2
// (optional): the dipoles mom[0..n) in pair layout too (to_pairs), for the
// packed product that follows.
__global__ void k_gather_sorted(const int32_t* __restrict__ perm, const float4* __restrict__ pos,
                                const float4* __restrict__ mom, int64_t n, float4* __restrict__ spos,
                                float4* __restrict__ smom, const int32_t* __restrict__ done_count, int done_total,
                                float4* __restrict__ mom2) {
  if (done_count && *done_count >= done_total) return;
  if (mom2)
    for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < (n + 1) / 2; p += int64_t(gridDim.x) * blockDim.x)
      pair_records(mom, mom2, n, p);
  for (int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += int64_t(gridDim.x) * blockDim.x) {
    const int32_t i = perm[q];
    spos[q] = pos[i];
    smom[q] = mom[i];
  }
}

// Correction of a source's pair with two targets at once (packed FP32, lanes
// .x / .y), exact minus clamped, added to acc[0..3): the force on the targets
// (over K, contracted with the targets' dipoles) or 4 pi times the field at
// them.  Without a branch: pairs beyond the near radius (and a particle with
// itself, for the force) get zero coefficients.
struct NearConsts {
  float near2, h, inv_h, ih3_30, ih5_30, ih4k, cA, cB;
  float c3;  // 3 ih5_unit: the field's alphas (ih5_30, cA) are in units of ih5_unit
};
struct NearTargets {  // two targets: positions, then dipoles (force)
  float4 xy, zm, mm;  // (x0, x1, y0, y1), (z0, z1, mx0, mx1), (my0, my1, mz0, mz1)
};
struct NearSource {
  float2 x, y, z, mx, my, mz;  // each value in both lanes
};
template <bool kForce>
__device__ __forceinline__ void near_pair2(const NearTargets& t, const NearSource& s, const NearConsts& c,
                                           const float* __restrict__ tbl, float2* acc) {
  const float2 dx = f2_sub(make_float2(t.xy.x, t.xy.y), s.x);
  const float2 dy = f2_sub(make_float2(t.xy.z, t.xy.w), s.y);
  const float2 dz = f2_sub(make_float2(t.zm.x, t.zm.y), s.z);
  const float2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
  const float2 ds = f2_fma(dz, s.mz, f2_fma(dy, s.my, f2_mul(dx, s.mx)));
  if constexpr (kForce) {
    const bool in0 = r2.x <= c.near2 && r2.x > 0.f, in1 = r2.y <= c.near2 && r2.y > 0.f;
    const float2 ri = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    const float2 q = f2_mul(f2_mul(r2, ri), f2_dup(c.inv_h));
    const float2 k = f2_mul(f2_dup(c.ih4k), ri);
    const float2 kr = f2_mul(k, f2_mul(ri, ri));
    float2 c1, c2;
    force_curves(q.x, tbl, c1.x, c2.x);
    force_curves(q.y, tbl, c1.y, c2.y);
    float2 dP = f2_fma(c1, k, f2_dup(-c.cA)), dQ = f2_fma(f2_fma(c1, f2_dup(-3.f), c2), kr, f2_dup(-c.cB));
    dP = make_float2(in0 ? dP.x : 0.f, in1 ? dP.y : 0.f);
    dQ = make_float2(in0 ? dQ.x : 0.f, in1 ? dQ.y : 0.f);
    const float2 tmx = make_float2(t.zm.z, t.zm.w), tmy = make_float2(t.mm.x, t.mm.y), tmz = make_float2(t.mm.z, t.mm.w);
    const float2 dm = f2_fma(dz, tmz, f2_fma(dy, tmy, f2_mul(dx, tmx)));
    const float2 sm = f2_fma(s.mz, tmz, f2_fma(s.my, tmy, f2_mul(s.mx, tmx)));
    const float2 u = f2_mul(dP, ds), v = f2_mul(dP, dm), w = f2_fma(f2_mul(dQ, ds), dm, f2_mul(dP, sm));
    acc[0] = f2_fma(dx, w, f2_fma(tmx, u, f2_fma(s.mx, v, acc[0])));
    acc[1] = f2_fma(dy, w, f2_fma(tmy, u, f2_fma(s.my, v, acc[1])));
    acc[2] = f2_fma(dz, w, f2_fma(tmz, u, f2_fma(s.mz, v, acc[2])));
  } else {
    const bool in0 = r2.x < c.near2, in1 = r2.y < c.near2;
    float2 al, be;
    field_near_unit2(r2, c.h, c.inv_h, al, be);
    float2 da = f2_fma(al, f2_dup(c.ih5_30), f2_dup(-c.cA)), db = f2_fma(be, f2_dup(-c.ih3_30), f2_dup(c.cB));
    da = make_float2(in0 ? da.x : 0.f, in1 ? da.y : 0.f);
    db = make_float2(in0 ? db.x : 0.f, in1 ? db.y : 0.f);
    const float2 t3 = f2_mul(f2_mul(ds, da), f2_dup(c.c3));
    acc[0] = f2_fma(dx, t3, f2_fma(s.mx, db, acc[0]));
    acc[1] = f2_fma(dy, t3, f2_fma(s.my, db, acc[1]));
    acc[2] = f2_fma(dz, t3, f2_fma(s.mz, db, acc[2]));
  }
}

// Near-field correction, W warps per cell (1 or 4): up to kT of the cell's
// particles are the targets of a pass, held in shared memory (read as
// broadcasts).  The candidate sources of the neighbourhood are rows of cells
// trimmed to the cell-level distance bound of the near radius, each one
// contiguous range of the cell-ordered copies.  The rows are listed once per
// cell (start and prefix offset in shared memory) and their ranges are
// concatenated, so the lanes split one flat candidate index space: every sweep
// of a warp covers 32 candidates whatever the rows' lengths.  Each lane sweeps
// its candidates in increasing order, two targets at a time without a branch,
// and every target's sum is finished by a fixed shuffle tree (and, with 4
// warps, added over the warps in order), so results are deterministic.
// Measured at 65,536 particles: force 573 us (819 with scalar pairs, a branch
// per target and one warp per cell; ~75 instructions per candidate and target
// then, of which ten scalar table loads, 39 now), field 127 us (157).
template <bool kForce, int W>
__global__ void __launch_bounds__(128) k_correction_cells(const CellGrid* __restrict__ grids, int n_scenes,
                                                          int64_t n_cells, const int32_t* __restrict__ perm,
                                                          const int32_t* __restrict__ start,
                                                          const float4* __restrict__ spos,
                                                          const float4* __restrict__ smom, float4* __restrict__ corr,
                                                          const int32_t* __restrict__ skip_scene,
                                                          const double* __restrict__ done_flags, int done_stride,
                                                          const int32_t* __restrict__ done_count, int done_total) {
  constexpr int kT = 8;
  constexpr int kRows = 81;  // (2R + 1)^2 row slots, R <= 4 (cells are at least h wide)
  static_assert(kT <= 10 && kT % 2 == 0, "32 sums per shuffle tree");
  if (done_count && *done_count >= done_total) return;
  __shared__ __align__(16) float s_tbl[80];
  __shared__ __align__(16) float s_t[4][kT / 2][12];  // NearTargets
  __shared__ int32_t s_rb[4][kRows], s_ro[4][kRows + 1];
  __shared__ float s_red[W][32];
  if (kForce)
    for (int k = threadIdx.x; k < 80; k += 128) s_tbl[k] = c_fit_tbl.v[k];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int wi = threadIdx.x >> 5;
  const int sub = W == 1 ? 0 : wi;  // which candidates of the cell this warp sweeps
  const int64_t n_groups = int64_t(gridDim.x) * (4 / W);
  for (int64_t c = int64_t(blockIdx.x) * (4 / W) + (W == 1 ? wi : 0); c < n_cells; c += n_groups) {
    const int32_t cb = start[c], ce = start[c + 1];
    if (cb == ce) continue;
    int lo = 0, hi = n_scenes - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (grids[mid].cell_off <= c) lo = mid;
      else hi = mid - 1;
    }
    if (done_flags && done_flags[int64_t(lo) * done_stride] != 0.0) continue;  // scene's solve stopped
    if (skip_scene && skip_scene[lo]) continue;  // scene evaluated by the exact-branch kernels
    const CellGrid& g = grids[lo];
    const int64_t lc = c - g.cell_off;
    const int ix = int(lc % g.nx), iy = int((lc / g.nx) % g.ny), iz = int(lc / (int64_t(g.nx) * g.ny));
    const int R = kForce ? g.reach_force : g.reach_field;
    NearConsts nc;
    nc.near2 = kForce ? g.pc.near2_force : g.pc.near2_field;
    nc.h = g.pc.h;
    nc.inv_h = g.pc.inv_h;
    nc.ih3_30 = g.pc.ih3_30;
    nc.ih5_30 = g.ih5_30;
    nc.ih4k = g.pc.ih4_over_k;
    if (kForce) clamped_force_coeffs(nc.near2, nc.cA, nc.cB);
    else clamped_field_coeffs(nc.near2, nc.cA, nc.cB);
    nc.c3 = 3.f * g.ih5_unit;
    if (!kForce) nc.cA *= 1.f / g.ih5_unit;
    const float cs = 1.f / g.inv_cs;
    // Row list of this cell: slot i = (dy, dz) in row-major order; a row
    // outside the grid or beyond the near radius has length 0.
    const int side = 2 * R + 1, n_slots = side * side;
    int32_t total = 0;
    __syncwarp();
    for (int i0 = 0; i0 < n_slots; i0 += 32) {
      const int i = i0 + lane;
      int32_t sb = 0, len = 0;
      if (i < n_slots) {
        const int dy = i % side - R, dz = i / side - R;
        const int cy = iy + dy, cz = iz + dz;
        const float gy = float(max(abs(dy) - 1, 0)) * cs, gz = float(max(abs(dz) - 1, 0)) * cs;
        const float rem = nc.near2 - gz * gz - gy * gy;
        if (cy >= 0 && cy < g.ny && cz >= 0 && cz < g.nz && rem >= 0.f) {
          const int dxm = min(R, int(sqrtf(rem) * g.inv_cs) + 1);
          const int cx0 = max(ix - dxm, 0), cx1 = min(ix + dxm, g.nx - 1);
          const int64_t row = g.cell_off + (int64_t(cz) * g.ny + cy) * g.nx;
          sb = start[row + cx0];
          len = start[row + cx1 + 1] - sb;
        }
      }
      int32_t inc = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (i < n_slots) {
        s_rb[wi][i] = sb;
        s_ro[wi][i] = total + inc - len;
      }
      total += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_ro[wi][n_slots] = total;
    __syncwarp();
    for (int32_t t0 = cb; t0 < ce; t0 += kT) {
      const int nt = min(kT, ce - t0);
      __syncwarp();
      if (lane < kT) {  // a slot past the cell's last particle lies beyond every near radius
        const float4 p = lane < nt ? spos[t0 + lane] : make_float4(1e15f, 0.f, 0.f, 0.f);
        const float4 m = lane < nt && kForce ? smom[t0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float v[6] = {p.x, p.y, p.z, m.x, m.y, m.z};
#pragma unroll
        for (int k = 0; k < 6; ++k) s_t[wi][lane >> 1][2 * k + (lane & 1)] = v[k];
      }
      __syncwarp();
      float2 acc[kT / 2][3];
#pragma unroll
      for (int t = 0; t < kT / 2; ++t) acc[t][0] = acc[t][1] = acc[t][2] = make_float2(0.f, 0.f);
      int r = 0;  // this lane's row cursor (its candidates only increase)
      for (int32_t k = sub * 32 + lane; k < total; k += 32 * W) {
        while (s_ro[wi][r + 1] <= k) ++r;
        const int32_t q = s_rb[wi][r] + (k - s_ro[wi][r]);
        const float4 pj = spos[q];
        const float4 mj = smom[q];
        const NearSource src{f2_dup(pj.x), f2_dup(pj.y), f2_dup(pj.z), f2_dup(mj.x), f2_dup(mj.y), f2_dup(mj.z)};
#pragma unroll
        for (int t = 0; t < kT / 2; ++t) {
          if (2 * t < nt) {
            const float4* tp = reinterpret_cast<const float4*>(s_t[wi][t]);
            NearTargets tg{tp[0], tp[1], make_float4(0.f, 0.f, 0.f, 0.f)};
            if (kForce) tg.mm = tp[2];
            near_pair2<kForce>(tg, src, nc, s_tbl, acc[t]);
          }
        }
      }
      float vals[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) vals[q] = 0.f;
#pragma unroll
      for (int t = 0; t < kT / 2; ++t)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          vals[6 * t + k] = acc[t][k].x;
          vals[6 * t + 3 + k] = acc[t][k].y;
        }
      // value 3 t + k (target t, component k) ends in lane 3 t + k; of one or two
      // targets by a tree for 8 values, 9 exchanges in place of 31 (the same
      // sums; direct force of 20,000 particles at h = 0.5 spacings 686 -> 671 us).
      float v;
      if (nt <= 2) {
        float few[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) few[q] = vals[q];
        v = __shfl_sync(0xffffffffu, warp_reduce_scatter<8>(few, lane), 4 * lane & 31);
      } else {
        v = warp_reduce_scatter<32>(vals, lane);
      }
      if (W > 1) {
        __syncthreads();  // the previous pass's sums have been read
        s_red[sub][lane] = v;
        __syncthreads();
        v = 0.f;
#pragma unroll
        for (int w = 0; w < W; ++w) v += s_red[w][lane];
      }
      if (sub == 0 && lane < 3 * nt)
        reinterpret_cast<float*>(corr + perm[t0 + lane / 3])[lane % 3] = v * (kForce ? float(kForceK) : float(kInv4Pi));
    }
  }
}

// Correction at separate targets tpos[0..nt) of a single-scene list: the field
// (kTensor false: corr[i]) or the force tensor (kTensor true: corr[2i] =
// (xx, yy, zz), corr[2i + 1] = (xy, xz, yz)), exact minus clamped, in the
// output units.  One warp per target: the rows of cells around it, trimmed
// to the near radius from the target itself, are listed as in
// k_correction_cells and concatenated, the lanes split the flat candidate
// index space of the cell-ordered copies, and a fixed shuffle tree finishes
// the sums.  Targets need no order of their own; what bounds the pass is the
// issue rate of the pair arithmetic (~35 instructions per candidate, the row
// list ~150 per target).  One thread per target over all cells in reach,
// reading the sources through the permutation, was latency-bound: 782 us for
// the field at 9,973 targets in 40,001 particles, 791 us (field) and 3,976 us
// (tensor) at 30,011 targets in 150,000.  Whole calls went from 2.80 to 2.04
// ms (direct field and tensor, the first sizes) and from 13.6 to 9.1 ms (FMM
// field and Hessian, the second).
// Border cells count as reaching outwards without limit.
template <bool kTensor>
__global__ void __launch_bounds__(128) k_correction_at(const CellGrid* __restrict__ grids, int64_t nt,
                                                       const int32_t* __restrict__ start,
                                                       const float4* __restrict__ spos,
                                                       const float4* __restrict__ smom,
                                                       const float4* __restrict__ tpos, float4* __restrict__ corr) {
  constexpr int kRows = 81;  // (2R + 1)^2 row slots, R <= 4 (cells are at least h wide)
  constexpr int kV = kTensor ? 6 : 3;
  __shared__ __align__(16) float s_tbl[80];
  __shared__ int32_t s_rb[4][kRows], s_ro[4][kRows + 1];
  if (kTensor)
    for (int k = threadIdx.x; k < 80; k += 128) s_tbl[k] = c_fit_tbl.v[k];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int wi = threadIdx.x >> 5;
  const CellGrid& g = grids[0];
  const int R = kTensor ? g.reach_force : g.reach_field;
  const float near2 = kTensor ? g.pc.near2_force : g.pc.near2_field;
  const float cs = 1.f / g.inv_cs;
  const float slack = 1e-3f * cs;  // covers the rounding of the cell map
  float cA, cB;
  if (kTensor) clamped_force_coeffs(near2, cA, cB);
  else clamped_field_coeffs(near2, cA, cB);
  const float c3 = 3.f * g.ih5_unit;  // the field's alphas are in units of ih5_unit
  if (!kTensor) cA *= 1.f / g.ih5_unit;
  const int side = 2 * R + 1, n_slots = side * side;
  const int64_t n_warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t i = int64_t(blockIdx.x) * (blockDim.x >> 5) + wi; i < nt; i += n_warps) {
    const float4 tp = tpos[i];
    int ix, iy, iz;
    cell_coords(g, tp.x, tp.y, tp.z, ix, iy, iz);
    // Distance from the target to the span of cell c along an axis of n cells.
    auto gap = [&](float x, float o, int c, int n) {
      const float lo = c > 0 ? o + float(c) * cs - x : 0.f;
      const float hi = c < n - 1 ? x - (o + float(c + 1) * cs) : 0.f;
      return fmaxf(fmaxf(lo, hi) - slack, 0.f);
    };
    int32_t total = 0;
    __syncwarp();  // the previous target's list has been read
    for (int i0 = 0; i0 < n_slots; i0 += 32) {
      const int k = i0 + lane;
      int32_t sb = 0, len = 0;
      if (k < n_slots) {
        const int cy = iy + k % side - R, cz = iz + k / side - R;
        if (cy >= 0 && cy < g.ny && cz >= 0 && cz < g.nz) {
          const float gy = gap(tp.y, g.oy, cy, g.ny), gz = gap(tp.z, g.oz, cz, g.nz);
          const float rem = near2 - gz * gz - gy * gy;
          if (rem >= 0.f) {
            // x cells within sqrt(rem) of the target, at most R from its cell
            const float w = sqrtf(rem) + slack;
            const int x0 = int(fmaxf((tp.x - w - g.ox) * g.inv_cs, 0.f));
            const int x1 = int(fmaxf((tp.x + w - g.ox) * g.inv_cs, 0.f));
            const int cx0 = min(max(x0, ix - R), g.nx - 1), cx1 = min(min(x1, ix + R), g.nx - 1);
            const int64_t row = g.cell_off + (int64_t(cz) * g.ny + cy) * g.nx;
            if (cx1 >= cx0) {
              sb = start[row + max(cx0, 0)];
              len = start[row + cx1 + 1] - sb;
            }
          }
        }
      }
      int32_t inc = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (k < n_slots) {
        s_rb[wi][k] = sb;
        s_ro[wi][k] = total + inc - len;
      }
      total += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_ro[wi][n_slots] = total;
    __syncwarp();
    float acc[kV];
#pragma unroll
    for (int q = 0; q < kV; ++q) acc[q] = 0.f;
    int r = 0;  // this lane's row cursor (its candidates only increase)
    for (int32_t k = lane; k < total; k += 32) {
      while (s_ro[wi][r + 1] <= k) ++r;
      const int32_t q = s_rb[wi][r] + (k - s_ro[wi][r]);
      const float4 pj = spos[q];
      const float dx = tp.x - pj.x, dy = tp.y - pj.y, dz = tp.z - pj.z;
      const float r2 = dx * dx + dy * dy + dz * dz;
      if (kTensor ? (r2 <= near2 && r2 > 0.f) : (r2 < near2)) {
        const float4 mj = smom[q];
        const float ds = dx * mj.x + dy * mj.y + dz * mj.z;
        if (kTensor) {
          float P, Q;
          force_near_pq_rn(r2, s_tbl, g.pc.inv_h, g.pc.ih4_over_k, P, Q);
          const float dP = P - cA, dQ = Q - cB;
          const float pd = dP * ds, qd = dQ * ds;
          const float ax = dP * mj.x, ay = dP * mj.y, az = dP * mj.z;
          acc[0] += pd + 2.f * ax * dx + qd * dx * dx;
          acc[1] += pd + 2.f * ay * dy + qd * dy * dy;
          acc[2] += pd + 2.f * az * dz + qd * dz * dz;
          acc[kV - 3] += ax * dy + ay * dx + qd * dx * dy;
          acc[kV - 2] += ax * dz + az * dx + qd * dx * dz;
          acc[kV - 1] += ay * dz + az * dy + qd * dy * dz;
        } else {
          float al, be;
          field_near_unit(r2, near_rsqrt(r2), g.pc.h, g.pc.inv_h, al, be);
          const float t3 = c3 * (ds * fmaf(al, g.ih5_30, -cA));
          const float db = fmaf(be, g.pc.ih3_30, -cB);
          acc[0] += dx * t3 - mj.x * db;
          acc[1] += dy * t3 - mj.y * db;
          acc[2] += dz * t3 - mj.z * db;
        }
      }
    }
    const float scale = kTensor ? float(kForceK) : float(kInv4Pi);
#pragma unroll
    for (int q = 0; q < kV; ++q) {
      float v = acc[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      acc[q] = v * scale;
    }
    if (lane == 0) {
      if (kTensor) {
        corr[2 * i] = make_float4(acc[0], acc[1], acc[2], 0.f);
        corr[2 * i + 1] = make_float4(acc[kV - 3], acc[kV - 2], acc[kV - 1], 0.f);
      } else {
        corr[i] = make_float4(acc[0], acc[1], acc[2], 0.f);
      }
    }
  }
}

__global__ void k_to_pairs(const float4* __restrict__ src, float4* __restrict__ dst, int64_t n,
                           const int32_t* __restrict__ done_count, int done_total) {
  if (done_count && *done_count >= done_total) return;
  const int64_t np = (n + 1) / 2;
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < np; p += int64_t(gridDim.x) * blockDim.x)
    pair_records(src, dst, n, p);
}

unsigned grid_for(int64_t n, int per_block = 256) {
  int64_t g = (n + per_block - 1) / per_block;
  if (g > 8192) g = 8192;
  return unsigned(g < 1 ? 1 : g);
}

}  // namespace

void to_pairs(const float4* src, float4* dst, int64_t n, cudaStream_t st, const int32_t* done_count,
              int done_total) {
  k_to_pairs<<<grid_for((n + 1) / 2), 256, 0, st>>>(src, dst, n, done_count, done_total);
}

mf_status CellList::build(const float4* pos4, const std::vector<CellSceneSpec>& scenes, cudaStream_t st,
                          double margin_h, const std::function<bool(const double*)>& wanted) {
  const int ns = int(scenes.size());
  if (ns == 0) return fail(MF_ERR_INVALID_ARG, "cell list: no scenes");
  n_scenes_ = ns;
  std::vector<int64_t> ranges(2 * size_t(ns));
  int64_t max_n = 0;
  n_total_ = 0;
  for (int s = 0; s < ns; ++s) {
    ranges[2 * s] = scenes[s].p_off;
    ranges[2 * s + 1] = scenes[s].n;
    max_n = std::max(max_n, scenes[s].n);
    n_total_ += scenes[s].n;
  }
  if (n_total_ >= (int64_t(1) << 31)) return fail(MF_ERR_INVALID_ARG, "cell list: too many particles");
  MF_TRY(bbox_.reserve(sizeof(int32_t) * 6 * ns + ranges.size() * sizeof(int64_t) + 64));
  int32_t* bbox = bbox_.as<int32_t>();
  int64_t* d_ranges = reinterpret_cast<int64_t*>(bbox_.as<char>() + ((sizeof(int32_t) * 6 * ns + 63) / 64) * 64);
  MF_CUDA_TRY(cudaMemcpyAsync(d_ranges, ranges.data(), ranges.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st));
  k_bbox_init<<<grid_for(6 * ns), 256, 0, st>>>(bbox, ns);
  const unsigned gx = std::min<unsigned>(grid_for(max_n), 256);
  k_bbox<<<dim3(gx, unsigned(ns)), 256, 0, st>>>(pos4, d_ranges, bbox);
  MF_CUDA_TRY(cudaGetLastError());
  std::vector<int32_t> hb(6 * size_t(ns));
  MF_CUDA_TRY(cudaMemcpyAsync(hb.data(), bbox, hb.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  MF_CUDA_TRY(cudaStreamSynchronize(st));

  host_grids_.assign(size_t(ns), CellGrid{});
  host_bbox_.assign(6 * size_t(ns), 0.0);
  for (size_t k = 0; k < hb.size(); ++k) host_bbox_[k] = double(ord2f(hb[k]));
  int64_t cells = 0, prefix = 0;
  double spanned = 0.0;
  for (int s = 0; s < ns; ++s) {
    CellGrid& g = host_grids_[size_t(s)];
    const double h = scenes[s].h;
    double lo[3], ext[3];
    for (int c = 0; c < 3; ++c) {
      lo[c] = ord2f(hb[6 * s + c]) - margin_h * h;
      ext[c] = std::max(0.0, double(ord2f(hb[6 * s + 3 + c])) + margin_h * h - lo[c]);
      if (!std::isfinite(lo[c]) || !std::isfinite(ext[c])) return fail(MF_ERR_INVALID_ARG, "non-finite positions");
    }
    if (wanted && !wanted(host_bbox_.data() + 6 * size_t(s))) return MF_OK;
    // Cells a hair wider than h (about 8 particles at h = 2 spacings): a point
    // closer than 2h (4h) to a target then always lies within 2 (4) cells of
    // it, whatever the rounding of the cell map.
    double cs = h * (1.0 + 1e-4);
    // Keep the grid at most ~8 cells per particle: widen cells for sparse scenes.
    const double cap = std::max(64.0, 8.0 * double(scenes[s].n));
    for (int it = 0; it < 512; ++it) {  // any FP32 extent over any FP32 h (1.25^512 = 1e49)
      const double c3 = (std::floor(ext[0] / cs) + 1) * (std::floor(ext[1] / cs) + 1) * (std::floor(ext[2] / cs) + 1);
      if (c3 <= cap) break;
      cs *= 1.25;
    }
    g.ox = float(lo[0]);
    g.oy = float(lo[1]);
    g.oz = float(lo[2]);
    g.inv_cs = float(1.0 / cs);
    g.nx = int32_t(std::floor(ext[0] / cs)) + 1;
    g.ny = int32_t(std::floor(ext[1] / cs)) + 1;
    g.nz = int32_t(std::floor(ext[2] / cs)) + 1;
    g.reach_field = int32_t(std::ceil(2.0 * h / cs));
    g.reach_force = int32_t(std::ceil(4.0 * h / cs));
    g.cell_off = cells;
    g.p_off = scenes[s].p_off;
    g.n = scenes[s].n;
    g.k_off = prefix;
    g.pc = make_pair_consts<float>(h);
    const double ih5 = 1.0 / (30.0 * h * h * h * h * h);
    g.ih5_unit = ih5 < 0x1p-100 ? 0x1p-96f : ih5 > 0x1p+100 ? 0x1p+20f : 1.f;
    g.ih5_30 = float(std::min(ih5 / double(g.ih5_unit), 1e37));  // times alpha's 24 at r = 0 still finite
    cells += int64_t(g.nx) * g.ny * g.nz;
    double box = 1.0;  // the particles' own bounding box, in cells
    for (int c = 0; c < 3; ++c) box *= std::max(1.0, (ext[c] - 2.0 * margin_h * h) / cs);
    spanned += box;
    prefix += scenes[s].n;
  }
  n_cells_ = cells;
  full_ = double(n_total_) >= 2.0 * spanned;
  MF_TRY(grids_.reserve(sizeof(CellGrid) * size_t(ns)));
  MF_CUDA_TRY(cudaMemcpyAsync(grids_.ptr, host_grids_.data(), sizeof(CellGrid) * size_t(ns), cudaMemcpyHostToDevice,
                              st));
  MF_TRY(cell_start_.reserve_slack(sizeof(int32_t) * size_t(cells + 1)));
  MF_TRY(cursor_.reserve_slack(sizeof(int32_t) * size_t(cells + 1)));
  MF_TRY(scan_tiles_.reserve_slack(sizeof(int32_t) * size_t((cells + kScanTile - 1) / kScanTile + 1)));
  MF_TRY(perm_.reserve(sizeof(int32_t) * size_t(n_total_)));
  MF_TRY(perm_tmp_.reserve(sizeof(int32_t) * size_t(n_total_)));
  MF_TRY(cell_of_.reserve(sizeof(int32_t) * size_t(n_total_)));
  MF_TRY(spos_.reserve(sizeof(float4) * size_t(n_total_)));
  MF_TRY(smom_.reserve(sizeof(float4) * size_t(n_total_)));
  return rebin(pos4, st);
}

mf_status CellList::rebin(const float4* pos4, cudaStream_t st) {
  const int64_t cells = n_cells_;
  const int ns = n_scenes_;
  int32_t* counts = cursor_.as<int32_t>();
  MF_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(int32_t) * size_t(cells + 1), st));
  const CellGrid* dg = grids_.as<CellGrid>();
  k_count<<<grid_for(n_total_), 256, 0, st>>>(pos4, dg, ns, n_total_, counts, cell_of_.as<int32_t>());
  {
    const int64_t tiles = (cells + kScanTile - 1) / kScanTile;
    int32_t* tsum = scan_tiles_.as<int32_t>();
    if (tiles > 0) k_scan_tiles<<<unsigned(tiles), kScanThreads, 0, st>>>(counts, cells, tsum);
    k_scan_tile_sums<<<1, kScanThreads, 0, st>>>(tsum, tiles, cell_start_.as<int32_t>(), cells);
    if (tiles > 0) k_scan_apply<<<unsigned(tiles), kScanThreads, 0, st>>>(counts, cells, tsum, cell_start_.as<int32_t>());
  }
  MF_CUDA_TRY(cudaMemcpyAsync(cursor_.ptr, cell_start_.ptr, sizeof(int32_t) * size_t(cells), cudaMemcpyDeviceToDevice,
                              st));
  k_scatter<<<grid_for(n_total_), 256, 0, st>>>(dg, ns, n_total_, cell_of_.as<int32_t>(), cursor_.as<int32_t>(),
                                                perm_tmp_.as<int32_t>());
  k_sort_cells<<<grid_for(cells * 32), 256, 0, st>>>(cell_start_.as<int32_t>(), cells, perm_tmp_.as<int32_t>(),
                                                     perm_.as<int32_t>());
  MF_CUDA_TRY(cudaGetLastError());
  return MF_OK;
}

// Warps per cell of the correction.  The force takes 4 where cells are full:
// they are long (116 sweeps of 32 candidates at h = 2 spacings), and one warp
// each left a last wave a fifth of the kernel long at 65,536 particles (743
// against 573 us; 273 against 143 at 16,411).  Below two particles per cell of
// the bounding boxes (h under 1.3-1.6 spacings) a cell's row list costs more
// than its sweeps, and one warp each is better: whole direct forces of 20,000
// particles, 4 warps / 1, 772 / 697 us at h = 0.5 spacings, 711 / 695 at 1.3,
// 710 / 735 at 1.6.  The field's cells are short (19 sweeps), so 4 warps pay
// while there are fewer cells than the device runs warps (14 against 39 us at
// 3,001 particles, 25 against 48 at 12,289), and one warp from there on (24
// scenes in one list: 25 against 41 us).
constexpr int64_t kSplitCells = 8192;
static unsigned cell_grid(int64_t cells) {
  int64_t g = cells;
  if (g > 65535) g = 65535;
  return unsigned(g < 1 ? 1 : g);
}

mf_status CellList::field_correction(const float4* pos4, const float4* mom4, float4* corr, cudaStream_t st,
                                     const double* done_flags, int done_stride, const int32_t* done_count,
                                     int done_total, float4* mom2) const {
  k_gather_sorted<<<grid_for(n_total_), 256, 0, st>>>(perm_.as<int32_t>(), pos4, mom4, n_total_, spos_.as<float4>(),
                                                      smom_.as<float4>(), done_count, done_total, mom2);
  auto* k = n_cells_ < kSplitCells ? k_correction_cells<false, 4> : k_correction_cells<false, 1>;
  k<<<cell_grid(n_cells_ < kSplitCells ? n_cells_ : (n_cells_ + 3) / 4), 128, 0, st>>>(
      grids_.as<CellGrid>(), n_scenes_, n_cells_, perm_.as<int32_t>(), cell_start_.as<int32_t>(), spos_.as<float4>(),
      smom_.as<float4>(), corr, skip_field_on_ ? skip_field_.as<int32_t>() : nullptr, done_flags, done_stride, done_count, done_total);
  MF_CUDA_TRY(cudaGetLastError());
  return MF_OK;
}

mf_status CellList::field_correction_at(const float4* tpos4, int64_t nt, const float4* pos4, const float4* mom4,
                                        float4* corr, cudaStream_t st) const {
  return correction_at<false>(tpos4, nt, pos4, mom4, corr, st);
}

mf_status CellList::tensor_correction_at(const float4* tpos4, int64_t nt, const float4* pos4, const float4* mom4,
                                         float4* corr2, cudaStream_t st) const {
  return correction_at<true>(tpos4, nt, pos4, mom4, corr2, st);
}

template <bool kTensor>
mf_status CellList::correction_at(const float4* tpos4, int64_t nt, const float4* pos4, const float4* mom4,
                                  float4* corr, cudaStream_t st) const {
  if (n_scenes_ != 1) return fail(MF_ERR_INVALID_ARG, "separate targets need a single-scene cell list");
  k_gather_sorted<<<grid_for(n_total_), 256, 0, st>>>(perm_.as<int32_t>(), pos4, mom4, n_total_, spos_.as<float4>(),
                                                      smom_.as<float4>(), nullptr, 0, nullptr);
  k_correction_at<kTensor><<<cell_grid((nt + 3) / 4), 128, 0, st>>>(
      grids_.as<CellGrid>(), nt, cell_start_.as<int32_t>(), spos_.as<float4>(), smom_.as<float4>(), tpos4, corr);
  MF_CUDA_TRY(cudaGetLastError());
  return MF_OK;
}

mf_status CellList::set_skips(const std::vector<int32_t>& field, const std::vector<int32_t>& force) {
  // A list without skips is not passed to the kernels; its buffer is kept
  // (freeing would wait for every stream of the device).
  auto put = [&](const std::vector<int32_t>& v, DevBuf& b, bool& on) -> mf_status {
    bool any = false;
    for (int32_t x : v) any = any || x != 0;
    on = any;
    if (!any) return MF_OK;
    if (int(v.size()) != n_scenes_) return fail(MF_ERR_INVALID_ARG, "skip list size");
    MF_TRY(b.reserve(v.size() * sizeof(int32_t)));
    MF_CUDA_TRY(cudaMemcpy(b.ptr, v.data(), v.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    return MF_OK;
  };
  MF_TRY(put(field, skip_field_, skip_field_on_));
  MF_TRY(put(force, skip_force_, skip_force_on_));
  return MF_OK;
}

mf_status CellList::force_correction(const float4* pos4, const float4* mom4, float4* corr, cudaStream_t st,
                                     float4* mom2) const {
  k_gather_sorted<<<grid_for(n_total_), 256, 0, st>>>(perm_.as<int32_t>(), pos4, mom4, n_total_, spos_.as<float4>(),
                                                      smom_.as<float4>(), nullptr, 0, mom2);
  auto* k = full_ ? k_correction_cells<true, 4> : k_correction_cells<true, 1>;
  k<<<cell_grid(full_ ? n_cells_ : (n_cells_ + 3) / 4), 128, 0, st>>>(
      grids_.as<CellGrid>(), n_scenes_, n_cells_, perm_.as<int32_t>(), cell_start_.as<int32_t>(), spos_.as<float4>(),
      smom_.as<float4>(), corr, skip_force_on_ ? skip_force_.as<int32_t>() : nullptr, nullptr, 0, nullptr, 0);
  MF_CUDA_TRY(cudaGetLastError());
  return MF_OK;
}

}  // namespace mfgb
