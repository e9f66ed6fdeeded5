// mf_fmm.cu -- uniform-octree fast multipole method for the field and force
// products of large scenes.
//
// The reference evaluates large products with FMMTL (KernelMatrix.hpp:26-164,
// DualTraversal.hpp:80-125, BatchNear.hpp:57-75): an adaptive octree,
// spherical expansions in FP64 on the host CPU and a GPU near field.  Here the
// whole product stays on the device:
//   * one uniform box grid per level (level 0 is one box around the scene);
//     the leaf level is the deepest with >= leaf_min particles per box on
//     average (default 12), deep enough that few pairs of a near box are far apart;
//   * particles binned into leaf boxes in row-major order (x fastest), each
//     box's list in increasing particle index and padded to an even length,
//     so every run of x-adjacent boxes is one contiguous, pair-aligned range of
//     sources for the packed two-source pair body;
//   * Cartesian Taylor expansions of the dipole potential
//       phi(x) = 1/(4 pi) sum_j m_j . (x - y_j) / |x - y_j|^3
//     (multipoles and locals of degree 1..Q, Q = P - 1, M2L truncated at
//     |alpha| + |beta| <= Q + 1), each level's coefficients scaled by its box
//     edge so M2M, M2L and L2L do not depend on the level;
//   * box pairs accepted by the criterion of FMMOptions.hpp:56-78 (theta on
//     the box radii, with the separation test that the reference enables) are
//     far only if their gap also exceeds the kernel's near radius 4h, so every
//     far pair is in the pure-dipole regime of Dipole_B.kern:46-104 /
//     Dipole_hessian.kern:155-207 and the truncation is the only approximation;
//   * near leaf boxes (not accepted at the leaf level) are summed with the
//     packed clamped pair body of the all-pairs kernel, and the cell-list
//     correction (mf_cells.cu) turns the clamped pairs inside the near radius
//     into the reference's SPH / fitted-curve kernel.
// Every launch reads a solver stop flag and does nothing once it is set.
#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <new>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

#include "mf_internal.h"
#include "mf_sym.cuh"

namespace mfgb {
namespace {

constexpr int kMaxDegree = 9;  // P = 10 (the field products stop at degree 8)
constexpr int kMaxFieldDegree = 8;
constexpr int kMaxLevel = 10;

// Multi-indices in graded order: degree n, then s = y + z, then z.
__host__ __device__ constexpr int ncoef(int q) { return q < 0 ? 0 : (q + 1) * (q + 2) * (q + 3) / 6; }
__host__ __device__ constexpr int gidx(int x, int y, int z) {
  return ncoef(x + y + z - 1) + (y + z) * (y + z + 1) / 2 + z;
}

// 1/|d| is harmonic, so D_(x, y, z + 2) = -D_(x + 2, y, z) - D_(x, y + 2, z):
// the translation works on the multi-indices with z <= 1 only, 2 n + 1 of a
// degree n instead of (n + 1)(n + 2)/2 (k_fmm_reduce, k_fmm_m2l, k_fmm_l2l).
__host__ __device__ constexpr int nharm(int q) { return (q + 1) * (q + 1) - 1; }  // degrees 1..q
__host__ __device__ constexpr int hidx(int x, int y, int z) {  // z <= 1
  return nharm(x + y + z - 1) + (z == 0 ? y : x + y + 2 + y);
}
// Derivatives D_gamma with gamma_z <= 2 (3 n of a degree n >= 1), in rows of ndtab floats.
__host__ __device__ constexpr int dofs(int n) { return n <= 0 ? 0 : 1 + 3 * n * (n - 1) / 2; }
__host__ __device__ constexpr int didx(int x, int y, int z) {
  const int n = x + y + z;
  return dofs(n) + (z == 0 ? y : z == 1 ? n + 1 + y : 2 * n + 1 + y);
}
__host__ __device__ constexpr int ndtab(int q) { return (dofs(q + 2) + 3) / 4 * 4; }  // degrees 0..q + 1, whole float4

// Multi-index table up to degree kMaxDegree + 1.
struct MultiIndexTable {
  char4 v[ncoef(kMaxDegree + 1)];
};
constexpr MultiIndexTable make_multi_indices() {
  MultiIndexTable t{};
  for (int d = 0; d <= kMaxDegree + 1; ++d)
    for (int s = 0; s <= d; ++s)
      for (int z = 0; z <= s; ++z) t.v[gidx(d - s, s - z, z)] = char4{(signed char)(d - s), (signed char)(s - z), (signed char)z, 0};
  return t;
}
__constant__ MultiIndexTable c_mi = make_multi_indices();
// 1-D translation factors: v[c][j] = ((c - 1/2) / 2)^j / j!, the child centre
// offset in parent box units raised to j over j!.
struct ShiftTable {
  float v[2][kMaxDegree + 2];
};
constexpr ShiftTable make_shifts() {
  ShiftTable t{};
  for (int c = 0; c < 2; ++c) {
    const double v = (double(c) - 0.5) / 2.0;
    double f = 1.0;
    for (int j = 0; j < kMaxDegree + 2; ++j) {
      t.v[c][j] = float(f);
      f = f * v / double(j + 1);
    }
  }
  return t;
}
__constant__ ShiftTable c_shift = make_shifts();

// ---------------------------------------------------------------------------
// Binning
// ---------------------------------------------------------------------------
__device__ __forceinline__ int64_t leaf_of(const FmmLevel& lv, float4 p) {
  const float inv = 1.f / lv.side;
  const int ix = min(max(int(floorf((p.x - lv.ox) * inv)), 0), lv.nx - 1);
  const int iy = min(max(int(floorf((p.y - lv.oy) * inv)), 0), lv.ny - 1);
  const int iz = min(max(int(floorf((p.z - lv.oz) * inv)), 0), lv.nz - 1);
  return (int64_t(iz) * lv.ny + iy) * lv.nx + ix;
}

__global__ void k_fmm_count(const float4* __restrict__ pos, int64_t n, FmmLevel lv, int32_t* __restrict__ cell_of,
                            int32_t* __restrict__ cnt) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t c = leaf_of(lv, pos[i]);
    cell_of[i] = int32_t(c);
    atomicAdd(&cnt[c], 1);
  }
}

// Exclusive scan of the even-padded counts into start[0..n], one CTA.
__global__ void __launch_bounds__(1024) k_fmm_scan(const int32_t* __restrict__ cnt, int64_t n,
                                                   int32_t* __restrict__ start, int32_t* __restrict__ extra_n) {
  if (extra_n && threadIdx.x == 0) *extra_n = 0;
  __shared__ int32_t sh[1024];
  const int t = threadIdx.x;
  const int64_t chunk = (n + 1023) / 1024;
  const int64_t b = t * chunk, e = min(n, b + chunk);
  int32_t s = 0;
  for (int64_t i = b; i < e; ++i) s += cnt[i] + (cnt[i] & 1);
  sh[t] = s;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int32_t v = t >= o ? sh[t - o] : 0;
    __syncthreads();
    sh[t] += v;
    __syncthreads();
  }
  int32_t run = sh[t] - s;
  for (int64_t i = b; i < e; ++i) {
    start[i] = run;
    run += cnt[i] + (cnt[i] & 1);
  }
  if (t == 1023) start[n] = sh[1023];
}

__global__ void k_fmm_scatter(const int32_t* __restrict__ cell_of, int64_t n, int32_t* __restrict__ cursor,
                              int32_t* __restrict__ tmp) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    tmp[atomicAdd(&cursor[cell_of[i]], 1)] = int32_t(i);
}

// Each box's list in increasing particle index (one warp per box ranks its
// entries), then -1 in the padding slot of an odd box.  extra (optional): (box,
// first target) of every further run of `chunk` targets of a box, extra_n of
// them, in any order (k_fmm_near_warp).
__global__ void k_fmm_sort(const int32_t* __restrict__ start, const int32_t* __restrict__ cnt, int64_t ncell,
                           const int32_t* __restrict__ tmp, int32_t* __restrict__ perm, int32_t chunk,
                           int2* __restrict__ extra, int32_t* __restrict__ extra_n) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t c = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncell; c += warps) {
    const int32_t b = start[c], m = cnt[c];
    for (int32_t k = lane; k < m; k += 32) {
      const int32_t v = tmp[b + k];
      int32_t rank = 0;
      for (int32_t l = 0; l < m; ++l) rank += tmp[b + l] < v;
      perm[b + rank] = v;
    }
    if (lane == 0 && (m & 1)) perm[b + m] = -1;
    if (extra && m > chunk) {
      const int32_t runs = (m - 1) / chunk;
      int32_t at = 0;
      if (lane == 0) at = atomicAdd(extra_n, runs);
      at = __shfl_sync(0xffffffffu, at, 0);
      for (int32_t k = lane; k < runs; k += 32) extra[at + k] = make_int2(int(c), (k + 1) * chunk);
    }
  }
}

// Occupancy of a level from its children's.
__global__ void k_fmm_occ_up(FmmLevel lc, FmmLevel lp, int32_t* __restrict__ occ) {
  for (int64_t b = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; b < lp.nbox; b += int64_t(gridDim.x) * blockDim.x) {
    const int px = int(b % lp.nx), py = int((b / lp.nx) % lp.ny), pz = int(b / (int64_t(lp.nx) * lp.ny));
    int32_t s = 0;
    for (int ch = 0; ch < 8; ++ch) {
      const int x = 2 * px + (ch & 1), y = 2 * py + ((ch >> 1) & 1), z = 2 * pz + (ch >> 2);
      if (x < lc.nx && y < lc.ny && z < lc.nz) s += occ[lc.box_off + (int64_t(z) * lc.ny + y) * lc.nx + x];
    }
    occ[lp.box_off + b] = s;
  }
}

// Sorted records in pair layout: slots 2p, 2p+1 as (x_a, x_b, y_a, y_b),
// (z_a, z_b, 0, 0).  A padding slot (always the odd one) repeats its
// partner's position (pos) or holds a zero dipole (moments).
__global__ void k_fmm_gather_pairs(const int32_t* __restrict__ perm, const float4* __restrict__ src,
                                   const int32_t* __restrict__ n_slots, float4* __restrict__ dst, int is_pos,
                                   const double* __restrict__ done) {
  if (done && *done != 0.0) return;
  const int64_t n_pairs = *n_slots / 2;
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n_pairs;
       p += int64_t(gridDim.x) * blockDim.x) {
    const int32_t ia = perm[2 * p], ib = perm[2 * p + 1];
    const float4 A = src[ia];
    const float4 B = ib >= 0 ? src[ib] : (is_pos ? A : make_float4(0.f, 0.f, 0.f, 0.f));
    dst[2 * p] = make_float4(A.x, B.x, A.y, B.y);
    dst[2 * p + 1] = make_float4(A.z, B.z, 0.f, 0.f);
  }
}

// Executed near-field pairs (real targets x real sources) and the largest leaf.
__global__ void k_fmm_p2p_stats(FmmLevel lv, const int32_t* __restrict__ cnt, const int32_t* __restrict__ tcnt,
                                const int4* __restrict__ rows, int n_rows, unsigned long long* __restrict__ out) {
  for (int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < lv.nbox; c += int64_t(gridDim.x) * blockDim.x) {
    const int32_t n = tcnt[c];
    if (n == 0) continue;
    const int ix = int(c % lv.nx), iy = int((c / lv.nx) % lv.ny), iz = int(c / (int64_t(lv.nx) * lv.ny));
    unsigned long long s = 0;
    for (int r = 0; r < n_rows; ++r) {
      const int4 rw = rows[r];
      const int cy = iy + rw.y, cz = iz + rw.z;
      if (cy < 0 || cy >= lv.ny || cz < 0 || cz >= lv.nz) continue;
      const int cx0 = max(ix - rw.x, 0), cx1 = min(ix + rw.x, lv.nx - 1);
      const int64_t rb = (int64_t(cz) * lv.ny + cy) * lv.nx;
      for (int x = cx0; x <= cx1; ++x) s += unsigned(cnt[rb + x]);
    }
    atomicAdd(&out[0], s * unsigned(n));
    atomicMax(&out[1], (unsigned long long)n);
    atomicAdd(&out[3], 1ull);
    atomicAdd(&out[4], (unsigned long long)cnt[c] * unsigned(n));
  }
}

// Multipole-to-local translations of one level (target box holding targets,
// source box holding sources), one warp per target box.
__global__ void k_fmm_m2l_stats(FmmLevel lv, const int32_t* __restrict__ occ, const int32_t* __restrict__ tocc,
                                const int4* __restrict__ list, const int64_t* __restrict__ off,
                                const int64_t* __restrict__ cnt, unsigned long long* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t b = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); b < lv.nbox; b += warps) {
    if (tocc[lv.box_off + b] == 0) continue;
    const int x = int(b % lv.nx), y = int((b / lv.nx) % lv.ny), z = int(b / (int64_t(lv.nx) * lv.ny));
    const int cls = (x & 1) | ((y & 1) << 1) | ((z & 1) << 2);
    unsigned k = 0;
    for (int64_t e = off[cls] + lane; e < off[cls] + cnt[cls]; e += 32) {
      const int4 d = list[e];
      const int sx = x - d.x, sy = y - d.y, sz = z - d.z;
      if (unsigned(sx) >= unsigned(lv.nx) || unsigned(sy) >= unsigned(lv.ny) || unsigned(sz) >= unsigned(lv.nz)) continue;
      k += occ[lv.box_off + (int64_t(sz) * lv.ny + sy) * lv.nx + sx] > 0 ? 1u : 0u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
    if (lane == 0) atomicAdd(&out[2], (unsigned long long)k);
  }
}

// ---------------------------------------------------------------------------
// Upward pass
// ---------------------------------------------------------------------------
// Leaf multipoles, one CTA per box, one thread per coefficient alpha (two for
// degree 8, whose 164 coefficients outnumber the threads):
//   M_alpha = (-1)^|alpha| sum_j sum_k m_jk u_j^(alpha - e_k) / (alpha - e_k)!,
// u_j = (y_j - centre) / edge.
template <int Q>
__global__ void __launch_bounds__(128) k_fmm_p2m(FmmLevel lv, const int32_t* __restrict__ start,
                                                 const int32_t* __restrict__ cnt, const int32_t* __restrict__ perm,
                                                 const float4* __restrict__ pos4, const float4* __restrict__ mom4,
                                                 float* __restrict__ M, const double* __restrict__ done) {
  constexpr int NC = ncoef(Q) - 1;
  constexpr int KPT = (NC + 127) / 128;  // coefficients per thread
  constexpr int W = 3 * Q + 3;  // powers u^i/i! (i < Q) per axis, then the dipole
  if (done && *done != 0.0) return;
  __shared__ float s_p[128][W + 1];
  const int tid = threadIdx.x;
  bool act[KPT];
  int ax[KPT], ay[KPT], az[KPT];
  float sign[KPT];
#pragma unroll
  for (int r = 0; r < KPT; ++r) {
    const int k = tid + 128 * r;
    act[r] = k < NC;
    ax[r] = ay[r] = az[r] = 0;
    if (act[r]) {
      const char4 e = c_mi.v[k + 1];
      ax[r] = e.x;
      ay[r] = e.y;
      az[r] = e.z;
    }
    sign[r] = ((ax[r] + ay[r] + az[r]) & 1) ? -1.f : 1.f;
  }
  const float inv_s = 1.f / lv.side;
  for (int64_t c = blockIdx.x; c < lv.nbox; c += gridDim.x) {
    const int32_t n = cnt[c];
    float acc[KPT];
#pragma unroll
    for (int r = 0; r < KPT; ++r) acc[r] = 0.f;
    if (n > 0) {
      const int ix = int(c % lv.nx), iy = int((c / lv.nx) % lv.ny), iz = int(c / (int64_t(lv.nx) * lv.ny));
      const float cx = lv.ox + (float(ix) + 0.5f) * lv.side;
      const float cy = lv.oy + (float(iy) + 0.5f) * lv.side;
      const float cz = lv.oz + (float(iz) + 0.5f) * lv.side;
      const int32_t b = start[c];
      for (int j0 = 0; j0 < n; j0 += 128) {
        const int nj = min(128, n - j0);
        __syncthreads();
        if (tid < nj) {
          const int32_t i = perm[b + j0 + tid];
          const float4 p = pos4[i], m = mom4[i];
          const float u[3] = {(p.x - cx) * inv_s, (p.y - cy) * inv_s, (p.z - cz) * inv_s};
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            float v = 1.f;
            s_p[tid][a * Q] = 1.f;
#pragma unroll
            for (int k = 1; k < Q; ++k) {
              v = v * u[a] * (1.f / float(k));
              s_p[tid][a * Q + k] = v;
            }
          }
          s_p[tid][3 * Q] = m.x;
          s_p[tid][3 * Q + 1] = m.y;
          s_p[tid][3 * Q + 2] = m.z;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < KPT; ++r) {
          if (act[r]) {
            for (int j = 0; j < nj; ++j) {
              const float* q = s_p[j];
              float t = 0.f;
              if (ax[r] > 0) t += q[3 * Q] * q[ax[r] - 1] * q[Q + ay[r]] * q[2 * Q + az[r]];
              if (ay[r] > 0) t += q[3 * Q + 1] * q[ax[r]] * q[Q + ay[r] - 1] * q[2 * Q + az[r]];
              if (az[r] > 0) t += q[3 * Q + 2] * q[ax[r]] * q[Q + ay[r]] * q[2 * Q + az[r] - 1];
              acc[r] += t;
            }
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < KPT; ++r)
      if (act[r]) M[int64_t(tid + 128 * r) * lv.nbox + c] = sign[r] * acc[r];
  }
}

// Children -> parent:  M^p_alpha = sum_c sum_{gamma <= alpha}
//   2^(1-|gamma|) M^c_gamma (-1)^|delta| v_c^delta / delta!,  delta = alpha - gamma,
// v_c the child centre offset in parent box units.  One thread per (alpha, box,
// child), a fixed shuffle tree over the eight children: a thread's chain of
// loads (up to 63 terms a child) is what bounds the pass, and one thread for
// all eight took 190 us for the force and 98 for the field of 200,003 particles
// (two levels), now 70 and 35.
template <int Q>
__global__ void k_fmm_m2m(FmmLevel lc, FmmLevel lp, const int32_t* __restrict__ occ, float* __restrict__ M,
                          const double* __restrict__ done) {
  constexpr int NC = ncoef(Q) - 1;
  if (done && *done != 0.0) return;
  const float* Mc = M + lc.box_off * NC;
  float* Mp = M + lp.box_off * NC;
  const int64_t total = int64_t(8 * NC) * lp.nbox;
  const int ch = threadIdx.x & 7, cx = ch & 1, cy = (ch >> 1) & 1, cz = ch >> 2;
  for (int64_t t0 = int64_t(blockIdx.x) * blockDim.x; t0 < total; t0 += int64_t(gridDim.x) * blockDim.x) {
    const int64_t t = (t0 + threadIdx.x) >> 3;
    const int k = int(t / lp.nbox);
    const int64_t b = t % lp.nbox;
    float acc = 0.f;
    if (k < NC && occ[lp.box_off + b] > 0) {
      const char4 e = c_mi.v[k + 1];
      const int x = 2 * int(b % lp.nx) + cx, y = 2 * int((b / lp.nx) % lp.ny) + cy,
                z = 2 * int(b / (int64_t(lp.nx) * lp.ny)) + cz;
      const int64_t cb = (int64_t(z) * lc.ny + y) * lc.nx + x;
      if (x < lc.nx && y < lc.ny && z < lc.nz && occ[lc.box_off + cb] > 0) {
        for (int gx = 0; gx <= e.x; ++gx)
          for (int gy = 0; gy <= e.y; ++gy)
            for (int gz = 0; gz <= e.z; ++gz) {
              const int g = gx + gy + gz;
              if (g == 0) continue;
              const int dx = e.x - gx, dy = e.y - gy, dz = e.z - gz;
              // (-1)^|delta| v^delta / delta! = prod over axes of ((1/2 - c) / 2)^d / d!
              const float w = c_shift.v[1 - cx][dx] * c_shift.v[1 - cy][dy] * c_shift.v[1 - cz][dz];
              acc += Mc[int64_t(gidx(gx, gy, gz) - 1) * lc.nbox + cb] * w * ldexpf(1.f, 1 - g);
            }
      }
    }
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (ch == 0 && k < NC) Mp[int64_t(k) * lp.nbox + b] = acc;
  }
}

// ---------------------------------------------------------------------------
// Multipoles onto the indices with z <= 1 (every level from 2 on): with
// D_(a, b, z + 2 j) = (-1)^j sum_i C(j, i) D_(a + 2 i, b + 2 (j - i), z),
//   M'_(x, y, z) = sum_j (-1)^j sum_i C(j, i) M_(x - 2 i, y - 2 (j - i), z + 2 j),
// the same potential outside the box, degree by degree.  One thread per
// (coefficient, box); blockIdx.y is the level.
// ---------------------------------------------------------------------------
struct FmmLevels {
  FmmLevel lv[kMaxLevel + 1];
};
__device__ __forceinline__ float binom_f(int j, int i) {  // j <= 5
  float c = 1.f;
  for (int k = 0; k < i; ++k) c = c * float(j - k) / float(k + 1);
  return c;
}

template <int Q>
__global__ void k_fmm_reduce(const FmmLevels lvs, int l0, const float* __restrict__ M, float* __restrict__ H,
                             const double* __restrict__ done) {
  constexpr int NC = ncoef(Q) - 1, NH = nharm(Q);
  if (done && *done != 0.0) return;
  const FmmLevel& lv = lvs.lv[l0 + blockIdx.y];
  const float* m = M + lv.box_off * NC;
  float* h = H + lv.box_off * NH;
  for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < int64_t(NH) * lv.nbox;
       t += int64_t(gridDim.x) * blockDim.x) {
    const int k = int(t / lv.nbox);
    const int64_t b = t % lv.nbox;
    // k -> (x, y, z) of degree n: nharm(n - 1) <= k < nharm(n)
    int n = 1;
    while (k >= nharm(n)) ++n;
    const int w = k - nharm(n - 1);
    const int z = w <= n ? 0 : 1, y = w <= n ? w : w - n - 1, x = n - z - y;
    float v = 0.f;
    for (int j = 0; 2 * j <= x + y; ++j) {
      float s = 0.f;
      for (int i = 0; i <= j; ++i) {
        const int a = x - 2 * i, c = y - 2 * (j - i);
        if (a >= 0 && c >= 0) s += binom_f(j, i) * m[int64_t(gidx(a, c, z + 2 * j) - 1) * lv.nbox + b];
      }
      v += (j & 1) ? -s : s;
    }
    h[int64_t(k) * lv.nbox + b] = v;
  }
}

// ---------------------------------------------------------------------------
// M2L:  L_beta += sum_alpha M'_alpha D_(alpha + beta)(d),  |alpha| + |beta| <= Q + 1,
// D_gamma(d) = d^gamma (1/|d|) at the box-centre offset d in box units, over
// the alpha and beta with z <= 1.  The locals with beta_z >= 2 follow from
// these (L_beta are derivatives of a harmonic potential too, and the
// truncation keeps whole degrees), so the result is the full sum's, at
// sum (2|alpha| + 1)(2|beta| + 1) FMAs instead of one per full index pair:
// 1,204 against 2,674 at Q = 7, 2,388 against ~6,500 for the force at Q = 9,
// and 63 / 80 multipole loads instead of 119 / 219 (several times over: the
// full sum needed two to four launches, each for a range of local degrees, to
// keep the multipole and the accumulators in registers).  The sum is an
// unrolled program over compile-time (gamma, alpha, beta) triples, gamma-major
// so each D value is read once (four per load); local degrees BLO..Q.
// Measured per step at 1,048,576 particles (one field product at Q = 7, one
// force product at Q = 9): 13.6 ms for the full sum, 4.2 here (1.1 + 3.0; 168
// and 249 registers).  Two launches split by local degree: 1.4 + 2.9 ms.
// The kernel is bound by lanes without work: at the force's aperture about
// half of the (target, list offset) pairs have no source box.
// ---------------------------------------------------------------------------
template <int Q, int BLO>
struct M2LPlan {
  static constexpr int AMAX = (Q < Q + 1 - BLO) ? Q : Q + 1 - BLO;
  static constexpr int NA = nharm(AMAX);
  static constexpr int BOFF = nharm(BLO - 1);
  static constexpr int NB = nharm(Q) - nharm(BLO - 1);
  struct Ent {
    int16_t g, a, b, first;  // first: this entry's gamma opens a new float4 of the row
  };
  template <class F>
  static constexpr void walk(F&& f) {
    for (int g = BLO + 1; g <= Q + 1; ++g)
      for (int gz = 0; gz <= 2 && gz <= g; ++gz)
        for (int gy = 0; gy <= g - gz; ++gy) {
          const int gx = g - gz - gy;
          for (int ax = 0; ax <= gx; ++ax)
            for (int ay = 0; ay <= gy; ++ay)
              for (int az = 0; az <= gz; ++az) {
                const int a = ax + ay + az, b = g - a;
                if (az > 1 || gz - az > 1 || a < 1 || a > AMAX || b < BLO || b > Q) continue;
                f(didx(gx, gy, gz), hidx(ax, ay, az), hidx(gx - ax, gy - ay, gz - az) - BOFF);
              }
        }
  }
  static constexpr int count() {
    int k = 0;
    walk([&](int, int, int) { ++k; });
    return k;
  }
  static constexpr int K = count();
  struct Tab {
    Ent e[K];
  };
  static constexpr Tab make() {
    Tab t{};
    int k = 0, quad = -1;
    walk([&](int g, int a, int b) {
      t.e[k].g = int16_t(g);
      t.e[k].a = int16_t(a);
      t.e[k].b = int16_t(b);
      t.e[k].first = int16_t(g / 4 != quad ? 1 : 0);
      quad = g / 4;
      ++k;
    });
    return t;
  }
  static constexpr Tab tab = make();
  template <int I>
  struct At {
    static constexpr int g = tab.e[I].g, a = tab.e[I].a, b = tab.e[I].b, first = tab.e[I].first;
  };
};

template <class Pl, int I>
__device__ __forceinline__ void m2l_step(float* acc, const float* M, const float4* __restrict__ dt, float4& dg) {
  using E = typename Pl::template At<I>;
  if constexpr (E::first != 0) dg = __ldg(dt + E::g / 4);
  constexpr int c = E::g % 4;
  const float d = c == 0 ? dg.x : c == 1 ? dg.y : c == 2 ? dg.z : dg.w;
  acc[E::b] = fmaf(M[E::a], d, acc[E::b]);
}

template <class Pl, int... Is>
__device__ __forceinline__ void m2l_apply(float* acc, const float* M, const float4* __restrict__ dt,
                                          std::integer_sequence<int, Is...>) {
  float4 dg = make_float4(0.f, 0.f, 0.f, 0.f);
  (m2l_step<Pl, Is>(acc, M, dt, dg), ...);
}

struct M2LArgs {
  FmmLevel lv;
  const int32_t* occ;   // sources per box
  const int32_t* tocc;  // targets per box
  const float* M;     // this level's multipoles with z <= 1 (NH rows of nbox)
  float* Lp;          // [chunks][NH][nbox] partial locals with z <= 1
  const int4* list;   // (dx, dy, dz, row of dtab)
  const float4* dtab; // [rows][ndtab(Q) / 4]
  int64_t list_off[8];
  int32_t list_cnt[8];
  int32_t chunks;
  int32_t hx, hy, hz;  // half-grid extents (boxes per class along each axis)
  int64_t per_class;   // hx * hy * hz rounded up to a multiple of 32
  const double* done;
};

// One thread per (list chunk, target box); the warps of a block share the
// chunk and the target parity class, so they walk the same offsets.
template <int Q, int BLO>
__global__ void __launch_bounds__(128) k_fmm_m2l(const M2LArgs p) {
  using Pl = M2LPlan<Q, BLO>;
  constexpr int NH = nharm(Q);
  if (p.done && *p.done != 0.0) return;
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t per = p.per_class;
  const int ch = int(t / (8 * per));
  if (ch >= p.chunks) return;
  const int cls = int((t / per) % 8);
  const int64_t r = t % per;
  const int hi = int(r % p.hx), hj = int((r / p.hx) % p.hy);
  const int64_t hk = r / (int64_t(p.hx) * p.hy);
  if (hk >= p.hz) return;
  const FmmLevel& lv = p.lv;
  const int tx = 2 * hi + (cls & 1), ty = 2 * hj + ((cls >> 1) & 1), tz = 2 * int(hk) + (cls >> 2);
  if (tx >= lv.nx || ty >= lv.ny || tz >= lv.nz) return;
  const int64_t tb = (int64_t(tz) * lv.ny + ty) * lv.nx + tx;
  if (p.tocc[lv.box_off + tb] == 0) return;
  const int64_t n = p.list_cnt[cls];
  const int64_t e0 = p.list_off[cls] + n * ch / p.chunks;
  const int64_t e1 = p.list_off[cls] + n * (ch + 1) / p.chunks;
  float acc[Pl::NB];
#pragma unroll
  for (int q = 0; q < Pl::NB; ++q) acc[q] = 0.f;
  for (int64_t e = e0; e < e1; ++e) {
    const int4 d = __ldg(p.list + e);
    const int sx = tx - d.x, sy = ty - d.y, sz = tz - d.z;
    if (unsigned(sx) >= unsigned(lv.nx) || unsigned(sy) >= unsigned(lv.ny) || unsigned(sz) >= unsigned(lv.nz))
      continue;
    const int64_t sb = (int64_t(sz) * lv.ny + sy) * lv.nx + sx;
    if (__ldg(p.occ + lv.box_off + sb) == 0) continue;
    float M[Pl::NA];
#pragma unroll
    for (int q = 0; q < Pl::NA; ++q) M[q] = __ldg(p.M + int64_t(q) * lv.nbox + sb);
    m2l_apply<Pl>(acc, M, p.dtab + int64_t(d.w) * (ndtab(Q) / 4), std::make_integer_sequence<int, Pl::K>{});
  }
  float* out = p.Lp + int64_t(ch) * NH * lv.nbox;
#pragma unroll
  for (int q = 0; q < Pl::NB; ++q) out[int64_t(Pl::BOFF + q) * lv.nbox + tb] = acc[q];
}

// Locals of a level: the M2L partials plus the parent's locals shifted to the
// child centre,  L^c_beta += 2^(-2-|beta|) sum_delta L^p_(beta+delta) v_c^delta / delta!.
// `occ` counts targets: boxes without targets need no locals.  The partials
// hold the locals with z <= 1; L_(x, y, z + 2 j) = (-1)^j sum_i C(j, i)
// L_(x + 2 i, y + 2 (j - i), z) gives the others.
// kmin: coefficients below it are not computed (zero): a Hessian-only product
// has no degree-1 partials (kmin 3).
template <int Q>
__global__ void k_fmm_l2l(FmmLevel lv, FmmLevel lp, int has_parent, const int32_t* __restrict__ occ,
                          const float* __restrict__ Lpart, int chunks, float* __restrict__ L,
                          const double* __restrict__ done, int kmin) {
  constexpr int NC = ncoef(Q) - 1, NH = nharm(Q);
  if (done && *done != 0.0) return;
  const float* Lpar = L + lp.box_off * NC;
  float* Lout = L + lv.box_off * NC;
  for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < int64_t(NC) * lv.nbox;
       t += int64_t(gridDim.x) * blockDim.x) {
    const int k = int(t / lv.nbox);
    const int64_t b = t % lv.nbox;
    float v = 0.f;
    if (k >= kmin && occ[lv.box_off + b] > 0) {
      const char4 e = c_mi.v[k + 1];
      const int j = e.z >> 1, z = e.z & 1;
      for (int i = 0; i <= j; ++i) {
        const float* lp = Lpart + int64_t(hidx(e.x + 2 * i, e.y + 2 * (j - i), z)) * lv.nbox + b;
        float p = 0.f;
        for (int ch = 0; ch < chunks; ++ch) p += lp[int64_t(ch) * NH * lv.nbox];
        v += binom_f(j, i) * p;
      }
      if (j & 1) v = -v;
      if (has_parent) {
        const int deg = e.x + e.y + e.z;
        const int x = int(b % lv.nx), y = int((b / lv.nx) % lv.ny), z = int(b / (int64_t(lv.nx) * lv.ny));
        const int64_t pb = (int64_t(z >> 1) * lp.ny + (y >> 1)) * lp.nx + (x >> 1);
        const int cx = x & 1, cy = y & 1, cz = z & 1;
        float s = 0.f;
        for (int dx = 0; dx <= Q - deg; ++dx)
          for (int dy = 0; dy <= Q - deg - dx; ++dy)
            for (int dz = 0; dz <= Q - deg - dx - dy; ++dz)
              s += Lpar[int64_t(gidx(e.x + dx, e.y + dy, e.z + dz) - 1) * lp.nbox + pb] * c_shift.v[cx][dx] *
                   c_shift.v[cy][dy] * c_shift.v[cz][dz];
        v += ldexpf(s, -2 - deg);
      }
    }
    Lout[int64_t(k) * lv.nbox + b] = v;
  }
}

// ---------------------------------------------------------------------------
// Near field + L2P + epilogue: one CTA per leaf box, one target per thread.
// Source runs (rows of x-adjacent near boxes) are cut into tiles staged in
// shared memory by bulk copies on an mbarrier pipeline, as in the all-pairs
// kernel, and swept with the packed clamped pair body.
// ---------------------------------------------------------------------------
// The CTA shape (threads per leaf box, one target each with rounds for
// larger boxes; sources per stage) is a template parameter of the kernel.
constexpr int kP2PStages = 3;
constexpr int kP2PMaxSteps = 128;  // tile steps per refill of the row walk (1 KB of shared memory)
template <int TILE>
constexpr int p2p_smem() { return kP2PStages * 2 * TILE * int(sizeof(float4)); }

struct P2PArgs {
  FmmLevel lv;
  const int32_t* start;   // sources: box starts (even-padded slots), counts, slot -> index
  const int32_t* cnt;
  const int32_t* perm;
  const int32_t* tstart;  // targets: box starts, counts, slot -> index (the same arrays
  const int32_t* tcnt;    //   when the targets are the sources)
  const int32_t* tperm;
  const float4* pos2s;
  const float4* mom2s;
  const float* L;     // leaf locals, NC rows of nbox
  const int4* rows;   // (half-width w, dy, dz, 0)
  int32_t n_rows;
  const double* done;
  // Near field from partial sums (k_fmm_near_sym): the half-stencil rows,
  // the planes [1 + offsets][3][n_slots] and their slot count.
  const int4* hrows;
  int32_t n_hrows;
  const float* part;
  int64_t n_slots;
  // k_fmm_near_warp: targets of a CTA, and the runs beyond a box's first.
  int32_t n_boxes, chunk;
  const int2* extra;
  const int32_t* extra_n;
};

// Plane of box offset dx in half row hr (1 + offsets before the row + index).
__device__ __forceinline__ int near_plane(const int4& hr, int dx) {
  return 1 + hr.w + ((hr.y == 0 && hr.z == 0) ? dx - 1 : dx + hr.x);
}

// w^k / k! for k < Q, `stride` apart.
template <int Q>
__device__ __forceinline__ void power_table(float w, float* pw, int stride) {
  float v = 1.f;
  pw[0] = 1.f;
#pragma unroll
  for (int k = 1; k < Q; ++k) {
    v = v * w * (1.f / float(k));
    pw[k * stride] = v;
  }
}

// The local expansion's terms g = g0, g0 + gstep, ...: h = sum_g L_(g + e_k)
// w^g / g! (kKind 0, x y z) or sum_g L_(g + e_a + e_b) w^g / g! (xx, yy, zz, xy,
// xz, yz).  pw: the target's columns of the three power tables.
template <int Q, int kKind>
__device__ __forceinline__ void local_terms(const float* pw, int stride, const float* s_L, int g0, int gstep, float* h) {
#pragma unroll
  for (int q = 0; q < 6; ++q) h[q] = 0.f;
  for (int g = g0; g < ncoef(kKind == 0 ? Q - 1 : Q - 2); g += gstep) {
    const char4 e = c_mi.v[g];
    const float mono = pw[e.x * stride] * pw[(Q + e.y) * stride] * pw[(2 * Q + e.z) * stride];
    if constexpr (kKind == 0) {
      h[0] = fmaf(s_L[gidx(e.x + 1, e.y, e.z) - 1], mono, h[0]);
      h[1] = fmaf(s_L[gidx(e.x, e.y + 1, e.z) - 1], mono, h[1]);
      h[2] = fmaf(s_L[gidx(e.x, e.y, e.z + 1) - 1], mono, h[2]);
    } else {
      h[0] = fmaf(s_L[gidx(e.x + 2, e.y, e.z) - 1], mono, h[0]);
      h[1] = fmaf(s_L[gidx(e.x, e.y + 2, e.z) - 1], mono, h[1]);
      h[2] = fmaf(s_L[gidx(e.x, e.y, e.z + 2) - 1], mono, h[2]);
      h[3] = fmaf(s_L[gidx(e.x + 1, e.y + 1, e.z) - 1], mono, h[3]);
      h[4] = fmaf(s_L[gidx(e.x + 1, e.y, e.z + 1) - 1], mono, h[4]);
      h[5] = fmaf(s_L[gidx(e.x, e.y + 1, e.z + 1) - 1], mono, h[5]);
    }
  }
}

// The far field from these sums: H = -grad phi = -h / (4 pi s^3); Hess phi =
// h / (4 pi s^4), F = -mu0 Hess phi m_t, the tensor -mu0 Hess phi.
template <int kKind>
__device__ __forceinline__ void add_far(const float* h, float inv_s, const AllPairsArgs<float>& a, int64_t i, double* v) {
  if constexpr (kKind == 0) {
    const double f = -kInv4Pi * double(inv_s) * double(inv_s) * double(inv_s);
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] += f * double(h[q]);
  } else {
    const double is2 = double(inv_s) * double(inv_s);
    const double f = -kMu0 * kInv4Pi * is2 * is2;
    if constexpr (kKind == 1) {
      const float4 tm = a.tmom[i];
      v[0] += f * (double(h[0]) * tm.x + double(h[3]) * tm.y + double(h[4]) * tm.z);
      v[1] += f * (double(h[3]) * tm.x + double(h[1]) * tm.y + double(h[5]) * tm.z);
      v[2] += f * (double(h[4]) * tm.x + double(h[5]) * tm.y + double(h[2]) * tm.z);
    } else {
#pragma unroll
      for (int q = 0; q < 6; ++q) v[q] += f * double(h[q]);
    }
  }
}

// kKind: 0 field (H); 1 Kelvin force, with kParts (targets = sources): the near
// field is not swept here but added from k_fmm_near_sym's partial sums -- the
// box's own plane, then the plane of every writer box (this box minus a
// half-stencil offset, inside the grid and not empty), in a fixed order with
// compensated FP32.
template <int Q, int kKind, bool kParts, int TPB, int TILE>
__global__ void __launch_bounds__(TPB) k_fmm_p2p(const P2PArgs p, const AllPairsArgs<float> a,
                                                         const SceneDesc<float> sc) {
  static_assert(kKind == (kParts ? 1 : 0), "the field swept, or the Kelvin force from partial sums");
  using Body = std::conditional_t<kKind == 0, FieldF2Body, ForceF2Body>;
  constexpr int kOut = Body::kOut;
  constexpr int NC = ncoef(Q) - 1;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar[kP2PStages];
  __shared__ int2 s_steps[kP2PMaxSteps];
  __shared__ int s_nsteps, s_row, s_pos;
  __shared__ float s_L[NC];
  if (p.done && *p.done != 0.0) return;
  const FmmLevel& lv = p.lv;
  const int64_t c = blockIdx.x;
  const int32_t n = p.tcnt[c];
  if (n == 0) return;
  const int tid = threadIdx.x;
  const int ix = int(c % lv.nx), iy = int((c / lv.nx) % lv.ny), iz = int(c / (int64_t(lv.nx) * lv.ny));
  const int32_t st0 = p.tstart[c];
  for (int k = tid; k < NC; k += TPB) s_L[k] = p.L[int64_t(k) * lv.nbox + c];
  auto stage_pos = [&](int s) { return reinterpret_cast<float4*>(smem_raw) + s * 2 * TILE; };
  auto stage_mom = [&](int s) { return stage_pos(s) + TILE; };
  if (tid == 0) {
    for (int s = 0; s < kP2PStages; ++s) mbar_init(&bar[s], 1);
    fence_mbar_init();
  }
  __syncthreads();

  auto issue = [&](int k, int s) {
    const int2 stp = s_steps[k];
    const uint32_t bytes = uint32_t(stp.y) * uint32_t(sizeof(float4));
    mbar_arrive_expect_tx(&bar[s], 2 * bytes);
    bulk_g2s(stage_pos(s), p.pos2s + stp.x, bytes, &bar[s]);
    bulk_g2s(stage_mom(s), p.mom2s + stp.x, bytes, &bar[s]);
  };
  // Thread 0: next tiles of the row walk into s_steps.
  auto fill = [&]() {
    int k = 0, r = s_row;
    int32_t pos = s_pos;
    while (r < p.n_rows && k < kP2PMaxSteps) {
      const int4 rw = p.rows[r];
      const int cy = iy + rw.y, cz = iz + rw.z;
      if (cy < 0 || cy >= lv.ny || cz < 0 || cz >= lv.nz) {
        ++r;
        pos = -1;
        continue;
      }
      const int cx0 = max(ix - rw.x, 0), cx1 = min(ix + rw.x, lv.nx - 1);
      const int64_t rb = (int64_t(cz) * lv.ny + cy) * lv.nx;
      const int32_t b = p.start[rb + cx0], e = p.start[rb + cx1 + 1];
      if (pos < 0) pos = b;
      if (pos >= e) {
        ++r;
        pos = -1;
        continue;
      }
      const int32_t m = min(TILE, e - pos);
      s_steps[k++] = make_int2(pos, m);
      pos += m;
    }
    s_row = r;
    s_pos = pos;
    s_nsteps = k;
  };

  uint32_t u = 0;  // steps consumed so far (stage and parity of the next)
  bool failed = false;
  int fail_k = 0, fail_ns = 0;
  for (int t0 = 0; t0 < n && !failed; t0 += TPB) {
    const bool act = t0 + tid < n;
    // A warp without a live target (the last warps of a small box) skips
    // the pair sweeps; it still takes part in every barrier and wait.
    const bool warp_live = __any_sync(0xffffffffu, act);
    const int32_t i = p.tperm[st0 + (act ? t0 + tid : 0)];
    typename Body::TData td;
    Body::load(a, i, td);
    float run[kOut], cmp[kOut];
#pragma unroll
    for (int q = 0; q < kOut; ++q) run[q] = cmp[q] = 0.f;
    if constexpr (kParts) {
      if (act) {
        const int64_t slot = int64_t(st0) + t0 + tid;
#pragma unroll
        for (int q = 0; q < 3; ++q) two_sum_acc(run[q], cmp[q], __ldcg(p.part + int64_t(q) * p.n_slots + slot));
        for (int r = 0; r < p.n_hrows; ++r) {
          const int4 hr = p.hrows[r];
          const int ay = iy - hr.y, az = iz - hr.z;
          if (ay < 0 || ay >= lv.ny || az < 0 || az >= lv.nz) continue;
          for (int dx = (hr.y == 0 && hr.z == 0) ? 1 : -hr.x; dx <= hr.x; ++dx) {
            const int ax = ix - dx;
            if (ax < 0 || ax >= lv.nx) continue;
            if (p.cnt[(int64_t(az) * lv.ny + ay) * lv.nx + ax] == 0) continue;
            const float* pl = p.part + int64_t(near_plane(hr, dx)) * 3 * p.n_slots + slot;
#pragma unroll
            for (int q = 0; q < 3; ++q) two_sum_acc(run[q], cmp[q], __ldcg(pl + int64_t(q) * p.n_slots));
          }
        }
      }
    }
    if (tid == 0) {
      s_row = 0;
      s_pos = -1;
    }
    // The row walk and its sweeps (not in the read-back mode).
    if constexpr (!kParts) for (;;) {
      __syncthreads();  // the previous segment's steps are consumed
      if (tid == 0) fill();
      __syncthreads();
      const int ns = s_nsteps;
      if (ns == 0) break;
      if (tid == 0)
        for (int k = 0; k < kP2PStages && k < ns; ++k) issue(k, int((u + k) % kP2PStages));
      for (int k = 0; k < ns; ++k) {
        const uint32_t uu = u + uint32_t(k);
        const int s = int(uu % kP2PStages);
        const bool ok = mbar_wait_bounded(&bar[s], (uu / kP2PStages) & 1u);
        if (__syncthreads_or(!ok)) {
          failed = true;
          fail_k = k;
          fail_ns = ns;
          break;
        }
        const int n_items = s_steps[k].y >> 1;
        const float4* __restrict__ sp = stage_pos(s);
        const float4* __restrict__ sm = stage_mom(s);
        if (warp_live) {
          typename Body::Acc acc;
          acc.zero();
#pragma unroll 4
          for (int j = 0; j < n_items; ++j) Body::pair(td, Body::load_item(sp, sm, j), sc.pc, acc);
          float o[kOut];
          Body::tile_out(acc, o);
#pragma unroll
          for (int q = 0; q < kOut; ++q) comp_add(run[q], cmp[q], o[q]);
        }
        __syncthreads();  // stage s is free
        if (tid == 0 && k + kP2PStages < ns) {
          fence_proxy_async_smem();
          issue(k + kP2PStages, s);
        }
      }
      if (failed) break;
      u += uint32_t(ns);
    }
    if (failed) break;
    __syncthreads();  // stages idle: reuse them for the power tables
    // Far field from the box's local expansion at w = (x - centre) / edge.
    float* pw = reinterpret_cast<float*>(smem_raw);  // [3Q][threads]
    const float4 tp = a.tpos[i];
    const float inv_s = 1.f / lv.side;
    const float w[3] = {(tp.x - (lv.ox + (float(ix) + 0.5f) * lv.side)) * inv_s,
                        (tp.y - (lv.oy + (float(iy) + 0.5f) * lv.side)) * inv_s,
                        (tp.z - (lv.oz + (float(iz) + 0.5f) * lv.side)) * inv_s};
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) power_table<Q>(w[ax], pw + ax * Q * TPB + tid, TPB);
    double v[kOut];
    for (int q = 0; q < kOut; ++q) v[q] = double(run[q]) + double(cmp[q]);
    float h[6];
    local_terms<Q, kKind>(pw + tid, TPB, s_L, 0, 1, h);
    add_far<kKind>(h, inv_s, a, i, v);
    if (act) Body::epilogue(a, sc, i, td, v);
  }
  if (failed && tid == 0) {
    // Copies in flight: steps fail_k .. min(fail_ns, fail_k + stages) - 1 of
    // the segment that failed, one per stage; wait for each (bounded).
    atomicExch(a.err, MF_DEVERR_STAGE_TIMEOUT);
    bool drained = true;
    const int k_stop = min(fail_ns, fail_k + kP2PStages);
    for (int k = fail_k; k < k_stop; ++k) {
      const uint32_t uu = u + uint32_t(k);
      if (!mbar_wait_bounded(&bar[uu % kP2PStages], (uu / kP2PStages) & 1u)) drained = false;
    }
    if (!drained) atomicExch(a.err, MF_DEVERR_DRAIN_TIMEOUT);
  }
}

// ---------------------------------------------------------------------------
// Near field + L2P + epilogue, four targets of a leaf box per warp and round.
// The lanes split the box's near source items: every lane holds the same four
// targets and reads its own item, straight from the pair-layout records (a
// warp's loads are one contiguous run), the next one while the current one is
// swept, so a box of any count leaves at most three slots of its last round
// empty and no wait is longer than a warp's own.  The CTA of 128 targets
// (k_fmm_p2p) leaves 38 % of its lanes idle at 20 particles a box and waits for
// its staging at four warps' pace.
// Bound: the packed FMAs' latency and register ports at three warps per
// scheduler (128 registers; FMA pipe 50 %, issue 52 % at 200,003 particles), with
// the record loads behind them: 8 bytes from L1 or L2 per pair (LSU wavefronts
// 49 %), which is why big boxes in great number stay with the staged kernel
// (launch_near).  Unrolling the item loop loses 8 % at 330,000 particles.
// Whole step of a cylinder of 200,003 particles (16 per box) 13.69 -> 11.57 ms, of
// a sphere of 330,000 (81, 124 per occupied box) 29.86 -> 23.78, field product of 150,000 sources at
// 30,011 separate targets 1.97 -> 1.32 ms, tensor 3.89 -> 2.68.  Other splits of the
// 32 lanes (targets per lane x lane groups), the same step at 200,003: 4 x 16
// 12.31, 4 x 8 12.58, 2 x 16 11.99, 8 x 32 12.69, 2 x 4 14.33 ms.
// ---------------------------------------------------------------------------
constexpr int kNearT = 4;         // targets of a round
constexpr int kNearFold = 64;     // items of a lane between folds of its FP32 sums
constexpr int kNearMaxWarps = 8;  // warps per CTA (one box), taking rounds in turn
constexpr int kNearRounds = 4;    // rounds of a warp; a box's further targets go to further CTAs
template <int Q>
struct NearWarp {
  static constexpr int kHead = (ncoef(Q) - 1 + 3) & ~3;       // words per CTA: the box's locals
  static constexpr int kWords = 64 + 3 * Q * kNearT;          // and per warp: rows, powers
  static constexpr int smem(int warps) { return (kHead + warps * kWords) * int(sizeof(float)); }
};

template <int Q, int kKind>
__global__ void __launch_bounds__(32 * kNearMaxWarps, 2)
    k_fmm_near_warp(const P2PArgs p, const AllPairsArgs<float> a, const SceneDesc<float> sc) {
  using Body = std::conditional_t<kKind == 0, FieldF2Body, std::conditional_t<kKind == 1, ForceF2Body, TensorF2Body>>;
  using Item = PairItems::Item;
  constexpr int kOut = Body::kOut;
  using S = NearWarp<Q>;
  static_assert(S::kHead % 2 == 0 && S::kWords % 2 == 0, "the rows are read as int2");
  extern __shared__ __align__(16) float near_smem[];
  if (p.done && *p.done != 0.0) return;
  const FmmLevel& lv = p.lv;
  int64_t c = blockIdx.x;
  int32_t first = 0;
  if (c >= p.n_boxes) {
    const int64_t e = c - p.n_boxes;
    if (e >= *p.extra_n) return;
    c = p.extra[e].x;
    first = p.extra[e].y;
  }
  const int32_t n = min(p.tcnt[c], first + p.chunk);
  if (n == 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ix = int(c % lv.nx), iy = int((c / lv.nx) % lv.ny), iz = int(c / (int64_t(lv.nx) * lv.ny));
  const int32_t st0 = p.tstart[c];
  float* s_L = near_smem;
  float* ws = near_smem + S::kHead + warp * S::kWords;
  int2* s_row = reinterpret_cast<int2*>(ws);  // per row: end in the flat item order, item offset
  float* pw = ws + 64;                        // [3 Q][kNearT]
  for (int k = threadIdx.x; k < ncoef(Q) - 1; k += blockDim.x) s_L[k] = p.L[int64_t(k) * lv.nbox + c];
  __syncthreads();  // the only block barrier: the warps part ways here
  for (int t0 = first + warp * kNearT; t0 < n; t0 += nw * kNearT) {
    typename Body::TData td[kNearT];
    float run[kNearT][kOut], cmp[kNearT][kOut];
#pragma unroll
    for (int t = 0; t < kNearT; ++t) {
      Body::load(a, p.tperm[st0 + (t0 + t < n ? t0 + t : 0)], td[t]);
#pragma unroll
      for (int q = 0; q < kOut; ++q) run[t][q] = cmp[t][q] = 0.f;
    }
    for (int r0 = 0; r0 < p.n_rows; r0 += 32) {
      // One lane per row of near boxes: its first item and its item count.
      int b = 0, m = 0;
      if (r0 + lane < p.n_rows) {
        const int4 rw = p.rows[r0 + lane];
        const int cy = iy + rw.y, cz = iz + rw.z;
        if (cy >= 0 && cy < lv.ny && cz >= 0 && cz < lv.nz) {
          const int cx0 = max(ix - rw.x, 0), cx1 = min(ix + rw.x, lv.nx - 1);
          const int64_t rb = (int64_t(cz) * lv.ny + cy) * lv.nx;
          b = p.start[rb + cx0] >> 1;
          m = (p.start[rb + cx1 + 1] >> 1) - b;
        }
      }
      int end = m;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += up;
      }
      const int total = __shfl_sync(0xffffffffu, end, 31);
      __syncwarp();  // the rows before these are done with
      s_row[lane] = make_int2(end, b - (end - m));
      __syncwarp();
      int row = -1, row_end = 0, row_off = 0;
      // Past the last item: a zero dipole, which adds nothing.
      auto fetch = [&](int j) {
        if (j >= total) return Item{{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        while (j >= row_end) {  // ends at the last row: j < total, its end
          const int2 e = s_row[++row];
          row_end = e.x;
          row_off = e.y;
        }
        return Body::load_item(p.pos2s, p.mom2s, j + row_off);
      };
      Item it = fetch(lane);
      for (int j0 = 0; j0 < total; j0 += 32 * kNearFold) {
        typename Body::Acc acc[kNearT];
#pragma unroll
        for (int t = 0; t < kNearT; ++t) acc[t].zero();
        const int j1 = min(total, j0 + 32 * kNearFold);
        for (int j = j0; j < j1; j += 32) {
          const Item nx = fetch(j + 32 + lane);
#pragma unroll
          for (int t = 0; t < kNearT; ++t) Body::pair(td[t], it, sc.pc, acc[t]);
          it = nx;
        }
#pragma unroll
        for (int t = 0; t < kNearT; ++t) {
          float o[kOut];
          Body::tile_out(acc[t], o);
#pragma unroll
          for (int q = 0; q < kOut; ++q) comp_add(run[t][q], cmp[t][q], o[q]);
        }
      }
    }
    // The lanes' sums, in a fixed order: the first two exchanges leave a lane
    // with target lane / 8, the others add up its eight lanes.
    auto fold = [&](float& r, float& e, float sr, float se, int d) {
      const float o = __shfl_xor_sync(0xffffffffu, sr, d), oe = __shfl_xor_sync(0xffffffffu, se, d);
      comp_add(r, e, o);
      e += oe;
    };
    auto scatter = [&](int keep, int d) {  // targets [0, 2 keep) -> [0, keep)
      const bool hi = lane & d;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (t >= keep) break;
#pragma unroll
        for (int q = 0; q < kOut; ++q) {
          const float sr = hi ? run[t][q] : run[t + keep][q], se = hi ? cmp[t][q] : cmp[t + keep][q];
          run[t][q] = hi ? run[t + keep][q] : run[t][q];
          cmp[t][q] = hi ? cmp[t + keep][q] : cmp[t][q];
          fold(run[t][q], cmp[t][q], sr, se, d);
        }
      }
    };
    scatter(2, 16);
    scatter(1, 8);
#pragma unroll
    for (int q = 0; q < kOut; ++q)
#pragma unroll
      for (int d = 4; d > 0; d >>= 1) fold(run[0][q], cmp[0][q], run[0][q], cmp[0][q], d);
    // Far field from the box's local expansion: eight lanes per target, each
    // every eighth term.
    const int tt = lane >> 3, tg = lane & 7;
    const bool act = t0 + tt < n;
    const int32_t i = p.tperm[st0 + (act ? t0 + tt : 0)];
    const float inv_s = 1.f / lv.side;
    if (tg < 3) {
      const float4 tp = a.tpos[i];
      const float x = tg == 0 ? tp.x : tg == 1 ? tp.y : tp.z, o = tg == 0 ? lv.ox : tg == 1 ? lv.oy : lv.oz;
      const int ib = tg == 0 ? ix : tg == 1 ? iy : iz;
      power_table<Q>((x - (o + (float(ib) + 0.5f) * lv.side)) * inv_s, pw + tg * Q * kNearT + tt, kNearT);
    }
    __syncwarp();
    float h[6];
    local_terms<Q, kKind>(pw + tt, kNearT, s_L, tg, 8, h);
#pragma unroll
    for (int q = 0; q < (kKind == 0 ? 3 : 6); ++q)
#pragma unroll
      for (int d = 4; d > 0; d >>= 1) h[q] += __shfl_xor_sync(0xffffffffu, h[q], d);
    if (tg == 0 && act) {
      double v[kOut];
#pragma unroll
      for (int q = 0; q < kOut; ++q) v[q] = double(run[0][q]) + double(cmp[0][q]);
      add_far<kKind>(h, inv_s, a, i, v);
      typename Body::TData t1;
      Body::load(a, i, t1);
      Body::epilogue(a, sc, i, t1, v);
    }
    __syncwarp();  // the powers are read before the next round writes them
  }
}

// ---------------------------------------------------------------------------
// Near field of the Kelvin force once per unordered box pair (targets are the
// sources): one warp per leaf box A.  Both half-warps hold the same 128
// target slots (8 per lane; rounds of 128 for larger boxes) and sweep
// alternate pairs of source items, so every shuffle tree of the source sums
// spans 16 lanes and serves 8 targets per lane.
//   * A's own pairs: every ordered pair, target side only.
//   * The boxes B of the half stencil: each pair item's force adds into the
//     targets' sums and, reduced over the half-warp by a fixed shuffle tree,
//     into the sources' sums (f_ji = -f_ij), stored at plane near_plane(B - A)
//     of the source's slot.  A later target round adds to the entries of the
//     earlier ones (the same lane, in order).
//   * The targets' sums (the two halves' added) go to plane 0.
// Every (plane, slot) entry has one writer, so results do not depend on
// scheduling.  Sums are in the all-pairs kernels' units (times K).
// ---------------------------------------------------------------------------
struct NearSymArgs {
  FmmLevel lv;
  const int32_t* start;  // box slot starts (even-padded), leaf level
  const int32_t* cnt;
  const int32_t* perm;   // slot -> particle
  const float4* pos2s;   // pair-layout records by slot
  const float4* mom2s;
  const int4* hrows;
  int32_t n_hrows;
  float* part;
  int64_t n_slots;
  const double* done;
};
constexpr int kNearSymWarps = 4, kNearSymTPT = 8, kNearSymChunk = 64;

// The walk over the half stencil's source boxes in units of up to
// kNearSymChunk pair items (a box in one or more chunks), in the order
// rows, x offsets, chunks.
struct NearUnit {
  int32_t sb;     // first slot of the box
  int32_t cs;     // first item of the chunk in the box
  int32_t cn;     // items in the chunk
  int32_t plane;  // partial-sum plane of the box's offset (-1: no unit)
};
struct NearCursor {
  int r, dx;         // next half-stencil row and x offset to examine
  int32_t sb, ni;    // the box being chunked (ni items; 0: none)
  int32_t cs, plane;
};

__device__ __forceinline__ NearUnit near_next(NearCursor& cur, const NearSymArgs& p, int ix, int iy, int iz) {
  constexpr int CH = kNearSymChunk;
  const FmmLevel& lv = p.lv;
  for (;;) {
    if (cur.cs < cur.ni) {
      const NearUnit u{cur.sb, cur.cs, min(CH, cur.ni - cur.cs), cur.plane};
      cur.cs += CH;
      return u;
    }
    if (cur.r >= p.n_hrows) return NearUnit{0, 0, 0, -1};
    const int4 hr = p.hrows[cur.r];
    const int cy = iy + hr.y, cz = iz + hr.z;
    const int dx = cur.dx;
    if (cy < 0 || cy >= lv.ny || cz < 0 || cz >= lv.nz || dx > hr.x) {  // next row
      ++cur.r;
      if (cur.r < p.n_hrows) {
        const int4 h2 = p.hrows[cur.r];
        cur.dx = (h2.y == 0 && h2.z == 0) ? 1 : -h2.x;
      }
      continue;
    }
    ++cur.dx;
    const int cx = ix + dx;
    if (cx < 0 || cx >= lv.nx) continue;
    const int64_t b = (int64_t(cz) * lv.ny + cy) * lv.nx + cx;
    const int32_t nb = p.cnt[b];
    if (nb == 0) continue;
    cur.sb = p.start[b];
    cur.ni = (nb + 1) >> 1;
    cur.cs = 0;
    cur.plane = near_plane(hr, dx);
  }
}

// Reduce-scatter of NV values over each half-warp (16 lanes): lane l ends
// with value l & 15 summed over its half, by a fixed shuffle tree.
template <int NV>
__device__ __forceinline__ float half_reduce_scatter(const float (&v)[NV], int lane) {
  static_assert(NV == 16, "one value per lane of a half-warp");
  float w[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) w[q] = v[q];
  int b = 8;
#pragma unroll
  for (int n = NV; n > 1; n >>= 1, b >>= 1) {
    const bool hi = lane & b;
#pragma unroll
    for (int q = 0; q < n / 2; ++q) {
      const float send = hi ? w[q] : w[q + n / 2];
      const float keep = hi ? w[q + n / 2] : w[q];
      w[q] = keep + __shfl_xor_sync(0xffffffffu, send, b);
    }
  }
  return w[0];
}

// 255 registers with 2 CTAs per SM; one warp per box with 4 targets per
// lane (168 registers, 3 CTAs per SM) measured 69.4 against 64.2 ms at
// 1,048,576 particles: its 32-lane trees served half the targets each.
__global__ void __launch_bounds__(32 * kNearSymWarps, 2) k_fmm_near_sym(const NearSymArgs p, const AllPairsArgs<float> a,
                                                                   const SceneDesc<float> sc) {
  constexpr int TPT = kNearSymTPT, CH = kNearSymChunk;
  constexpr int TL = 16;    // lanes per target set (a half-warp)
  constexpr int STEP = 4;   // items per sweep step of the warp (2 per half)
  // per warp, two buffers: a unit of a source box's pair items (positions,
  // then dipoles); the next unit is copied into one while the current one is
  // swept from the other
  __shared__ __align__(16) float4 s_pos[kNearSymWarps][2][2 * CH], s_mom[kNearSymWarps][2][2 * CH];
  if (p.done && *p.done != 0.0) return;
  const FmmLevel& lv = p.lv;
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  const int tl = lane & (TL - 1);  // slot lane within the target set
  const int half = lane >> 4;      // which items of a step this lane sweeps
  const int64_t c = int64_t(blockIdx.x) * kNearSymWarps + w;
  if (c >= lv.nbox) return;  // warp-uniform; the kernel has no block barrier
  const int32_t n = p.cnt[c];
  if (n == 0) return;
  const int ix = int(c % lv.nx), iy = int((c / lv.nx) % lv.ny), iz = int(c / (int64_t(lv.nx) * lv.ny));
  const int32_t st0 = p.start[c];
  const float near2 = sc.pc.near2_force;
  const float kk = float(kForceK);
  const PairItems::Item zero_item{{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  // Every lane copies its share of a unit and commits one group per unit
  // (possibly empty), so the lanes' group counts stay in step.
  auto stage = [&](const NearUnit& u, int buf) {
    if (u.plane >= 0) {
      const float4* sp = p.pos2s + u.sb + 2 * u.cs;
      const float4* sm = p.mom2s + u.sb + 2 * u.cs;
      for (int k = lane; k < 2 * u.cn; k += 32) {
        cp_async16(&s_pos[w][buf][k], sp + k);
        cp_async16(&s_mom[w][buf][k], sm + k);
      }
    }
    cp_async_commit();
  };
  for (int t0 = 0; t0 < n; t0 += TL * TPT) {
    float2 tx[TPT], ty[TPT], tz[TPT], tmx[TPT], tmy[TPT], tmz[TPT];
    float2 acc[TPT][3];
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
      const int li = t0 + t * TL + tl;
      const bool live = li < n;
      const int32_t i = p.perm[st0 + (live ? li : 0)];
      const float4 q = a.tpos[i];
      const float4 wm = live ? a.tmom[i] : make_float4(0.f, 0.f, 0.f, 0.f);  // a dead slot adds nothing to sources
      tx[t] = f2_dup(q.x);
      ty[t] = f2_dup(q.y);
      tz[t] = f2_dup(q.z);
      tmx[t] = f2_dup(wm.x);
      tmy[t] = f2_dup(wm.y);
      tmz[t] = f2_dup(wm.z);
      acc[t][0] = acc[t][1] = acc[t][2] = make_float2(0.f, 0.f);
    }
    NearCursor cur{0, 0, 0, 0, 0, 0};
    if (p.n_hrows > 0) {
      const int4 h0 = p.hrows[0];
      cur.dx = (h0.y == 0 && h0.z == 0) ? 1 : -h0.x;
    }
    NearUnit u = near_next(cur, p, ix, iy, iz);
    int buf = 0;
    __syncwarp();  // the previous round's reads of both buffers are done
    stage(u, 0);
    {  // the box's own pairs, target side only (the first unit's copy is in flight)
      const float4* sp = p.pos2s + st0;
      const float4* sm = p.mom2s + st0;
      const int ni = (n + 1) >> 1;
      for (int j = half; j < ni; j += 2) {
        const PairItems::Item it = PairItems::load_item(sp, sm, j);
        float2 src[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int t = 0; t < TPT; ++t) sym_force_pair2(tx[t], ty[t], tz[t], tmx[t], tmy[t], tmz[t], it, near2, acc[t], src);
      }
    }
    while (u.plane >= 0) {
      const NearUnit nxt = near_next(cur, p, ix, iy, iz);
      stage(nxt, buf ^ 1);
      cp_async_wait<1>();  // this lane's copies of unit u have landed
      __syncwarp();        // and every lane's
      const float4* wpos = s_pos[w][buf];
      const float4* wmom = s_mom[w][buf];
      float* plane = p.part + int64_t(u.plane) * 3 * p.n_slots;
      const int cn = u.cn;
      // Past the unit's last item: a zero dipole at the origin, nothing on either side.
      for (int j0 = 0; j0 < cn; j0 += STEP) {
        const int jb = j0 + 2 * half;  // this lane's first item of the step
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = 0.f;
#pragma unroll
        for (int q2 = 0; q2 < 2; ++q2) {
          const PairItems::Item it = (jb + q2 < cn) ? PairItems::load_item(wpos, wmom, jb + q2) : zero_item;
          float2 src[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
          for (int t = 0; t < TPT; ++t) sym_force_pair2(tx[t], ty[t], tz[t], tmx[t], tmy[t], tmz[t], it, near2, acc[t], src);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            v[q2 * 6 + 2 * k] = src[k].x;
            v[q2 * 6 + 2 * k + 1] = src[k].y;
          }
        }
        // value kv: item jb + kv / 6, component (kv % 6) / 2, source kv % 2
        const float wr = half_reduce_scatter<16>(v, lane);
        const int kv = tl;
        if (kv < 12) {
          const int jl = jb + kv / 6, rem = kv % 6;
          if (jl < cn) {
            float* dst = plane + int64_t(rem >> 1) * p.n_slots + (int64_t(u.sb) + 2 * (u.cs + jl) + (rem & 1));
            const float val = -wr * kk;  // f_ji = -f_ij
            if (t0 == 0) *dst = val;
            else *dst += val;
          }
        }
      }
      __syncwarp();  // every lane is done with buffer buf before it is refilled
      buf ^= 1;
      u = nxt;
    }
    cp_async_wait<0>();
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        float s2 = acc[t][k].x + acc[t][k].y;
        s2 += __shfl_xor_sync(0xffffffffu, s2, 16);  // the other half's items
        acc[t][k].x = s2;
      }
      const int li = t0 + t * TL + tl;
      if (li < n && half == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) p.part[int64_t(k) * p.n_slots + st0 + li] = acc[t][k].x * kk;
      }
    }
  }
}

unsigned blocks_for(int64_t n, int per = 256, int64_t cap = 65535) {
  int64_t g = (n + per - 1) / per;
  if (g > cap) g = cap;
  return unsigned(g < 1 ? 1 : g);
}

// Taylor coefficients of 1/|R| times gamma!: D_gamma = d^gamma (1/|R|), all
// gamma of degree <= nmax, in graded order.  Recurrence on the coefficients
// T_n = d^n(1/|R|)/n!:  |n| R^2 T_n + (2|n|-1) sum_i R_i T_(n-e_i) + (|n|-1) sum_i T_(n-2e_i) = 0.
void taylor_inv_r(const double R[3], int nmax, std::vector<double>& D) {
  const int N = ncoef(nmax);
  std::vector<double> T(size_t(N), 0.0);
  std::vector<int> mx(static_cast<size_t>(N)), my(static_cast<size_t>(N)), mz(static_cast<size_t>(N));
  const double r2 = R[0] * R[0] + R[1] * R[1] + R[2] * R[2];
  for (int n = 0; n <= nmax; ++n)
    for (int s = 0; s <= n; ++s)
      for (int z = 0; z <= s; ++z) {
        const int x = n - s, y = s - z;
        const int k = gidx(x, y, z);
        mx[size_t(k)] = x;
        my[size_t(k)] = y;
        mz[size_t(k)] = z;
        if (n == 0) {
          T[size_t(k)] = 1.0 / std::sqrt(r2);
          continue;
        }
        const int a[3] = {x, y, z};
        double acc = 0.0;
        for (int i = 0; i < 3; ++i) {
          int b[3] = {x, y, z};
          if (a[i] >= 1) {
            b[i] -= 1;
            acc += double(2 * n - 1) * R[i] * T[size_t(gidx(b[0], b[1], b[2]))];
            b[i] += 1;
          }
          if (a[i] >= 2) {
            b[i] -= 2;
            acc += double(n - 1) * T[size_t(gidx(b[0], b[1], b[2]))];
          }
        }
        T[size_t(k)] = -acc / (double(n) * r2);
      }
  D.assign(size_t(N), 0.0);
  auto fact = [](int v) {
    double f = 1.0;
    for (int i = 2; i <= v; ++i) f *= double(i);
    return f;
  };
  for (int k = 0; k < N; ++k) D[size_t(k)] = T[size_t(k)] * fact(mx[size_t(k)]) * fact(my[size_t(k)]) * fact(mz[size_t(k)]);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// The interaction lists of the levels, the near rows of the leaf level and the
// derivative table, built on the host and uploaded.  far(l, dx, dy, dz): the
// acceptance test, |d|^2 > m[l].
template <class Far>
mf_status Fmm::build_lists(int L, const std::vector<int64_t>& m, const Far& far, cudaStream_t st) {
  const int Q = degree_;
  const FmmLevel& leaf = lv_[size_t(L)];
  auto reach = [&](int l) { return int(std::min<int64_t>(int64_t(std::sqrt(double(m[size_t(l)]))) + 1, 1 << 20)); };
  auto fdiv = [](int a, int b) { return (a >= 0) ? a / b : -((-a + b - 1) / b); };
  std::map<std::tuple<int, int, int>, int> did;
  host_list_.clear();
  list_off_.assign(size_t(8 * (L + 1)), 0);
  list_cnt_.assign(size_t(8 * (L + 1)), 0);
  for (int l = 2; l <= L; ++l) {
    const FmmLevel& v = lv_[size_t(l)];
    const int R = 2 * reach(l - 1) + 1;  // parent offsets that are not accepted reach this far
    for (int cls = 0; cls < 8; ++cls) {
      const int c[3] = {cls & 1, (cls >> 1) & 1, cls >> 2};
      list_off_[size_t(8 * l + cls)] = int64_t(host_list_.size());
      const int Rx = std::min(R, v.nx - 1), Ry = std::min(R, v.ny - 1), Rz = std::min(R, v.nz - 1);
      for (int dz = -Rz; dz <= Rz; ++dz)
        for (int dy = -Ry; dy <= Ry; ++dy)
          for (int dx = -Rx; dx <= Rx; ++dx) {
            if (!far(l, dx, dy, dz)) continue;
            const int d[3] = {dx, dy, dz};
            int D[3];
            for (int k = 0; k < 3; ++k) D[k] = -fdiv(c[k] - d[k], 2);
            if (far(l - 1, D[0], D[1], D[2])) continue;
            const int id = did.emplace(std::make_tuple(dx, dy, dz), int(did.size())).first->second;
            host_list_.push_back(make_int4(dx, dy, dz, id));
          }
      list_cnt_[size_t(8 * l + cls)] = int64_t(host_list_.size()) - list_off_[size_t(8 * l + cls)];
    }
  }
  // Near rows of the leaf level: for each (dy, dz), x offsets |dx| <= w.
  host_rows_.clear();
  {
    const int R = reach(L);
    const int Rx = std::min(R, leaf.nx - 1), Ry = std::min(R, leaf.ny - 1), Rz = std::min(R, leaf.nz - 1);
    for (int dz = -Rz; dz <= Rz; ++dz)
      for (int dy = -Ry; dy <= Ry; ++dy) {
        if (far(L, 0, dy, dz)) continue;
        int w = 0;
        while (w + 1 <= Rx && !far(L, w + 1, dy, dz)) ++w;
        host_rows_.push_back(make_int4(w, dy, dz, 0));
      }
  }
  n_rows_ = int(host_rows_.size());
  // Half stencil for the near field once per unordered box pair: rows with
  // dz > 0, or dz = 0 and dy > 0 (x offsets -w..w), and the centre row (x
  // offsets 1..w).  w of a half row holds the box offsets before it; its
  // offsets dx take planes 1 + w_before + (dx + w) (centre: dx - 1).
  host_hrows_.clear();
  n_off_ = 0;
  for (const int4& r : host_rows_) {
    if (r.z > 0 || (r.z == 0 && r.y > 0)) {
      host_hrows_.push_back(make_int4(r.x, r.y, r.z, n_off_));
      n_off_ += 2 * r.x + 1;
    } else if (r.y == 0 && r.z == 0 && r.x > 0) {
      host_hrows_.push_back(make_int4(r.x, 0, 0, n_off_));
      n_off_ += r.x;
    }
  }
  n_hrows_ = int(host_hrows_.size());
  const int ND = ndtab(Q);
  host_dt_.assign(did.size() * size_t(ND), 0.f);
  std::vector<double> D;
  for (const auto& kv : did) {
    const double R[3] = {double(std::get<0>(kv.first)), double(std::get<1>(kv.first)), double(std::get<2>(kv.first))};
    taylor_inv_r(R, Q + 1, D);
    for (int n = 0; n <= Q + 1; ++n)
      for (int z = 0; z <= std::min(n, 2); ++z)
        for (int y = 0; y <= n - z; ++y)
          host_dt_[size_t(kv.second) * size_t(ND) + size_t(didx(n - z - y, y, z))] = float(D[size_t(gidx(n - z - y, y, z))]);
  }
  host_lofs_ = list_off_;
  host_lofs_.insert(host_lofs_.end(), list_cnt_.begin(), list_cnt_.end());
  // Uploads are ordered on the stream, from host copies kept as members.
  auto put = [&](DevBuf& dst, const void* src, size_t bytes) -> mf_status {
    MF_TRY(dst.reserve_slack(std::max<size_t>(16, bytes)));
    if (bytes) MF_CUDA_TRY(cudaMemcpyAsync(dst.ptr, src, bytes, cudaMemcpyHostToDevice, st));
    return MF_OK;
  };
  MF_TRY(put(dtab_, host_dt_.data(), host_dt_.size() * sizeof(float)));
  MF_TRY(put(lists_, host_list_.data(), host_list_.size() * sizeof(int4)));
  MF_TRY(put(rows_, host_rows_.data(), host_rows_.size() * sizeof(int4)));
  MF_TRY(put(hrows_, host_hrows_.data(), host_hrows_.size() * sizeof(int4)));
  return put(lofs_, host_lofs_.data(), host_lofs_.size() * sizeof(int64_t));
}

mf_status Fmm::build(const float4* pos4, int64_t n, const float4* tpos4, int64_t nt, double h, const double* bbox,
                     const FmmConfig& cfg, cudaStream_t st) {
  if (n <= 0) return fail(MF_ERR_INVALID_ARG, "fmm: no particles");
  if (n >= (int64_t(1) << 30) || nt >= (int64_t(1) << 30)) return fail(MF_ERR_INVALID_ARG, "fmm: too many particles");
  if (tpos4 && nt <= 0) return fail(MF_ERR_INVALID_ARG, "fmm: no targets");
  separate_ = tpos4 != nullptr;
  nt_ = separate_ ? nt : n;
  if (cfg.order < 4 || cfg.order > kMaxDegree + 1) return fail(MF_ERR_INVALID_ARG, "fmm: order must be in [4, 10]");
  if (!(cfg.theta > 0.0 && cfg.theta <= 1.0)) return fail(MF_ERR_INVALID_ARG, "fmm: theta must be in (0, 1]");
  if (cfg.leaf_min < 1) return fail(MF_ERR_INVALID_ARG, "fmm: leaf_min must be >= 1");
  cfg_ = cfg;
  degree_ = cfg.order - 1;
  n_ = n;
  const int Q = degree_;
  const int NC = ncoef(Q) - 1;

  // Box grids.
  double lo[3], ext[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = bbox[k];
    ext[k] = std::max(0.0, bbox[3 + k] - bbox[k]);
    if (!std::isfinite(lo[k]) || !std::isfinite(ext[k])) return fail(MF_ERR_INVALID_ARG, "fmm: non-finite positions");
  }
  const double emax = std::max({ext[0], ext[1], ext[2]});
  const double S0 = std::max(emax * (1.0 + 1e-5), h * 1e-3);
  for (int k = 0; k < 3; ++k) lo[k] -= 0.25e-5 * S0;
  auto dims_at = [&](int l, int d[3]) {
    const double s = S0 / double(int64_t(1) << l);
    for (int k = 0; k < 3; ++k) {
      int64_t m = int64_t(std::ceil((ext[k] + 0.5e-5 * S0) / s));
      m = std::max<int64_t>(1, std::min<int64_t>(m, int64_t(1) << l));
      d[k] = int(m);
    }
  };
  int L = 2;
  for (int l = 3; l <= kMaxLevel; ++l) {
    int d[3];
    dims_at(l, d);
    const double boxes = double(d[0]) * d[1] * d[2];
    if (double(n) / boxes < double(cfg.leaf_min) || boxes > double(1 << 24)) break;
    L = l;
  }
  lv_.assign(size_t(L + 1), FmmLevel{});
  {
    int d[3];
    dims_at(L, d);
    for (int l = L; l >= 0; --l) {
      FmmLevel& v = lv_[size_t(l)];
      v.nx = d[0];
      v.ny = d[1];
      v.nz = d[2];
      v.nbox = int64_t(d[0]) * d[1] * d[2];
      v.side = float(S0 / double(int64_t(1) << l));
      v.ox = float(lo[0]);
      v.oy = float(lo[1]);
      v.oz = float(lo[2]);
      for (int k = 0; k < 3; ++k) d[k] = (d[k] + 1) / 2;
    }
    int64_t off = 0;
    for (int l = 0; l <= L; ++l) {
      lv_[size_t(l)].box_off = off;
      off += lv_[size_t(l)].nbox;
    }
  }
  const FmmLevel& leaf = lv_[size_t(L)];
  const int64_t nbox_total = leaf.box_off + leaf.nbox;
  const int64_t ncell = leaf.nbox;

  // Bin.
  MF_TRY(occ_.reserve_slack(size_t(nbox_total) * sizeof(int32_t)));
  int32_t* occ = occ_.as<int32_t>();
  int32_t* cnt = occ + leaf.box_off;
  MF_TRY(cell_of_.reserve(size_t(n) * sizeof(int32_t)));
  MF_TRY(start_.reserve_slack(size_t(ncell + 1) * sizeof(int32_t)));
  // The list of runs lies behind the cursors (whole 16 bytes on): its count,
  // then 16 bytes on the entries.
  near_warps_ = int(std::min<int64_t>(kNearMaxWarps, (nt_ + ncell * kNearT - 1) / (ncell * kNearT)));
  near_chunk_ = near_warps_ * kNearT * kNearRounds;
  const size_t cursors = (size_t(ncell + 1) * sizeof(int32_t) + 15) / 16 * 16;
  MF_TRY(cursor_.reserve_slack(cursors + 16 + sizeof(int2) * size_t(1 + nt_ / near_chunk_)));
  extra_ = cursor_.as<char>() + cursors;
  int32_t* extra_n = reinterpret_cast<int32_t*>(extra_);
  int2* extra = reinterpret_cast<int2*>(extra_ + 16);
  MF_TRY(perm_tmp_.reserve_slack(size_t(n + ncell + 2) * sizeof(int32_t)));
  MF_TRY(perm_.reserve_slack(size_t(n + ncell + 2) * sizeof(int32_t)));
  MF_CUDA_TRY(cudaMemsetAsync(cnt, 0, size_t(ncell) * sizeof(int32_t), st));
  k_fmm_count<<<blocks_for(n), 256, 0, st>>>(pos4, n, leaf, cell_of_.as<int32_t>(), cnt);
  k_fmm_scan<<<1, 1024, 0, st>>>(cnt, ncell, start_.as<int32_t>(), separate_ ? nullptr : extra_n);
  MF_CUDA_TRY(cudaMemcpyAsync(cursor_.ptr, start_.ptr, size_t(ncell) * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  k_fmm_scatter<<<blocks_for(n), 256, 0, st>>>(cell_of_.as<int32_t>(), n, cursor_.as<int32_t>(),
                                                perm_tmp_.as<int32_t>());
  k_fmm_sort<<<blocks_for(ncell * 32), 256, 0, st>>>(start_.as<int32_t>(), cnt, ncell, perm_tmp_.as<int32_t>(),
                                                      perm_.as<int32_t>(), near_chunk_, separate_ ? nullptr : extra,
                                                      extra_n);
  for (int l = L - 1; l >= 0; --l)
    k_fmm_occ_up<<<blocks_for(lv_[size_t(l)].nbox), 256, 0, st>>>(lv_[size_t(l + 1)], lv_[size_t(l)], occ);
  MF_CUDA_TRY(cudaGetLastError());
  // Separate targets: their own binning into the same leaf boxes (lists in
  // increasing index, padded like the sources), and their own occupancy.
  if (separate_) {
    MF_TRY(tocc_.reserve_slack(size_t(nbox_total) * sizeof(int32_t)));
    int32_t* tocc = tocc_.as<int32_t>();
    int32_t* tcnt = tocc + leaf.box_off;
    MF_TRY(tcell_of_.reserve(size_t(nt) * sizeof(int32_t)));
    MF_TRY(tstart_.reserve_slack(size_t(ncell + 1) * sizeof(int32_t)));
    MF_TRY(tcursor_.reserve_slack(size_t(ncell + 1) * sizeof(int32_t)));
    MF_TRY(tperm_tmp_.reserve_slack(size_t(nt + ncell + 2) * sizeof(int32_t)));
    MF_TRY(tperm_.reserve_slack(size_t(nt + ncell + 2) * sizeof(int32_t)));
    MF_CUDA_TRY(cudaMemsetAsync(tcnt, 0, size_t(ncell) * sizeof(int32_t), st));
    k_fmm_count<<<blocks_for(nt), 256, 0, st>>>(tpos4, nt, leaf, tcell_of_.as<int32_t>(), tcnt);
    k_fmm_scan<<<1, 1024, 0, st>>>(tcnt, ncell, tstart_.as<int32_t>(), extra_n);
    MF_CUDA_TRY(cudaMemcpyAsync(tcursor_.ptr, tstart_.ptr, size_t(ncell) * sizeof(int32_t), cudaMemcpyDeviceToDevice,
                                st));
    k_fmm_scatter<<<blocks_for(nt), 256, 0, st>>>(tcell_of_.as<int32_t>(), nt, tcursor_.as<int32_t>(),
                                                   tperm_tmp_.as<int32_t>());
    k_fmm_sort<<<blocks_for(ncell * 32), 256, 0, st>>>(tstart_.as<int32_t>(), tcnt, ncell, tperm_tmp_.as<int32_t>(),
                                                        tperm_.as<int32_t>(), near_chunk_, extra, extra_n);
    for (int l = L - 1; l >= 0; --l)
      k_fmm_occ_up<<<blocks_for(lv_[size_t(l)].nbox), 256, 0, st>>>(lv_[size_t(l + 1)], lv_[size_t(l)], tocc);
    MF_CUDA_TRY(cudaGetLastError());
  }
  // Slots: every box padded to an even count, so at most n + ncell; the
  // kernels read the exact count (start[ncell]) on the device.
  n_slots_ = n + ncell + 1;
  MF_TRY(pos2s_.reserve_slack(size_t(n_slots_ + 2) * sizeof(float4)));
  MF_TRY(mom2s_.reserve_slack(size_t(n_slots_ + 2) * sizeof(float4)));
  k_fmm_gather_pairs<<<blocks_for(n_slots_ / 2), 256, 0, st>>>(perm_.as<int32_t>(), pos4, start_.as<int32_t>() + ncell,
                                                                pos2s_.as<float4>(), 1, nullptr);
  MF_CUDA_TRY(cudaGetLastError());

  // Acceptance: box pairs of one level at centre offset d (box units) are far
  // when theta |d| > r1 + r2 (the box radii, FMMOptions.hpp:56-78) and the gap
  // |d| - (r1 + r2) exceeds the near radius 4h.  The offsets are whole numbers
  // and both tests grow with |d|, so a level's test is |d|^2 > m, m the largest
  // near |d|^2.  Lists, rows and the derivative table are a function of the
  // degree, the grid shape and the m's alone: particles that move a little keep
  // all of it.  (Tested afresh for every offset, with their lookup in a tree,
  // the lists took 2 ms of host time per tree and step: 4.2 of a 16.8 ms step
  // at 200,003 particles.)
  const double rnear = 4.0 * h * (1.0 + 1e-4);
  const double r12 = std::sqrt(3.0);
  std::vector<int64_t> m(size_t(L + 1), 0);
  for (int l = 1; l <= L; ++l) {
    const double s = double(lv_[size_t(l)].side);
    auto is_far = [&](int64_t d2) {
      const double r0 = std::sqrt(double(d2));
      return cfg.theta * r0 > r12 && (r0 - r12) * s > rnear;
    };
    // No two boxes are as far apart as kNoFar: beyond, nothing is far (and the
    // square of a radius at a tiny theta need not fit).
    constexpr double kNoFar = double(2 << kMaxLevel);
    const double t = std::max(r12 / cfg.theta, r12 + rnear / s);
    if (!(t < kNoFar)) {
      m[size_t(l)] = int64_t(kNoFar * kNoFar);
      continue;
    }
    int64_t d2 = int64_t(t * t);
    while (d2 > 0 && is_far(d2)) --d2;
    while (!is_far(d2 + 1)) ++d2;
    m[size_t(l)] = d2;
  }
  auto far = [&](int l, int dx, int dy, int dz) {
    return l > 0 && int64_t(dx) * dx + int64_t(dy) * dy + int64_t(dz) * dz > m[size_t(l)];
  };
  std::vector<int64_t> key{Q, L};
  for (int l = 0; l <= L; ++l) {
    const FmmLevel& v = lv_[size_t(l)];
    key.insert(key.end(), {v.nx, v.ny, v.nz, m[size_t(l)]});
  }
  if (key != lists_key_) {
    // Kernels of earlier products may still read the old tables, and uploads
    // the host copies.
    MF_CUDA_TRY(cudaStreamSynchronize(st));
    lists_key_.clear();
    MF_TRY(build_lists(L, m, far, st));
    lists_key_ = std::move(key);
  }

  // Coefficients and the M2L split per level.
  const int sms = device_sms(current_device());
  chunks_.assign(size_t(L + 1), 1);
  int64_t lpart = 1;
  for (int l = 2; l <= L; ++l) {
    const FmmLevel& v = lv_[size_t(l)];
    const int64_t per = ((int64_t((v.nx + 1) / 2) * ((v.ny + 1) / 2) * ((v.nz + 1) / 2)) + 31) / 32 * 32;
    int64_t ch = (int64_t(sms) * 1024 + 8 * per - 1) / (8 * per);
    int64_t maxcnt = 1;
    for (int cls = 0; cls < 8; ++cls) maxcnt = std::max(maxcnt, list_cnt_[size_t(8 * l + cls)]);
    ch = std::max<int64_t>(1, std::min<int64_t>({ch, 16, maxcnt}));
    chunks_[size_t(l)] = int32_t(ch);
    lpart = std::max(lpart, ch * nharm(Q) * v.nbox);
  }
  MF_TRY(mcoef_.reserve_slack(size_t(NC + nharm(Q)) * size_t(nbox_total) * sizeof(float)));
  hcoef_ = mcoef_.as<float>() + int64_t(NC) * nbox_total;
  MF_TRY(lcoef_.reserve_slack(size_t(NC) * size_t(nbox_total) * sizeof(float)));
  MF_TRY(lpart_.reserve_slack(size_t(lpart) * sizeof(float)));

  // Statistics, counted on the device and read back lazily (stats()).
  MF_TRY(stat_.reserve(5 * sizeof(unsigned long long)));
  MF_CUDA_TRY(cudaMemsetAsync(stat_.ptr, 0, 5 * sizeof(unsigned long long), st));
  const int32_t* tocc_all = separate_ ? tocc_.as<int32_t>() : occ;
  k_fmm_p2p_stats<<<blocks_for(ncell), 256, 0, st>>>(leaf, cnt, tocc_all + leaf.box_off, rows_.as<int4>(), n_rows_,
                                                      stat_.as<unsigned long long>());
  for (int l = 2; l <= L; ++l)
    k_fmm_m2l_stats<<<blocks_for(lv_[size_t(l)].nbox * 32), 256, 0, st>>>(
        lv_[size_t(l)], occ, tocc_all, lists_.as<int4>(), lofs_.as<int64_t>() + 8 * l,
        lofs_.as<int64_t>() + list_off_.size() + 8 * l, stat_.as<unsigned long long>());
  MF_CUDA_TRY(cudaGetLastError());
  if (!hstat_) MF_CUDA_TRY(cudaMallocHost(&hstat_, 5 * sizeof(unsigned long long)));
  if (!stat_ev_) MF_CUDA_TRY(cudaEventCreateWithFlags(&stat_ev_, cudaEventDisableTiming));
  MF_CUDA_TRY(cudaMemcpyAsync(hstat_, stat_.ptr, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
  MF_CUDA_TRY(cudaEventRecord(stat_ev_, st));
  stat_pending_ = true;
  stats_ = FmmStats{};
  stats_.levels = L + 1;
  stats_.leaf_level = L;
  stats_.degree = Q;
  stats_.leaf_boxes = ncell;
  stats_.near_rows = n_rows_;
  return MF_OK;
}

const FmmStats& Fmm::stats() {
  if (stat_pending_ && stat_ev_ && cudaEventSynchronize(stat_ev_) == cudaSuccess) {
    stats_.p2p_pairs = double(hstat_[0]);
    stats_.max_leaf = int32_t(hstat_[1]);
    stats_.m2l_per_product = double(hstat_[2]);
    stats_.occupied_leaves = int64_t(hstat_[3]);
    stats_.p2p_self_pairs = double(hstat_[4]);
    stat_pending_ = false;
  }
  return stats_;
}

Fmm::~Fmm() {
  if (hstat_) pinned_free(hstat_);
  if (stat_ev_) cudaEventDestroy(stat_ev_);
}

mf_status Fmm::product(int kind, const float4* pos4, const float4* smom, const AllPairsArgs<float>& a,
                       const SceneDesc<float>& sc, cudaStream_t st, const double* done, cudaEvent_t* marks,
                       bool sym_near) {
  if (kind < 0 || kind > 2) return fail(MF_ERR_INVALID_ARG, "fmm: unknown product kind");
  switch (degree_) {
    case 3: return product_q<3>(kind, pos4, smom, a, sc, st, done, marks, sym_near);
    case 4: return product_q<4>(kind, pos4, smom, a, sc, st, done, marks, sym_near);
    case 5: return product_q<5>(kind, pos4, smom, a, sc, st, done, marks, sym_near);
    case 6: return product_q<6>(kind, pos4, smom, a, sc, st, done, marks, sym_near);
    case 7: return product_q<7>(kind, pos4, smom, a, sc, st, done, marks, sym_near);
    case 8: return product_q<8>(kind, pos4, smom, a, sc, st, done, marks, sym_near);
    case 9:
      if (kind == 0) return fail(MF_ERR_INVALID_ARG, "fmm: order 10 is for the force products only");
      return product_q<9>(kind, pos4, smom, a, sc, st, done, marks, sym_near);
    default: return fail(MF_ERR_INVALID_ARG, "fmm: unsupported degree");
  }
}

namespace {
// The near field of a product: four targets per warp (k_fmm_near_warp), as many
// warps per CTA as a mean box has rounds, up to eight (steps of a cylinder of
// 200,003 particles, 16 per box: 2-4 warps 11.6-11.7 ms, 8 12.1; of a sphere of
// 330,000, 81 per box: 2 warps 28.6, 8 23.8).  A CTA takes four rounds of its warps, a
// fuller box goes over several: the mean counts empty boxes and says nothing of
// boxes that hold many targets (10,000 targets in one box of 150,000 sources: 39
// ms for the field where one warp walked them all, 7.1 by 128-target CTAs, 0.49
// now; on a line 9.6, 3.6, 0.82; spread evenly 0.88).
// The staged CTA of 128 targets per box (k_fmm_p2p) is kept for the field of a
// set on itself where there are many boxes that fill it.  Near fields, staged /
// warps: 12,800 boxes of 82 (1,048,576 particles) 54.4 / 55.7 ms for the step,
// 800,000 (62) 43.3 / 41.2, a sphere of 330,000 (4,074 of 81) 29.9 / 23.8;
// 4,096 boxes of 244 27.2 / 27.2, of 488 98.5 / 104.0, of 977 385 / 412, 512
// boxes of 977 54.0 / 40.4 ms.
template <int Q, int kKind>
void launch_near(unsigned boxes, int64_t nt, bool separate, int warps, cudaStream_t st, const P2PArgs& pp,
                 const AllPairsArgs<float>& a, const SceneDesc<float>& sc) {
  if constexpr (kKind == 0) {
    const int64_t b = boxes;
    if (!separate && ((b >= 8192 && nt > 64 * b && nt <= 128 * b) || (b >= 4096 && nt > 256 * b))) {
      k_fmm_p2p<Q, 0, false, 128, 256><<<boxes, 128, p2p_smem<256>(), st>>>(pp, a, sc);
      return;
    }
  }
  const unsigned ctas = boxes + unsigned(nt / pp.chunk);  // the extra runs are at most so many
  k_fmm_near_warp<Q, kKind><<<ctas, 32 * warps, NearWarp<Q>::smem(warps), st>>>(pp, a, sc);
}
}  // namespace

template <int Q>
mf_status Fmm::product_q(int kind, const float4* pos4, const float4* smom, const AllPairsArgs<float>& a,
                         const SceneDesc<float>& sc, cudaStream_t st, const double* done, cudaEvent_t* marks,
                         bool sym_near) {
  constexpr int NC = ncoef(Q) - 1;
  const int L = int(lv_.size()) - 1;
  const FmmLevel& leaf = lv_[size_t(L)];
  int32_t* occ = occ_.as<int32_t>();
  const int32_t* cnt = occ + leaf.box_off;
  const int32_t* tocc = separate_ ? tocc_.as<int32_t>() : occ;
  constexpr int NH = nharm(Q);
  float* M = mcoef_.as<float>();
  float* H = hcoef_;  // multipoles with z <= 1
  float* Lc = lcoef_.as<float>();
  int nl = 0;
  if (marks) MF_CUDA_TRY(cudaEventRecord(marks[0], st));
  k_fmm_gather_pairs<<<blocks_for(n_slots_ / 2), 256, 0, st>>>(perm_.as<int32_t>(), smom, start_.as<int32_t>() + leaf.nbox,
                                                                mom2s_.as<float4>(), 0, done);
  ++nl;
  const int sms = device_sms(current_device());
  k_fmm_p2m<Q><<<blocks_for(leaf.nbox, 1, int64_t(sms) * 16), 128, 0, st>>>(
      leaf, start_.as<int32_t>(), cnt, perm_.as<int32_t>(), pos4, smom, M + leaf.box_off * NC, done);
  ++nl;
  for (int l = L - 1; l >= 2; --l) {
    k_fmm_m2m<Q><<<blocks_for(int64_t(8 * NC) * lv_[size_t(l)].nbox, 256, int64_t(sms) * 32), 256, 0, st>>>(
        lv_[size_t(l + 1)], lv_[size_t(l)], occ, M, done);
    ++nl;
  }
  {
    FmmLevels lvs{};
    for (int l = 0; l <= L; ++l) lvs.lv[l] = lv_[size_t(l)];
    const dim3 grid{blocks_for(int64_t(NH) * leaf.nbox, 256, int64_t(sms) * 32), unsigned(L - 1)};
    k_fmm_reduce<Q><<<grid, 256, 0, st>>>(lvs, 2, M, H, done);
    ++nl;
  }
  for (int l = 2; l <= L; ++l) {
    const FmmLevel& v = lv_[size_t(l)];
    M2LArgs p{};
    p.lv = v;
    p.occ = occ;
    p.tocc = tocc;
    p.M = H + v.box_off * NH;
    p.Lp = lpart_.as<float>();
    p.list = lists_.as<int4>();
    p.dtab = dtab_.as<float4>();
    for (int cls = 0; cls < 8; ++cls) {
      p.list_off[cls] = list_off_[size_t(8 * l + cls)];
      p.list_cnt[cls] = int32_t(list_cnt_[size_t(8 * l + cls)]);
    }
    p.chunks = chunks_[size_t(l)];
    p.hx = (v.nx + 1) / 2;
    p.hy = (v.ny + 1) / 2;
    p.hz = (v.nz + 1) / 2;
    p.per_class = ((int64_t(p.hx) * p.hy * p.hz) + 31) / 32 * 32;
    p.done = done;
    const int64_t threads = int64_t(p.chunks) * 8 * p.per_class;
    // The products that need only the Hessian of the local expansion (the
    // Kelvin force, the force tensor) leave out the degree-1 locals: no degree
    // below 2 reaches it (L2L maps degree >= 2 only from degree >= 2).
    const unsigned g = unsigned((threads + 127) / 128);
    if (kind != 0) k_fmm_m2l<Q, 2><<<g, 128, 0, st>>>(p);
    else if constexpr (Q <= kMaxFieldDegree) k_fmm_m2l<Q, 1><<<g, 128, 0, st>>>(p);
    ++nl;
    k_fmm_l2l<Q><<<blocks_for(int64_t(NC) * v.nbox, 256, int64_t(sms) * 32), 256, 0, st>>>(
        v, lv_[size_t(l - 1)], l > 2 ? 1 : 0, tocc, lpart_.as<float>(), p.chunks, Lc, done, kind != 0 ? 3 : 0);
    ++nl;
  }
  P2PArgs pp{};
  pp.lv = leaf;
  pp.start = start_.as<int32_t>();
  pp.cnt = cnt;
  pp.perm = perm_.as<int32_t>();
  pp.tstart = separate_ ? tstart_.as<int32_t>() : pp.start;
  pp.tcnt = tocc + leaf.box_off;
  pp.tperm = separate_ ? tperm_.as<int32_t>() : pp.perm;
  pp.pos2s = pos2s_.as<float4>();
  pp.mom2s = mom2s_.as<float4>();
  pp.L = Lc + leaf.box_off * NC;
  pp.rows = rows_.as<int4>();
  pp.n_rows = n_rows_;
  pp.done = done;
  pp.n_boxes = int32_t(leaf.nbox);
  pp.chunk = near_chunk_;
  pp.extra_n = reinterpret_cast<const int32_t*>(extra_);
  pp.extra = reinterpret_cast<const int2*>(extra_ + 16);
  const bool sym = kind == 1 && sym_near && !separate_;
  if (sym) {
    MF_TRY(npart_.reserve_grow(size_t(1 + n_off_) * 3 * size_t(n_slots_) * sizeof(float)));
    pp.hrows = hrows_.as<int4>();
    pp.n_hrows = n_hrows_;
    pp.part = npart_.as<float>();
    pp.n_slots = n_slots_;
  }
  if (leaf.nbox > int64_t(0x7fffffff)) return fail(MF_ERR_INVALID_ARG, "fmm: too many leaf boxes");
  if (marks) {
    MF_CUDA_TRY(cudaEventRecord(marks[1], st));
    MF_CUDA_TRY(cudaEventRecord(marks[2], st));
  }
  if (sym) {
    NearSymArgs ns{};
    ns.lv = leaf;
    ns.start = pp.start;
    ns.cnt = cnt;
    ns.perm = pp.perm;
    ns.pos2s = pp.pos2s;
    ns.mom2s = pp.mom2s;
    ns.hrows = pp.hrows;
    ns.n_hrows = n_hrows_;
    ns.part = npart_.as<float>();
    ns.n_slots = n_slots_;
    ns.done = done;
    k_fmm_near_sym<<<unsigned((leaf.nbox + kNearSymWarps - 1) / kNearSymWarps), 32 * kNearSymWarps, 0, st>>>(ns, a, sc);
    ++nl;
    k_fmm_p2p<Q, 1, true, 128, 256><<<unsigned(leaf.nbox), 128, p2p_smem<256>(), st>>>(pp, a, sc);
  } else if (kind == 1)
    launch_near<Q, 1>(unsigned(leaf.nbox), nt_, separate_, near_warps_, st, pp, a, sc);
  else if (kind == 2)
    launch_near<Q, 2>(unsigned(leaf.nbox), nt_, separate_, near_warps_, st, pp, a, sc);
  else
    if constexpr (Q <= kMaxFieldDegree) launch_near<Q, 0>(unsigned(leaf.nbox), nt_, separate_, near_warps_, st, pp, a, sc);
  ++nl;
  if (marks) MF_CUDA_TRY(cudaEventRecord(marks[3], st));
  launches_ = nl;
  MF_CUDA_TRY(cudaGetLastError());
  return MF_OK;
}

}  // namespace mfgb

// ===========================================================================
// C ABI: an FMM matrix over a source set and a target set
// ===========================================================================
struct mf_fmm {
  int device = 0;
  cudaStream_t st = nullptr;
  mfgb::Fmm fmm;
  // The Hessian product's lists at the force aperture, built on its first
  // call when that aperture is smaller than the field's.
  mfgb::Fmm fmmh;
  bool fmmh_built = false;
  mfgb::FmmConfig cfg;
  double h = 0.0, bbox[6] = {0, 0, 0, 0, 0, 0};
  mfgb::CellList cells;  // over the sources: the near-field correction
  mfgb::Scratch scr;
  mfgb::DevBuf spos, smom, tpos, corr, out4, out9, staging;
  int64_t ns = 0, nt = 0;
  bool same = true;
  mfgb::SceneDesc<float> sc{};
  ~mf_fmm() {
    if (st) {
      cudaStreamSynchronize(st);
      cudaStreamDestroy(st);
    }
  }
};

namespace mfgb {
namespace {
__global__ void k_aos_to_f4(const float* __restrict__ src, int64_t n, float4* __restrict__ dst,
                            int32_t* __restrict__ bad) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const float x = src[3 * i], y = src[3 * i + 1], z = src[3 * i + 2];
    if (!isfinite(x) || !isfinite(y) || !isfinite(z)) atomicExch(bad, 1);
    dst[i] = make_float4(x, y, z, 0.f);
  }
}
// 9 SoA arrays (k = column * 3 + row) -> [n][9] in the same order per target.
__global__ void k_soa9_to_aos(const float* __restrict__ src, int64_t n, float* __restrict__ dst) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
#pragma unroll
    for (int k = 0; k < 9; ++k) dst[9 * i + k] = src[int64_t(k) * n + i];
}
__global__ void k_f4_to_aos(const float4* __restrict__ src, int64_t n, float* __restrict__ dst) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const float4 v = src[i];
    dst[3 * i] = v.x;
    dst[3 * i + 1] = v.y;
    dst[3 * i + 2] = v.z;
  }
}

// Host AoS float[n][3] -> device float4 records (through `staging`); checks finiteness.
mf_status upload_f4(mf_fmm& f, const float* host, int64_t n, DevBuf& dst) {
  MF_TRY(f.staging.reserve(size_t(3 * n) * sizeof(float) + 16));
  MF_TRY(dst.reserve(size_t(n + 2) * sizeof(float4), false, true));
  int32_t* bad = reinterpret_cast<int32_t*>(f.staging.as<char>() + size_t(3 * n) * sizeof(float));
  MF_CUDA_TRY(cudaMemsetAsync(bad, 0, sizeof(int32_t), f.st));
  MF_CUDA_TRY(cudaMemcpyAsync(f.staging.ptr, host, size_t(3 * n) * sizeof(float), cudaMemcpyHostToDevice, f.st));
  k_aos_to_f4<<<blocks_for(n), 256, 0, f.st>>>(f.staging.as<float>(), n, dst.as<float4>(), bad);
  MF_CUDA_TRY(cudaGetLastError());
  int32_t hb = 0;
  MF_CUDA_TRY(cudaMemcpyAsync(&hb, bad, sizeof(int32_t), cudaMemcpyDeviceToHost, f.st));
  MF_CUDA_TRY(cudaStreamSynchronize(f.st));
  if (hb) return fail(MF_ERR_INVALID_ARG, "non-finite input value");
  return MF_OK;
}

template <class F>
mf_status fguard(mf_fmm* f, F&& fn) {
  if (!f) return fail(MF_ERR_INVALID_ARG, "NULL fmm handle");
  try {
    cudaError_t e = cudaSetDevice(f->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    return fn(*f);
  } catch (const std::bad_alloc&) {
    return fail(MF_ERR_OOM, "host allocation failed");
  } catch (...) {
    return fail(MF_ERR_CUDA, "unexpected exception");
  }
}
}  // namespace
}  // namespace mfgb

using namespace mfgb;

extern "C" {

mf_status mf_fmm_create(const float* sources, int64_t ns, const float* targets, int64_t nt, float h, int32_t order,
                        double theta, int32_t leaf_min, int32_t device, mf_fmm** out) {
  if (!out || !sources || ns <= 0) return fail(MF_ERR_INVALID_ARG, "fmm: no sources");
  *out = nullptr;
  if (targets && nt <= 0) return fail(MF_ERR_INVALID_ARG, "fmm: no targets");
  if (!(h > 0.f) || !std::isfinite(h)) return fail(MF_ERR_INVALID_ARG, "fmm: h must be finite and > 0");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(MF_ERR_UNSUPPORTED, "no CUDA device available");
  if (device < 0 || device >= ndev) return fail(MF_ERR_INVALID_ARG, "bad device ordinal");
  try {
    MF_CUDA_TRY(cudaSetDevice(device));
    std::unique_ptr<mf_fmm> f(new mf_fmm);
    f->device = device;
    MF_CUDA_TRY(cudaStreamCreateWithFlags(&f->st, cudaStreamNonBlocking));
    f->ns = ns;
    f->same = targets == nullptr;
    f->nt = f->same ? ns : nt;
    MF_TRY(upload_f4(*f, sources, ns, f->spos));
    if (!f->same) MF_TRY(upload_f4(*f, targets, nt, f->tpos));
    MF_TRY(f->cells.build(f->spos.as<float4>(), {CellSceneSpec{0, ns, double(h)}}, f->st));
    double bbox[6];
    for (int k = 0; k < 6; ++k) bbox[k] = f->cells.bbox(0)[k];
    if (!f->same)
      for (int64_t i = 0; i < nt; ++i)
        for (int k = 0; k < 3; ++k) {
          bbox[k] = std::min(bbox[k], double(targets[3 * i + k]));
          bbox[3 + k] = std::max(bbox[3 + k], double(targets[3 * i + k]));
        }
    FmmConfig& cfg = f->cfg;
    cfg.order = order;
    cfg.theta = theta;
    cfg.leaf_min = leaf_min;
    f->h = double(h);
    for (int k = 0; k < 6; ++k) f->bbox[k] = bbox[k];
    MF_TRY(f->fmm.build(f->spos.as<float4>(), ns, f->same ? nullptr : f->tpos.as<float4>(), f->nt, double(h), bbox,
                        cfg, f->st));
    MF_TRY(f->corr.reserve(size_t(f->nt + 2) * sizeof(float4), false, true));
    MF_TRY(f->out4.reserve(size_t(f->nt + 2) * sizeof(float4), false, true));
    MF_TRY(f->scr.ensure(0, 0));
    f->sc.pc = make_pair_consts<float>(double(h));
    f->sc.scale = 1.f;
    MF_CUDA_TRY(cudaStreamSynchronize(f->st));
    *out = f.release();
    return MF_OK;
  } catch (const std::bad_alloc&) {
    return fail(MF_ERR_OOM, "host allocation failed");
  }
}

mf_status mf_fmm_destroy(mf_fmm* f) {
  if (!f) return MF_OK;
  cudaSetDevice(f->device);
  delete f;
  return MF_OK;
}

mf_status mf_fmm_field(mf_fmm* f, const float* charges, float* results) {
  return fguard(f, [&](mf_fmm& x) {
    if (!charges || !results) return fail(MF_ERR_INVALID_ARG, "NULL argument");
    MF_TRY(upload_f4(x, charges, x.ns, x.smom));
    const float4* tp = x.same ? x.spos.as<float4>() : x.tpos.as<float4>();
    if (x.same)
      MF_TRY(x.cells.field_correction(x.spos.as<float4>(), x.smom.as<float4>(), x.corr.as<float4>(), x.st));
    else
      MF_TRY(x.cells.field_correction_at(tp, x.nt, x.spos.as<float4>(), x.smom.as<float4>(), x.corr.as<float4>(),
                                         x.st));
    AllPairsArgs<float> a{};
    a.tpos = tp;
    a.corr4 = x.corr.as<float4>();
    a.out4 = x.out4.as<float4>();
    a.err = x.scr.err.as<int32_t>();
    MF_TRY(x.fmm.product(0, x.spos.as<float4>(), x.smom.as<float4>(), a, x.sc, x.st, nullptr));
    MF_TRY(x.staging.reserve(size_t(3 * x.nt) * sizeof(float) + 16));
    k_f4_to_aos<<<blocks_for(x.nt), 256, 0, x.st>>>(x.out4.as<float4>(), x.nt, x.staging.as<float>());
    MF_CUDA_TRY(cudaGetLastError());
    MF_CUDA_TRY(cudaMemcpyAsync(results, x.staging.ptr, size_t(3 * x.nt) * sizeof(float), cudaMemcpyDeviceToHost,
                                x.st));
    MF_CUDA_TRY(cudaStreamSynchronize(x.st));
    return x.scr.check(x.st);
  });
}

mf_status mf_fmm_hessian(mf_fmm* f, const float* charges, float* results9) {
  return fguard(f, [&](mf_fmm& x) {
    if (!charges || !results9) return fail(MF_ERR_INVALID_ARG, "NULL argument");
    MF_TRY(upload_f4(x, charges, x.ns, x.smom));
    const float4* tp = x.same ? x.spos.as<float4>() : x.tpos.as<float4>();
    MF_TRY(x.corr.reserve(size_t(2 * x.nt + 2) * sizeof(float4), false, true));
    MF_TRY(x.cells.tensor_correction_at(tp, x.nt, x.spos.as<float4>(), x.smom.as<float4>(), x.corr.as<float4>(),
                                        x.st));
    MF_TRY(x.out9.reserve(size_t(9 * x.nt) * sizeof(float)));
    AllPairsArgs<float> a{};
    a.tpos = tp;
    a.corr4 = x.corr.as<float4>();
    for (int k = 0; k < 9; ++k) a.out[k] = x.out9.as<float>() + size_t(k) * size_t(x.nt);
    a.err = x.scr.err.as<int32_t>();
    Fmm* fh = &x.fmm;
    if (x.cfg.force_tree()) {
      if (!x.fmmh_built) {
        FmmConfig ct = x.cfg;
        ct.theta = x.cfg.force_theta();
        ct.order = x.cfg.force_order();
        MF_TRY(x.fmmh.build(x.spos.as<float4>(), x.ns, x.same ? nullptr : x.tpos.as<float4>(), x.nt, x.h, x.bbox, ct,
                            x.st));
        x.fmmh_built = true;
      }
      fh = &x.fmmh;
    }
    MF_TRY(fh->product(2, x.spos.as<float4>(), x.smom.as<float4>(), a, x.sc, x.st, nullptr));
    MF_TRY(x.staging.reserve(size_t(9 * x.nt) * sizeof(float) + 16));
    k_soa9_to_aos<<<blocks_for(x.nt), 256, 0, x.st>>>(x.out9.as<float>(), x.nt, x.staging.as<float>());
    MF_CUDA_TRY(cudaGetLastError());
    MF_CUDA_TRY(cudaMemcpyAsync(results9, x.staging.ptr, size_t(9 * x.nt) * sizeof(float), cudaMemcpyDeviceToHost,
                                x.st));
    MF_CUDA_TRY(cudaStreamSynchronize(x.st));
    return x.scr.check(x.st);
  });
}

mf_status mf_fmm_get_stats(mf_fmm* f, mf_fmm_stats* out) {
  return fguard(f, [&](mf_fmm& x) {
    if (!out) return fail(MF_ERR_INVALID_ARG, "NULL");
    *out = mf_fmm_stats{};
    const FmmStats& s = x.fmm.stats();
    out->active = 1;
    out->levels = s.levels;
    out->leaf_level = s.leaf_level;
    out->degree = s.degree;
    out->leaf_boxes = s.leaf_boxes;
    out->occupied_leaves = s.occupied_leaves;
    out->max_leaf = s.max_leaf;
    out->near_rows = s.near_rows;
    out->p2p_pairs = s.p2p_pairs;
    out->m2l_per_product = s.m2l_per_product;
    out->launches_per_product = x.fmm.launches_per_product();
    out->force_active = 1;
    out->theta = x.cfg.theta;
    out->force_theta = x.cfg.force_theta();
    if (x.fmmh_built) {
      out->force_p2p_pairs = x.fmmh.stats().p2p_pairs;
      out->force_m2l_per_product = x.fmmh.stats().m2l_per_product;
    } else if (!x.cfg.force_tree()) {
      out->force_p2p_pairs = s.p2p_pairs;
      out->force_m2l_per_product = s.m2l_per_product;
    }
    return MF_OK;
  });
}

}  // extern "C"
