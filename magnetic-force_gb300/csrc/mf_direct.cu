// mf_direct.cu -- direct all-pairs evaluation of the reference's pair kernels
// on caller-owned device buffers (the fmmtl::direct replacement of mf.h).
//
// The caller's AoS [n][3] arrays are packed into 16-byte records so source
// tiles can be staged by bulk copies; that packing space, the plan table and
// the kernel scratch live in one context per device, created on first use
// and kept until mf_release_scratch() or process exit.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "mf_internal.h"

namespace mfgb {
namespace {

// AoS [n][3] -> records.  reset (optional) is cleared; seen (optional) gets bit
// k if a value of axis k is not NaN and bit 3 if any value is infinite.
__global__ void k_pack_aos(int64_t n, const float* __restrict__ src, float4* __restrict__ dst,
                           int32_t* __restrict__ reset = nullptr, int32_t* __restrict__ seen = nullptr) {
  if (reset && blockIdx.x == 0 && threadIdx.x == 0) *reset = 0;
  int32_t f = 0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const float x = src[3 * i], y = src[3 * i + 1], z = src[3 * i + 2];
    dst[i] = make_float4(x, y, z, 0.f);
    f |= (isnan(x) ? 0 : 1) | (isnan(y) ? 0 : 2) | (isnan(z) ? 0 : 4) | (isinf(x) || isinf(y) || isinf(z) ? 8 : 0);
  }
  if (seen) {
    __shared__ int32_t s_f;
    if (threadIdx.x == 0) s_f = 0;
    __syncthreads();
    f = __reduce_or_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && f) atomicOr(&s_f, f);
    __syncthreads();
    if (threadIdx.x == 0 && s_f) atomicOr(seen, s_f);
  }
}

// SoA (k arrays of n) -> AoS [n][k].  seen (optional, k_pack_aos over the
// sources): without a finite bounding box nothing is written and err is set.
__global__ void k_soa_to_aos_k(int64_t n, int k, const float* __restrict__ soa, float* __restrict__ aos,
                               const int32_t* __restrict__ seen = nullptr, int32_t* __restrict__ err = nullptr) {
  if (seen && *seen != 7) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(err, 0, MF_DEVERR_NONFINITE);
    return;
  }
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    for (int c = 0; c < k; ++c) aos[i * k + c] = soa[int64_t(c) * n + i];
}

// AoS [n][k] -> SoA
__global__ void k_aos_to_soa_k(int64_t n, int k, const float* __restrict__ aos, float* __restrict__ soa) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    for (int c = 0; c < k; ++c) soa[int64_t(c) * n + i] = aos[i * k + c];
}

unsigned grid_for(int64_t n) {
  int64_t g = (n + 255) / 256;
  if (g > 4096) g = 4096;
  if (g < 1) g = 1;
  return unsigned(g);
}

constexpr int kBodies = 6;

// Whether a call's packed kernels can beat the exact-branch ones.  They cost a
// cell list over the sources (ten launches, a host round trip, then with the
// count) and the near-field correction, a warp per target; they save about half
// of every pair of the padded target blocks.  Whole calls, exact / packed us:
//   field, 64 x 200,000 612 / 653, 64 x 1,000,000 1,165 / 976, 1,000 x 200,000 562 /
//   531, 4,000 x 40,000 355 / 346, 40,000 x 4,000 312 / 300-516, 200,000 x 1,000 399
//   / 562; of one set (the correction by cells) 9,500 249 / 274, 12,000 323 / 305.
//   force of one set, 9,500 347 / 324-407, 12,000 471 / 366-518 (few to many near
//   pairs).
//   tensor, 256 x 1,000,000 898 / 1,208, 1,000 x 200,000 644 / 624, 1,000 x
//   1,000,000 2,033 / 1,480, 2,000 x 40,000 433 / 442, 11,000 x 10,000 424 /
//   418, 40,000 x 10,000 1,331 / 976, 1,000,000 x 1,000 3,119 / 5,115.
double padded_pairs(Body body, int64_t nt, int64_t ns) {
  const int64_t block = body == Body::Tensor ? 128 : 512;
  return double((nt + block - 1) / block * block) * double(ns);
}
bool packed_pays(Body body, bool one_set, int64_t nt, int64_t ns) {
  const double t = double(nt), s = double(ns), pairs = padded_pairs(body, nt, ns);
  if (body == Body::Tensor) return pairs >= 9e7 + 360.0 * s + 2450.0 * t;
  if (one_set) return t * s >= 1.25e8;
  return pairs >= 1.4e8 + 1000.0 * t;
}

// And whether they do, given the sources' bounding box: where many pairs are
// near, the correction costs more than the packed kernel saves.  The part of the
// sources expected within the near radius (2h field, 4h force and tensor) at
// which both take the same time, in uniform cubes:
//   field, one set: 0.04 at 12,000, 0.07 at 20,000, 0.09 at 40,000; separate: 0.03
//   at 40,000 x 4,000 and 12,000 x 12,000, 0.12 at 20,000 x 100,000;
//   force: 0.14 at 9,500, 0.24 at 12,000, 0.26 at 20,000, 0.39 at 40,000;
//   tensor: 0.2 at 12,000, 0.4 at 20,000, 0.52 at 40,000, 0.27 at 40,000 x 4,000.
// Beyond it packed fields lose most: 12,000 of one set at 0.52, exact / packed
// 330 / 1,695 us, force 474 / 685, tensor 487 / 647.
bool few_near(Body body, bool one_set, int64_t nt, int64_t ns, double h, const double* bbox) {
  const double reach = body == Body::Field ? 2.0 * h : 4.0 * h, pairs = padded_pairs(body, nt, ns);
  double near = kPi / 6.0;
  for (int k = 0; k < 3; ++k) near *= std::min(1.0, 2.0 * reach / std::max(bbox[3 + k] - bbox[k], 1e-300));
  if (body == Body::Tensor) return near <= 0.55 - 5e7 / pairs;
  if (body == Body::Force) return near <= 0.38 - 2e7 / pairs;
  return near <= (one_set ? 0.105 - 9e6 / pairs : std::max(0.02, 0.135 - 1.6e7 / pairs));
}

struct DirectCtx {
  std::mutex mu;
  DevBuf t4, s4, m4, tm4, soa, aux, s2, m2, corr, seen;
  Scratch scr;
  CellList cells;
  Plan<float> plan[kBodies];
  bool plan_ok[kBodies] = {};
  int64_t plan_nt[kBodies] = {}, plan_ns[kBodies] = {};
  double plan_h[kBodies] = {};
  void release() {
    for (DevBuf* b : {&t4, &s4, &m4, &tm4, &soa, &aux, &s2, &m2, &corr, &seen}) b->release();
    scr.partials.release();
    scr.counters.release();
    scr.err.release();
    cells = CellList();
    for (int b = 0; b < kBodies; ++b) {
      plan[b].d_scenes.release();
      plan_ok[b] = false;
    }
  }
};

DirectCtx g_ctx[64];

mf_status get_plan(DirectCtx& c, Body body, int64_t nt, int64_t ns, double h, int shape, const Plan<float>** out) {
  const int b = int(body);
  if (!c.plan_ok[b] || c.plan_nt[b] != nt || c.plan_ns[b] != ns || c.plan_h[b] != h || c.plan[b].shape != shape) {
    SceneSpec s;
    s.t_off = 0;
    s.nt = nt;
    s.s_off = 0;
    s.ns = ns;
    s.h = h;
    s.scale = 1.0;
    MF_TRY(build_plan<float>(body, {s}, c.plan[b], shape));
    c.plan_ok[b] = true;
    c.plan_nt[b] = nt;
    c.plan_ns[b] = ns;
    c.plan_h[b] = h;
  }
  *out = &c.plan[b];
  return MF_OK;
}

mf_status check_common(const void* a, int64_t na, const void* b, const void* c, int64_t nb, float h) {
  if (na < 0 || nb < 0) return fail(MF_ERR_INVALID_ARG, "negative count");
  if (na > 0 && !a) return fail(MF_ERR_INVALID_ARG, "NULL target array");
  if (nb > 0 && (!b || !c)) return fail(MF_ERR_INVALID_ARG, "NULL source array");
  if (!(h > 0.f) || !std::isfinite(h)) return fail(MF_ERR_INVALID_ARG, "h must be finite and > 0");
  return MF_OK;
}

mf_status direct_impl(Body body, const float* targets, int64_t nt, const float* sources, const float* charges,
                      int64_t ns, float h, const float* rext9, int naive, float* results, cudaStream_t st) {
  const int dev = current_device();
  if (dev < 0 || dev >= 64) return fail(MF_ERR_UNSUPPORTED, "device ordinal out of range");
  DirectCtx& c = g_ctx[dev];
  std::lock_guard<std::mutex> lk(c.mu);
  const int kOut = body == Body::Tensor ? 9 : 3;
  if (nt == 0) return MF_OK;
  if (ns == 0) {
    MF_CUDA_TRY(cudaMemsetAsync(results, 0, size_t(nt) * kOut * sizeof(float), st));
    MF_CUDA_TRY(cudaStreamSynchronize(st));
    return MF_OK;
  }
  MF_TRY(c.t4.reserve(size_t(nt) * sizeof(float4)));
  MF_TRY(c.s4.reserve(size_t(ns) * sizeof(float4)));
  MF_TRY(c.m4.reserve(size_t(ns) * sizeof(float4)));
  MF_TRY(c.soa.reserve(size_t(nt) * kOut * sizeof(float)));
  MF_TRY(c.seen.reserve(sizeof(int32_t)));
  // The cell list of the packed path refuses sources without a finite bounding
  // box; the field and the force refuse them on the exact path as well.
  const bool one_set = body == Body::Force || (targets == sources && nt == ns);
  const bool large = packed_pays(body, one_set, nt, ns);
  int32_t* seen = !large && body != Body::Tensor ? c.seen.as<int32_t>() : nullptr;
  k_pack_aos<<<grid_for(nt), 256, 0, st>>>(nt, targets, c.t4.as<float4>(), seen);
  k_pack_aos<<<grid_for(ns), 256, 0, st>>>(ns, sources, c.s4.as<float4>(), nullptr, seen);
  k_pack_aos<<<grid_for(ns), 256, 0, st>>>(ns, charges, c.m4.as<float4>());
  MF_CUDA_TRY(cudaGetLastError());
  LaunchIO<float> io;
  io.tpos = c.t4.as<float4>();
  io.spos = c.s4.as<float4>();
  io.smom = c.m4.as<float4>();
  // Large calls go through the packed two-source kernels: sources in pair
  // layout, a cell list over the sources, and the near-field correction.  Dense
  // ones go to the exact kernel, and so does a tensor whose sources no cell list
  // can be made of (positions that are not finite: that kernel takes any).
  Body launch_body = body;
  bool packed = large;
  if (packed) {
    auto wanted = [&](const double* bbox) { return packed = few_near(body, one_set, nt, ns, double(h), bbox); };
    const mf_status built = c.cells.build(c.s4.as<float4>(), {CellSceneSpec{0, ns, double(h)}}, st, 0.0, wanted);
    if (built != MF_OK) {
      if (body != Body::Tensor) return built;
      cudaGetLastError();
      packed = false;
    }
  }
  if (packed) {
    const size_t pair_bytes = size_t(ns + 1) * sizeof(float4);
    MF_TRY(c.s2.reserve(pair_bytes));
    MF_TRY(c.m2.reserve(pair_bytes));
    MF_TRY(c.corr.reserve(size_t(nt) * (body == Body::Tensor ? 2 : 1) * sizeof(float4)));
    to_pairs(c.s4.as<float4>(), c.s2.as<float4>(), ns, st);
    to_pairs(c.m4.as<float4>(), c.m2.as<float4>(), ns, st);
    MF_CUDA_TRY(cudaGetLastError());
    if (body == Body::Field) {
      if (one_set)
        MF_TRY(c.cells.field_correction(c.s4.as<float4>(), c.m4.as<float4>(), c.corr.as<float4>(), st));
      else
        MF_TRY(c.cells.field_correction_at(c.t4.as<float4>(), nt, c.s4.as<float4>(), c.m4.as<float4>(),
                                           c.corr.as<float4>(), st));
      launch_body = Body::FieldF2;
    } else if (body == Body::Tensor) {
      MF_TRY(c.cells.tensor_correction_at(c.t4.as<float4>(), nt, c.s4.as<float4>(), c.m4.as<float4>(),
                                          c.corr.as<float4>(), st));
      launch_body = Body::TensorF2;
    } else {
      MF_TRY(c.cells.force_correction(c.s4.as<float4>(), c.m4.as<float4>(), c.corr.as<float4>(), st));
      launch_body = Body::ForceF2;
    }
    io.spos = c.s2.as<float4>();
    io.smom = c.m2.as<float4>();
    io.corr4 = c.corr.as<float4>();
  }
  // One particle set (the force always; the field when the caller passes
  // the sources as the targets): each unordered pair once for both
  // particles from kSymDirectMin particles on (no tuning on this path: a
  // call can be seconds long), per MF_PAIR_SYMMETRIC.
  int shape = 0;
  if ((launch_body == Body::FieldF2 || launch_body == Body::ForceF2) && one_set) {
    const int mode = default_sym_mode();
    if (mode == 2 || (mode == 1 && nt >= kSymDirectMin)) shape = kShapeSym;
  }
  if (shape == kShapeSym) io.tpos = c.s4.as<float4>();  // the same records as the sources
  const Plan<float>* plan = nullptr;
  MF_TRY(get_plan(c, launch_body, nt, ns, h, shape, &plan));
  float* soa = c.soa.as<float>();
  for (int k = 0; k < kOut; ++k) io.out[k] = soa + int64_t(k) * nt;
  if (body == Body::Force) {
    io.tmom = c.m4.as<float4>();  // one particle set: target dipoles = sources' dipoles
    io.naive_quirks = naive;
    if (rext9) {
      MF_TRY(c.aux.reserve(size_t(nt) * 9 * sizeof(float)));
      k_aos_to_soa_k<<<grid_for(nt), 256, 0, st>>>(nt, 9, rext9, c.aux.as<float>());
      MF_CUDA_TRY(cudaGetLastError());
      for (int k = 0; k < 9; ++k) io.rext[k] = c.aux.as<float>() + int64_t(k) * nt;
    }
  }
  MF_TRY(run_plan<float>(*plan, io, c.scr, st));
  k_soa_to_aos_k<<<grid_for(nt), 256, 0, st>>>(nt, kOut, soa, results, seen, c.scr.err.as<int32_t>());
  MF_CUDA_TRY(cudaGetLastError());
  MF_TRY(c.scr.check(st));  // synchronises the stream
  return MF_OK;
}

}  // namespace
}  // namespace mfgb

using namespace mfgb;

extern "C" {

mf_status mf_direct_field(const float* targets, int64_t nt, const float* sources, const float* charges,
                          int64_t ns, float h, float* results, void* stream) {
  MF_TRY(check_common(targets, nt, sources, charges, ns, h));
  if (nt > 0 && !results) return fail(MF_ERR_INVALID_ARG, "NULL results");
  return direct_impl(Body::Field, targets, nt, sources, charges, ns, h, nullptr, 0, results,
                     static_cast<cudaStream_t>(stream));
}

mf_status mf_direct_force_tensor(const float* targets, int64_t nt, const float* sources, const float* charges,
                                 int64_t ns, float h, float* results9, void* stream) {
  MF_TRY(check_common(targets, nt, sources, charges, ns, h));
  if (nt > 0 && !results9) return fail(MF_ERR_INVALID_ARG, "NULL results");
  return direct_impl(Body::Tensor, targets, nt, sources, charges, ns, h, nullptr, 0, results9,
                     static_cast<cudaStream_t>(stream));
}

mf_status mf_direct_force(const float* pos, const float* mom, int64_t n, float h, const float* rext9,
                          int32_t naive_quirks, float* force, void* stream) {
  MF_TRY(check_common(pos, n, pos, mom, n, h));
  if (n > 0 && !force) return fail(MF_ERR_INVALID_ARG, "NULL force");
  return direct_impl(Body::Force, pos, n, pos, mom, n, h, rext9, naive_quirks ? 1 : 0, force,
                     static_cast<cudaStream_t>(stream));
}

mf_status mf_debug_stage_wait_limit(int64_t limit) {
  if (limit < 0) set_stage_wait_debug(0);
  else set_stage_wait_debug(uint32_t(std::min<int64_t>(limit, int64_t(kWaitLimit)) + 1));
  return MF_OK;
}

mf_status mf_release_scratch(void) {
  const int dev = current_device();
  if (dev < 0 || dev >= 64) return MF_OK;
  std::lock_guard<std::mutex> lk(g_ctx[dev].mu);
  g_ctx[dev].release();
  return MF_OK;
}

}  // extern "C"
