// mf_sym64.cu -- the FP64 field and force products evaluated once per
// unordered pair of particles.
//
// GB300 issues two FP64 operations per SM and clock, 1/64 of its FP32
// rate, so the FP64 instructions are all that counts here: loads, shuffles,
// integer work and selects ride along free.  The kernels below spend as few
// of them as the exact pair terms allow:
//   * both terms of a pair come from one evaluation (the field tensor is even
//     in d, the Kelvin force odd; see mf_sympair.cu);
//   * no square root and no division: a hardware seed y of r^-1 and e = 1 -
//     r^2 y^2, at most 2^-19.04 (measured over r^2 in [1, 4)), give r^-3 = y^3
//     (1 + 3/2 e + 15/8 e^2), r^-5 and r^-2 by their binomial series; the first
//     terms left out, 35/16 e^3, 105/16 e^3 and e^3, are at most 2^-56.0, 2^-54.4
//     and 2^-57.1;
//   * the near forms (SPH weights inside 2h, fitted curves inside 4h) are
//     polynomials in q with coefficients looked up per lane, evaluated where
//     any lane of the warp needs them, and selected;
//   * each lane holds one target and meets the 32 sources of a sub-tile in
//     rotation, the sources' sums travelling from lane to lane, so no sum
//     needs a reduction tree.
// Per unordered pair the field takes 36 FP64 operations, comparisons included
// (50 with a near lane in the warp), the force 47 (72).  At 4,096 uniformly random
// particles 79 % of the rotations have a near lane for the field, all for the
// force: 47 and 72 operations, 0.64 and 0.97 ms of the FP64 units at their nominal
// rate (a warp's operation 16 cycles of an SM).  Measured with the finish: field
// product 0.80 ms against 3.0 for the all-pairs kernel (~105 operations per
// ordered pair: both branches with their square roots and divisions), force
// 1.21 against 3.2.  The FP64 pipe is active 88 and 85 % of the kernels' time
// (conversions and selects of the tables are on it too): what is left is the
// operation count.
//
// Work layout: blocks of TB = 32 W particles (W warps per CTA), steps = block
// pairs (I, J), I <= J, split evenly over the resident CTAs; every step writes
// its sums for I and for J to part[][] once, and k_sym64_finish adds a
// particle's entries in a fixed order, as mf_sympair.cu does for FP32.
#include <cstring>
#include <mutex>

#include "mf_internal.h"

namespace mfgb {
namespace {

struct Sym64Args {
  AllPairsArgs<double> a;
  double* part;  // [nb][nb][3][TB]
  int32_t nb;
  int64_t n, off;  // particles, index of the first
};

// Step l -> (I, J), row I holding nb - I steps.
__device__ __forceinline__ void block_pair64(int64_t l, int nb, int& I, int& J) {
  const double b = 2.0 * nb + 1.0;
  int i = int((b - sqrt(b * b - 8.0 * double(l))) * 0.5);
  i = max(0, min(i, nb - 1));
  auto start = [&](int r) { return int64_t(r) * nb - int64_t(r) * (r - 1) / 2; };
  while (i > 0 && start(i) > l) --i;
  while (i < nb - 1 && start(i + 1) <= l) ++i;
  I = i;
  J = i + int(l - start(i));
}

// rsqrt.approx.ftz.f64: the hardware seed of 1 / sqrt(x) from x's upper word.
// Zero and subnormal x give 0, which drops the far terms of a coincident pair.
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return __double2hiint(x) < 0x00100000 ? 0.0 : y;
}

// Coefficients of the near field forms by piece (0: q < 1, 1: 1 <= q < 2,
// 2: far), from Dipole_B.kern:46-76 with the polynomials multiplied out:
//   alpha h^5 = kA q^-5 + a0 + a1 q + a2 / q,
//   beta h^3  = kA q^-3 + b0 + b1 q + b2 q^2 + b3 q^3.
__constant__ double c_field_near[3][8] = {
    {0.0, 0.8, -0.5, 0.0, -8.0 / 3.0, 0.0, 4.8, -2.5},
    {-1.0 / 15.0, -0.8, 1.0 / 6.0, 1.0, -16.0 / 3.0, 9.0, -4.8, 5.0 / 6.0},
    {1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0},
};
// The fitted force curves C1 and C2 - 3 C1 by piece (Dipole_hessian.kern:53-61),
// highest power first.
#define MF_ROW(a, b, c, d, e, f, g, h, i, j) \
  { a, b, c, d, e, f - 3.0 * (a), g - 3.0 * (b), h - 3.0 * (c), i - 3.0 * (d), j - 3.0 * (e) }
__constant__ double c_force_near[4][10] = {
    MF_ROW(9.97813616438174e-09, -2.97897856524718e-08, 2.38918644566813e-09, 4.53199938857366e-08,
           2.44617454752747e-11, 6.69550479838731e-08, -1.61753307173877e-07, 1.68213714992711e-08,
           1.34558143036838e-07, 1.10976027980100e-10),
    MF_ROW(-2.76473728643294e-09, 2.86975546540539e-08, -9.94582836806651e-08, 1.25129924573675e-07,
           -2.37010166723652e-08, -3.08460139955194e-08, 2.29192245602275e-07, -5.88399621128587e-07,
           5.61170054591844e-07, -1.14421132829680e-07),
    MF_ROW(-1.09679990621465e-09, 9.77055663264614e-09, -2.54781238661150e-08, 2.65020634884934e-09,
           5.00787562417835e-08, 3.50477408060213e-09, -5.25956271895141e-08, 2.78876509535747e-07,
           -6.24199554212217e-07, 4.91807818904985e-07),
    MF_ROW(3.79927162333632e-10, -6.26368404962679e-09, 3.94760528277489e-08, -1.13580541622200e-07,
           1.27491333574323e-07, 7.33485346367840e-10, -9.58855788627803e-09, 4.37085309763591e-08,
           -7.48004594092261e-08, 2.34161209605651e-08),
};
#undef MF_ROW

struct Vec3d {
  double x, y, z;
};

// Field: acc += (3 d (d.ms) r^-5 - ms r^-3) at the target, src the same with
// the target's dipole.  m3: the dipoles times 3.  tbl: c_field_near.
template <bool kSrc>
__device__ __forceinline__ void pair64_field(const Vec3d& t, const Vec3d& tm, const Vec3d& tm3, const Vec3d& s,
                                             const Vec3d& sm, const Vec3d& sm3, const PairConsts<double>& pc,
                                             const double* tbl, Vec3d& acc, Vec3d& src) {
  const double dx = t.x - s.x, dy = t.y - s.y, dz = t.z - s.z;
  const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
  const double y = rsqrt_seed(r2);
  const double y2 = y * y;
  const double e = fma(-r2, y2, 1.0);
  const double u = y * y2;
  double beta = fma(u * e, fma(1.875, e, 1.5), u);  // r^-3
  const double ir2 = fma(y2, fma(e, e, e), y2);     // r^-2
  double alpha = beta * ir2;                        // r^-5
  const bool near = r2 < pc.near2_field;
  if (__any_sync(0xffffffffu, near)) {
    const double ri = beta * r2;
    const double iq = ri * (1.0 / pc.inv_h);  // h / r
    const double q = (ri * pc.inv_h) * r2;
    const double* c = tbl + (near ? (q >= 1.0 ? 8 : 0) : 16);
    const double ih5 = pc.ih3 * (pc.inv_h * pc.inv_h);
    const double a = fma(c[3], iq, fma(c[2], q, c[1]));
    const double b = fma(fma(fma(c[7], q, c[6]), q, c[5]), q, c[4]);
    alpha = fma(c[0], alpha, a * ih5);
    beta = fma(c[0], beta, b * pc.ih3);
  }
  const double ts = fma(dz, sm3.z, fma(dy, sm3.y, dx * sm3.x)) * alpha;
  acc.x = fma(-sm.x, beta, fma(dx, ts, acc.x));
  acc.y = fma(-sm.y, beta, fma(dy, ts, acc.y));
  acc.z = fma(-sm.z, beta, fma(dz, ts, acc.z));
  if (kSrc) {
    const double tt = fma(dz, tm3.z, fma(dy, tm3.y, dx * tm3.x)) * alpha;
    src.x = fma(-tm.x, beta, fma(dx, tt, src.x));
    src.y = fma(-tm.y, beta, fma(dy, tt, src.y));
    src.z = fma(-tm.z, beta, fma(dz, tt, src.z));
  }
}

// Force (over K): acc += f_ij, src -= f_ij, f = d (P sm + Q ds dm) + m_t P ds + m_s P dm.
template <bool kSrc>
__device__ __forceinline__ void pair64_force(const Vec3d& t, const Vec3d& tm, const Vec3d& s, const Vec3d& sm,
                                             const PairConsts<double>& pc, const double* tbl, Vec3d& acc,
                                             Vec3d& src) {
  const double dx = t.x - s.x, dy = t.y - s.y, dz = t.z - s.z;
  const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
  const double y = rsqrt_seed(r2);
  const double y2 = y * y;
  const double e = fma(-r2, y2, 1.0);
  const double u5 = (y * y2) * y2;
  double P = fma(u5 * e, fma(4.375, e, 2.5), u5);  // r^-5
  double Q = P * (-5.0 * fma(y2, fma(e, e, e), y2));
  const bool near = !(r2 > pc.near2_force);
  if (__any_sync(0xffffffffu, near)) {
    const double ri = fma(y * e, fma(0.375, e, 0.5), y);
    // r rounded as a square root would be: the curves jump where their
    // pieces meet, and exact distances must stay on their side.
    double r = r2 * ri;
    r = fma(fma(-r, r, r2), 0.5 * ri, r);
    const double q = r * pc.inv_h;
    const double* c = tbl + 10 * (q <= 1.0 ? 0 : q <= 2.0 ? 1 : q <= 3.0 ? 2 : 3);
    const double c1 = fma(fma(fma(fma(c[0], q, c[1]), q, c[2]), q, c[3]), q, c[4]);
    const double c2 = fma(fma(fma(fma(c[5], q, c[6]), q, c[7]), q, c[8]), q, c[9]);
    const double k = pc.ih4_over_k * ri;
    const double kr = k * (ri * ri);
    if (near) {
      P = c1 * k;
      Q = c2 * kr;
    }
  }
  const double ds = fma(dz, sm.z, fma(dy, sm.y, dx * sm.x));
  const double dm = fma(dz, tm.z, fma(dy, tm.y, dx * tm.x));
  const double mm = fma(sm.z, tm.z, fma(sm.y, tm.y, sm.x * tm.x));
  const double u = P * ds, v = P * dm;
  const double w = fma(Q * ds, dm, P * mm);
  const double fx = fma(dx, w, fma(tm.x, u, sm.x * v));
  const double fy = fma(dy, w, fma(tm.y, u, sm.y * v));
  const double fz = fma(dz, w, fma(tm.z, u, sm.z * v));
  acc.x += fx;
  acc.y += fy;
  acc.z += fz;
  if (kSrc) {
    src.x -= fx;
    src.y -= fy;
    src.z -= fz;
  }
}

// The body's epilogue for particle i of the scene, v its sums.
template <bool kForce>
__device__ __forceinline__ void finish64(const Sym64Args& p, const SceneDesc<double>& sc, int64_t i, const double* v) {
  const int64_t gi = p.off + i;
  if constexpr (kForce) {
    const dbl4 m = p.a.tmom[gi];
    force_epilogue<double>(p.a, sc, gi, m.x, m.y, m.z, v);
  } else {
    FieldBody<double>::epilogue(p.a, sc, gi, FieldBody<double>::TData{}, v);
  }
}

template <bool kForce, int W>
__global__ void __launch_bounds__(32 * W) k_sym64(const Sym64Args p) {
  constexpr int TB = 32 * W;
  // A sub-tile of block J: 32 sources, and the warps' sums for them.
  __shared__ double s_p[3][32], s_m[3][32], s_m3[3][32];
  __shared__ double s_src[W][3][32];
  __shared__ double s_tbl[kForce ? 40 : 24];
  const AllPairsArgs<double>& a = p.a;
  const SceneDesc<double>& sc = a.scenes[0];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int64_t T = a.total_steps, G = gridDim.x;
  const int64_t k_begin = step_start(T, G, blockIdx.x), k_end = step_start(T, G, int64_t(blockIdx.x) + 1);
  if (k_begin >= k_end) return;
  if (a.done_flags && a.done_flags[int64_t(sc.flag_index) * a.done_stride] != 0.0) return;  // the solve has stopped
  for (int k = tid; k < (kForce ? 40 : 24); k += TB)
    s_tbl[k] = kForce ? c_force_near[k / 10][k % 10] : c_field_near[k / 8][k % 8];
  const PairConsts<double> pc = sc.pc;
  const double kk = kForce ? kForceK : kInv4Pi;
  auto load = [&](int64_t i, Vec3d& x, Vec3d& m) {  // a slot past the end: a zero dipole at particle 0
    const bool live = i < p.n;
    const dbl4 q = a.spos[p.off + (live ? i : 0)];
    x = Vec3d{q.x, q.y, q.z};
    m = Vec3d{0.0, 0.0, 0.0};
    if (live) {
      const dbl4 w = a.smom[p.off + i];
      m = Vec3d{w.x, w.y, w.z};
    }
  };
  Vec3d t, tm, tm3;
  int cur_I = -1;
  for (int64_t k = k_begin; k < k_end; ++k) {
    int I, J;
    block_pair64(k, p.nb, I, J);
    if (I != cur_I) {
      load(int64_t(I) * TB + tid, t, tm);
      tm3 = Vec3d{3.0 * tm.x, 3.0 * tm.y, 3.0 * tm.z};
      cur_I = I;
    }
    Vec3d acc{0.0, 0.0, 0.0};
    double* pj = p.part + (int64_t(J) * p.nb + I) * 3 * TB;
    for (int h = 0; h < W; ++h) {  // sub-tiles of block J
      __syncthreads();
      if (wid == 0) {
        Vec3d x, m;
        load(int64_t(J) * TB + h * 32 + lane, x, m);
        s_p[0][lane] = x.x;
        s_p[1][lane] = x.y;
        s_p[2][lane] = x.z;
        s_m[0][lane] = m.x;
        s_m[1][lane] = m.y;
        s_m[2][lane] = m.z;
        if (!kForce) {
          s_m3[0][lane] = 3.0 * m.x;
          s_m3[1][lane] = 3.0 * m.y;
          s_m3[2][lane] = 3.0 * m.z;
        }
      }
      __syncthreads();
      Vec3d src{0.0, 0.0, 0.0};  // the sums of source (lane + r) & 31 at rotation r
      const bool sym = I != J;   // block-uniform
      if (sym) {
#pragma unroll 1
        for (int r = 0; r < 32; ++r) {
          const int j = (lane + r) & 31;
          const Vec3d s{s_p[0][j], s_p[1][j], s_p[2][j]}, sm{s_m[0][j], s_m[1][j], s_m[2][j]};
          if constexpr (kForce) {
            pair64_force<true>(t, tm, s, sm, pc, s_tbl, acc, src);
          } else {
            const Vec3d sm3{s_m3[0][j], s_m3[1][j], s_m3[2][j]};
            pair64_field<true>(t, tm, tm3, s, sm, sm3, pc, s_tbl, acc, src);
          }
          const int from = (lane + 1) & 31;  // hand the sums to the lane that meets the source next
          src.x = __shfl_sync(0xffffffffu, src.x, from);
          src.y = __shfl_sync(0xffffffffu, src.y, from);
          src.z = __shfl_sync(0xffffffffu, src.z, from);
        }
      } else {
        // A block with itself hands nothing on: its live sources in turn (32
        // rotations take 80 us however few there are: forces of 1 and 10
        // particles 118 us against 43 and 66 by all pairs, 41 and 64 this way).
        const int64_t live = p.n - (int64_t(J) * TB + h * 32);
        const int n_src = live < 32 ? int(live < 0 ? 0 : live) : 32;
#pragma unroll 1
        for (int j = 0; j < n_src; ++j) {
          const Vec3d s{s_p[0][j], s_p[1][j], s_p[2][j]}, sm{s_m[0][j], s_m[1][j], s_m[2][j]};
          if constexpr (kForce) {
            pair64_force<false>(t, tm, s, sm, pc, s_tbl, acc, src);
          } else {
            const Vec3d sm3{s_m3[0][j], s_m3[1][j], s_m3[2][j]};
            pair64_field<false>(t, tm, tm3, s, sm, sm3, pc, s_tbl, acc, src);
          }
        }
      }
      if (sym) {  // back at source `lane`
        s_src[wid][0][lane] = src.x;
        s_src[wid][1][lane] = src.y;
        s_src[wid][2][lane] = src.z;
        __syncthreads();
        for (int q = tid; q < 96; q += TB) {
          const int c = q / 32, l = q % 32;
          double v = 0.0;
#pragma unroll
          for (int w = 0; w < W; ++w) v += s_src[w][c][l];
          pj[c * TB + h * 32 + l] = v * kk;
        }
      }
    }
    if (p.nb == 1) {  // one block: its sums are whole, no finish follows
      const double v[3] = {acc.x * kk, acc.y * kk, acc.z * kk};
      if (tid < p.n) finish64<kForce>(p, sc, tid, v);
      return;
    }
    double* pi = p.part + (int64_t(I) * p.nb + J) * 3 * TB;
    pi[tid] = acc.x * kk;
    pi[TB + tid] = acc.y * kk;
    pi[2 * TB + tid] = acc.z * kk;
  }
}

// Per particle: its nb partial sums (eight threads per particle, each every
// eighth entry in order, then added in order), and the body's epilogue.
template <bool kForce>
__global__ void __launch_bounds__(256) k_sym64_finish(const Sym64Args p, int tb) {
  __shared__ double s[8][3][32];
  const AllPairsArgs<double>& a = p.a;
  const SceneDesc<double>& sc = a.scenes[0];
  if (a.done_flags && a.done_flags[int64_t(sc.flag_index) * a.done_stride] != 0.0) return;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int64_t i = int64_t(blockIdx.x) * 32 + x;  // 32 particles of one block (tb is a multiple of 32)
  const int64_t K = i / tb;
  const int r = int(i % tb);
  const double* row = p.part + K * p.nb * 3 * tb + r;
  double v[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int X = y; X < p.nb; X += 8)
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __ldcg(row + (int64_t(X) * 3 + c) * tb);
#pragma unroll
  for (int c = 0; c < 3; ++c) s[y][c][x] = v[c];
  __syncthreads();
  if (y != 0 || i >= p.n) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    v[c] = s[0][c][x];
#pragma unroll
    for (int w = 1; w < 8; ++w) v[c] += s[w][c][x];
  }
  finish64<kForce>(p, sc, i, v);
}

// Warps per CTA: the finest split, one 32-particle block pair per warp, keeps
// the four FP64 units of every SM evenly loaded (field kernel at 4,096
// particles: 7 % slower with two); larger blocks keep
// the partial sums (24 n^2 / TB bytes) of larger scenes small.  16 or 8 warps
// per SM measure the same, 32 take 8 % longer (the steps no longer divide
// evenly).  Also the scratch bound: see sym64_eligible.
int warps_for(int64_t n) { return n < 8192 ? 1 : n < 16384 ? 2 : n < 32768 ? 4 : 8; }

template <bool kForce, int W>
mf_status launch64(const Sym64Args& p, cudaStream_t st) {
  static std::mutex mu;
  static int cache[64] = {};
  const int dev = current_device();
  int gmax = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    int& g = cache[dev >= 0 && dev < 64 ? dev : 0];
    if (!g) {
      int per_sm = 0;
      MF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sym64<kForce, W>, 32 * W, 0));
      g = std::max(1, std::min(per_sm, 16 / W)) * device_sms(dev);
    }
    gmax = g;
  }
  const int64_t g = std::min<int64_t>(p.a.total_steps, gmax);
  k_sym64<kForce, W><<<unsigned(g), 32 * W, 0, st>>>(p);
  MF_CUDA_TRY(cudaGetLastError());
  if (p.nb == 1) return MF_OK;
  k_sym64_finish<kForce><<<unsigned((p.n + 31) / 32), 256, 0, st>>>(p, 32 * W);
  MF_CUDA_TRY(cudaGetLastError());
  return MF_OK;
}

}  // namespace

// One scene whose targets are its sources.  Up to 65,536 particles the
// partial sums take at most 0.4 GB; larger scenes keep the all-pairs kernel.
bool sym64_eligible(Body body, const std::vector<SceneSpec>& specs) {
  if ((body != Body::Field && body != Body::Force) || specs.size() != 1) return false;
  const SceneSpec& s = specs[0];
  return s.nt > 0 && s.nt == s.ns && s.t_off == s.s_off && s.nt <= 65536;
}

mf_status build_sym64_plan(Body body, const std::vector<SceneSpec>& specs, Plan<double>& plan) {
  if (!sym64_eligible(body, specs))
    return fail(MF_ERR_INVALID_ARG, "pair-symmetric FP64 plan: field or force of one scene, targets equal to the sources");
  const SceneSpec& s = specs[0];
  if (!(s.h > 0.0)) return fail(MF_ERR_INVALID_ARG, "build_plan: smoothing length must be > 0");
  SceneDesc<double> d;
  memset(&d, 0, sizeof(d));
  const int W = warps_for(s.nt);
  const int64_t nb = (s.nt + 32 * W - 1) / (32 * W);
  d.t_off = d.s_off = s.t_off;
  d.nt = d.ns = s.nt;
  d.n_tb = int32_t(nb);
  d.n_tiles = W;
  d.flag_index = s.flag_index >= 0 ? s.flag_index : 0;
  fill_scene_coefs<double>(s, d);
  plan.body = body;
  plan.shape = kShapeSym;
  plan.host.assign(1, d);
  plan.total_steps = nb * (nb + 1) / 2;
  plan.total_tb = nb * nb;
  plan.n_scenes = 1;
  plan.pairs = double(s.nt) * double(s.nt);
  plan.evals = double(s.nt) * double(s.nt - 1) * 0.5;
  MF_TRY(plan.d_scenes.reserve_grow(sizeof(d)));
  MF_CUDA_TRY(cudaMemcpy(plan.d_scenes.ptr, plan.host.data(), sizeof(d), cudaMemcpyHostToDevice));
  return MF_OK;
}

size_t sym64_partials(const Plan<double>& plan) {
  return size_t(plan.total_tb) * 3 * 32 * size_t(plan.host.front().n_tiles);
}

mf_status run_sym64(const Plan<double>& plan, const LaunchIO<double>& io, double* partials, int32_t* err,
                    cudaStream_t st) {
  Sym64Args p;
  memset(&p, 0, sizeof(p));
  p.a = allpairs_args<double>(plan, io, partials, nullptr, err);
  p.part = partials;
  p.nb = plan.host.front().n_tb;
  p.n = plan.host.front().nt;
  p.off = plan.host.front().t_off;
  const bool force = plan.body == Body::Force;
  switch (plan.host.front().n_tiles) {
    case 1: return force ? launch64<true, 1>(p, st) : launch64<false, 1>(p, st);
    case 2: return force ? launch64<true, 2>(p, st) : launch64<false, 2>(p, st);
    case 4: return force ? launch64<true, 4>(p, st) : launch64<false, 4>(p, st);
    default: return force ? launch64<true, 8>(p, st) : launch64<false, 8>(p, st);
  }
}

}  // namespace mfgb
