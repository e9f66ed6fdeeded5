// mf_pair.cuh -- pair arithmetic of the SPH-smoothed dipole kernels.
//
// Field (B/mu0) of a source dipole s at offset d = target - source:
//   fmmtl_minimum/kernel/Dipole_B.kern:46-104, magnetic_force.cu:63-98
//   K_B(d) s = rhat (rhat.s)(w_avr - w_dens) - (w_avr/3 - w_dens) s.
// Written here as  (1/4pi) * (3 d (d.s) alpha - s beta)  with
//   far  (q >= 2):  alpha = r^-5,  beta = r^-3        (w_dens = 0)
//   near (q <  2):  alpha = 4pi (w_avr - w_dens) / (3 r^2),  beta = 4pi (w_avr/3 - w_dens)
// so the common far pair costs one rsqrt and a handful of FMAs.  At r = 0 the
// d-term vanishes and beta carries the self term, as in the reference.
//
// Force tensor of a source dipole s, contracted with the target dipole m:
//   fmmtl_minimum/kernel/Dipole_hessian.kern:53-253, magnetic_force.cu:239-427.
// The reference builds a rotated frame (xi, eta, zeta = rhat) and forms
// M U M^T.  Expanding that product with an orthonormal frame gives the
// frame-free form used here,
//   T_ab = P (ds delta_ab + s_a d_b + d_a s_b) + Q ds d_a d_b,   ds = d.s,
//   far  (q >  4):  P = K r^-5,            Q = -5 K r^-7,   K = 3 mu0 / (4 pi)
//   near (0<q<=4):  P = C1(q) / (h^4 r),   Q = (C2(q) - 3 C1(q)) / (h^4 r^3)
//   q == 0:         T = 0  (overlapping particles exert no force, :101-104)
// and F = T m = P (ds m + dm s + sm d) + Q ds dm d  with dm = d.m, sm = s.m.
// The far branch is the reference's analytic tensor term for term
// (A = mu0 w_avr / r^2, dAdr, dBdr of :168-206).
#pragma once
#include "mf_device.cuh"

namespace mfgb {

constexpr double kPi = 3.14159265358979323846;
constexpr double kMu0 = 1.25663706e-6;              // Dipole_hessian.kern:170
constexpr double kForceK = 3.0 * kMu0 / (4.0 * kPi);  // far-field force prefactor
constexpr double kInv4Pi = 1.0 / (4.0 * kPi);

// Per-scene constants derived from the smoothing length.
template <class Real>
struct PairConsts {
  Real inv_h;        // 1/h
  Real h;            // smoothing length
  Real ih3;          // 1/h^3
  Real ih3_30;       // 1/(30 h^3), 1/(30 h^5): scale the field's near forms (field_near_unit)
  Real ih5_30;
  Real ih4_over_k;   // 1/(h^4 K): scales the fitted curves into the K-free form
  Real near2_field;  // (2h)^2: field pairs closer than this take the SPH branch
  Real near2_force;  // (4h)^2: force pairs at or inside this take the fitted branch
  // FP32 kernels: the fitted-curve table in shared memory (set by the kernel
  // in its own copy; null in stored scene tables).
  const float* tbl;
};

template <class Real>
__host__ __device__ inline PairConsts<Real> make_pair_consts(double h) {
  PairConsts<Real> k;
  k.inv_h = Real(1.0 / h);
  k.h = Real(h);
  k.ih3 = Real(1.0 / (h * h * h));
  k.ih3_30 = Real(1.0 / (30.0 * h * h * h));
  // h^-5 leaves FP32 from 1e-8 down, where it is held finite: what it scales
  // overflows there, except at r = 0, which the kernels leave out.  Above 1e7
  // it is subnormal: the corrections take theirs times a power of two
  // (CellGrid); here the multiplication that would undo it costs 1.5 % of every
  // small solve (field of 200 particles at h = 4e7: 9e-7 from FP64).
  const double ih5 = 1.0 / (30.0 * h * h * h * h * h);
  k.ih5_30 = Real(sizeof(Real) == 4 ? fmin(ih5, 3.4e38) : ih5);
  k.ih4_over_k = Real(1.0 / (h * h * h * h * kForceK));
  k.near2_field = Real(4.0 * h * h);
  k.near2_force = Real(16.0 * h * h);
  k.tbl = nullptr;
  return k;
}

template <class Real>
__device__ __forceinline__ Real rsqrt_r(Real x);
template <>
__device__ __forceinline__ float rsqrt_r<float>(float x) {
  return rsqrt_approx(x);
}
template <>
__device__ __forceinline__ double rsqrt_r<double>(double x) {
  return rsqrt(x);
}

// Near-field SPH weights of the field kernel (Dipole_B.kern:46-76), returned as
// the (alpha, beta) pair of the form above.  Only reached for r < 2h.
template <class Real>
__device__ __noinline__ void field_near_coeffs(Real r2, const PairConsts<Real>& k, Real& alpha, Real& beta) {
  Real r = sqrt(r2);
  Real q = r * k.inv_h;
  Real tmq = Real(2) - q;
  Real tmq3 = tmq * tmq * tmq;
  Real wa, wd;  // 4 pi h^3 w_avr, 4 pi h^3 w_dens
  if (q >= Real(1)) {
    Real q2 = q * q, q3 = q2 * q;
    Real P = q3 * q3 / Real(6) - Real(6) * q3 * q2 / Real(5) + Real(3) * q2 * q2 - Real(8) * q3 / Real(3) +
             Real(1) / Real(15);
    wa = Real(-3) * P / q3;
    wd = tmq3;
  } else {
    Real q2 = q * q;
    Real omq = Real(1) - q;
    wa = (Real(15) * q2 * q - Real(36) * q2 + Real(40)) / Real(10);
    wd = tmq3 - Real(4) * omq * omq * omq;
  }
  beta = (wa / Real(3) - wd) * k.ih3;
  alpha = (r2 > Real(0)) ? (wa - wd) * k.ih3 / (Real(3) * r2) : Real(0);
}

// One field pair: s1 += d (d.s) alpha, s2 += s beta.  Field = (3 s1 - s2) / 4pi.
template <class Real>
__device__ __forceinline__ void field_pair(Real dx, Real dy, Real dz, Real sx, Real sy, Real sz,
                                           const PairConsts<Real>& k, Real* s1, Real* s2) {
  Real r2 = dx * dx + dy * dy + dz * dz;
  Real alpha, beta;
  if (r2 >= k.near2_field) {
    Real ri = rsqrt_r(r2);
    Real ri2 = ri * ri;
    beta = ri2 * ri;
    alpha = beta * ri2;
  } else {
    field_near_coeffs(r2, k, alpha, beta);
  }
  Real t = (dx * sx + dy * sy + dz * sz) * alpha;
  s1[0] += dx * t;
  s1[1] += dy * t;
  s1[2] += dz * t;
  s2[0] += sx * beta;
  s2[1] += sy * beta;
  s2[2] += sz * beta;
}

// Fitted near-field curves C1(q), C2(q), q in (0, 4]
// (Dipole_hessian.kern:53-85, magnetic_force.cu:301-330).
template <class Real>
__device__ __forceinline__ void fitted_curves(Real q, Real& c1, Real& c2) {
#define MF_P4(a, b, c, d, e) (q * (q * (q * (q * Real(a) + Real(b)) + Real(c)) + Real(d)) + Real(e))
  if (q <= Real(1)) {
    c1 = MF_P4(9.97813616438174e-09, -2.97897856524718e-08, 2.38918644566813e-09, 4.53199938857366e-08,
               2.44617454752747e-11);
    c2 = MF_P4(6.69550479838731e-08, -1.61753307173877e-07, 1.68213714992711e-08, 1.34558143036838e-07,
               1.10976027980100e-10);
  } else if (q <= Real(2)) {
    c1 = MF_P4(-2.76473728643294e-09, 2.86975546540539e-08, -9.94582836806651e-08, 1.25129924573675e-07,
               -2.37010166723652e-08);
    c2 = MF_P4(-3.08460139955194e-08, 2.29192245602275e-07, -5.88399621128587e-07, 5.61170054591844e-07,
               -1.14421132829680e-07);
  } else if (q <= Real(3)) {
    c1 = MF_P4(-1.09679990621465e-09, 9.77055663264614e-09, -2.54781238661150e-08, 2.65020634884934e-09,
               5.00787562417835e-08);
    c2 = MF_P4(3.50477408060213e-09, -5.25956271895141e-08, 2.78876509535747e-07, -6.24199554212217e-07,
               4.91807818904985e-07);
  } else {
    c1 = MF_P4(3.79927162333632e-10, -6.26368404962679e-09, 3.94760528277489e-08, -1.13580541622200e-07,
               1.27491333574323e-07);
    c2 = MF_P4(7.33485346367840e-10, -9.58855788627803e-09, 4.37085309763591e-08, -7.48004594092261e-08,
               2.34161209605651e-08);
  }
#undef MF_P4
}

// (P, Q) of the force tensor for 0 <= r <= 4h, in units of K.
template <class Real>
__device__ __noinline__ void force_near_coeffs(Real r2, const PairConsts<Real>& k, Real& P, Real& Q) {
  if (r2 == Real(0)) {
    P = Real(0);
    Q = Real(0);
    return;
  }
  Real r = sqrt(r2);
  Real q = r * k.inv_h;
  q = q > Real(4) ? Real(4) : q;  // the branch test is on r^2; keep q on the fitted range
  Real c1, c2;
  fitted_curves(q, c1, c2);
  Real ir = Real(1) / r;
  Real s = k.ih4_over_k * ir;
  P = c1 * s;
  Q = (c2 - Real(3) * c1) * s * ir * ir;
}

// (P, Q) of the force tensor for any pair, in units of K.
template <class Real>
__device__ __forceinline__ void force_coeffs(Real r2, const PairConsts<Real>& k, Real& P, Real& Q) {
  if (r2 > k.near2_force) {
    Real ri = rsqrt_r(r2);
    Real ri2 = ri * ri;
    P = ri2 * ri2 * ri;
    Q = Real(-5) * P * ri2;
  } else {
    force_near_coeffs(r2, k, P, Q);
  }
}

// One force pair contracted with the target dipole m: f += T(d, s) m / K.
template <class Real>
__device__ __forceinline__ void force_pair(Real dx, Real dy, Real dz, Real sx, Real sy, Real sz, Real mx,
                                           Real my, Real mz, const PairConsts<Real>& k, Real* f) {
  Real r2 = dx * dx + dy * dy + dz * dz;
  Real ds = dx * sx + dy * sy + dz * sz;
  Real dm = dx * mx + dy * my + dz * mz;
  Real sm = sx * mx + sy * my + sz * mz;
  Real u, v, w;
  if (r2 > k.near2_force) {
    Real ri = rsqrt_r(r2);
    Real ri2 = ri * ri;
    Real ri5 = ri2 * ri2 * ri;
    u = ds * ri5;
    v = dm * ri5;
    w = (Real(-5) * ri2 * ds) * v + sm * ri5;
  } else {
    Real P, Q;
    force_near_coeffs(r2, k, P, Q);
    u = P * ds;
    v = P * dm;
    w = P * sm + Q * ds * dm;
  }
  f[0] += dx * w + mx * u + sx * v;
  f[1] += dy * w + my * u + sy * v;
  f[2] += dz * w + mz * u + sz * v;
}

// ---------------------------------------------------------------------------
// Packed two-source forms (FP32).  Lanes .x / .y hold two different sources;
// the target's values are duplicated into both lanes.  Every pair takes the
// far form with r^2 clamped to the near radius: exact beyond it, finite inside
// it (including r = 0).  The near-field correction pass (mf_cells.cu) adds,
// for each pair inside the near radius, the exact term minus this clamped one.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 clamp_rsqrt2(float2 r2, float near2) {
  return make_float2(rsqrt_approx(fmaxf(r2.x, near2)), rsqrt_approx(fmaxf(r2.y, near2)));
}

// s1 += d (d.m) r^-5, s2 += m r^-3 (field = (3 s1 - s2) / 4pi after the lanes are added).
__device__ __forceinline__ void field_pair2(float2 tx, float2 ty, float2 tz, float2 sx, float2 sy, float2 sz,
                                            float2 mx, float2 my, float2 mz, float near2, float2* s1, float2* s2) {
  const float2 dx = f2_sub(tx, sx), dy = f2_sub(ty, sy), dz = f2_sub(tz, sz);
  const float2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
  const float2 ri = clamp_rsqrt2(r2, near2);
  const float2 ri2 = f2_mul(ri, ri);
  const float2 beta = f2_mul(ri2, ri);
  const float2 alpha = f2_mul(beta, ri2);
  const float2 dm = f2_fma(dz, mz, f2_fma(dy, my, f2_mul(dx, mx)));
  const float2 t = f2_mul(dm, alpha);
  s1[0] = f2_fma(dx, t, s1[0]);
  s1[1] = f2_fma(dy, t, s1[1]);
  s1[2] = f2_fma(dz, t, s1[2]);
  s2[0] = f2_fma(mx, beta, s2[0]);
  s2[1] = f2_fma(my, beta, s2[1]);
  s2[2] = f2_fma(mz, beta, s2[2]);
}

// f += T(d, s) m / K with the far (P, Q) = (r^-5, -5 r^-7) of the clamped
// distance, in two parts: f gets d w + s v, and u the scalar sum of
// r^-5 (d.s) whose product with the target's dipole m completes the force
// (the caller applies it once per tile: 3 packed operations fewer per pair).
__device__ __forceinline__ void force_pair2(float2 tx, float2 ty, float2 tz, float2 tmx, float2 tmy, float2 tmz,
                                            float2 sx, float2 sy, float2 sz, float2 smx, float2 smy, float2 smz,
                                            float near2, float2* f, float2& u) {
  const float2 dx = f2_sub(tx, sx), dy = f2_sub(ty, sy), dz = f2_sub(tz, sz);
  const float2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
  const float2 ri = clamp_rsqrt2(r2, near2);
  const float2 ri2 = f2_mul(ri, ri);
  const float2 ri5 = f2_mul(f2_mul(ri2, ri2), ri);
  const float2 ds = f2_fma(dz, smz, f2_fma(dy, smy, f2_mul(dx, smx)));
  const float2 dm = f2_fma(dz, tmz, f2_fma(dy, tmy, f2_mul(dx, tmx)));
  const float2 sm = f2_fma(smz, tmz, f2_fma(smy, tmy, f2_mul(smx, tmx)));
  const float2 v = f2_mul(dm, ri5);
  const float2 e = f2_mul(f2_mul(ri2, ds), f2_dup(-5.f));
  const float2 w = f2_fma(e, v, f2_mul(sm, ri5));
  u = f2_fma(ds, ri5, u);
  f[0] = f2_fma(dx, w, f2_fma(smx, v, f[0]));
  f[1] = f2_fma(dy, w, f2_fma(smy, v, f[1]));
  f[2] = f2_fma(dz, w, f2_fma(smz, v, f[2]));
}

// Packed two-source force tensor, clamped far form: with e = P d and
// v = m - 5/2 r^-2 (d.m) d,
//   T / K = e v^T + v e^T + P (d.m) I,
// summed as the off-diagonal entries t[0..2] (xy, xz, yz), half the diagonal
// ones without the trace term t[3..5], and the trace term t[6]: 30 packed
// operations (entry by entry 46).
__device__ __forceinline__ void tensor_pair2(float2 tx, float2 ty, float2 tz, float2 sx, float2 sy, float2 sz,
                                             float2 smx, float2 smy, float2 smz, float near2, float2* t) {
  const float2 dx = f2_sub(tx, sx), dy = f2_sub(ty, sy), dz = f2_sub(tz, sz);
  const float2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
  const float2 ri = clamp_rsqrt2(r2, near2);
  const float2 ri2 = f2_mul(ri, ri);
  const float2 P = f2_mul(f2_mul(ri2, ri2), ri);
  const float2 ds = f2_fma(dz, smz, f2_fma(dy, smy, f2_mul(dx, smx)));
  const float2 k = f2_mul(f2_mul(ri2, f2_dup(-2.5f)), ds);
  const float2 vx = f2_fma(dx, k, smx), vy = f2_fma(dy, k, smy), vz = f2_fma(dz, k, smz);
  const float2 ex = f2_mul(dx, P), ey = f2_mul(dy, P), ez = f2_mul(dz, P);
  t[0] = f2_fma(ex, vy, f2_fma(ey, vx, t[0]));
  t[1] = f2_fma(ex, vz, f2_fma(ez, vx, t[1]));
  t[2] = f2_fma(ey, vz, f2_fma(ez, vy, t[2]));
  t[3] = f2_fma(ex, vx, t[3]);
  t[4] = f2_fma(ey, vy, t[4]);
  t[5] = f2_fma(ez, vz, t[5]);
  t[6] = f2_fma(P, ds, t[6]);
}

// The clamped far coefficients every near pair received in the packed loop
// (the same rsqrt and products; equal to within rounding).
__device__ __forceinline__ void clamped_field_coeffs(float near2, float& alpha, float& beta) {
  const float ri = rsqrt_approx(near2);
  const float ri2 = ri * ri;
  beta = ri2 * ri;
  alpha = beta * ri2;
}
__device__ __forceinline__ void clamped_force_coeffs(float near2, float& P, float& Q) {
  const float ri = rsqrt_approx(near2);
  const float ri2 = ri * ri;
  P = (ri2 * ri2) * ri;
  Q = ri2 * -5.f * P;
}

// Branch-free FP32 forms of the near-field coefficients, for kernels where the
// lanes of a warp sit on different pieces.  Same mathematics as
// field_near_coeffs / force_near_coeffs with the polynomials multiplied out.

// Field: 30 alpha h^5 and 30 beta h^3 at q = r / h < 2.  Times 30 every
// coefficient is a whole number: 0.8f alone would put 4e-7 of alpha at q = 2
// into every pair.  The outer piece's beta is written in t = 2 - q, where its
// terms do not cancel.  alpha is infinite at r = 0 from h = 2e-8 down; it
// multiplies d = 0 there and is to be taken as 0.
//   q < 1: 24 - 15 q,                       -80 + 144 q^2 - 75 q^3
//   else:  5 q - 24 + 30 / q - 2 q^-5,      4 + 6 t + 6 t^2 - 25 t^3 - 2 q^-3
// ri: near_rsqrt(r2), finite at r = 0 (where q comes out 0).
__device__ __forceinline__ float near_rsqrt(float r2) { return rsqrt_approx(fmaxf(r2, 1e-36f)); }
__device__ __forceinline__ void field_near_unit(float r2, float ri, float h, float inv_h, float& al, float& be) {
  const float q = (r2 * ri) * inv_h, iq = ri * h;
  const float iq2 = iq * iq, iq3 = iq2 * iq, t = 2.f - q;
  const bool hi = q >= 1.f;
  const float al_hi = fmaf(iq3 * iq2, -2.f, fmaf(q, 5.f, fmaf(iq, 30.f, -24.f)));
  const float be_hi = fmaf(iq3, -2.f, fmaf(t, fmaf(t, fmaf(t, -25.f, 6.f), 6.f), 4.f));
  const float al_lo = fmaf(q, -15.f, 24.f);
  const float be_lo = fmaf(q * q, fmaf(q, -75.f, 144.f), -80.f);
  al = hi ? al_hi : al_lo;
  be = hi ? be_hi : be_lo;
}
// The same for two distances at once (packed FP32).
__device__ __forceinline__ void field_near_unit2(float2 r2, float h, float inv_h, float2& al, float2& be) {
  const float2 ri = make_float2(near_rsqrt(r2.x), near_rsqrt(r2.y));
  const float2 q = f2_mul(f2_mul(r2, ri), f2_dup(inv_h)), iq = f2_mul(ri, f2_dup(h));
  const float2 iq2 = f2_mul(iq, iq), iq3 = f2_mul(iq2, iq), t = f2_sub(f2_dup(2.f), q);
  const float2 m2 = f2_dup(-2.f);
  const float2 al_hi = f2_fma(f2_mul(iq3, iq2), m2, f2_fma(q, f2_dup(5.f), f2_fma(iq, f2_dup(30.f), f2_dup(-24.f))));
  const float2 b2 = f2_fma(t, f2_fma(t, f2_dup(-25.f), f2_dup(6.f)), f2_dup(6.f));
  const float2 be_hi = f2_fma(iq3, m2, f2_fma(t, b2, f2_dup(4.f)));
  const float2 al_lo = f2_fma(q, f2_dup(-15.f), f2_dup(24.f));
  const float2 be_lo = f2_fma(f2_mul(q, q), f2_fma(q, f2_dup(-75.f), f2_dup(144.f)), f2_dup(-80.f));
  const bool h0 = q.x >= 1.f, h1 = q.y >= 1.f;
  al = make_float2(h0 ? al_hi.x : al_lo.x, h1 ? al_hi.y : al_lo.y);
  be = make_float2(h0 ? be_hi.x : be_lo.x, h1 ? be_hi.y : be_lo.y);
}

// The fitted-curve table for the force (Dipole_hessian.kern:53-61) in the
// layout force_curves reads from shared memory: entry i = ceil(q) of three
// arrays, (C1's q^4 .. q^1), (C2's q^4 .. q^1), (both constants).  Entries 0
// and 1 hold the piece q <= 1, 2 and 3 the next two, the others q > 3 (any
// index of three bits is inside the table).
struct ForceTable {
  float v[80];
};
constexpr ForceTable make_force_table() {
  constexpr double c[4][10] = {
      {9.97813616438174e-09, -2.97897856524718e-08, 2.38918644566813e-09, 4.53199938857366e-08,
       2.44617454752747e-11, 6.69550479838731e-08, -1.61753307173877e-07, 1.68213714992711e-08,
       1.34558143036838e-07, 1.10976027980100e-10},
      {-2.76473728643294e-09, 2.86975546540539e-08, -9.94582836806651e-08, 1.25129924573675e-07,
       -2.37010166723652e-08, -3.08460139955194e-08, 2.29192245602275e-07, -5.88399621128587e-07,
       5.61170054591844e-07, -1.14421132829680e-07},
      {-1.09679990621465e-09, 9.77055663264614e-09, -2.54781238661150e-08, 2.65020634884934e-09,
       5.00787562417835e-08, 3.50477408060213e-09, -5.25956271895141e-08, 2.78876509535747e-07,
       -6.24199554212217e-07, 4.91807818904985e-07},
      {3.79927162333632e-10, -6.26368404962679e-09, 3.94760528277489e-08, -1.13580541622200e-07,
       1.27491333574323e-07, 7.33485346367840e-10, -9.58855788627803e-09, 4.37085309763591e-08,
       -7.48004594092261e-08, 2.34161209605651e-08}};
  ForceTable t{};
  for (int i = 0; i < 8; ++i) {
    const int p = i < 1 ? 0 : i > 4 ? 3 : i - 1;
    for (int k = 0; k < 4; ++k) {
      t.v[4 * i + k] = float(c[p][k]);
      t.v[32 + 4 * i + k] = float(c[p][5 + k]);
    }
    t.v[64 + 2 * i] = float(c[p][4]);
    t.v[64 + 2 * i + 1] = float(c[p][9]);
  }
  return t;
}

// C1(q) and C2(q) for 0 <= q <= 4 (C2 - 3 C1 is formed from the two values: as
// curves of its own its rounding no longer cancelled C1's along d, and the
// force came out 2.7e-6 instead of 1.1e-6 from the oracle).  tbl: a ForceTable in shared memory, 16-byte
// aligned.  ceil(q) by one add rounded up to a whole number (no conversion
// through the slow units).  Other q give values the caller must not use.
__device__ __forceinline__ void force_curves(float q, const float* __restrict__ tbl, float& c1, float& c2) {
  const int i = __float_as_int(__fadd_ru(q, 8388608.f)) & 7;
  const float4 a = *reinterpret_cast<const float4*>(tbl + 4 * i);
  const float4 b = *reinterpret_cast<const float4*>(tbl + 32 + 4 * i);
  const float2 c = *reinterpret_cast<const float2*>(tbl + 64 + 2 * i);
  c1 = fmaf(q, fmaf(q, fmaf(q, fmaf(q, a.x, a.y), a.z), a.w), c.x);
  c2 = fmaf(q, fmaf(q, fmaf(q, fmaf(q, b.x, b.y), b.z), b.w), c.y);
}

// (P, Q) of the force tensor for 0 < r <= 4h, in units of K.
__device__ __forceinline__ void force_near_pq(float r2, const float* __restrict__ tbl, float inv_h, float ih4_over_k,
                                              float& P, float& Q) {
  const float ri = rsqrt_approx(r2);
  float c1, c2;
  force_curves((r2 * ri) * inv_h, tbl, c1, c2);
  const float s = ih4_over_k * ri;
  P = c1 * s;
  Q = fmaf(-3.f, c1, c2) * s * (ri * ri);
}

// FP32 exact pair forms without a branch: the far coefficients and the fast
// near coefficients above are both evaluated and selected by the radius, so
// warps whose lanes straddle the near radius do not diverge.  Same
// mathematics as field_pair / force_pair (the far value at r = 0 is infinite
// and discarded by the select).  The force needs k.tbl.
__device__ __forceinline__ void field_pair_sel(float dx, float dy, float dz, float sx, float sy, float sz,
                                               const PairConsts<float>& k, float* s1, float* s2) {
  const float r2 = dx * dx + dy * dy + dz * dz;
  const float ri = near_rsqrt(r2), ri2 = ri * ri, ri3 = ri2 * ri;
  float al, be;
  field_near_unit(r2, ri, k.h, k.inv_h, al, be);
  const bool far = r2 >= k.near2_field;
  al = r2 > 0.f ? al : 0.f;
  const float beta = far ? ri3 : be * k.ih3_30;
  const float alpha = far ? ri3 * ri2 : al * k.ih5_30;
  const float t = (dx * sx + dy * sy + dz * sz) * alpha;
  s1[0] += dx * t;
  s1[1] += dy * t;
  s1[2] += dz * t;
  s2[0] += sx * beta;
  s2[1] += sy * beta;
  s2[2] += sz * beta;
}

__device__ __forceinline__ void force_pair_sel(float dx, float dy, float dz, float sx, float sy, float sz, float mx,
                                               float my, float mz, const PairConsts<float>& k, float* f) {
  const float r2 = dx * dx + dy * dy + dz * dz;
  const float ds = dx * sx + dy * sy + dz * sz;
  const float dm = dx * mx + dy * my + dz * mz;
  const float sm = sx * mx + sy * my + sz * mz;
  float Pn, Qn;
  force_near_pq(r2, k.tbl, k.inv_h, k.ih4_over_k, Pn, Qn);
  const float ri = rsqrt_approx(r2), ri2 = ri * ri, ri5 = ri2 * ri2 * ri;
  const bool far = r2 > k.near2_force, apart = r2 > 0.f;
  const float P = far ? ri5 : apart ? Pn : 0.f;
  const float Q = far ? -5.f * ri5 * ri2 : apart ? Qn : 0.f;
  const float u = P * ds, v = P * dm, w = P * sm + Q * ds * dm;
  f[0] += dx * w + mx * u + sx * v;
  f[1] += dy * w + my * u + sy * v;
  f[2] += dz * w + mz * u + sz * v;
}

// (P, Q) of the force tensor for 0 < r <= 4h, in units of K, with r and 1/r to
// FP32 rounding (one Newton step each from the hardware's reciprocal root):
// the curves jump where their pieces meet, and a distance exactly on a join
// has to stay on its side, as with a rounded square root (a root that is a
// unit off puts the tensor at q = 3 1.3e-5 from its value, 4e-6 with this).
__device__ __forceinline__ void force_near_pq_rn(float r2, const float* __restrict__ tbl, float inv_h,
                                                 float ih4_over_k, float& P, float& Q) {
  const float y = rsqrt_approx(r2);
  float r = r2 * y;
  r = fmaf(fmaf(-r, r, r2), 0.5f * y, r);
  const float ri = fmaf(y, fmaf(-r, y, 1.f), y);
  float c1, c2;
  force_curves(r * inv_h, tbl, c1, c2);
  const float s = ih4_over_k * ri;
  P = c1 * s;
  Q = fmaf(-3.f, c1, c2) * s * (ri * ri);
}

// (P, Q) of the force tensor for any pair, FP32 without a branch (k.tbl set).
__device__ __forceinline__ void force_coeffs_sel(float r2, const PairConsts<float>& k, float& P, float& Q) {
  float Pn, Qn;
  force_near_pq_rn(r2, k.tbl, k.inv_h, k.ih4_over_k, Pn, Qn);
  const float ri = rsqrt_approx(r2), ri2 = ri * ri, ri5 = ri2 * ri2 * ri;
  const bool far = r2 > k.near2_force, apart = r2 > 0.f;
  P = far ? ri5 : apart ? Pn : 0.f;
  Q = far ? -5.f * ri5 * ri2 : apart ? Qn : 0.f;
}

// One tensor pair (6 unique entries xx, yy, zz, xy, xz, yz): t += T(d, s) / K.
template <class Real>
__device__ __forceinline__ void tensor_terms(Real dx, Real dy, Real dz, Real sx, Real sy, Real sz, Real P, Real Q,
                                             Real* t) {
  Real ds = dx * sx + dy * sy + dz * sz;
  Real pd = P * ds, qd = Q * ds;
  Real ax = P * sx, ay = P * sy, az = P * sz;
  t[0] += pd + Real(2) * ax * dx + qd * dx * dx;
  t[1] += pd + Real(2) * ay * dy + qd * dy * dy;
  t[2] += pd + Real(2) * az * dz + qd * dz * dz;
  t[3] += ax * dy + ay * dx + qd * dx * dy;
  t[4] += ax * dz + az * dx + qd * dx * dz;
  t[5] += ay * dz + az * dy + qd * dy * dz;
}
template <class Real>
__device__ __forceinline__ void tensor_pair(Real dx, Real dy, Real dz, Real sx, Real sy, Real sz,
                                            const PairConsts<Real>& k, Real* t) {
  Real r2 = dx * dx + dy * dy + dz * dz;
  Real P, Q;
  if constexpr (sizeof(Real) == 4) force_coeffs_sel(r2, k, P, Q);
  else force_coeffs(r2, k, P, Q);
  tensor_terms<Real>(dx, dy, dz, sx, sy, sz, P, Q, t);
}

}  // namespace mfgb
