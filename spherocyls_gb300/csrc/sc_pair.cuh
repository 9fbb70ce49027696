// sc_pair.cuh -- segment-segment contact of two spherocylinders (device code).
//
// Two forms of the same geometry (tmarschall/spherocyls
// src/cpp/strain_dynamics.cpp:17-75, calc_force_pair; stress arms from
// src/cpp/spherocyl_box.cpp:425-500, calc_se_force_pair):
//
//  * pair_fp64: every floating-point operation in the reference's order.  It is
//    compiled in a translation unit built with -fmad=false so no fused
//    multiply-add changes the rounding; together with role assignment by particle
//    index (the lower index plays the reference's "p") each pair contribution is
//    the reference's up to the last-ulp difference of the device cos/sin.
//  * pair_fp32: the same closest-point algorithm in FP32 on a displacement that
//    the caller already reduced to the minimum image, with fast reciprocal and
//    reciprocal-square-root; the caller accumulates stress and energy in FP64.
//
// Both take the displacement of P relative to Q in sheared coordinates and apply
// the Lees-Edwards shift dX += gamma*dY themselves.
#pragma once

#include <cuda_runtime.h>

namespace sc {

struct PairF64 {
  double fx, fy, tp, tq;          // force on P (Q gets -f), torques on P and Q
  double e, pxx, pyy, pxy, pyx;   // stress/energy contributions (when requested)
};

// ---- FP64 operations taken off the FP64 pipe ----
//
// GB300 runs FP64 at about 1/60 of its FP32 rate, and that pipe bounds the pair code.
// Comparisons with constants and clamps are decided on the bits of the operand by the
// integer pipe instead, with the same result for every value (NaN as in fmin, fmax).

// d - L where d > L/2, d + L where d < -L/2 (L > 0)
__device__ __forceinline__ double nearest_image(double d, double L) {
  if ((__double2hiint(d) & 0x7fffffff) < __double2hiint(0.5 * L)) return d;
  return d + L * (double)((d < -0.5 * L) - (d > 0.5 * L));
}
__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
constexpr unsigned long long kBitsOne = 0x3ff0000000000000ull, kBitsInf = 0x7ff0000000000000ull;
// fmin(fmax(v, -1), 1): a NaN becomes -1
__device__ __forceinline__ double clamp_one(double v) {
  const unsigned long long b = abs_bits(v);
  if (b < kBitsOne) return v;
  return b > kBitsInf || __double2hiint(v) < 0 ? -1.0 : 1.0;
}
// |v| > 1 and |v| >= 1 (false for NaN)
__device__ __forceinline__ bool beyond_one(double v) {
  const unsigned long long b = abs_bits(v);
  return b > kBitsOne && b <= kBitsInf;
}
__device__ __forceinline__ bool reaches_one(double v) {
  const unsigned long long b = abs_bits(v);
  return b >= kBitsOne && b <= kBitsInf;
}
// u < v for sums of squares, whose bits order as their values (false where u is NaN)
__device__ __forceinline__ bool less_square(double u, double v) {
  return (unsigned long long)__double_as_longlong(u) < (unsigned long long)__double_as_longlong(v);
}

// (double)f and (float)d (rounded to nearest even) by the integer pipe; the conversions
// run at the FP64 pipe's rate.
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f), e = b & 0x7f800000u;
  if (e == 0u || e == 0x7f800000u) return (double)f;  // zero, subnormal, infinite, NaN
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)),
                          (int)(b << 29));
}
__device__ __forceinline__ float narrow(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned e = hi & 0x7ff00000u;
  // exponents whose rounded value is a normal float
  if (e - 0x38100000u >= 0x0fd00000u) return (float)v;
  const unsigned m = __funnelshift_l(lo, (hi & 0x7fffffffu) - 0x38000000u, 3);
  const unsigned rest = lo & 0x1fffffffu;
  const unsigned up = rest > 0x10000000u || (rest == 0x10000000u && (m & 1u)) ? 1u : 0u;
  return __uint_as_float((hi & 0x80000000u) | (m + up));
}

// Quotients that share a divisor: r = 1/y rounded to nearest, then q = x r with one correction
// by its remainder (P. W. Markstein, IBM J. Res. Dev. 34, 111 (1990)); three operations in
// place of a division's eight or so.  The result is the correctly rounded x/y.  With the
// mantissas 1 <= x, y < 2: a q within one ulp of x/y has an exact remainder, and Markstein's
// theorem holds; that covers x >= y (|q - x/y| <= x 2^-54 + 2^-53) and, with 2^-54 (x + 1),
// x <= 1.  For 1 < x < y, q may be up to 1.5 ulp (of 2^-53) off.  Past one ulp the remainder
// is rounded once, by at most 2^-105, and the corrected value is within 2^-104 of x/y, so
// that it rounds otherwise only if x/y - q is within 2^-104 of 1.5 ulp: x > 2 - 2^-50, which
// leaves (x, y) = 2 - (m, n) 2^-52 with n < m < 4, and those round right.
// That is for |x| within 2^-500 to 2^500, like r; a divisor out of that range has r = 0 and is
// divided by.  The pair code's dividends are products of its lengths and forces, in range
// where its divisors are; an x of -0 gives +0, which no sum of forces that starts at +0 can
// tell, and an infinite one NaN, which only a state that is already non-finite has (a test of
// x's exponent as well costs 2 to 7% of k_pairs64).
__device__ __forceinline__ double shared_rcp(double y) {
  const double r = 1.0 / y;
  const unsigned h = (unsigned)__double2hiint(r);
  return h - 0x20b00000u < 0x3e800000u ? r : 0.0;  // 2^-500 < r < 2^500
}
__device__ __forceinline__ double div_by(double x, double y, double r) {
  if (__double2hiint(r) == 0) return x / y;
  const double q = x * r;
  return fma(fma(-y, q, x), r, q);
}

// x / y by the shared reciprocal of y, or, in the minimiser's form (FAST), x times a
// reciprocal of y.  The FAST form trades the last bits of the reference's
// rounding for fewer FP64 divisions (GB300's FP64 rate is a small fraction of its
// FP32 rate); the force-evaluation and dynamics paths never use it.
template <bool FAST>
__device__ __forceinline__ double qdiv(double x, double y, double inv_y) {
  return FAST ? x * inv_y : div_by(x, y, inv_y);
}

// Reciprocals of a = |u_A|^2, c = |u_B|^2, delta and sig from one division.  Their product is
// zero for a disc and out of range for some other shapes: handles with such particles
// (Dev::odd_shapes) take the form with a division each.
struct Recip64 {
  double a, c, delta, sig;
};
__device__ __forceinline__ Recip64 recip64(double a, double c, double delta, double sig) {
  Recip64 r;
  const double ac = a * c;
  if (delta > 0) {
    const double inv = 1.0 / (ac * delta * sig);
    const double i_ac = delta * sig * inv;
    r.delta = ac * sig * inv;
    r.sig = ac * delta * inv;
    r.a = c * i_ac;
    r.c = a * i_ac;
  } else {
    const double inv = 1.0 / (ac * sig);
    r.delta = 0.0;
    r.sig = ac * inv;
    r.a = c * sig * inv;
    r.c = a * sig * inv;
  }
  return r;
}

// dX, dY: raw coordinate differences P - Q (no minimum image yet).
// Returns true when the spherocylinders overlap.  inv_aP, inv_aQ: shared_rcp of aP^2, aQ^2
// (unused with FAST).
// FAST with SE (the mixed form's FP64 stress): inv_LL = 1/(Lx Ly) and inv_two_n =
// 1/(2n) from the caller replace the per-term divisions.
template <bool SE, bool FAST = false>
__device__ __forceinline__ bool pair_fp64(double dX, double dY, double nxA, double nyA, double aP,
                                          double nxB, double nyB, double aQ, double sig,
                                          double gamma, double Lx, double Ly, bool virial,
                                          double two_n, PairF64& o, double inv_aP, double inv_aQ,
                                          double inv_LL = 0.0, double inv_two_n = 0.0) {
  dX = nearest_image(dX, Lx);
  dY = nearest_image(dY, Ly);
  dX += gamma * dY;

  double a = aP * aP;
  double b = -(nxA * nxB + nyA * nyB);
  double c = aQ * aQ;
  double d = nxA * dX + nyA * dY;
  double e = -nxB * dX - nyB * dY;
  double delta = a * c - b * b;
  Recip64 iv{};
  if (FAST) {
    iv = recip64(a, c, delta, sig);
  } else {
    iv.a = inv_aP;
    iv.c = inv_aQ;
  }

  double t = clamp_one((FAST && delta > 0) ? (b * d - a * e) * iv.delta : (b * d - a * e) / delta);
  double s = qdiv<FAST>(-(b * t + d), a, iv.a);
  const bool end = beyond_one(s);
  s = clamp_one(s);
  if (end) t = clamp_one(qdiv<FAST>(-(b * s + e), c, iv.c));

  double dDx = dX + s * nxA - t * nxB;
  double dDy = dY + s * nyA - t * nyB;
  double dsq = dDx * dDx + dDy * dDy;
  if (!less_square(dsq, sig * sig)) return false;
  double Fx, Fy, dij, dvij, inv_sig = 0.0;
  if (FAST) {
    const double rs = rsqrt(dsq);
    dij = dsq * rs;
    dvij = (1.0 - dij * iv.sig) * iv.sig;
    Fx = dDx * (dvij * rs);
    Fy = dDy * (dvij * rs);
  } else {
    dij = sqrt(dsq);
    inv_sig = shared_rcp(sig);
    const double rd = shared_rcp(dij);
    dvij = div_by(1.0 - div_by(dij, sig, inv_sig), sig, inv_sig);
    Fx = div_by(dDx * dvij, dij, rd);
    Fy = div_by(dDy * dvij, dij, rd);
  }
  o.fx = Fx;
  o.fy = Fy;
  o.tp = s * nxA * Fy - s * nyA * Fx;
  o.tq = t * nyB * Fx - t * nxB * Fy;
  if (SE && FAST) {
    const double CxA = s * nxA - 0.5 * dDx, CyA = s * nyA - 0.5 * dDy;
    const double CxB = t * nxB + 0.5 * dDx;
    const double CyB = (virial ? t * nyB : t * nxB) + 0.5 * dDy;
    const double gx = Fx * inv_LL, gy = Fy * inv_LL;
    o.e = dvij * sig * (1.0 - dij * iv.sig) * inv_two_n;
    if (!virial) {  // the reference's slips, as below
      o.pxx = gx * (CxA - CxB) - gy * CxB;
      o.pyy = gy * (CyA - CyB);
      o.pxy = gy * CxA;
      o.pyx = gx * (CyA - CyB);
    } else {
      o.pxx = gx * (CxA - CxB);
      o.pyy = gy * (CyA - CyB);
      o.pxy = gy * (CxA - CxB);
      o.pyx = gx * (CyA - CyB);
    }
  } else if (SE) {
    const double LL = Lx * Ly, rLL = shared_rcp(LL);
    double CxA = s * nxA - 0.5 * dDx;
    double CyA = s * nyA - 0.5 * dDy;
    double CxB = t * nxB + 0.5 * dDx;
    o.e = dvij * sig * (1.0 - div_by(dij, sig, inv_sig)) / two_n;
    if (!virial) {
      // the reference's accumulation, slips included: CyB is built from nxB,
      // one Pxy term lands in Pxx, and Pxy misses its B arm.
      double CyB = t * nxB + 0.5 * dDy;
      o.pxx = div_by(Fx * CxA, LL, rLL) - div_by(Fx * CxB, LL, rLL) - div_by(Fy * CxB, LL, rLL);
      o.pyy = div_by(Fy * CyA, LL, rLL) - div_by(Fy * CyB, LL, rLL);
      o.pxy = div_by(Fy * CxA, LL, rLL);
      o.pyx = div_by(Fx * CyA, LL, rLL) - div_by(Fx * CyB, LL, rLL);
    } else {
      double CyB = t * nyB + 0.5 * dDy;
      o.pxx = div_by(Fx * CxA, LL, rLL) - div_by(Fx * CxB, LL, rLL);
      o.pyy = div_by(Fy * CyA, LL, rLL) - div_by(Fy * CyB, LL, rLL);
      o.pxy = div_by(Fy * CxA, LL, rLL) - div_by(Fy * CxB, LL, rLL);
      o.pyx = div_by(Fx * CyA, LL, rLL) - div_by(Fx * CyB, LL, rLL);
    }
  }
  return true;
}

// Approximate quotient, reciprocal and reciprocal square root of normal numbers: those of
// __fdividef and rsqrtf without the scaling around subnormal operands, about a dozen
// instructions a pair.
__device__ __forceinline__ float rcp_fast(float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}
__device__ __forceinline__ float div_fast(float x, float y) { return x * rcp_fast(y); }
__device__ __forceinline__ float rsqrt_fast(float y) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}
// Cell offset 1 - code of a mixed list entry as a float: code is the low two bits of c.
// (8388608 + code is exact; a conversion would take the slow pipe)
__device__ __forceinline__ float cell_offset(unsigned c) {
  return 8388609.f - __uint_as_float(0x4b000000u | (c & 3u));
}

struct PairF32 {
  float fx, fy, tp, tq;
  float ov;                      // overlap 1 - d/sigma
  float cxa, cya, cxb, cyb;      // contact arms (virial or reference form)
};

// dX, dY: displacement P - Q already reduced to the minimum image (FP32);
// a = |u_A|^2 and c = |u_B|^2 are the squared half shaft lengths.
// Either particle may be A, except where one of the two is a disc and the other a rod: the
// reference's rule then depends on which has the lower index (its "p").  DISCS, q_first (B has
// the lower index, looked at only for such a pair): the closest point on the rod B where the
// disc is A, the -1 end of the rod A where the disc is B.
template <bool SE, bool DISCS = false>
__device__ __forceinline__ bool pair_fp32(float dX, float dY, float nxA, float nyA, float a,
                                          float nxB, float nyB, float c, float sig, float gamma,
                                          bool virial, PairF32& o, bool q_first = false) {
  dX = fmaf(gamma, dY, dX);
  float b = -(nxA * nxB + nyA * nyB);
  float d = nxA * dX + nyA * dY;
  float e = -(nxB * dX + nyB * dY);
  // Unclamped spine parameter of Q.  The reference's (b d - a e)/(a c - b^2) is,
  // by the Binet-Cauchy identity, cross(u_A, D)/cross(u_A, u_B); the cross-product
  // form keeps FP32 accurate for nearly parallel spines, where a c - b^2 cancels.
  // Exactly parallel spines give 0/0 in the reference, which its clamp turns into
  // t = -1; the same value is used here.
  float w = nyA * nxB;
  float uxv = fmaf(nxA, nyB, -w) + fmaf(-nyA, nxB, w);  // cross(u_A, u_B), error-compensated
  float w2 = nyA * dX;
  float uxD = fmaf(nxA, dY, -w2) + fmaf(-nyA, dX, w2);  // cross(u_A, D)
  float t = uxv == 0.f ? -1.f : fminf(fmaxf(div_fast(uxD, uxv), -1.f), 1.f);
  float s = -div_fast(b * t + d, a);
  float sarg = fabsf(s);
  s = fminf(fmaxf(s, -1.f), 1.f);
  if (sarg > 1.f) t = fminf(fmaxf(-div_fast(b * s + e, c), -1.f), 1.f);
  if (DISCS && q_first) {
    if (a == 0.f)
      t = fminf(fmaxf(-div_fast(e, c), -1.f), 1.f);
    else
      s = -1.f;
  }
  float dDx = dX + s * nxA - t * nxB;
  float dDy = dY + s * nyA - t * nyB;
  float dsq = dDx * dDx + dDy * dDy;
  if (!(dsq < sig * sig)) return false;
  float inv_d = rsqrt_fast(dsq);
  float inv_sig = rcp_fast(sig);
  float ov = 1.f - dsq * inv_d * inv_sig;   // 1 - d/sigma
  float f = ov * inv_sig * inv_d;           // (1 - d/sigma)/(sigma d)
  float Fx = dDx * f, Fy = dDy * f;
  o.fx = Fx;
  o.fy = Fy;
  o.tp = s * (nxA * Fy - nyA * Fx);
  o.tq = t * (nyB * Fx - nxB * Fy);
  if (SE) {
    o.ov = ov;
    o.cxa = s * nxA - 0.5f * dDx;
    o.cya = s * nyA - 0.5f * dDy;
    o.cxb = t * nxB + 0.5f * dDx;
    o.cyb = (virial ? t * nyB : t * nxB) + 0.5f * dDy;
  }
  return true;
}

constexpr float kMinNormal = 1.17549435e-38f;  // the smallest normal FP32 number

// Conservative FP32 screen: false only when the two spines (P at the origin, Q at
// -D in the sheared, minimum-image frame) are certainly farther apart than sig.
// The closest-point parameters come from the cross-product form; an error in them
// only moves the evaluated point pair along the spines, which can only raise the
// distance by the spines' misalignment angle times their length, and both that and
// the FP32 rounding of the distance stay far below the 1e-4 relative margin.  Both
// contact rules need the minimum distance below sig for any contact.  A spine P whose
// squared length is no normal number is a point (a disc), and the closest point to it is
// looked for on Q (as past an end of P): the first formula, which looks along P, says nothing
// about Q then.
__device__ __forceinline__ bool may_touch_fp32(float dX, float dY, float nxA, float nyA,
                                               float nxB, float nyB, float sig) {
  float a = fmaf(nxA, nxA, nyA * nyA), c = fmaf(nxB, nxB, nyB * nyB);
  float b = -(nxA * nxB + nyA * nyB);
  float d = nxA * dX + nyA * dY;
  float e = -(nxB * dX + nyB * dY);
  float w = nyA * nxB;
  float uxv = fmaf(nxA, nyB, -w) + fmaf(-nyA, nxB, w);
  float w2 = nyA * dX;
  float uxD = fmaf(nxA, dY, -w2) + fmaf(-nyA, dX, w2);
  float t = uxv == 0.f ? -1.f : fminf(fmaxf(div_fast(uxD, uxv), -1.f), 1.f);
  float s = a >= kMinNormal ? -div_fast(b * t + d, a) : 2.f;
  float sarg = fabsf(s);
  s = fminf(fmaxf(s, -1.f), 1.f);
  if (sarg > 1.f && c > 0.f) t = fminf(fmaxf(-div_fast(b * s + e, c), -1.f), 1.f);
  float dDx = dX + s * nxA - t * nxB;
  float dDy = dY + s * nyA - t * nyB;
  float lim = sig * 1.0001f + 1e-5f;
  return dDx * dDx + dDy * dDy < lim * lim;
}

// Spines P + s u_A and Q + t u_B (P - Q = D, lab frame) closer than lim: the
// closest points in FP32 with the cross-product form of the parameter (an error in
// it only moves the evaluated pair along the spines, raising the distance by the
// misalignment angle times the spine length, far below the caller's margin).
__device__ __forceinline__ bool capsules_within(float dX, float dY, float nxA, float nyA,
                                                float nxB, float nyB, float lim) {
  const float a = fmaf(nxA, nxA, nyA * nyA), c = fmaf(nxB, nxB, nyB * nyB);
  const float b = -(nxA * nxB + nyA * nyB);
  const float d = nxA * dX + nyA * dY;
  const float e = -(nxB * dX + nyB * dY);
  const float w = nyA * nxB;
  const float uxv = fmaf(nxA, nyB, -w) + fmaf(-nyA, nxB, w);
  const float w2 = nyA * dX;
  const float uxD = fmaf(nxA, dY, -w2) + fmaf(-nyA, dX, w2);
  float t = uxv == 0.f ? -1.f : fminf(fmaxf(div_fast(uxD, uxv), -1.f), 1.f);
  float s = a >= kMinNormal ? -div_fast(b * t + d, a) : 2.f;  // (a point: see may_touch_fp32)
  const float sarg = fabsf(s);
  s = fminf(fmaxf(s, -1.f), 1.f);
  if (sarg > 1.f && c > 0.f) t = fminf(fmaxf(-div_fast(b * s + e, c), -1.f), 1.f);
  const float x = dX + s * nxA - t * nxB, y = dY + s * nyA - t * nyB;
  return x * x + y * y < lim * lim;
}

// ---- two-point contacts (src/cuda/2point_dynamics.cu:385-546, euler_est_2p) ----
//
// For nearly parallel overlapping spines the single closest-point pair jumps from
// one end of the overlap to the other as the relative angle changes sign, which
// puts a cusp in the energy at alignment.  The reference's jamming code adds a
// second contact at the other end of the overlap (the closer of two candidates),
// each contact carrying its own harmonic overlap energy.  These functions return
// the spine parameters of both contacts in the reference's case analysis; has2 is
// false when the second candidate coincides with the first.
template <class T>
struct Contacts2 {
  T s1, t1, s2, t2;
  bool has2;
};

template <bool FAST = false>
__device__ __forceinline__ Contacts2<double> contacts2_fp64(double a, double b, double c, double d,
                                                            double e, double delta, double dX,
                                                            double dY, double nxA, double nyA,
                                                            double nxB, double nyB,
                                                            const Recip64& iv) {
  double s1, t1, s2, t2, s3, t3;
  if (delta <= 0) {
    s1 = clamp_one(qdiv<FAST>(-(b + d), a, iv.a));
    s2 = clamp_one(qdiv<FAST>(-(d - b), a, iv.a));
    if (abs_bits(s1) == kBitsOne)
      t1 = clamp_one(qdiv<FAST>(-(b * s1 + e), c, iv.c));
    else if (b < 0)
      t1 = clamp_one(qdiv<FAST>(-(b + e), c, iv.c));
    else
      t1 = clamp_one(qdiv<FAST>(-(e - b), c, iv.c));
    if (abs_bits(s2) == kBitsOne)
      t2 = clamp_one(qdiv<FAST>(-(b * s2 + e), c, iv.c));
    else if (b < 0)
      t2 = clamp_one(qdiv<FAST>(-(e - b), c, iv.c));
    else
      t2 = clamp_one(qdiv<FAST>(-(b + e), c, iv.c));
    s3 = s2;
    t3 = t2;
  } else {
    t1 = clamp_one(FAST ? (b * d - a * e) * iv.delta : (b * d - a * e) / delta);
    s1 = qdiv<FAST>(-(b * t1 + d), a, iv.a);
    bool end = reaches_one(s1);
    s1 = clamp_one(s1);
    if (end) {
      t1 = clamp_one(qdiv<FAST>(-(b * s1 + e), c, iv.c));
      s2 = -s1;
      t2 = qdiv<FAST>(-(b * s2 + e), c, iv.c);
      const bool out = beyond_one(t2);
      t2 = clamp_one(t2);
      if (out) {
        s2 = clamp_one(qdiv<FAST>(-(b * t2 + d), a, iv.a));
        s3 = s2;
        t3 = t2;
      } else {
        t3 = b < 0 ? -s1 : s1;
        s3 = qdiv<FAST>(-(b * t3 + d), a, iv.a);
        end = reaches_one(s3);
        s3 = clamp_one(s3);
        if (end) t3 = clamp_one(qdiv<FAST>(-(b * s3 + e), c, iv.c));
      }
    } else {
      t2 = -t1;
      s2 = qdiv<FAST>(-(b * t2 + d), a, iv.a);
      end = beyond_one(s2);
      s2 = clamp_one(s2);
      if (end) {
        t2 = clamp_one(qdiv<FAST>(-(b * s2 + e), c, iv.c));
        s3 = s2;
        t3 = t2;
      } else {
        s3 = b < 0 ? -t1 : t1;
        t3 = qdiv<FAST>(-(b * s3 + e), c, iv.c);
        const bool out = reaches_one(t3);
        t3 = clamp_one(t3);
        if (out) s3 = clamp_one(qdiv<FAST>(-(b * t3 + d), a, iv.a));
      }
    }
  }
  Contacts2<double> r;
  r.s1 = s1;
  r.t1 = t1;
  r.has2 = (s1 != s2 && t1 != t2);
  if (r.has2 && s3 != s1 && s3 != s2) {
    double x2 = dX + s2 * nxA - t2 * nxB, y2 = dY + s2 * nyA - t2 * nyB;
    double x3 = dX + s3 * nxA - t3 * nxB, y3 = dY + s3 * nyA - t3 * nyB;
    if (x3 * x3 + y3 * y3 < x2 * x2 + y2 * y2) {
      s2 = s3;
      t2 = t3;
    }
  }
  r.s2 = s2;
  r.t2 = t2;
  return r;
}

// One harmonic contact at spine parameters (s, t); accumulates into o (no SE arms
// beyond the virial form: the two-point model is the reference's jamming path).
template <bool SE, bool FAST = false>
__device__ __forceinline__ bool contact_fp64(double dX, double dY, double s, double t, double nxA,
                                             double nyA, double nxB, double nyB, double sig,
                                             double LL, double two_n, PairF64& o,
                                             double inv_sig = 0.0, double inv_LL = 0.0,
                                             double inv_two_n = 0.0) {
  double dDx = dX + s * nxA - t * nxB;
  double dDy = dY + s * nyA - t * nyB;
  double dsq = dDx * dDx + dDy * dDy;
  if (!less_square(dsq, sig * sig)) return false;
  double dij, dvij, Fx, Fy;
  if (FAST) {
    const double rs = rsqrt(dsq);
    dij = dsq * rs;
    dvij = (1.0 - dij * inv_sig) * inv_sig;
    Fx = dDx * (dvij * rs);
    Fy = dDy * (dvij * rs);
  } else {
    dij = sqrt(dsq);
    const double rd = shared_rcp(dij);
    dvij = div_by(1.0 - div_by(dij, sig, inv_sig), sig, inv_sig);
    Fx = div_by(dDx * dvij, dij, rd);
    Fy = div_by(dDy * dvij, dij, rd);
  }
  o.fx += Fx;
  o.fy += Fy;
  o.tp += s * nxA * Fy - s * nyA * Fx;
  o.tq += t * nyB * Fx - t * nxB * Fy;
  if (SE && FAST) {
    const double CxA = s * nxA - 0.5 * dDx, CyA = s * nyA - 0.5 * dDy;
    const double CxB = t * nxB + 0.5 * dDx, CyB = t * nyB + 0.5 * dDy;
    const double gx = Fx * inv_LL, gy = Fy * inv_LL;
    o.e += dvij * sig * (1.0 - dij * inv_sig) * inv_two_n;
    o.pxx += gx * (CxA - CxB);
    o.pyy += gy * (CyA - CyB);
    o.pxy += gy * (CxA - CxB);
    o.pyx += gx * (CyA - CyB);
  } else if (SE) {
    double CxA = s * nxA - 0.5 * dDx, CyA = s * nyA - 0.5 * dDy;
    double CxB = t * nxB + 0.5 * dDx, CyB = t * nyB + 0.5 * dDy;
    o.e += dvij * sig * (1.0 - div_by(dij, sig, inv_sig)) / two_n;
    o.pxx += div_by(Fx * CxA, LL, inv_LL) - div_by(Fx * CxB, LL, inv_LL);
    o.pyy += div_by(Fy * CyA, LL, inv_LL) - div_by(Fy * CyB, LL, inv_LL);
    o.pxy += div_by(Fy * CxA, LL, inv_LL) - div_by(Fy * CxB, LL, inv_LL);
    o.pyx += div_by(Fx * CyA, LL, inv_LL) - div_by(Fx * CyB, LL, inv_LL);
  }
  return true;
}

// Two-point contact pair in FP64 (minimum image and Lees-Edwards shift applied
// here, as in pair_fp64).  Stress uses the virial arms.
template <bool SE, bool FAST = false>
__device__ __forceinline__ bool pair2_fp64(double dX, double dY, double nxA, double nyA,
                                           double aP, double nxB, double nyB, double aQ,
                                           double sig, double gamma, double Lx, double Ly,
                                           double two_n, PairF64& o, double inv_aP, double inv_aQ,
                                           double inv_LL = 0.0, double inv_two_n = 0.0) {
  dX = nearest_image(dX, Lx);
  dY = nearest_image(dY, Ly);
  dX += gamma * dY;
  double a = aP * aP;
  double b = -(nxA * nxB + nyA * nyB);
  double c = aQ * aQ;
  double d = nxA * dX + nyA * dY;
  double e = -nxB * dX - nyB * dY;
  double delta = a * c - b * b;
  Recip64 iv{};
  if (FAST) {
    iv = recip64(a, c, delta, sig);
  } else {
    iv.a = inv_aP;
    iv.c = inv_aQ;
    iv.sig = shared_rcp(sig);
    if (SE) inv_LL = shared_rcp(Lx * Ly);
  }
  Contacts2<double> k =
      contacts2_fp64<FAST>(a, b, c, d, e, delta, dX, dY, nxA, nyA, nxB, nyB, iv);
  o.fx = o.fy = o.tp = o.tq = 0.0;
  o.e = o.pxx = o.pyy = o.pxy = o.pyx = 0.0;
  const double LL = Lx * Ly;
  bool hit = contact_fp64<SE, FAST>(dX, dY, k.s1, k.t1, nxA, nyA, nxB, nyB, sig, LL, two_n, o,
                                    iv.sig, inv_LL, inv_two_n);
  if (k.has2)
    hit |= contact_fp64<SE, FAST>(dX, dY, k.s2, k.t2, nxA, nyA, nxB, nyB, sig, LL, two_n, o,
                                  iv.sig, inv_LL, inv_two_n);
  return hit;
}

// Two-point contact pair in FP32 on a displacement already reduced to the minimum
// image (as pair_fp32); the primary parameter uses the cross-product form.
__device__ __forceinline__ bool contact_fp32(float dX, float dY, float s, float t, float nxA,
                                             float nyA, float nxB, float nyB, float sig,
                                             PairF32& o) {
  float dDx = dX + s * nxA - t * nxB;
  float dDy = dY + s * nyA - t * nyB;
  float dsq = dDx * dDx + dDy * dDy;
  if (!(dsq < sig * sig)) return false;
  float inv_d = rsqrt_fast(dsq);
  float inv_sig = rcp_fast(sig);
  float ov = 1.f - dsq * inv_d * inv_sig;
  float f = ov * inv_sig * inv_d;
  float Fx = dDx * f, Fy = dDy * f;
  o.fx += Fx;
  o.fy += Fy;
  o.tp += s * (nxA * Fy - nyA * Fx);
  o.tq += t * (nyB * Fx - nxB * Fy);
  o.ov += ov * ov;  // sum of squared overlaps of the contacts
  // stress: virial arms summed over the contacts, as force-weighted terms
  o.cxa += Fx * (s * nxA - 0.5f * dDx - t * nxB - 0.5f * dDx);
  o.cya += Fy * (s * nyA - 0.5f * dDy - t * nyB - 0.5f * dDy);
  o.cxb += Fy * (s * nxA - 0.5f * dDx - t * nxB - 0.5f * dDx);
  o.cyb += Fx * (s * nyA - 0.5f * dDy - t * nyB - 0.5f * dDy);
  return true;
}

// For the two-point model the PairF32 fields ov, cxa, cya, cxb, cyb hold summed
// quantities: sum ov^2, and the force-weighted virial terms Pxx, Pyy, Pxy, Pyx (before
// the division by the box area).
__device__ __forceinline__ bool pair2_fp32(float dX, float dY, float nxA, float nyA, float a,
                                           float nxB, float nyB, float c, float sig, float gamma,
                                           PairF32& o) {
  dX = fmaf(gamma, dY, dX);
  float b = -(nxA * nxB + nyA * nyB);
  float d = nxA * dX + nyA * dY;
  float e = -(nxB * dX + nyB * dY);
  float w = nyA * nxB;
  float uxv = fmaf(nxA, nyB, -w) + fmaf(-nyA, nxB, w);
  float w2 = nyA * dX;
  float uxD = fmaf(nxA, dY, -w2) + fmaf(-nyA, dX, w2);
  float s1, t1, s2, t2, s3, t3;
  auto cl = [](float v) { return fminf(fmaxf(v, -1.f), 1.f); };
  if (uxv == 0.f) {
    s1 = cl(-div_fast(b + d, a));
    s2 = cl(-div_fast(d - b, a));
    if (fabsf(s1) == 1.f)
      t1 = cl(-div_fast(b * s1 + e, c));
    else
      t1 = cl(b < 0.f ? -div_fast(b + e, c) : -div_fast(e - b, c));
    if (fabsf(s2) == 1.f)
      t2 = cl(-div_fast(b * s2 + e, c));
    else
      t2 = cl(b < 0.f ? -div_fast(e - b, c) : -div_fast(b + e, c));
    s3 = s2;
    t3 = t2;
  } else {
    t1 = cl(div_fast(uxD, uxv));
    s1 = -div_fast(b * t1 + d, a);
    float sarg = fabsf(s1);
    s1 = cl(s1);
    if (sarg >= 1.f) {
      t1 = cl(-div_fast(b * s1 + e, c));
      s2 = -s1;
      t2 = -div_fast(b * s2 + e, c);
      float targ = fabsf(t2);
      t2 = cl(t2);
      if (targ > 1.f) {
        s2 = cl(-div_fast(b * t2 + d, a));
        s3 = s2;
        t3 = t2;
      } else {
        t3 = b < 0.f ? -s1 : s1;
        s3 = -div_fast(b * t3 + d, a);
        sarg = fabsf(s3);
        s3 = cl(s3);
        if (sarg >= 1.f) t3 = cl(-div_fast(b * s3 + e, c));
      }
    } else {
      t2 = -t1;
      s2 = -div_fast(b * t2 + d, a);
      sarg = fabsf(s2);
      s2 = cl(s2);
      if (sarg > 1.f) {
        t2 = cl(-div_fast(b * s2 + e, c));
        s3 = s2;
        t3 = t2;
      } else {
        s3 = b < 0.f ? -t1 : t1;
        t3 = -div_fast(b * s3 + e, c);
        float targ = fabsf(t3);
        t3 = cl(t3);
        if (targ >= 1.f) s3 = cl(-div_fast(b * t3 + d, a));
      }
    }
  }
  o.fx = o.fy = o.tp = o.tq = 0.f;
  o.ov = o.cxa = o.cya = o.cxb = o.cyb = 0.f;
  bool hit = contact_fp32(dX, dY, s1, t1, nxA, nyA, nxB, nyB, sig, o);
  if (s1 != s2 && t1 != t2) {
    if (s3 != s1 && s3 != s2) {
      float x2 = dX + s2 * nxA - t2 * nxB, y2 = dY + s2 * nyA - t2 * nyB;
      float x3 = dX + s3 * nxA - t3 * nxB, y3 = dY + s3 * nyA - t3 * nyB;
      if (x3 * x3 + y3 * y3 < x2 * x2 + y2 * y2) {
        s2 = s3;
        t2 = t3;
      }
    }
    hit |= contact_fp32(dX, dY, s2, t2, nxA, nyA, nxB, nyB, sig, o);
  }
  return hit;
}

// isolated_rotation, src/cpp/strain_dynamics.cpp:174-177
__device__ __forceinline__ double iso_rot64(double RC, double phi) {
  return 0.5 * (1 - RC * cos(2 * phi));
}

__device__ __forceinline__ int wrap_index(int v, int n) {
  return v < 0 ? v + n : (v >= n ? v - n : v);
}

}  // namespace sc
