// FP64 sphere contact law of LIGGGHTS-INL, as device code.
//
//   SurfaceModel<SURFACE_DEFAULT>::surfacesIntersect  src/surface_model_default.h:146-211
//   NormalModel<HERTZ>::surfacesIntersect             src/normal_model_hertz.h:205-408
//   NormalModel<HOOKE>::surfacesIntersect             src/normal_model_hooke.h:230-400
//   TangentialModel<TANGENTIAL_HISTORY>               src/tangential_model_history.h:135-439
//   RollingModel<ROLLING_CDT>                         src/rolling_model_cdt.h:89-167
//
// GB300 has ~1.25 TFLOP/s of FP64, so the law is restated with fewer FP64
// instructions; every change is an algebraic identity and moves results only
// at the rounding level:
//   * Hertz damping: gamma_n = -2 sqrt(5/6) beta sqrt(Sn meff) with
//     Sn = 2 Y sqrt(reff deltan) equals Kn * (reff deltan)^(1/4) with the
//     per-pair constant Kn = -2 sqrt(5/6) beta sqrt(2 Y meff) (likewise Kt
//     with 8 G): one sqrt per contact-step instead of three;
//   * Hooke: kn and gamma_n depend only on the pair (reff, meff, types), so
//     the pow() of the reference is evaluated once per neighbour build;
//   * Coulomb test kt|s| > mu|Fn| on squares; sqrt and division only when
//     the contact slides; shear = -Ft/kt as shear*ratio;
//   * 1/r and 1/|w_roll| as rsqrt;
//   * 4/3 Yeff and 8 Geff from the type table; (cri, crj)/r formed once;
//     the rolling torque folded into the torque products (one rounding
//     fewer).
// The quantities that decide the contact set (rsq, radsum) and the overlap
// deltan = radsum - sqrt(rsq) are formed exactly as in the reference.
#pragma once
#include "dem_device.cuh"

namespace gb300 {

enum { kHertz = 0, kHooke = 1 };

// Per type pair: Yeff, Geff, betaeff, coeffFrict, coeffRollFrict,
// coeffRestLog, and the Hertz stiffness prefactors 4/3 Yeff and 8 Geff
// (formed on the host as the reference forms them inside its law, so kn and
// kt keep their bits).  The table stacks kTypeTables matrices of (nt+1)^2.
constexpr int kTypeTables = 8;

struct TypePair {
  double Y, G, beta, mu, mur, restlog;
  double Y43, G8;
};

__device__ __forceinline__ TypePair load_typepair(const double *__restrict__ params, int nt,
                                                  int it, int jt) {
  const int m = (nt + 1) * (nt + 1);
  const int k = it * (nt + 1) + jt;
  TypePair t;
  t.Y = __ldg(params + k);
  t.G = __ldg(params + m + k);
  t.beta = __ldg(params + 2 * m + k);
  t.mu = __ldg(params + 3 * m + k);
  t.mur = __ldg(params + 4 * m + k);
  t.restlog = __ldg(params + 5 * m + k);
  t.Y43 = __ldg(params + 6 * m + k);
  t.G8 = __ldg(params + 7 * m + k);
  return t;
}

// host side: the two derived matrices from Yeff and Geff
inline void derive_type_tables(int m, double *tab) {
  for (int q = 0; q < m; q++) {
    tab[6 * m + q] = 4. / 3. * tab[q];
    tab[7 * m + q] = 8. * tab[m + q];
  }
}

// Per-pair constants of the normal law.  Hertz: (Kn, Kt) damping prefactors;
// Hooke: (kn, gamma_n) of src/normal_model_hooke.h:272-279.
template <int NORMAL>
__device__ __forceinline__ void contact_consts(const TypePair &tp, double meff, double reff,
                                               double charVel, bool tdamp, double &c0,
                                               double &c1) {
  if (NORMAL == kHertz) {
    const double sqrtFiveOverSix = 0.91287092917527685576161630466800355658790782499663875;
    const double k = -2. * sqrtFiveOverSix * tp.beta;
    c0 = k * sqrt(2. * tp.Y * meff);
    c1 = tdamp ? k * sqrt(8. * tp.G * meff) : 0.0;
  } else {
    const double sqrtval = sqrt(reff);
    const double kn = 16. / 15. * sqrtval * (tp.Y) *
                      pow(15. * meff * charVel * charVel / (16. * sqrtval * tp.Y), 0.2);
    const double lsq = tp.restlog * tp.restlog;
    c0 = kn;
    c1 = sqrt(4. * meff * kn * lsq / (lsq + 9.86960440108935861883 /* M_PI*M_PI */));
  }
}

struct ContactIn {
  double radi, radj, radsum, r, rinv;
  double reff, c0, c1;
  double en[3], d[3];
  double vr[3];          // v_i - v_j
  double wi[3], wj[3];
  double deltan_wall;    // wall: sidata.deltan as passed in (overlap)
};

struct ContactOut {
  double F[3];           // i_forces.delta_F
  double Ti[3];          // i_forces.delta_torque
  double Tj[3];          // j_forces.delta_torque
};

// a > b for doubles that are not negative, on the integer pipe (their bit
// patterns order the same way; a DSETP and the selects behind it hold the FP64
// pipe for 108 cycles per warp).  Unsigned: no a is above a NaN b (a distance),
// whose sign may be either.
__device__ __forceinline__ bool gt_nonneg(double a, double b) {
  return (unsigned long long)__double_as_longlong(a) > (unsigned long long)__double_as_longlong(b);
}

// A key that orders doubles as the comparison does, -0 and +0 alike, for
// comparisons of any sign on the integer pipe.  A NaN lies beyond the infinity
// of its sign: where one may come, key_lt and key_gt say no to it, as the
// comparison does.
__device__ __forceinline__ long long order_key(double x) {
  const long long b = __double_as_longlong(x);
  return b < 0 ? (long long)(0x8000000000000000ull - (unsigned long long)b) : b;
}
constexpr long long kInfKey = 0x7ff0000000000000ll;
// a < b for a's key and a b that may be NaN; a > b for such an a and b's key
__device__ __forceinline__ bool key_lt(long long a, double b) {
  const long long k = order_key(b);
  return a < k && k <= kInfKey;
}
__device__ __forceinline__ bool key_gt(double a, long long b) {
  const long long k = order_key(a);
  return k > b && k <= kInfKey;
}

// shear[3] is the tangential history, updated in place when update_history.
// base: forces and torques of a bonded pair (cohesion bond/nonlinear), which
// replace the normal model's force before the tangential and rolling models
// add theirs (src/contact_models.h:228-238); nullptr otherwise.
template <int NORMAL, bool WALL>
__device__ __forceinline__ void contact_law(const ContactIn &c, const TypePair &tp, double dt,
                                            bool tdamp, bool limitf, bool rolling,
                                            bool update_history, double shear[3], ContactOut &o,
                                            const ContactOut *base = nullptr) {
  const double enx = c.en[0], eny = c.en[1], enz = c.en[2];
  // ---- surface model (sphere kinematics)
  const double vr1 = c.vr[0], vr2 = c.vr[1], vr3 = c.vr[2];
  const double vn = vr1 * enx + vr2 * eny + vr3 * enz;
  const double vt1 = vr1 - vn * enx;
  const double vt2 = vr2 - vn * eny;
  const double vt3 = vr3 - vn * enz;
  const double deltan = __dadd_rn(c.radsum, -c.r);
  const double dx = c.d[0], dy = c.d[1], dz = c.d[2];
  double wr1, wr2, wr3, cri, crj = 0.0;
  if (WALL) {
    cri = c.radi - 0.5 * c.deltan_wall;
    const double cr = cri * c.rinv;
    wr1 = cr * c.wi[0];
    wr2 = cr * c.wi[1];
    wr3 = cr * c.wi[2];
  } else {
    cri = c.radi - 0.5 * deltan;
    crj = c.radj - 0.5 * deltan;
    const double ai = cri * c.rinv, aj = crj * c.rinv;
    wr1 = ai * c.wi[0] + aj * c.wj[0];
    wr2 = ai * c.wi[1] + aj * c.wj[1];
    wr3 = ai * c.wi[2] + aj * c.wj[2];
  }
  const double vtr1 = vt1 - (dz * wr2 - dy * wr3);
  const double vtr2 = vt2 - (dx * wr3 - dz * wr1);
  const double vtr3 = vt3 - (dy * wr1 - dx * wr2);

  // ---- normal model
  double kn, kt, gamman, gammat;
  if (NORMAL == kHertz) {
    // sqrt(reff*deltan) and its square root from two reciprocal square
    // roots (x^-1/2, then (x^-1/2)^-1/2 = x^1/4): within an ulp or two of
    // the correctly rounded sqrt, with fewer FP64 instructions and no divide
    // (zero for a contact at zero overlap, as sqrt(0) gives)
    const double xr = c.reff * deltan;
    const bool pos = __double_as_longlong(xr) > 0;  // (on the integer pipe)
    const double rs = rsqrt(pos ? xr : 1.0);
    const double sqrtval = pos ? xr * rs : 0.0;
    const double q = pos ? rsqrt(rs) : 0.0;
    kn = tp.Y43 * sqrtval;
    kt = tp.G8 * sqrtval;
    gamman = c.c0 * q;
    gammat = c.c1 * q;
  } else {
    kn = c.c0;
    kt = kn;
    gamman = c.c1;
    gammat = tdamp ? gamman : 0.0;
  }
  double Fn = kn * deltan - gamman * vn;
  if (limitf && Fn < 0.0) Fn = 0.0;

  // ---- tangential history
  double s0 = shear[0], s1 = shear[1], s2 = shear[2];
  if (update_history) {
    s0 += vtr1 * dt;
    s1 += vtr2 * dt;
    s2 += vtr3 * dt;
    const double rsht = s0 * enx + s1 * eny + s2 * enz;
    s0 -= rsht * enx;
    s1 -= rsht * eny;
    s2 -= rsht * enz;
  }
  double Ft1, Ft2, Ft3;
  const double ss = s0 * s0 + s1 * s1 + s2 * s2;
  const double Ft_friction = tp.mu * fabs(Fn);
  const double kt2ss = kt * kt * ss;
  if (gt_nonneg(kt2ss, Ft_friction * Ft_friction)) {
    // sliding (ss > 0 here): cap the spring force at mu|Fn|;
    // mu|Fn| / (kt |shear|) with one reciprocal square root, no divide
    const double ratio = Ft_friction * rsqrt(kt2ss);
    Ft1 = -(kt * s0) * ratio;
    Ft2 = -(kt * s1) * ratio;
    Ft3 = -(kt * s2) * ratio;
    if (update_history) {
      s0 *= ratio;
      s1 *= ratio;
      s2 *= ratio;
    }
  } else {
    Ft1 = -(kt * s0) - gammat * vtr1;
    Ft2 = -(kt * s1) - gammat * vtr2;
    Ft3 = -(kt * s2) - gammat * vtr3;
  }
  if (update_history) {
    shear[0] = s0;
    shear[1] = s1;
    shear[2] = s2;
  }
  const double tor1 = eny * Ft3 - enz * Ft2;
  const double tor2 = enz * Ft1 - enx * Ft3;
  const double tor3 = enx * Ft2 - eny * Ft1;
  // rolling friction, constant directional torque: rt, taken from Ti and
  // given to Tj (folded into their products below)
  double rt1 = 0., rt2 = 0., rt3 = 0.;
  if (rolling) {
    double w1, w2, w3;
    if (WALL) {
      w1 = wr1;
      w2 = wr2;
      w3 = wr3;
    } else {
      w1 = c.wi[0] - c.wj[0];
      w2 = c.wi[1] - c.wj[1];
      w3 = c.wi[2] - c.wj[2];
    }
    const double wsq = w1 * w1 + w2 * w2 + w3 * w3;
    if (__double_as_longlong(wsq) != 0) {  // wsq > 0 (a sum of squares: +0 or positive)
      const double fac = tp.mur * kn * deltan * c.reff * rsqrt(wsq);
      rt1 = fac * w1;
      rt2 = fac * w2;
      rt3 = fac * w3;
      const double rtd = rt1 * enx + rt2 * eny + rt3 * enz;
      rt1 -= enx * rtd;
      rt2 -= eny * rtd;
      rt3 -= enz * rtd;
    }
  }
  if (base) {
    o.F[0] = base->F[0] + Ft1;
    o.F[1] = base->F[1] + Ft2;
    o.F[2] = base->F[2] + Ft3;
    o.Ti[0] = base->Ti[0] + (-cri * tor1 - rt1);
    o.Ti[1] = base->Ti[1] + (-cri * tor2 - rt2);
    o.Ti[2] = base->Ti[2] + (-cri * tor3 - rt3);
    o.Tj[0] = base->Tj[0] + (-crj * tor1 + rt1);
    o.Tj[1] = base->Tj[1] + (-crj * tor2 + rt2);
    o.Tj[2] = base->Tj[2] + (-crj * tor3 + rt3);
  } else {
    o.F[0] = Fn * enx + Ft1;
    o.F[1] = Fn * eny + Ft2;
    o.F[2] = Fn * enz + Ft3;
    o.Ti[0] = -cri * tor1 - rt1;
    o.Ti[1] = -cri * tor2 - rt2;
    o.Ti[2] = -cri * tor3 - rt3;
    o.Tj[0] = -crj * tor1 + rt1;
    o.Tj[1] = -crj * tor2 + rt2;
    o.Tj[2] = -crj * tor3 + rt3;
  }
}

// a b + c d with one product rounded; written out, so that every kernel that
// inlines a law forms the same bits (which product the compiler rounds depends
// on the code around it)
__device__ __forceinline__ double two_products(double a, double b, double c, double d) {
  return fma(c, d, __dmul_rn(a, b));
}

// contact_law for a pair of spheres without cohesion and rolling friction,
// with the identities that save FP64 instructions (about 110 against 125 per
// entry; each holds the pipe of its SM quarter for 64 cycles, whatever the
// number of active lanes):
//   * the surface velocity from en x (cri wi + crj wj): no 1/r on the radii,
//     the vector sums as chains of fused multiply-adds;
//   * one path for sticking and sliding: the spring of a sliding contact is
//     cut to mu|Fn| (history and force alike), its damping drops out, so a
//     warp with both kinds does not run two force evaluations;
//   * kn*deltan formed once; comparisons of magnitudes on the integer pipe.
// Each moves a result by rounding only.  With rolling friction the general
// law stays (see plane_contact_fast on what CDT makes of a changed rounding).
template <int NORMAL>
__device__ __forceinline__ void pair_law(const ContactIn &c, const TypePair &tp, double dt, bool tdamp, bool limitf,
                                         bool update_history, double shear[3], ContactOut &o) {
  const double ex = c.en[0], ey = c.en[1], ez = c.en[2];
  const double vn = fma(c.vr[2], ez, two_products(c.vr[0], ex, c.vr[1], ey));
  const double deltan = __dadd_rn(c.radsum, -c.r);
  const double cri = c.radi - 0.5 * deltan, crj = c.radj - 0.5 * deltan;
  const double W0 = two_products(cri, c.wi[0], crj, c.wj[0]);
  const double W1 = two_products(cri, c.wi[1], crj, c.wj[1]);
  const double W2 = two_products(cri, c.wi[2], crj, c.wj[2]);
  const double vt0 = fma(-ez, W1, fma(ey, W2, fma(-vn, ex, c.vr[0])));
  const double vt1 = fma(-ex, W2, fma(ez, W0, fma(-vn, ey, c.vr[1])));
  const double vt2 = fma(-ey, W0, fma(ex, W1, fma(-vn, ez, c.vr[2])));

  // ---- normal model (see contact_law)
  double kn, kt, gamman, gammat;
  if (NORMAL == kHertz) {
    const double xr = c.reff * deltan;
    const bool pos = __double_as_longlong(xr) > 0;
    const double rs = rsqrt(pos ? xr : 1.0);
    const double sqrtval = pos ? xr * rs : 0.0;
    const double q = pos ? rsqrt(rs) : 0.0;
    kn = tp.Y43 * sqrtval;
    kt = tp.G8 * sqrtval;
    gamman = c.c0 * q;
    gammat = c.c1 * q;
  } else {
    kn = c.c0;
    kt = kn;
    gamman = c.c1;
    gammat = tdamp ? gamman : 0.0;
  }
  const double knd = kn * deltan;
  double Fn = fma(-gamman, vn, knd);
  if (limitf && Fn < 0.0) Fn = 0.0;

  // ---- tangential history
  double s0 = shear[0], s1 = shear[1], s2 = shear[2];
  if (update_history) {
    s0 = fma(vt0, dt, s0);
    s1 = fma(vt1, dt, s1);
    s2 = fma(vt2, dt, s2);
    const double rsht = fma(s2, ez, two_products(s0, ex, s1, ey));
    s0 = fma(-rsht, ex, s0);
    s1 = fma(-rsht, ey, s1);
    s2 = fma(-rsht, ez, s2);
  }
  const double kt2ss = kt * kt * fma(s2, s2, two_products(s0, s0, s1, s1));
  const double Ff = tp.mu * fabs(Fn);
  if (gt_nonneg(kt2ss, Ff * Ff)) {  // sliding
    const double ratio = Ff * rsqrt(kt2ss);
    s0 *= ratio;
    s1 *= ratio;
    s2 *= ratio;
    gammat = 0.0;
  }
  const double Ft0 = fma(-gammat, vt0, -(kt * s0));
  const double Ft1 = fma(-gammat, vt1, -(kt * s1));
  const double Ft2 = fma(-gammat, vt2, -(kt * s2));
  if (update_history) {
    shear[0] = s0;
    shear[1] = s1;
    shear[2] = s2;
  }
  const double tor0 = two_products(ey, Ft2, -ez, Ft1);
  const double tor1 = two_products(ez, Ft0, -ex, Ft2);
  const double tor2 = two_products(ex, Ft1, -ey, Ft0);
  o.F[0] = fma(Fn, ex, Ft0);
  o.F[1] = fma(Fn, ey, Ft1);
  o.F[2] = fma(Fn, ez, Ft2);
  o.Ti[0] = -cri * tor0;
  o.Ti[1] = -cri * tor1;
  o.Ti[2] = -cri * tor2;
  o.Tj[0] = -crj * tor0;
  o.Tj[1] = -crj * tor1;
  o.Tj[2] = -crj * tor2;
}

// contact_law for a sphere on a plane normal to axis n (sign: the side it is
// on), in the frame (n, t1, t2), cyclic axes: v and w are the velocity and
// spin in that frame, sh the tangential history in t1 and t2 (its normal part
// is zero after every update), F and T the results.  With en = +-e_n the
// vector algebra falls away: about 50 FP64 instructions against 140 for the
// general law.
template <int NORMAL>
__device__ __forceinline__ void plane_law(double sign, double radi, double deltan, const double v[3], const double w[3],
                                          double c0, double c1, const TypePair &tp, double dt, bool tdamp,
                                          bool limitf, bool update_history, double &s1, double &s2,
                                          double F[3], double T[3]) {
  const double vn = sign * v[0];
  const double cri = radi - 0.5 * deltan, cs = sign * cri;
  const double vt1 = fma(-cs, w[2], v[1]), vt2 = fma(cs, w[1], v[2]);
  double kn, kt, gamman, gammat;
  if (NORMAL == kHertz) {
    const double xr = radi * deltan;
    const bool pos = __double_as_longlong(xr) > 0;
    const double rs = rsqrt(pos ? xr : 1.0);
    const double sqrtval = pos ? xr * rs : 0.0;
    const double q = pos ? rsqrt(rs) : 0.0;
    kn = tp.Y43 * sqrtval;
    kt = tp.G8 * sqrtval;
    gamman = c0 * q;
    gammat = c1 * q;
  } else {
    kn = c0;
    kt = kn;
    gamman = c1;
    gammat = tdamp ? gamman : 0.0;
  }
  const double knd = kn * deltan;
  double Fn = fma(-gamman, vn, knd);
  if (limitf && Fn < 0.0) Fn = 0.0;
  if (update_history) {
    s1 = fma(vt1, dt, s1);
    s2 = fma(vt2, dt, s2);
  }
  const double kt2ss = kt * kt * two_products(s1, s1, s2, s2);
  const double Ff = tp.mu * fabs(Fn);
  if (gt_nonneg(kt2ss, Ff * Ff)) {
    const double ratio = Ff * rsqrt(kt2ss);
    s1 *= ratio;
    s2 *= ratio;
    gammat = 0.0;
  }
  const double Ft1 = fma(-gammat, vt1, -(kt * s1)), Ft2 = fma(-gammat, vt2, -(kt * s2));
  F[0] = sign * Fn;
  F[1] = Ft1;
  F[2] = Ft2;
  T[0] = 0.0;
  T[1] = cs * Ft2;
  T[2] = -(cs * Ft1);
}

}  // namespace gb300
