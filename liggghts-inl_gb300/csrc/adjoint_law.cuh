// Reverse mode (vector-Jacobian product) of the Hertz + tangential-history
// contact law for one pair or one primitive-wall contact, as device code.
//
// Forward law: the same equations as contact_law.cuh (NormalModel<HERTZ>,
// TangentialModel<TANGENTIAL_HISTORY>, SurfaceModel<SURFACE_DEFAULT>;
// src/normal_model_hertz.h:205-408, src/tangential_model_history.h:135-439,
// src/surface_model_default.h:146-211), written out in the form the
// adjoint needs:
//   en = d/|d|, deltan = radsum - |d|, vn = vr.en, vt = vr - vn en,
//   cri = ri - deltan/2, crj = rj - deltan/2,
//   wr = (cri wi + crj wj)/|d|, vtr = vt + d x wr,
//   sv = sqrt(reff deltan), q = sqrt(sv), kn = 4/3 Y sv, kt = 8 G sv,
//   gamma_n = K beta sqrt(2 Y meff) q, gamma_t = K beta sqrt(8 G meff) q,
//   Fn = kn deltan - gamma_n vn,
//   s1 = shear + dt vtr, s2 = s1 - (s1.en) en          (update_history)
//   sliding (kt^2 |s2|^2 > (mu|Fn|)^2): Ft = -mu|Fn| s2/|s2|, s3 = (mu|Fn|/kt) s2/|s2|
//   else: Ft = -kt s2 - gamma_t vtr, s3 = s2
//   F = Fn en + Ft, Ti = -cri (en x Ft), Tj = -crj (en x Ft)
// With CDT rolling friction (RollingModel<ROLLING_CDT>, src/rolling_model_cdt.h:
// 89-167): w = wi - wj (walls: wr), rt = mur kn deltan reff w/|w| projected
// off en, Ti -= rt, Tj += rt (w = 0: none).
// For a bonded pair the bond's force replaces Fn en (src/contact_models.h:
// 228-238): F = Ft here, Fn still caps the friction.
// Walls: radsum = reff = ri, meff = mi, no j terms.  Without
// update_history (the setup force pass) s2 = shear.
// The adjoint is exact for this piecewise-smooth law away from its switch
// points (touching/sliding transitions).
#pragma once

namespace gb300 {

// Values of the law that depend on the run's material alone.
struct LawUniform {
  double Y43, G8;   // 4/3 Y, 8 G
  double Kb;        // -2 sqrt(5/6) beta
  double iG8;       // 1/(8 G)
  double i2Y, i2G;  // 1/(2 Y), 1/(2 G)
};

// Values that depend on the pair of spheres (or the sphere at a wall) and the
// material: reff, meff, 1/ri, 1/rj, 1/mi, 1/mj, sqrt(2 Y meff), sqrt(8 G meff).
struct LawPair {
  double reff, meff, iri, irj, imi, imj, sY, sG;
};

struct VjpIn {
  double d[3], vr[3], wi[3], wj[3], sh[3];
  double ri, rj, mi, mj;
  double Y, G, beta, mu, dt;
  bool upd;     // update_history
  bool wall;
  bool bonded;  // a bond (cohesion bond/nonlinear) replaces the normal force
  bool rolling;  // CDT rolling friction with coefficient mur
  double mur;
  bool pre = false;  // pu and pp are filled in (the engine keeps them per run and per list entry);
                     // else the law forms them from the inputs above
  LawUniform pu;
  LawPair pp;
};

struct VjpBar {  // adjoints of the outputs (in) and of the inputs (out)
  double F[3], Ti[3], Tj[3], s3[3];
  double d[3], vr[3], wi[3], wj[3], sh[3];
  double ri, rj, mi, mj, Y, G, beta, mu, mur;
};

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double c[3]) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// On the device the law avoids divisions and square roots (some ten FP64
// instructions each, and every one of them holds the pipe of its SM quarter
// for 64 cycles): reciprocal square roots give a root and its inverse
// together, the comparisons of magnitudes run on the integer pipe, and the
// values of LawUniform and LawPair come from the caller.
__device__ __forceinline__ double law_rsqrt(double x) {
#ifdef __CUDA_ARCH__
  return rsqrt(x);
#else
  return 1.0 / sqrt(x);
#endif
}
__device__ __forceinline__ bool law_gt(double a, double b) {  // a > b, neither negative
#ifdef __CUDA_ARCH__
  return __double_as_longlong(a) > __double_as_longlong(b);
#else
  return a > b;
#endif
}
__device__ __forceinline__ double law_sign(double x) {  // -1, 0 or 1
#ifdef __CUDA_ARCH__
  const long long b = __double_as_longlong(x);
  return (b << 1) == 0 ? 0.0 : (b < 0 ? -1.0 : 1.0);
#else
  return x > 0 ? 1.0 : (x < 0 ? -1.0 : 0.0);
#endif
}

constexpr double kLawK = -2.0 * 0.91287092917527685576161630466800355658790782499663875;

__device__ __forceinline__ LawUniform law_uniform(double Y, double G, double beta) {
  LawUniform u;
  u.Y43 = 4.0 / 3.0 * Y;
  u.G8 = 8.0 * G;
  u.Kb = kLawK * beta;
  u.iG8 = 1.0 / u.G8;
  u.i2Y = 0.5 / Y;
  u.i2G = 0.5 / G;
  return u;
}

// walls: rj and mj are not used
__device__ __forceinline__ LawPair law_pair(bool wall, double ri, double rj, double mi, double mj, double Y,
                                            double G) {
  LawPair p;
  p.reff = wall ? ri : ri * rj / (ri + rj);
  p.meff = wall ? mi : mi * mj / (mi + mj);
  p.iri = 1.0 / ri;
  p.imi = 1.0 / mi;
  p.irj = wall ? 0.0 : 1.0 / rj;
  p.imj = wall ? 0.0 : 1.0 / mj;
  p.sY = sqrt(2.0 * Y * p.meff);
  p.sG = sqrt(8.0 * G * p.meff);
  return p;
}

// The law of the forward kernels.  Its arithmetic stays as it is (what
// LawUniform and LawPair bring are the same values formed earlier): a changed
// rounding of a force moves positions by an ulp, and the gradient divides by
// powers of overlaps that small, so it would change by 1e-8.
struct LawState {
  double r, rinv, en[3], radsum, deltan, vn, vt[3], cri, crj, wsum[3], wr[3], vtr[3];
  double reff, meff, sv, q, kn, kt, c0, c1, gn, gt, Fn, s1[3], rsht, s2[3], ss, Ffr, u, shat[3];
  double Ft[3], tor[3];
  bool slide;
  double rw[3], rwsq, rfac;  // rolling: relative spin, |w|^2, mur kn deltan reff / |w|
};

// ROLL = false compiles the rolling part out (kernels of systems without it)
template <bool ROLL = true>
__device__ __forceinline__ void law_forward(const VjpIn &a, LawState &S, double F[3], double Ti[3],
                                            double Tj[3], double s3[3]) {
  const LawUniform u = a.pre ? a.pu : law_uniform(a.Y, a.G, a.beta);
  const LawPair pp = a.pre ? a.pp : law_pair(a.wall, a.ri, a.rj, a.mi, a.mj, a.Y, a.G);
  const double rsq = dot3(a.d, a.d);
  S.r = sqrt(rsq);
  S.rinv = 1.0 / S.r;
  for (int k = 0; k < 3; k++) S.en[k] = a.d[k] * S.rinv;
  S.radsum = a.wall ? a.ri : a.ri + a.rj;
  S.deltan = S.radsum - S.r;
  S.vn = dot3(a.vr, S.en);
  for (int k = 0; k < 3; k++) S.vt[k] = a.vr[k] - S.vn * S.en[k];
  S.cri = a.ri - 0.5 * S.deltan;
  S.crj = a.wall ? 0.0 : a.rj - 0.5 * S.deltan;
  for (int k = 0; k < 3; k++) {
    S.wsum[k] = S.cri * a.wi[k] + (a.wall ? 0.0 : S.crj * a.wj[k]);
    S.wr[k] = S.wsum[k] * S.rinv;
  }
  double c[3];
  cross3(a.d, S.wr, c);
  for (int k = 0; k < 3; k++) S.vtr[k] = S.vt[k] + c[k];
  S.reff = pp.reff;
  S.meff = pp.meff;
  S.sv = sqrt(S.reff * S.deltan);
  S.q = sqrt(S.sv);
  S.kn = u.Y43 * S.sv;
  S.kt = u.G8 * S.sv;
  S.c0 = u.Kb * pp.sY;
  S.c1 = u.Kb * pp.sG;
  S.gn = S.c0 * S.q;
  S.gt = S.c1 * S.q;
  S.Fn = S.kn * S.deltan - S.gn * S.vn;
  if (a.upd) {
    for (int k = 0; k < 3; k++) S.s1[k] = a.sh[k] + S.vtr[k] * a.dt;
    S.rsht = dot3(S.s1, S.en);
    for (int k = 0; k < 3; k++) S.s2[k] = S.s1[k] - S.rsht * S.en[k];
  } else {
    for (int k = 0; k < 3; k++) S.s1[k] = S.s2[k] = a.sh[k];
    S.rsht = 0.0;
  }
  S.ss = dot3(S.s2, S.s2);
  S.Ffr = a.mu * fabs(S.Fn);
  S.slide = law_gt(S.kt * S.kt * S.ss, S.Ffr * S.Ffr);
  if (S.slide) {
    S.u = sqrt(S.ss);
    for (int k = 0; k < 3; k++) {
      S.shat[k] = S.s2[k] / S.u;
      S.Ft[k] = -S.Ffr * S.shat[k];
      s3[k] = a.upd ? S.Ffr / S.kt * S.shat[k] : a.sh[k];
    }
  } else {
    S.u = 0.0;
    for (int k = 0; k < 3; k++) {
      S.shat[k] = 0.0;
      S.Ft[k] = -S.kt * S.s2[k] - S.gt * S.vtr[k];
      s3[k] = S.s2[k];
    }
  }
  cross3(S.en, S.Ft, S.tor);
  for (int k = 0; k < 3; k++) {
    F[k] = (a.bonded ? 0.0 : S.Fn * S.en[k]) + S.Ft[k];
    Ti[k] = -S.cri * S.tor[k];
    Tj[k] = -S.crj * S.tor[k];
  }
  S.rwsq = 0.0;
  if (ROLL && a.rolling) {
    for (int k = 0; k < 3; k++) S.rw[k] = a.wall ? S.wr[k] : a.wi[k] - a.wj[k];
    S.rwsq = dot3(S.rw, S.rw);
    if (S.rwsq > 0.) {
      S.rfac = a.mur * S.kn * S.deltan * S.reff / sqrt(S.rwsq);
      const double we = dot3(S.rw, S.en);
      for (int k = 0; k < 3; k++) {
        const double rt = S.rfac * (S.rw[k] - we * S.en[k]);
        Ti[k] -= rt;
        Tj[k] += rt;
      }
    }
  }
}

// The forward values that the product needs, with reciprocal square roots for
// the divisions and roots of law_forward.  The overlap is formed as there
// (r correctly rounded): it may be a few ulps of r.
struct LawValues {
  LawUniform u;
  LawPair p;
  double r, rinv, en[3], radsum, deltan, vn, cri, crj, W[3], vtr[3];
  double isv, iq, sv, q, kn, kt, c0, c1, gn, gt, Fn, s1[3], rsht, s2[3], ss, Ffr, iu, Fk, shat[3];
  double Ft[3], tor[3];
  bool slide;
  double rw[3], rwsq, irw, rfac;  // rolling: relative spin, |w|^2, 1/|w|, mur kn deltan reff / |w|
};

// ROLL = false compiles the rolling part out (kernels of systems without it)
template <bool ROLL = true>
__device__ __forceinline__ void law_values(const VjpIn &a, LawValues &S) {
  if (a.pre) {
    S.u = a.pu;
    S.p = a.pp;
  } else {
    S.u = law_uniform(a.Y, a.G, a.beta);
    S.p = law_pair(a.wall, a.ri, a.rj, a.mi, a.mj, a.Y, a.G);
  }
  const double rsq = dot3(a.d, a.d);
  S.rinv = law_rsqrt(rsq);
  S.r = sqrt(rsq);
  for (int k = 0; k < 3; k++) S.en[k] = a.d[k] * S.rinv;
  S.radsum = a.wall ? a.ri : a.ri + a.rj;
  S.deltan = S.radsum - S.r;
  S.vn = dot3(a.vr, S.en);
  S.cri = a.ri - 0.5 * S.deltan;
  S.crj = a.wall ? 0.0 : a.rj - 0.5 * S.deltan;
  for (int k = 0; k < 3; k++) S.W[k] = S.cri * a.wi[k] + (a.wall ? 0.0 : S.crj * a.wj[k]);
  // vt + d x wr with wr = W/|d|
  for (int k = 0; k < 3; k++) {
    const int m = (k + 1) % 3, l = (k + 2) % 3;
    S.vtr[k] = a.vr[k] - S.vn * S.en[k] + S.en[m] * S.W[l] - S.en[l] * S.W[m];
  }
  const double x = S.p.reff * S.deltan;
  S.isv = law_rsqrt(x);
  S.sv = x * S.isv;
  S.iq = law_rsqrt(S.sv);
  S.q = S.sv * S.iq;
  S.kn = S.u.Y43 * S.sv;
  S.kt = S.u.G8 * S.sv;
  S.c0 = S.u.Kb * S.p.sY;
  S.c1 = S.u.Kb * S.p.sG;
  S.gn = S.c0 * S.q;
  S.gt = S.c1 * S.q;
  S.Fn = S.kn * S.deltan - S.gn * S.vn;
  if (a.upd) {
    for (int k = 0; k < 3; k++) S.s1[k] = a.sh[k] + S.vtr[k] * a.dt;
    S.rsht = dot3(S.s1, S.en);
    for (int k = 0; k < 3; k++) S.s2[k] = S.s1[k] - S.rsht * S.en[k];
  } else {
    for (int k = 0; k < 3; k++) S.s1[k] = S.s2[k] = a.sh[k];
    S.rsht = 0.0;
  }
  S.ss = dot3(S.s2, S.s2);
  S.Ffr = a.mu * fabs(S.Fn);
  S.slide = law_gt(S.kt * S.kt * S.ss, S.Ffr * S.Ffr);
  S.iu = S.Fk = 0.0;
  if (S.slide) {
    S.iu = law_rsqrt(S.ss);
    S.Fk = S.Ffr * S.u.iG8 * S.isv;  // mu|Fn|/kt
    for (int k = 0; k < 3; k++) {
      S.shat[k] = S.s2[k] * S.iu;
      S.Ft[k] = -S.Ffr * S.shat[k];
    }
  } else {
    for (int k = 0; k < 3; k++) {
      S.shat[k] = 0.0;
      S.Ft[k] = -S.kt * S.s2[k] - S.gt * S.vtr[k];
    }
  }
  cross3(S.en, S.Ft, S.tor);
  S.rwsq = 0.0;
  if (ROLL && a.rolling) {
    // (a wall's wr = W/|d| has the direction of W, which is all that counts)
    for (int k = 0; k < 3; k++) S.rw[k] = a.wall ? S.W[k] : a.wi[k] - a.wj[k];
    S.rwsq = dot3(S.rw, S.rw);
    if (S.rwsq > 0.) {
      S.irw = law_rsqrt(S.rwsq);
      S.rfac = a.mur * S.kn * S.deltan * S.p.reff * S.irw;
    }
  }
}

// b.F/Ti/Tj/s3 hold the output adjoints; fills the input adjoints of b.
template <bool ROLL = true>
__device__ void law_vjp(const VjpIn &a, VjpBar &b) {
  LawValues S;
  law_values<ROLL>(a, S);
  double torb[3], enb[3], Ftb[3];
  // rolling friction (the last forward operation): rt = rfac (w - (w.en) en)
  double rwb[3] = {0., 0., 0.}, renb[3] = {0., 0., 0.};
  double knb_r = 0.0, deltanb_r = 0.0, reffb_r = 0.0, murb = 0.0;
  if (ROLL && a.rolling && S.rwsq > 0.) {
    double rtb[3], pw[3];
    const double we = dot3(S.rw, S.en);
    for (int k = 0; k < 3; k++) {
      rtb[k] = b.Tj[k] - b.Ti[k];
      pw[k] = S.rw[k] - we * S.en[k];
    }
    const double facb = dot3(rtb, pw), rte = dot3(rtb, S.en);
    const double iw = S.irw, fw = facb * S.rfac * iw * iw;
    for (int k = 0; k < 3; k++) {
      rwb[k] = S.rfac * (rtb[k] - rte * S.en[k]) - fw * S.rw[k];
      renb[k] = -S.rfac * (rte * S.rw[k] + we * rtb[k]);
    }
    const double fi = facb * iw;
    murb = fi * S.kn * S.deltan * S.p.reff;
    knb_r = fi * a.mur * S.deltan * S.p.reff;
    deltanb_r = fi * a.mur * S.kn * S.p.reff;
    reffb_r = fi * a.mur * S.kn * S.deltan;
  }
  for (int k = 0; k < 3; k++) torb[k] = -S.cri * b.Ti[k] - S.crj * b.Tj[k];
  double crib = -dot3(S.tor, b.Ti), crjb = -dot3(S.tor, b.Tj);
  cross3(S.Ft, torb, enb);
  if (ROLL)
    for (int k = 0; k < 3; k++) enb[k] += renb[k];
  cross3(torb, S.en, Ftb);
  double Fnb = a.bonded ? 0.0 : dot3(b.F, S.en);
  for (int k = 0; k < 3; k++) {
    enb[k] += a.bonded ? 0.0 : S.Fn * b.F[k];
    Ftb[k] += b.F[k];
  }
  double s2b[3], vtrb[3] = {0., 0., 0.};
  double ktb, gtb = 0.0, mub = 0.0, shb_direct[3] = {0., 0., 0.};
  if (S.slide) {
    const double s3dot = a.upd ? dot3(b.s3, S.shat) : 0.0;
    const double ikt = S.u.iG8 * S.isv;
    const double Ffrb = -dot3(Ftb, S.shat) + s3dot * ikt;
    ktb = -(S.Fk * ikt) * s3dot;
    double shatb[3];
    for (int k = 0; k < 3; k++) shatb[k] = -S.Ffr * Ftb[k] + (a.upd ? S.Fk * b.s3[k] : 0.0);
    const double sd = dot3(shatb, S.shat);
    for (int k = 0; k < 3; k++) s2b[k] = (shatb[k] - sd * S.shat[k]) * S.iu;
    mub = fabs(S.Fn) * Ffrb;
    Fnb += a.mu * law_sign(S.Fn) * Ffrb;
    if (!a.upd)
      for (int k = 0; k < 3; k++) shb_direct[k] = b.s3[k];
  } else {
    for (int k = 0; k < 3; k++) {
      s2b[k] = -S.kt * Ftb[k] + b.s3[k];
      vtrb[k] = -S.gt * Ftb[k];
    }
    ktb = -dot3(S.s2, Ftb);
    gtb = -dot3(S.vtr, Ftb);
  }
  if (a.upd) {
    const double s2e = dot3(s2b, S.en);
    for (int k = 0; k < 3; k++) {
      const double s1b = s2b[k] - s2e * S.en[k];
      enb[k] += -S.rsht * s2b[k] - s2e * S.s1[k];
      b.sh[k] = s1b;
      vtrb[k] += a.dt * s1b;
    }
  } else {
    for (int k = 0; k < 3; k++) b.sh[k] = s2b[k] + shb_direct[k];
  }
  const double knb = Fnb * S.deltan + knb_r;
  double deltanb = Fnb * S.kn + deltanb_r;
  const double gnb = -Fnb * S.vn;
  double vnb = -Fnb * S.gn;
  const double c0b = gnb * S.q, c1b = gtb * S.q, qb = gnb * S.c0 + gtb * S.c1;
  const double cY = c0b * S.c0, cG = c1b * S.c1;
  const double svb = S.u.Y43 * knb + S.u.G8 * ktb + 0.5 * qb * S.iq;
  const double wb = 0.5 * svb * S.isv;
  const double reffb = wb * S.deltan + reffb_r;
  deltanb += wb * S.p.reff;
  b.beta = kLawK * (c0b * S.p.sY + c1b * S.p.sG);
  b.Y = 4.0 / 3.0 * S.sv * knb + cY * S.u.i2Y;
  b.G = 8.0 * S.sv * ktb + cG * S.u.i2G;
  // vtr = vr - vn en + en x W
  double Wb[3], t[3];
  cross3(vtrb, S.en, Wb);
  cross3(S.W, vtrb, t);
  if (ROLL && a.wall)  // rolling of a wall contact spins with W
    for (int k = 0; k < 3; k++) Wb[k] += rwb[k];
  for (int k = 0; k < 3; k++) {
    b.wi[k] = S.cri * Wb[k] + (ROLL && !a.wall ? rwb[k] : 0.0);
    b.wj[k] = a.wall ? 0.0 : S.crj * Wb[k] - (ROLL ? rwb[k] : 0.0);
  }
  crib += dot3(a.wi, Wb);
  if (!a.wall) crjb += dot3(a.wj, Wb);
  deltanb += -0.5 * (crib + (a.wall ? 0.0 : crjb));
  vnb -= dot3(S.en, vtrb);
  for (int k = 0; k < 3; k++) {
    b.vr[k] = vtrb[k] + vnb * S.en[k];
    enb[k] += t[k] - S.vn * vtrb[k] + vnb * a.vr[k];
  }
  b.ri = crib + deltanb;
  b.rj = a.wall ? 0.0 : crjb + deltanb;
  const double meffb = 0.5 * (cY + cG);  // times 1/meff
  if (a.wall) {
    b.ri += reffb;
    b.mi = meffb * S.p.imi;
    b.mj = 0.0;
  } else {
    // d reff/d ri = (reff/ri)^2; d meff/d mi / meff = meff/mi^2
    const double ei = S.p.reff * S.p.iri, ej = S.p.reff * S.p.irj;
    b.ri += reffb * ei * ei;
    b.rj += reffb * ej * ej;
    const double mm = meffb * S.p.meff;
    b.mi = mm * S.p.imi * S.p.imi;
    b.mj = mm * S.p.imj * S.p.imj;
  }
  // en = d/|d|, deltan = radsum - |d|
  const double ee = dot3(S.en, enb), db = -deltanb - S.rinv * ee;
  for (int k = 0; k < 3; k++) b.d[k] = S.rinv * enb[k] + db * S.en[k];
  b.mu = mub;
  b.mur = murb;
}

}  // namespace gb300
