// tmk_fault.cuh -- FP64 fault-face friction solves, boundary-data updates and
// the Drucker-Prager return, one face (or cell) per thread.
//
// Friction laws follow ibcLinElast/RSIBCF.ChF (RSFAULTBCF, RSNEWTON, RSSETBND)
// and ibcLinElast/SWIBCF.ChF (SWFAULTBCF, SWSETBND) with the reference's
// operation order; plasticity follows srcLinElast/PlasticPhysicsF.ChF.
#pragma once
#include "tmk_device.cuh"

namespace tmk {

TMK_D double gaussian(double w, double r) { double q = r / w; return exp(-(0.5 * (q * q))); }
TMK_D double smoothfn(double w, double r) {
  if (r >= w) return 0.0;
  if (r <= 0) return 1.0;
  return exp(r * r / (r * r - w * w));
}
TMK_D double boxcar(double w, double r) { return (r >= w) ? 0.0 : 1.0; }

constexpr int RS_IMAX = 100;

// Rate-and-state parameters of one fault face: the scenario's a, b, L, or the
// face's own when the level carries per-face friction (an extension: the
// reference varies only a and Vw along x, by the linear ramp that RSSETF sets,
// ibcLinElast/RSIBCF.ChF:8-55).
struct RSFace { double a, b, L; };
TMK_D RSFace rs_face(const DevParams& P, const double* fric, int off, int stride) {
  if (!fric) return RSFace{P.rs_a, P.rs_b, P.rs_L};
  return RSFace{fric[off], fric[off + stride], fric[off + 2 * stride]};
}

// RSNEWTON (ibcLinElast/RSIBCF.ChF:336-401): bracketed Newton on the slip rate
// for  sn a asinh(V exp(psi/a)/(2V0)) + Zs/2 V = phi  on (0, phi/Zs).  The loop
// is bounded by IMAX; returns the iterations used.  halve: the first iterations,
// known to halve V without a look at the function, done at once (same bits).
// climb: the root lies beyond phi/Zs; f and f' fall towards that end, so once
// f(end) / f'(V) reaches past it every further step only halves the distance.
TMK_D int rs_newton(const DevParams& P, double phi, double psi, double sn, double c_rs_a, double& V,
                    double& tau, int halve = 0, bool climb = false) {
  const double atolG = 2.220446049250313e-16 * 1e4;
  double Vmin = 0.0, Vmax = phi / P.Zs;
  if (V < Vmin || V > Vmax) V = (Vmin + Vmax) / 2.0;
  if (halve > 0) { V = V * __hiloint2double((1023 - halve) << 20, 0); Vmax = 2.0 * V; }
  double alpha = sn * c_rs_a;
  double beta = exp(psi / c_rs_a) / (2.0 * P.rs_V0);
  double eta = 0.5 * P.Zs;
  double fval = alpha * asinh(beta * V) + eta * V - phi;
  const double fend = climb ? alpha * asinh(beta * Vmax) + eta * Vmax - phi : 0.0;
  climb = fend < -1e-6;
  int it;
  for (it = halve + 1; it <= RS_IMAX; ++it) {
    if (fval < 0) Vmin = V; else Vmax = V;
    double dfval = alpha * beta / sqrt((beta * beta) * (V * V) + 1) + eta;
    if (climb && -0.999 * fend > (Vmax - V) * dfval) {
      for (; it <= RS_IMAX; ++it) V = (V + Vmax) / 2.0;
      break;
    }
    double dV = -fval / dfval;
    V = V + dV;
    if (V < Vmin || V > Vmax) V = (Vmin + Vmax) / 2.0;
    fval = alpha * asinh(beta * V) + eta * V - phi;
    if (fabs(fval) <= atolG) break;
    if (fabs(dV) <= 0.0) break;
  }
  tau = alpha * asinh(beta * V);
  return it;
}

// RSFAULTBCF (ibcLinElast/RSIBCF.ChF:158-323) at one fault face; Wi, Wg: 22 comps.
TMK_D int rs_fault(const DevParams& P, const RSFace& fr, const double* Wi, double psi, double x, double* Wg) {
  const double Zs = P.Zs, Zp = P.Zp, lam = P.lam, G = P.G;
  double vx1 = Wi[0], vy1 = Wi[1], vz1 = Wi[2], sxx1 = Wi[3], syy1 = Wi[4], szz1 = Wi[5];
  double sxy1 = Wi[6], sxz1 = Wi[7], syz1 = Wi[8];
  double vx2 = Wi[11], vy2 = Wi[12], vz2 = Wi[13], sxx2 = Wi[14], syy2 = Wi[15], szz2 = Wi[16];
  double sxy2 = Wi[17], sxz2 = Wi[18], syz2 = Wi[19];
  double wpxy1 = -sxy1 - Zs * vx1;
  double wpyy1 = -syy1 - Zp * vy1;
  double wpxy2 = sxy2 - Zs * vx2;
  double wpyy2 = syy2 - Zp * vy2;
  double wpyz1 = 0.0, wpyz2 = 0.0;
  (void)syz1; (void)syz2;
  double tau_xy_0 = P.rs_nsig * gaussian(P.rs_r0, x);
  double tau_yz_0 = 0.0;
  double phi_xy = 0.5 * (wpxy2 - wpxy1) + tau_xy_0;
  double phi_yz = 0.5 * (wpyz2 - wpyz1) + tau_yz_0;
  double phi = sqrt(phi_xy * phi_xy + phi_yz * phi_yz);
  syy1 = -(wpyy1 - wpyy2) / 2.0;
  syy2 = -(wpyy1 - wpyy2) / 2.0;
  vy1 = -(wpyy1 + wpyy2) / 2.0 / Zp;
  vy2 = -(wpyy1 + wpyy2) / 2.0 / Zp;
  double V = sqrt((vx1 - vx2) * (vx1 - vx2) + (vz1 - vz2) * (vz1 - vz2));
  double c_ramp = fmin(1.0, fmax(0.0, (x - P.ramp_x) / P.ramp_w));
  double c_rs_a = fr.a + P.ramp_a * c_ramp;
  double tau;
  int it = rs_newton(P, phi, psi, -syy1, c_rs_a, V, tau);
  sxy1 = (phi_xy / phi) * tau - tau_xy_0;
  syz1 = (phi_yz / phi) * tau - tau_yz_0;
  double Vx = (phi_xy / phi) * V;
  double Vz = (phi_yz / phi) * V;
  vx1 = -(sxy1 + wpxy1) / Zs;
  vz1 = -(syz1 + wpyz1) / Zs;
  double SHF = -(vy1 - syy1) * lam / (lam + 2.0 * G);
  Wg[0] = vx1; Wg[1] = vy1; Wg[2] = vz1;
  Wg[3] = sxx1 + SHF; Wg[4] = syy1; Wg[5] = szz1 + SHF;
  Wg[6] = sxy1; Wg[7] = sxz1; Wg[8] = syz1;
  Wg[9] = 0.0; Wg[10] = 0.0;
  sxy2 = (phi_xy / phi) * tau - tau_xy_0;
  syz2 = (phi_yz / phi) * tau - tau_yz_0;
  vx2 = vx1 - Vx;
  vz2 = vz1 - Vz;
  SHF = -(vy2 - syy2) * lam / (lam + 2.0 * G);
  Wg[11] = vx2; Wg[12] = vy2; Wg[13] = vz2;
  Wg[14] = sxx2 + SHF; Wg[15] = syy2; Wg[16] = szz2 + SHF;
  Wg[17] = sxy2; Wg[18] = sxz2; Wg[19] = syz2;
  Wg[20] = 0.0; Wg[21] = 0.0;
  return it;
}

// RSSETBND (ibcLinElast/RSIBCF.ChF:61-151) for one face, B in/out (11 comps,
// strided).  When `final_` is false only psi is produced (the predictor's
// tmp data, of which the fault solve reads nothing else).  Returns the new
// psi (NaN is reported by the caller; the reference stops there).
TMK_D double rs_setbnd(const DevParams& P, const RSFace& fr, const double* U, double* B, int bstride, double dt,
                       double x, double time, bool final_) {
  double tau_xy_0 = P.rs_nsig * gaussian(P.rs_r0, x);
  double c_ramp = fmin(1.0, fmax(0.0, (x - P.ramp_x) / P.ramp_w));
  double c_rs_a = fr.a + P.ramp_a * c_ramp;
  double c_rs_Vw = P.rs_Vw + P.ramp_Vw * c_ramp;
  double Vx = U[0] - U[11];
  double Vz = U[2] - U[13];
  double V = sqrt(Vx * Vx + Vz * Vz);
  double psi = B[10 * bstride];
  double dPsi;
  if (P.state_law == 1) {
    // aging law (extension), exact at constant V over dt:
    // theta' = theta exp(-x) + dt (1-exp(-x))/x, x = V dt / L
    double xx = V * dt / fr.L;
    double phi1 = (xx > 1e-12) ? -expm1(-xx) / xx : 1.0 - 0.5 * xx;
    double q = (psi - P.rs_f0) / fr.b - xx;
    dPsi = P.rs_f0 + fr.b * log(exp(q) + (P.rs_V0 * dt / fr.L) * phi1);
  } else {
    double f = c_rs_a * asinh(V * exp(psi / c_rs_a) / (2.0 * P.rs_V0));
    double fss = P.rs_f0 - (fr.b - c_rs_a) * log(V / P.rs_V0);
    if (P.rs_fexp > 0.0) {
      double q = V / c_rs_Vw, q2 = q * q, q4 = q2 * q2, q8 = q4 * q4;
      fss = P.rs_fw + (fss - P.rs_fw) / pow(1.0 + q8, 0.125);
    }
    dPsi = psi - dt * (V / fr.L) * (f - fss);
  }
  if (final_) {
    double rt = B[9 * bstride];
    B[0] = Vx;
    B[1 * bstride] = Vz;
    B[2 * bstride] = V;
    B[3 * bstride] = U[6] + tau_xy_0;
    B[4 * bstride] = U[8] + 0.0;
    B[6 * bstride] = B[6 * bstride] + dt * Vx;
    B[7 * bstride] = B[7 * bstride] + dt * Vz;
    B[8 * bstride] = B[8 * bstride] + dt * V;
    if (rt > time && V > P.rs_thr) B[9 * bstride] = time;
    else if (rt > time) B[9 * bstride] = 1e10;
    B[5 * bstride] = U[4];
    B[10 * bstride] = dPsi;
  }
  return dPsi;
}

// ---------------------------------------------- solves on characteristic values
// The same friction laws arranged for latency: on GB300 an FP64 instruction
// holds its pipe for 64 cycles a warp (a division is ten of them, exp 17, log
// 32), so a face's chain of FP64 instructions is the fault kernel's run time.
// Quantities that depend only on the face (nucleation shear, ramped a, the
// reciprocals of a, b, L) are computed once beside the predictors, divisions
// by constants become products with reciprocals, the friction equation is
// solved for a variable in which Newton converges at once, and logarithms are
// evaluated only where a short series does not do.

struct RSFaceK {
  double tau0;    // nucleation shear at the face
  double a, inv_a, b, inv_b, inv_L;
  double c_Vw;    // ramped weakening velocity (slip law with fexp > 0)
  double eq0;     // aging law: e^-(psi - f0)/b at the stored psi
};

// own: the face carries its own a, b, L (else the scenario's, whose reciprocals
// come from the host)
TMK_D RSFaceK rs_face_k(const DevParams& P, const RSFace& fr, bool own, double x, double psi) {
  RSFaceK k;
  const double q = x * P.inv_r0;
  k.tau0 = P.rs_nsig * exp(-0.5 * (q * q));
  const double c_ramp = fmin(1.0, fmax(0.0, (x - P.ramp_x) * P.inv_ramp_w));
  k.a = fr.a + P.ramp_a * c_ramp;
  k.b = fr.b;
  k.inv_a = P.inv_a; k.inv_b = P.inv_b; k.inv_L = P.inv_L;
  if (own) { k.inv_b = 1.0 / fr.b; k.inv_L = 1.0 / fr.L; }
  if (own || P.ramp_a != 0.0) k.inv_a = 1.0 / k.a;
  k.c_Vw = P.rs_Vw + P.ramp_Vw * c_ramp;
  k.eq0 = P.state_law == 1 ? exp((P.rs_f0 - psi) * k.inv_b) : 0.0;
  return k;
}

// State of a fault face: both sides' tangential velocities, the shared normal
// velocity and tractions, and the slip rate.
struct FaultFace { double vx1, vx2, vz1, vz2, vy, syy, sxy, syz, Vx, Vz, V; };

// The friction equation of RSNEWTON solved for z = asinh(beta V) instead of V:
//   f(z) = alpha z + c sinh z - phi = 0,  c = eta / beta,  V = sinh(z)/beta,  tau = alpha z.
// f is smooth and monotone in z on the same bracket (0, asinh(beta phi/Zs)], so
// Newton converges in a few steps where the iteration in V creeps up through
// tens of decades; it starts from the slip rate of the given states.  As in the
// reference, a root beyond the bracket's upper end V = phi/Zs yields that end;
// parameters outside the range of this form (a tensile fault, say) and, in the
// FP64 form, roots that RSNEWTON does not reach (near or beyond the bracket's
// end, too far below its start, or where beta^2 is out of range) go to RSNEWTON itself.
//
// The iterations run in FP32 (c e^{+-z} as e^{+-z + ln c}, whose exponent stays
// below log(phi) inside the bracket).  The mixed form finishes with one FP64
// Newton step from the FP32 root: from a start within ~1e-5 of the root it lands
// within ~1e-10, far below the FP32 volume arithmetic.  The FP64 form (EXACT)
// repeats it until the step is 1e-13 of z.  Repeated steps are divided by the
// FP32 derivative, which leaves the fixed point as it is, the mixed form's one
// by the FP64 one (the FP32 one cost a digit of tau in the median, 9e-16 for
// 8e-17, and saves nothing: rs 64x32, 20 us a step either way); e^-z is dropped
// past z = 19, where e^-2z is below FP64 resolution; V follows the last step to
// first order.  Errors against 80-bit arithmetic over V = 1e-16 to 20 m/s: V
// 7.5e-15 rms and tau 8e-17 in FP64 (RSNEWTON 3.5e-13 and 8.5e-15), V 9.8e-12
// and tau 2.5e-14 in the mixed form, as with an FP32 search by expf and division.
template <bool EXACT, typename T>
TMK_D int rs_solve_z(const DevParams& P, const RSFaceK& fk, double phi, double psi, double sn, T dvx, T dvz,
                     double& V, double& tau) {
  const double alpha = sn * fk.a;
  const double lb = psi * fk.inv_a - P.ln_2V0;        // ln beta, beta = e^(psi/a) / (2 V0)
  const double lc = P.ln_halfZs - lb;                 // ln c
  const float a32 = (float)alpha, lb32 = (float)lb, lc32 = (float)lc, phi32 = (float)phi;
  auto newton = [&](int halve = 0, bool climb = false) {
    V = sqrt((double)dvx * (double)dvx + (double)dvz * (double)dvz);
    return rs_newton(P, phi, psi, sn, fk.a, V, tau, halve, climb);
  };
  // RSNEWTON's derivative squares beta, which overflows past e^354.9
  if (!(a32 > 0.f) || !(phi32 > 0.f) || !(lb32 > -600.f && lb32 < (EXACT ? 354.f : 600.f)) || !(P.rs_V0 > 0.0))
    return newton();
  // bracket end z_max = asinh(beta Vmax) (= ln(2 beta Vmax) past e^20); the
  // root lies inside where alpha z_max > phi / 2
  const float vmax32 = phi32 * P.inv_Zs32;
  const float lbv = lb32 + logf(vmax32);
  const float zmax = lbv > 20.f ? 0.6931472f + lbv : asinhf(expf(lbv));
  if (!(a32 * zmax - 0.5f * phi32 > 1e-4f * phi32)) {
    if (EXACT) return newton(0, true);
    const double Vmax = phi * P.inv_Zs, l = lb + log(Vmax);
    const double zm = l > 20.0 ? 0.6931471805599453 + l : asinh(exp(l));
    if (alpha * zm + 0.5 * P.Zs * Vmax - phi <= 0.0) {
      V = Vmax;
      tau = alpha * zm;
      return RS_IMAX + 1;
    }
  }
  const float v0 = sqrtf((float)dvx * (float)dvx + (float)dvz * (float)dvz);
  float z = phi32 / a32;
  if (v0 > 0.f && v0 < vmax32) {
    const float lg = lb32 + logf(v0);                 // ln(beta V0)
    z = lg > 9.f ? 0.6931472f + lg : asinhf(expf(lg));
  }
  z = fminf(z, zmax);
  int it;
  for (it = 1; it <= 30; ++it) {
    const float ep = __expf(z + lc32), em = __expf(lc32 - z);
    const float f = a32 * z + 0.5f * (ep - em) - phi32;
    const float dz = __fdividef(-f, a32 + 0.5f * (ep + em));
    float zn = z + dz;
    if (zn < 0.f) zn = 0.5f * z;
    if (zn > zmax) zn = 0.5f * (z + zmax);
    z = zn;
    if (fabsf(dz) <= 2e-6f * fmaxf(1.f, z)) break;
  }
  // RSNEWTON halves its way down from a slip rate V far above the root and stops
  // after RS_IMAX iterations wherever it is: the FP64 form leaves a root more
  // than 80 halvings below the start (or, from rest, the bracket's middle) to it,
  // beginning where the halvings end.  A step leaves the bracket while
  // asinh(beta V) is above the root's z by more than 1 (+ eta V_root / alpha,
  // nothing here); 2.5 allows for the FP32 root and for a start that FP64 puts at
  // the bracket's middle.  (An iteration takes 3 us and holds up the step: a plastic
  // FP64 level of 512x256 whose fault heals 298 us a step, 837 with every
  // halving; from rest there are none.)
  if (EXACT) {
    const bool from = v0 > 0.f && v0 <= vmax32;
    const float lv0 = logf(from ? v0 : 0.5f * vmax32);
    const float lroot = (z > 1.f ? z - 0.6931472f : logf(fmaxf(z, 1e-30f))) - lb32;       // ln V, within 0.2
    if (lv0 - lroot > 55.45f) {
      const float h = (0.6931472f + lb32 + lv0 - z - 2.5f) * 1.442695f;
      return newton(v0 > 0.f && a32 > 1e-6f ? min(max((int)h, 0), RS_IMAX) : 0);
    }
  }
  double zz = (double)z;
  for (int k = 0; k < 12; ++k) {
    const float z32 = (float)zz;
    const double ep = exp(zz + lc);
    double sh = 0.5 * ep, ch = sh;
    if (z32 < 19.f) {
      const double em = 0.5 * exp(lc - zz);
      ch = sh + em;
      sh = sh - em;
    }
    const double f = alpha * zz + sh - phi;
    const float r32 = 1.f / (a32 + (float)ch), d32 = -(float)f * r32;
    double r = (double)r32;
    if (!EXACT) r = fma(r, fma(-(alpha + ch), r, 1.0), r);      // the mixed form's only FP64 step: not FP32's error
    const double dz = -f * r;
    const float small = (EXACT || k > 0) ? 1e-13f : 1e-4f;
    const bool done = fabsf(d32) <= small * fmaxf(1.f, z32) && z32 + d32 >= 0.f && z32 + d32 <= zmax;
    zz = zz + dz;
    if (done) {
      V = (sh + ch * dz) * P.two_inv_Zs;              // c sinh(z) / eta
      tau = alpha * zz;
      return it + k;
    }
    if (!(zz > 0.0)) zz = 0.5 * (double)z32;
    if (zz > (double)zmax) zz = 0.5 * ((double)z32 + (double)zmax);
  }
  return newton();
}

// RSFAULTBCF (ibcLinElast/RSIBCF.ChF:158-323) from the values the fault sees of
// the two sides' states: the left-going characteristic values of the P pair
// (aP = syy + Zp rv vy) and of the S pair (aS = sxy + Zs rv vx), rv = +1, -1.
// The antiplane traction term is zero in the law.  dvx, dvz: the states'
// velocity differences (the first guess).  The slip rates are those of RSSETBND,
// the differences of the two sides' velocities: zero where V is below their last
// bit and NaN without a traction, on which the state evolution's NaN, and with it
// the status of the step, depends.  Returns the iterations used.
template <bool EXACT, typename T>
TMK_D int rs_face_solve(const DevParams& P, const RSFaceK& fk, double aP1, double aP2, double aS1, double aS2,
                        double psi, T dvx, T dvz, FaultFace& f) {
  const double phi_xy = 0.5 * (aS1 + aS2) + fk.tau0;
  const double phi = fabs(phi_xy);
  f.syy = 0.5 * (aP1 + aP2);
  f.vy = (aP1 - aP2) * P.half_inv_Zp;
  double V, tau;
  const int it = rs_solve_z<EXACT>(P, fk, phi, psi, -f.syy, dvx, dvz, V, tau);
  // phi_xy / phi: +-1, NaN when phi is zero or NaN (as the reference's quotient)
  const double sgn = phi > 0.0 ? copysign(1.0, phi_xy) : __longlong_as_double(0x7ff8000000000000ll);
  f.sxy = sgn * tau - fk.tau0;
  f.syz = 0.0 * tau;                    // (phi_yz / phi) tau - tau_yz_0 with phi_yz = tau_yz_0 = 0
  f.vx1 = (aS1 - f.sxy) * P.inv_Zs;
  f.vx2 = __dsub_rn(f.vx1, sgn * V);
  f.vz1 = -f.syz;
  f.vz2 = f.vz1 - 0.0 * V;
  f.Vx = __dsub_rn(f.vx1, f.vx2);       // of the rounded velocities: not fused with vx1's product
  f.Vz = f.vz1 - f.vz2;
  f.V = fabs(f.Vx);                     // Vz is zero, or NaN as Vx is
  return it;
}

// The state variable of RSSETBND (ibcLinElast/RSIBCF.ChF:61-151) after dt at
// slip rate V: the reference's slip law, or the aging law at constant V,
// theta' = theta e^-x + dt (1 - e^-x)/x with x = V dt / L, that is
// psi' = psi - b x + b log(1 + r), r = (V0 dt / L) (e^x - 1)/x e^-(psi - f0)/b.
TMK_D double rs_state_next(const DevParams& P, const RSFaceK& fk, double psi, double V, double dt) {
  if (P.state_law == 1) {
    const double dl = dt * fk.inv_L, x = V * dl, c = P.rs_V0 * dl;
    double g;           // (e^x - 1)/x; the next term of the series is x^7 / 40320
    if (x < 0.01)
      g = 1.0 + x * (0.5 + x * (1.0 / 6.0 + x * (1.0 / 24.0 + x * (1.0 / 120.0 + x * (1.0 / 720.0 + x * (1.0 / 5040.0))))));
    else
      g = expm1(x) / x;
    const double r = c * g * fk.eq0;
    double l;           // log(1 + r); the next term of the series is r^7 / 7
    if (r < 1e-3) {
      l = r * (1.0 + r * (-0.5 + r * (1.0 / 3.0 + r * (-0.25 + r * (0.2 + r * (-1.0 / 6.0))))));
    } else if (r < 1e300) {
      l = log1p(r);
    } else {            // out of range (or NaN): the sum itself
      const double phi1 = x > 1e-12 ? -expm1(-x) / x : 1.0 - 0.5 * x;
      return P.rs_f0 + fk.b * log(exp((psi - P.rs_f0) * fk.inv_b - x) + c * phi1);
    }
    return psi + fk.b * (l - x);
  }
  const double f = fk.a * asinh(V * exp(psi * fk.inv_a) * P.inv_2V0);
  double fss = P.rs_f0 - (fk.b - fk.a) * log(V / P.rs_V0);
  if (P.rs_fexp > 0.0) {
    const double q = V / fk.c_Vw, q2 = q * q, q4 = q2 * q2, q8 = q4 * q4;
    fss = P.rs_fw + (fss - P.rs_fw) / pow(1.0 + q8, 0.125);
  }
  return psi - dt * (V * fk.inv_L) * (f - fss);
}

// The 3-D mixed form's fault face (22-component states): RSFAULTBCF and
// RSSETBND on the solves above.  The components that no flux, transverse term
// or boundary value reads are left as the caller set them.
TMK_D int rs_fault_k(const DevParams& P, const RSFaceK& fk, const double* Wi, double psi, double* Wg) {
  FaultFace f;
  const int it = rs_face_solve<false>(P, fk, Wi[4] + P.Zp * Wi[1], Wi[15] - P.Zp * Wi[12], Wi[6] + P.Zs * Wi[0],
                                      Wi[17] - P.Zs * Wi[11], psi, Wi[0] - Wi[11], Wi[2] - Wi[13], f);
  Wg[0] = f.vx1; Wg[1] = f.vy; Wg[2] = f.vz1; Wg[4] = f.syy; Wg[6] = f.sxy; Wg[8] = f.syz;
  Wg[11] = f.vx2; Wg[12] = f.vy; Wg[13] = f.vz2; Wg[15] = f.syy; Wg[17] = f.sxy; Wg[19] = f.syz;
  return it;
}
TMK_D double rs_setbnd_k(const DevParams& P, const RSFaceK& fk, const double* U, double* B, int bstride, double dt,
                         double time, bool final_) {
  const double Vx = U[0] - U[11];
  const double Vz = U[2] - U[13];
  const double V = sqrt(Vx * Vx + Vz * Vz);
  const double dPsi = rs_state_next(P, fk, B[10 * bstride], V, dt);
  if (final_) {
    const double rt = B[9 * bstride];
    B[0] = Vx;
    B[1 * bstride] = Vz;
    B[2 * bstride] = V;
    B[3 * bstride] = U[6] + fk.tau0;
    B[4 * bstride] = U[8] + 0.0;
    B[6 * bstride] = B[6 * bstride] + dt * Vx;
    B[7 * bstride] = B[7 * bstride] + dt * Vz;
    B[8 * bstride] = B[8 * bstride] + dt * V;
    if (rt > time && V > P.rs_thr) B[9 * bstride] = time;
    else if (rt > time) B[9 * bstride] = 1e10;
    B[5 * bstride] = U[4];
    B[10 * bstride] = dPsi;
  }
  return dPsi;
}

// Slip weakening on characteristic values (side 2 at component 11, the
// corrected layout): the quantities of one face, and SWFAULTBCF
// (ibcLinElast/SWIBCF.ChF:79-267) as rs_face_solve.  az: the values of the
// antiplane S pair (syz + Zs rv vz).
struct SWFaceK { double tau0, mu_s; };

// Centre of cell i relative to c.  A face exactly on the rim of a nucleation
// patch or friction box (odd nx, box at the grid's middle) is inside or outside
// by the rounding of this number, with a jump of the whole patch: the 2-D mixed
// form and a mixed 3-D patch by itself round it once (FUSED), FP64, as the
// reference's Fortran, and the mixed batch round the product first.  Each form
// keeps the side it has always had; written out, not left to the compiler.
template <bool FUSED> TMK_D double cell_from(int i, double dx, double c) {
  return FUSED ? __fma_rn(i + 0.5, dx, -c) : __dsub_rn(__dmul_rn(i + 0.5, dx), c);
}
// x, z: the face's position relative to the friction box's centre
template <bool Z3 = false>
TMK_D SWFaceK sw_face_k(const DevParams& P, double x, double z = 0.0) {
  SWFaceK k;
  k.tau0 = 0.0;
  for (int ip = 0; ip < P.sw_np; ++ip) {
    double v = P.sw_tau[ip] * smoothfn(P.sw_smooth, fabs(x - P.sw_xc[ip]) - P.sw_xw[ip]);
    if (Z3) v = v * smoothfn(P.sw_smooth, fabs(z - P.sw_zc[ip]) - P.sw_zw[ip]);
    k.tau0 = k.tau0 + v;
  }
  double valx = boxcar(P.sw_fbw0, fabs(x));
  if (Z3) valx = valx * boxcar(P.sw_fbw1, fabs(z));
  k.mu_s = P.sw_fs * valx + (1 - valx) * P.sw_outside;
  return k;
}
TMK_D void sw_face_solve(const DevParams& P, const SWFaceK& k, double aP1, double aP2, double aS1, double aS2,
                         double az1, double az2, double slip, FaultFace& f) {
  const double fx = 0.5 * (aS1 + aS2), fz = 0.5 * (az1 + az2), a1 = fx + k.tau0;
  f.syy = 0.5 * (aP1 + aP2);
  f.vy = (aP1 - aP2) * P.half_inv_Zp;
  const double mu = k.mu_s - (k.mu_s - P.sw_fd) * fmin(1.0, slip * P.inv_dw);
  const double tau = fmin(sqrt(a1 * a1 + fz * fz), -f.syy * mu) - k.tau0;
  const double q = tau * rsqrt(fx * fx + fz * fz);
  f.sxy = fx * q;
  f.syz = fz * q;
  f.vx1 = (aS1 - f.sxy) * P.inv_Zs;
  f.vz1 = (az1 - f.syz) * P.inv_Zs;
  f.vx2 = (f.sxy - aS2) * P.inv_Zs;
  f.vz2 = (f.syz - az2) * P.inv_Zs;
  f.Vx = f.vx1 - f.vx2;
  f.Vz = f.vz1 - f.vz2;
  f.V = sqrt(f.Vx * f.Vx + f.Vz * f.Vz);
}

// SWFAULTBCF (ibcLinElast/SWIBCF.ChF:79-267) at one fault face.  Side 2 is read
// and written at component offset P.sw_off (9 as in the reference source).
// Components the law does not write keep the values already in Wg.  Z3 (the
// 3-D fault plane): the nucleation patches and the friction box are products
// of x and z profiles, tau_0 += (tau valx) valz and box value valx valz
// (:118-126,175-180).
template <bool Z3 = false>
TMK_D void sw_fault(const DevParams& P, const double* Wi, double slip_total, double xcell, double* Wg,
                    double zcell = 0.0) {
  const int off = P.sw_off;
  const double Zs = P.Zs, Zp = P.Zp, lam = P.lam, G = P.G;
  double x = xcell - P.sw_fbc0;
  const double z = zcell - P.sw_fbc1;
  double vx1 = Wi[0], vy1 = Wi[1], vz1 = Wi[2], sxx1 = Wi[3], syy1 = Wi[4], szz1 = Wi[5];
  double sxy1 = Wi[6], sxz1 = Wi[7], syz1 = Wi[8];
  double vx2 = Wi[off + 0], vy2 = Wi[off + 1], vz2 = Wi[off + 2], sxx2 = Wi[off + 3], syy2 = Wi[off + 4];
  double szz2 = Wi[off + 5], sxy2 = Wi[off + 6], sxz2 = Wi[off + 7], syz2 = Wi[off + 8];
  double wpxy1 = -sxy1 - Zs * vx1;
  double wpyy1 = -syy1 - Zp * vy1;
  double wpyz1 = -syz1 - Zs * vz1;
  double wpxy2 = sxy2 - Zs * vx2;
  double wpyy2 = syy2 - Zp * vy2;
  double wpyz2 = syz2 - Zs * vz2;
  double tau_0 = 0;
  for (int ip = 0; ip < P.sw_np; ++ip) {
    double valx = smoothfn(P.sw_smooth, fabs(x - P.sw_xc[ip]) - P.sw_xw[ip]);
    if constexpr (Z3) {
      double valz = smoothfn(P.sw_smooth, fabs(z - P.sw_zc[ip]) - P.sw_zw[ip]);
      tau_0 = tau_0 + P.sw_tau[ip] * valx * valz;
    } else {
      tau_0 = tau_0 + P.sw_tau[ip] * valx;
    }
  }
  double a1 = 0.5 * (wpxy2 - wpxy1) + tau_0, a2 = 0.5 * (wpyz2 - wpyz1);
  double tau_lock = sqrt(a1 * a1 + a2 * a2);
  syy1 = -(wpyy1 - wpyy2) / 2.0;
  syy2 = -(wpyy1 - wpyy2) / 2.0;
  vy1 = -(wpyy1 + wpyy2) / 2.0 / Zp;
  vy2 = -(wpyy1 + wpyy2) / 2.0 / Zp;
  double valx = boxcar(P.sw_fbw0, fabs(x));
  double fric;
  if constexpr (Z3) {
    double valz = boxcar(P.sw_fbw1, fabs(z));
    fric = P.sw_fs * valx * valz + (1 - valx * valz) * P.sw_outside;
  } else {
    fric = P.sw_fs * valx + (1 - valx) * P.sw_outside;
  }
  fric = fric - (fric - P.sw_fd) * fmin(1.0, slip_total / P.sw_dw);
  double tau = fmin(tau_lock, -syy1 * fric) - tau_0;
  double phi_xy = 0.5 * (wpxy2 - wpxy1);
  double phi_yz = 0.5 * (wpyz2 - wpyz1);
  double phi = sqrt(phi_xy * phi_xy + phi_yz * phi_yz);
  sxy1 = (phi_xy / phi) * tau;
  syz1 = (phi_yz / phi) * tau;
  vx1 = -(sxy1 + wpxy1) / Zs;
  vz1 = -(syz1 + wpyz1) / Zs;
  double SHF = -(vy1 - syy1) * lam / (lam + 2.0 * G);
  Wg[0] = vx1; Wg[1] = vy1; Wg[2] = vz1;
  Wg[3] = sxx1 + SHF; Wg[4] = syy1; Wg[5] = szz1 + SHF;
  Wg[6] = sxy1; Wg[7] = sxz1; Wg[8] = syz1;
  sxy2 = (phi_xy / phi) * tau;
  syz2 = (phi_yz / phi) * tau;
  vx2 = (sxy2 - wpxy2) / Zs;
  vz2 = (syz2 - wpyz2) / Zs;
  SHF = -(vy2 - syy2) * lam / (lam + 2.0 * G);
  Wg[off + 0] = vx2; Wg[off + 1] = vy2; Wg[off + 2] = vz2;
  Wg[off + 3] = sxx2 + SHF; Wg[off + 4] = syy2; Wg[off + 5] = szz2 + SHF;
  Wg[off + 6] = sxy2; Wg[off + 7] = sxz2; Wg[off + 8] = syz2;
}

// SWSETBND (ibcLinElast/SWIBCF.ChF:32-72).  Predictor (final_=false): returns the
// predicted slip_total only.  Final: updates B in place; as in the reference's
// in-place call the rupture test reads the V just written.
TMK_D double sw_setbnd(const DevParams& P, const double* U, double* B, int bstride, double dt, double time,
                       bool final_) {
  const int off = P.sw_off;
  double vx = U[0] - U[off + 0];
  double vz = U[2] - U[off + 2];
  double V = sqrt((vx * vx + vz * vz));
  double st = B[7 * bstride] + dt * V;
  if (final_) {
    double rt = B[8 * bstride];
    B[0] = vx;
    B[1 * bstride] = vz;
    B[2 * bstride] = U[6];
    B[3 * bstride] = U[8];
    B[4 * bstride] = V;
    B[5 * bstride] = B[5 * bstride] + dt * vx;
    B[6 * bstride] = B[6 * bstride] + dt * vz;
    B[7 * bstride] = st;
    if (rt > time && V > P.sw_thr) B[8 * bstride] = time;
  }
  return st;
}

// The plasticity parameters (PLASTICSETF) and moduli in arithmetic T.
template <typename T>
struct PlasticK {
  T mu, beta, eta, pb, ph, G, K;
  TMK_HD void load(const DevParams& P) {
    mu = (T)P.p_mu; beta = (T)P.p_beta; eta = (T)P.p_eta; pb = (T)P.p_b; ph = (T)P.p_h;
    G = (T)P.G; K = (T)P.K;
  }
};

// PLASTICFLOW (srcLinElast/PlasticPhysicsF.ChF:74-181) on one side's stresses;
// returns whether the point yielded (else only p_lam, set to 0, changed).  The
// parameters come in T already: a pass over many cells converts them once (on
// GB300 each FP64-to-FP32 conversion uses the narrow FP64 pipe).
template <typename T>
TMK_D bool plastic_flow_k(const PlasticK<T>& c, T& sxx, T& syy, T& szz, T& sxy, T& sxz, T& syz, T& p_lam,
                          T& p_gam, T dt) {
  const T mu = c.mu, beta = c.beta, eta = c.eta, pb = c.pb, ph = c.ph;
  const T G = c.G, K = c.K;
  T sigma = (sxx + syy + szz) / T(3);
  T J2 = ((sxx - syy) * (sxx - syy) + (syy - szz) * (syy - szz) + (szz - sxx) * (szz - sxx)) / T(6) +
         sxy * sxy + sxz * sxz + syz * syz;
  T tau = sqrt(J2);
  T b = pb + p_gam * ph;
  T Y = tau - fmax(-mu * sigma + b, T(0));
  if (Y <= T(0)) { p_lam = T(0); return false; }
  p_lam = Y / (dt * (ph + G + mu * beta * K) + eta);
  p_gam = p_gam + dt * p_lam;
  T sig_e = sigma;
  tau = tau - dt * p_lam * G;
  sigma = sigma - dt * p_lam * K * beta;
  T factor = tau / (tau + dt * p_lam * G);
  sxx = sigma + factor * (sxx - sig_e);
  syy = sigma + factor * (syy - sig_e);
  szz = sigma + factor * (szz - sig_e);
  sxy = factor * sxy;
  sxz = factor * sxz;
  syz = factor * syz;
  return true;
}

// the same from the scenario's parameters
template <typename T>
TMK_D bool plastic_flow(const DevParams& P, T& sxx, T& syy, T& szz, T& sxy, T& sxz, T& syz, T& p_lam,
                        T& p_gam, T dt) {
  PlasticK<T> c;
  c.load(P);
  return plastic_flow_k<T>(c, sxx, syy, szz, sxy, sxz, syz, p_lam, p_gam, dt);
}

}  // namespace tmk
