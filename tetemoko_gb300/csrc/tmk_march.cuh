// tmk_march.cuh -- column-marching volume kernel.
//
// A warp owns 32 adjacent columns of a patch (28 updated columns plus a
// 2-column halo on each side) and streams up a run of rows, emitting one
// updated row per step: the CTU sequence of LinElastPatchGodunov::computeWHalf
// and LinElastPhysics::computeUpdate (srcLinElast/LinElastPatchGodunov.cpp:174-469).
//
// The medium of a level is uniform, so past the limiters every stage is linear
// with constant coefficients and is carried out on the characteristic values
// that meet at a face instead of on states: for a wave pair (v, s) of
// direction D and impedance Z,
//   An = s + Z v + traced left-going delta    at the cell's lo face,
//   Ap = s - Z v + traced right-going delta   at the cell's hi face
// are all that RIEMANNF (srcLinElast/LinElastPhysicsF.ChF:601-765) reads of the
// predicted states WM, WP of a cell.  The face state between cells i-1 and i is
// s = (An_i + Ap_{i-1})/2, v = (An_i - Ap_{i-1})/(2Z), so the difference of the
// two face states of a cell follows from the jumps
//   jn = An_{i+1} - An_i,   jp = Ap_i - Ap_{i-1}
// as ds = (jn + jp)/2, dv = (jn - jp)/(2Z).  The transverse term (GETADWDXF,
// :791-901) of one direction moves the values An, Ap of the other one by
// multiples of ds and dv, and the update (GETFLUXF, :265-353) is a multiple of
// ds and dv of the moved values.  No predicted state, face state or flux is
// formed (but the fluxes of coarse-fine faces, for the flux registers): a wave
// pair takes 10 operations to trace, 4 for the jumps' sums and differences, 4
// to correct, where states took about 60, and one or two values per pair are
// exchanged between lanes and carried from row to row instead of all
// components.  The stresses in An and Ap are taken relative to the scenario's
// background, which every jump cancels: in FP32 their rounding is that of the
// waves' amplitude, not of the 100 MPa they ride on.
//
// The state of the two fault sides is packed into one pair per component
// (.x = side 1, .y = side 2; the y direction of side 2 is mirrored, rv = -1),
// so the linear algebra runs as packed FP32x2 instructions in the FP32 form.
// The components split into two groups that never mix inside the volume:
//   in-plane  (vx vy sxx syy szz sxy): a P-wave pair, an S-wave pair and the
//             two normal stresses tied to the P-wave stress by lam/(lam+2G);
//   antiplane (vz sxz syz): an S-wave pair and one stress with zero speed.
// The PPM tracing is Colella & Woodward 1984 eq. 1.12, written as
// a*w_near + b*w_far with a = (1-s)^2, b = s^2 - s.
#pragma once
#include "tmk_device.cuh"
#include "tmk_kernels.cuh"

namespace tmk {

// ------------------------------------------------------------ pair arithmetic
template <typename T> struct PairOf;
template <> struct PairOf<float> { using P = float2; };
template <> struct PairOf<double> { using P = double2; };

TMK_HD float2 mk2(float a, float b) { return make_float2(a, b); }
TMK_HD double2 mk2(double a, double b) { return make_double2(a, b); }
TMK_D float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
TMK_D float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
TMK_D float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
TMK_D float2 psub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
TMK_D double2 padd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
TMK_D double2 pmul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
TMK_D double2 pfma(double2 a, double2 b, double2 c) { return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)); }
TMK_D double2 psub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
TMK_D float2 pneg(float2 a) { return make_float2(-a.x, -a.y); }
TMK_D double flip(double a) { return __hiloint2double(__double2hiint(a) ^ 0x80000000, __double2loint(a)); }
TMK_D double2 pneg(double2 a) { return make_double2(flip(a.x), flip(a.y)); }

TMK_D float2 shfl_up2(float2 v, int d) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
TMK_D float2 shfl_dn2(float2 v, int d) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
TMK_D double2 shfl_up2(double2 v, int d) {
  return make_double2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
TMK_D double2 shfl_dn2(double2 v, int d) {
  return make_double2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}

// ------------------------------------------------------------ groups and roles
template <int G> struct Grp;
template <> struct Grp<0> {   // in-plane
  static constexpr int N = 6;
  TMK_HD static constexpr int glob(int k) { return k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 3 : k == 3 ? 4 : k == 4 ? 5 : 6; }
};
template <> struct Grp<1> {   // antiplane
  static constexpr int N = 3;
  TMK_HD static constexpr int glob(int k) { return k == 0 ? 2 : k == 1 ? 7 : 8; }
};

// Wave roles of the group's components in direction D (indices into the group):
//   P pair (vP, sP), S pair (vS, sS), zero-speed components coupled to sP
//   (zc0, zc1: normal stresses, z - lam/(lam+2G) sP is invariant), and a
//   zero-speed component with no coupling (zf).
template <int G, int D> struct Role;
template <> struct Role<0, 0> { static constexpr bool hasP = true, hasZc = true, hasZf = false;
  static constexpr int vP = 0, sP = 2, vS = 1, sS = 5, zc0 = 3, zc1 = 4, zf = 0; };
template <> struct Role<0, 1> { static constexpr bool hasP = true, hasZc = true, hasZf = false;
  static constexpr int vP = 1, sP = 3, vS = 0, sS = 5, zc0 = 4, zc1 = 2, zf = 0; };
template <> struct Role<1, 0> { static constexpr bool hasP = false, hasZc = false, hasZf = true;
  static constexpr int vP = 0, sP = 0, vS = 0, sS = 1, zc0 = 0, zc1 = 0, zf = 2; };
template <> struct Role<1, 1> { static constexpr bool hasP = false, hasZc = false, hasZf = true;
  static constexpr int vP = 0, sP = 0, vS = 0, sS = 2, zc0 = 0, zc1 = 0, zf = 1; };

// Components of a group whose direction-D states feed no flux and no
// transverse term: the zero-speed components of the direction (the normal
// stresses tied to the P-wave stress, the uncoupled stress).  RIEMANNF, the
// edge conditions, GETFLUXF and GETADWDXF read only the P and S wave pairs of
// a face state, and those are formed from the wave pairs of the cell states
// alone, so these components of the predicted states, of the face states and
// of a transverse correction aimed at direction D are never read: the kernels
// skip them (szz, for instance, is updated from the fluxes of the velocities
// but feeds no face state in either direction).
template <int G, int D> TMK_HD constexpr bool live(int c) {
  using R = Role<G, D>;
  return !((R::hasZc && (c == R::zc0 || c == R::zc1)) || (R::hasZf && c == R::zf));
}

// Wave pairs of a group: in-plane 0 = P, 1 = S; antiplane 0 = S.
template <int G> constexpr int kWaves = G == 0 ? 2 : 1;
template <int G> TMK_HD constexpr bool is_p(int w) { return G == 0 && w == 0; }
template <int G, int D> TMK_HD constexpr int wave_v(int w) { return is_p<G>(w) ? Role<G, D>::vP : Role<G, D>::vS; }
template <int G, int D> TMK_HD constexpr int wave_s(int w) { return is_p<G>(w) ? Role<G, D>::sP : Role<G, D>::sS; }

// Constants of one direction D (E: the other one).  A packed FP32x2
// instruction takes a constant operand straight from the parameter bank only
// when both halves are the same scalar (a broadcast); a pair of two values has
// to be loaded into registers.  The products of two constants that both carry
// rv (side 2 = -side 1 in y) are the same on both sides, so only the ones with
// a single rv are pairs: the impedances of y, the velocity terms.
template <typename T>
struct MK {
  using P = typename PairOf<T>::P;
  P Zp, Zs;            // characteristics w = s +- Z v (rv Z)
  T aP, bP, aS, bS;    // PPM tracing coefficients of the P and S speeds, halved (the deltas are kept doubled)
  // transverse term of D on the characteristic values of E: the stress part
  // from the differences jn - jp, the velocity part (times E's impedance) from
  // the sums jn + jp
  T c_lam, c_G;
  P cvP, cvS;
  // update: velocities from the sums, stresses from the differences
  P e_v;
  T e_l2g, e_lam, e_G;
  // face states and GETFLUXF: v = (An - Ap) hZ, F = -rv * {1/rho, lam+2G, lam, G}
  P hZp, hZs, f_irho, f_l2g, f_lam, f_G;
  // per wave pair (P, in-plane S, antiplane S): the background's
  // characteristic values, whose stress part is zero, and its stress
  P bgn[3], bgp[3];
  T s0[3];
  TMK_HD void load(const DevParams& p, int D, double dtdx) {
    const double s2 = (D == 1) ? -1.0 : 1.0;    // rv of side 2
    auto two = [](double a, double b) { return mk2((T)a, (T)b); };
    // An and Ap carry the velocity times the rounded impedances: what undoes or
    // matches that product takes them too, or FP32 would scale every velocity by
    // Z's rounding (4e-8)
    const double zp = (double)(T)p.Zp, zs = (double)(T)p.Zs;
    Zp = two(p.Zp, s2 * p.Zp); Zs = two(p.Zs, s2 * p.Zs);
    const double sp = p.cp * dtdx, ss = p.cs * dtdx;
    aP = (T)(0.5 * (1.0 - sp) * (1.0 - sp)); bP = (T)(0.5 * (sp * sp - sp));
    aS = (T)(0.5 * (1.0 - ss) * (1.0 - ss)); bS = (T)(0.5 * (ss * ss - ss));
    const double l2g = p.lam + 2.0 * p.G;
    c_lam = (T)(0.5 * dtdx * p.lam * (0.5 / zp));
    c_G = (T)(0.5 * dtdx * p.G * (0.5 / zs));
    // the velocity term carries the rv of y in both directions (D's or E's)
    const double vP = zp * (0.25 * dtdx / p.rho), vS = zs * (0.25 * dtdx / p.rho);
    cvP = two(vP, -vP); cvS = two(vS, -vS);
    const double ev = 0.5 * dtdx / p.rho;
    e_v = two(ev, s2 * ev);
    e_l2g = (T)(dtdx * l2g * (0.5 / zp)); e_lam = (T)(dtdx * p.lam * (0.5 / zp));
    e_G = (T)(dtdx * p.G * (0.5 / zs));
    hZp = two(0.5 / zp, s2 * 0.5 / zp); hZs = two(0.5 / zs, s2 * 0.5 / zs);
    f_irho = two(-1.0 / p.rho, -s2 / p.rho);
    f_l2g = two(-l2g, -s2 * l2g); f_lam = two(-p.lam, -s2 * p.lam); f_G = two(-p.G, -s2 * p.G);
    const int v[3] = {D, 1 - D, 2}, s[3] = {3 + D, 6, 7 + D};
    for (int w = 0; w < 3; ++w) {
      const double Z = w == 0 ? p.Zp : p.Zs;
      bgn[w] = two(Z * p.bg[v[w]], s2 * Z * p.bg[11 + v[w]]);
      bgp[w] = two(-Z * p.bg[v[w]], -s2 * Z * p.bg[11 + v[w]]);
      s0[w] = (T)p.bg[s[w]];            // both sides start from one background (tmk_context_create)
    }
  }
};

// A constant of direction D that carries rv in y: in x a broadcast of one
// scalar, in y the stored pair.
template <int D, typename P> TMK_D P kpair(const P& pair) {
  if constexpr (D == 0) return mk2(pair.x, pair.x);
  else return pair;
}
template <typename T> TMK_D auto kall(T s) { return mk2(s, s); }

// position of a component among those live in y; of those live in x, and the
// component at a position
template <int G, int D = 1> TMK_HD constexpr int slope_slot(int c) {
  int k = 0;
  for (int q = 0; q < c; ++q) k += live<G, D>(q) ? 1 : 0;
  return k;
}
template <int G, int D> TMK_HD constexpr int slot_comp(int k) {
  int c = 0;
  while (!live<G, D>(c) || slope_slot<G, D>(c) != k) ++c;
  return c;
}

// Everything the marching kernel needs that is uniform over a launch (all
// patches of a level share the scenario, dt and dx).  Built on the host and
// passed by value as a __grid_constant__ parameter, so the kernel reads the
// constants from the parameter bank instead of holding them in registers
// through the row loop.
template <typename T>
struct MarchConst {
  using P = typename PairOf<T>::P;
  MK<T> kx, ky;
  P sc;              // -dt/dx
  T nbg[9];          // minus the background of the evolving components
  int plim, clim, lim, ppm;
  int xout_lo, xout_hi, yout_lo, yout_hi;
  void* stash[2];    // row-0 intermediates of the fault-row items, per component group
  const int4* caps[2];   // coarse-fine faces each group's items store (row, kind, lane, slot)
  // Drucker-Prager return of a plastic level when it is fused into the
  // in-plane group's stores (the antiplane group's updated stresses are stored
  // first); the level's tuning sets `plastic`
  PlasticK<T> pk;
  T pdt;
  int plastic;
  int patch_run;     // rows of an item of the patch form, which has no work list
  TMK_HD void load(const DevParams& p, double dt, double dx) {
    kx.load(p, 0, dt / dx);
    ky.load(p, 1, dt / dx);
    sc = mk2((T)(-dt / dx), (T)(-dt / dx));
    for (int c = 0; c < 9; ++c) nbg[c] = (T)-p.bg[c];
    plim = p.prim_lim != 0; clim = p.char_lim != 0; lim = plim || clim; ppm = p.order != 0;
    xout_lo = p.bc[0] == 0; xout_hi = p.bc[1] == 0; yout_lo = p.bc[2] == 0; yout_hi = p.bc[3] == 0;
    plastic = 0; patch_run = 0;
    pk.load(p);
    pdt = (T)dt;
  }
};

// ---- limiters.  On GB300 an FP64 instruction holds its pipe for 64 cycles a
// warp, so the FP64 form's comparisons, signs and powers of two are done on the
// bit patterns with integer instructions; magnitudes order as their patterns,
// and a NaN is larger than every number, so a minimum drops it as fmin does.
// (the masks act on the high word: a 64-bit one is turned back into an FP64
// absolute value, which holds the FP64 pipe like a sum)
TMK_D unsigned long long mag64(double x) {
  unsigned long long m;
  asm("mov.b64 %0, {%1, %2};" : "=l"(m) : "r"(__double2loint(x)), "r"(__double2hiint(x) & 0x7fffffff));
  return m;
}
// min(|a|, |b|) with the sign of a
TMK_D float clip_mag(float a, float b) { return copysignf(fminf(fabsf(a), fabsf(b)), a); }
TMK_D double with_sign(unsigned long long m, double a) {
  return __hiloint2double((int)(m >> 32) | (__double2hiint(a) & 0x80000000), (int)m);
}
TMK_D double clip_mag(double a, double b) {
  const unsigned long long ma = mag64(a), mb = mag64(b);
  return with_sign(ma < mb ? ma : mb, a);
}
TMK_D float clip_mag(float a, float b, float c) { return copysignf(fminf(fminf(fabsf(a), fabsf(b)), fabsf(c)), a); }
TMK_D double clip_mag(double a, double b, double c) {
  const unsigned long long ma = mag64(a), mb = mag64(b), mc = mag64(c);
  const unsigned long long m = mb < mc ? mb : mc;
  return with_sign(ma < m ? ma : m, a);
}
// x * 2^K by the exponent bits (|K| <= 3), for the limiters' bounds alone: zeros,
// numbers below 2^-1020 and numbers near the overflow limit are returned as they
// are (limited slopes down there are of no account: the product of two differences
// below 1e-154, which a limiter by products tests, is zero).  Unlimited slopes and
// deltas take the product and the sum.
template <int K> TMK_D double mul_pow2(double x) {
  const int hi = __double2hiint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
  return __hiloint2double(e - 3u < 2040u ? hi + (K << 20) : hi, __double2loint(x));
}
TMK_D float2 quarter(float2 a) { return pmul(a, make_float2(0.25f, 0.25f)); }
TMK_D double2 quarter(double2 a) { return make_double2(mul_pow2<-2>(a.x), mul_pow2<-2>(a.y)); }
TMK_D float2 twice(float2 a) { return padd(a, a); }
TMK_D double2 twice(double2 a) { return make_double2(mul_pow2<1>(a.x), mul_pow2<1>(a.y)); }
TMK_D float2 eight_times(float2 a) { return pmul(a, make_float2(8.f, 8.f)); }
TMK_D double2 eight_times(double2 a) { return make_double2(mul_pow2<3>(a.x), mul_pow2<3>(a.y)); }
// a b > 0 per half (both nonzero numbers of one sign)
TMK_D void same_sign(float2 a, float2 b, bool& x, bool& y) {
  const float2 p = pmul(a, b);
  x = p.x > 0.f;
  y = p.y > 0.f;
}
TMK_D bool same_sign1(double a, double b) {
  const unsigned long long inf = 0x7ff0000000000000ull;
  return (__double2hiint(a) ^ __double2hiint(b)) >= 0 && mag64(a) - 1 < inf && mag64(b) - 1 < inf;
}
TMK_D void same_sign(double2 a, double2 b, bool& x, bool& y) { x = same_sign1(a.x, b.x); y = same_sign1(a.y, b.y); }

// Limited slope of the middle value from the negated one-sided differences
// nl = w_{i-1} - w_i and nr = w_i - w_{i+1} (at a domain edge the missing one
// is given the other's value: the one-sided difference the reference uses):
// minus half the van Leer slope, sign(dc) min(|dc|, 2|dl|, 2|dr|) when
// dl dr > 0, else 0.
template <typename P> TMK_D P half_slope(P nl, P nr, bool limit) {
  using T = decltype(nl.x);
  if (!limit) return pmul(padd(nl, nr), kall(T(0.25)));     // the slope itself: exact down to the smallest numbers
  const P q = quarter(padd(nl, nr));
  bool x, y;
  same_sign(nl, nr, x, y);
  return mk2(x ? clip_mag(q.x, nl.x, nr.x) : T(0), y ? clip_mag(q.y, nl.y, nr.y) : T(0));
}
// the doubled lo delta of a cell at a domain edge
template <typename P> TMK_D P edge_delta(P n, bool limit) { return limit ? twice(n) : padd(n, n); }

// Twice the PPM delta (lo face value - w) of a cell from its negated
// difference to the cell below and both cells' half slopes:
// w_lo = (w_{i-1} + w_i)/2 - (s_i - s_{i-1})/6.
template <typename T, typename P> TMK_D P delta_lo(P nl, P n_i, P n_im1) {
  return pfma(psub(n_i, n_im1), kall(T(2.0 / 3.0)), nl);
}
// twice the hi delta from the next cell's: w_hi(i) = w_lo(i+1)
template <typename T, typename P> TMK_D P delta_hi(P nr, P dlo_next) { return pfma(nr, kall(T(-2)), dlo_next); }

// PPM limiter (Colella & Woodward 1984 eq. 1.10) of the doubled deltas m, p of
// a cell with half slope n: both zero at an extremum, otherwise each clipped to
// twice the other's magnitude.  With slopes limited as above, m lies between
// -0.17 and -0.83 of dl (doubled: twice that) and p between 0.17 and 0.83 of
// dr, so m p < 0 exactly where dl dr > 0, that is where n is not zero; there
// the clipped values stay below 2 * 1.66 min(|dl|, |dr|) <= 6.7 |n|, so the
// further bound 8 |n| only acts where n is zero and makes both zero without a
// test.
template <typename P> TMK_D void limit_mono(P& m, P& p, P n) {
  const P m2 = twice(m), p2 = twice(p), b = eight_times(n);
  const P a = mk2(clip_mag(m.x, p2.x, b.x), clip_mag(m.y, p2.y, b.y));
  p = mk2(clip_mag(p.x, m2.x, b.x), clip_mag(p.y, m2.y, b.y));
  m = a;
}
// the same limiter for deltas of unknown sign (characteristic limiting)
template <typename P> TMK_D void limit2(P& m, P& p) {
  using T = decltype(m.x);
  bool x, y;
  same_sign(m, pneg(p), x, y);
  m = mk2(x ? m.x : T(0), y ? m.y : T(0));
  const P m2 = twice(m), p2 = twice(p);
  const P a = mk2(clip_mag(m.x, p2.x), clip_mag(m.y, p2.y));
  p = mk2(clip_mag(p.x, m2.x), clip_mag(p.y, m2.y));
  m = a;
}

// The traced characteristic values of a cell in direction D (see the head of
// the file) from its state w and its doubled deltas m (lo) and p (hi).
// kd: the constants that are the same in both directions
template <int G, int D, typename T>
TMK_D void trace(const MK<T>& k, const MK<T>& kd, const typename PairOf<T>::P* w, const typename PairOf<T>::P* m,
                 const typename PairOf<T>::P* p, bool clim, typename PairOf<T>::P* An, typename PairOf<T>::P* Ap) {
  using P = typename PairOf<T>::P;
#pragma unroll
  for (int q = 0; q < kWaves<G>; ++q) {
    const int v = wave_v<G, D>(q), s = wave_s<G, D>(q);
    const P Z = kpair<D>(is_p<G>(q) ? k.Zp : k.Zs), nZ = pneg(Z);
    const P a = kall(is_p<G>(q) ? kd.aP : kd.aS), b = kall(is_p<G>(q) ? kd.bP : kd.bS);
    P nm = pfma(Z, m[v], m[s]), np = pfma(Z, p[v], p[s]);
    P pm = pfma(nZ, m[v], m[s]), pp = pfma(nZ, p[v], p[s]);
    if (clim) { limit2(nm, np); limit2(pm, pp); }
    An[q] = pfma(b, np, pfma(a, nm, pfma(Z, w[v], w[s])));
    Ap[q] = pfma(b, pm, pfma(a, pp, pfma(nZ, w[v], w[s])));
  }
}
// the cell's own characteristic values (CTU: no delta)
template <int G, int D, typename T>
TMK_D void chars(const MK<T>& k, const typename PairOf<T>::P* w, typename PairOf<T>::P* An,
                 typename PairOf<T>::P* Ap) {
#pragma unroll
  for (int q = 0; q < kWaves<G>; ++q) {
    const int v = wave_v<G, D>(q), s = wave_s<G, D>(q);
    An[q] = pfma(kpair<D>(is_p<G>(q) ? k.Zp : k.Zs), w[v], w[s]);
    Ap[q] = pfma(pneg(kpair<D>(is_p<G>(q) ? k.Zp : k.Zs)), w[v], w[s]);
  }
}

// The characteristic value arriving from outside a domain edge
// (LINELASTOUTBCF, LINELASTFREEBCF): the background's, or minus the one that
// leaves the domain (of the whole stress: both are relative to s0).
template <int G, typename T, typename P>
TMK_D void edge_value(const MK<T>& k, const P* bg, bool outflow, const P* leaving, P* arriving) {
#pragma unroll
  for (int q = 0; q < kWaves<G>; ++q) {
    const int w = G == 0 ? q : 2;
    arriving[q] = outflow ? bg[w] : pfma(kall(T(-2)), kall(k.s0[w]), pneg(leaving[q]));
  }
}

// sums and differences of the jumps
template <int G, typename P> TMK_D void jumps(const P* jn, const P* jp, P* sum, P* dif) {
#pragma unroll
  for (int q = 0; q < kWaves<G>; ++q) { sum[q] = padd(jn[q], jp[q]); dif[q] = psub(jn[q], jp[q]); }
}

// Transverse term of direction D with scale -1/2 dt/dx (its constants are the
// same in both directions) on the characteristic
// values Bn, Bp of the other direction.  E's P pair takes the normal stress
// from D's P wave (lam) and the velocity from D's S wave; E's S pair takes the
// shear stress from D's S wave (G) and the velocity from D's P wave; the
// antiplane stress of D does not enter E's wave.
template <int G, int D, typename T>
TMK_D void correct(const MK<T>& k, const typename PairOf<T>::P* sum, const typename PairOf<T>::P* dif,
                   typename PairOf<T>::P* Bn, typename PairOf<T>::P* Bp) {
  if constexpr (G == 0) {
    Bn[0] = pfma(k.cvP, sum[1], pfma(kall(k.c_lam), dif[0], Bn[0]));
    Bp[0] = pfma(pneg(k.cvP), sum[1], pfma(kall(k.c_lam), dif[0], Bp[0]));
    Bn[1] = pfma(k.cvS, sum[0], pfma(kall(k.c_G), dif[1], Bn[1]));
    Bp[1] = pfma(pneg(k.cvS), sum[0], pfma(kall(k.c_G), dif[1], Bp[1]));
  } else {
    Bn[0] = pfma(k.cvS, sum[0], Bn[0]);
    Bp[0] = pfma(pneg(k.cvS), sum[0], Bp[0]);
  }
}

// The conservative update's increments -dt/dx (F_hi - F_lo): the x part (D = 0)
// starts them, the y part adds to them; the state is rounded once, when they
// are added to it.
template <int G, int D, typename T>
TMK_D void add_update(const MK<T>& k, const MK<T>& kd, const typename PairOf<T>::P* sum, const typename PairOf<T>::P* dif,
                      typename PairOf<T>::P* du) {
  using P = typename PairOf<T>::P;
  using R = Role<G, D>;
  auto acc = [&](int c, P a, P b) { du[c] = D == 0 ? pmul(a, b) : pfma(a, b, du[c]); };
#pragma unroll
  for (int q = 0; q < kWaves<G>; ++q) {
    acc(wave_v<G, D>(q), kpair<D>(k.e_v), sum[q]);
    acc(wave_s<G, D>(q), kall(is_p<G>(q) ? kd.e_l2g : kd.e_G), dif[q]);
  }
  if constexpr (R::hasP) {
    acc(R::zc0, kall(kd.e_lam), dif[0]);
    acc(R::zc1, kall(kd.e_lam), dif[0]);
  }
  if constexpr (R::hasZf && D == 0) du[R::zf] = mk2(T(0), T(0));
}

// GETFLUXF of the face state with characteristic values Bn, Bp
template <int G, int D, typename T>
TMK_D void face_flux(const MK<T>& k, const typename PairOf<T>::P* Bn, const typename PairOf<T>::P* Bp,
                     typename PairOf<T>::P* F) {
  using P = typename PairOf<T>::P;
  using R = Role<G, D>;
#pragma unroll
  for (int q = 0; q < kWaves<G>; ++q) {
    const P fs = pfma(kall(T(0.5)), padd(Bn[q], Bp[q]), kall(k.s0[G == 0 ? q : 2]));
    const P fv = pmul(is_p<G>(q) ? k.hZp : k.hZs, psub(Bn[q], Bp[q]));
    F[wave_v<G, D>(q)] = pmul(k.f_irho, fs);
    F[wave_s<G, D>(q)] = pmul(is_p<G>(q) ? k.f_l2g : k.f_G, fv);
    if constexpr (R::hasP) {
      if (is_p<G>(q)) { F[R::zc0] = pmul(k.f_lam, fv); F[R::zc1] = F[R::zc0]; }
    }
  }
  if constexpr (R::hasZf) F[R::zf] = mk2(T(0), T(0));
}

// ---------------------------------------------------------------- the kernel
// A strip of MARCH_COLS columns of a patch by the rows [y0, y1].  fslot >= 0
// marks the first item of a strip on the fault row: its row 0 needs the fault
// kernel's results, so the kernel leaves that row to march_fault_row_kernel
// and keeps what it needs in stash slot fslot.
// [cap0, cap0+ncap) are the item's entries in its group's capture list.
struct MarchItem { int patch, x0, y0, y1, fslot, cap0, ncap; };
// vectors of a group's N components' size that a fault-row item keeps for its
// row 0: the traced x values (An, Ap), the first-pass and the final values at
// y face 1 (An of row 1, Ap of row 0 each; two per wave pair, N = 3 pairs'
// worth per component count of 6), the old state
constexpr int MARCH_STASH_VECS = 3;

constexpr int MARCH_COLS = 28;   // updated columns per warp
constexpr int MARCH_HALO = 2;    // halo lanes on either side (lane l holds column x0 - 2 + l)
constexpr int MARCH_WARPS = 4;   // warps per CTA

// Rows q-1 (the old state of the row updated at step q) to q+2 of the rolling
// window and the row in flight, q+3, live in a per-warp ring of five rows of
// shared memory filled by cp.async.  A ring row holds MARCH_RW entries per
// component: the column left of lane 0, the warp's 32 columns, the column right
// of lane 31.
constexpr int MARCH_RING = 5;
constexpr int MARCH_AHEAD = 3;
constexpr int MARCH_RW = 34;
template <typename T, int G>
constexpr int march_row_pairs() { return Grp<G>::N * MARCH_RW; }
// The FP32 in-plane kernel keeps the y half slopes and lo deltas of a lane (8
// values) in shared memory, which fits its registers into four CTAs per SM.
template <typename T, int G> constexpr bool kSlopesInSmem = sizeof(T) == 4 && G == 0;
// The FP64 form computes each difference of two cells once, since a sum holds
// its pipe for 64 cycles: a row's difference to the next one is kept for the
// next row (in shared memory, its registers being full), and the one to the
// right comes from the neighbour lane (2048x1024 2160 -> 2080 us a step).
template <typename T> constexpr bool kDiffsOnce = sizeof(T) == 8;
template <typename T, int G>
constexpr size_t march_warp_pairs() {
  return (size_t)MARCH_RING * march_row_pairs<T, G>() + (kSlopesInSmem<T, G> ? 8 * 32 : 0) +
         (kDiffsOnce<T> ? (G == 0 ? 4 : 2) * 32 : 0);
}
template <typename T, int G, bool PATCH = false>
constexpr size_t march_smem_bytes() {
  const size_t stash = PATCH ? (size_t)MARCH_STASH_VECS * Grp<G>::N * 32 : 0;
  return (size_t)MARCH_WARPS * (march_warp_pairs<T, G>() + stash) * sizeof(typename PairOf<T>::P);
}

// resident CTAs per SM the register allocation targets: FP32 in-plane 4 (128
// registers), antiplane 6 (80); FP64 in-plane 2, antiplane 4.  FP32 with 3 / 5
// instead, us a step: slip weakening 512x256 19.2 against 17.0, rate and state
// 512x512 32.7 against 25.7, 2048x1024 121 against 118; 4 / 7 and 5 / 7 spill.
template <typename T, int G> struct MarchMinBlocks {
  static constexpr int value = sizeof(T) == 4 ? ((G == 0) ? 4 : 6) : ((G == 0) ? 2 : 4);
};

// asynchronous copy of one element to shared address dst + OFF (completion
// tracked per thread); nbytes = sizeof(T), or 0: nothing is read and zeros are
// written
template <typename T, int OFF> TMK_D void cp_async_elem(unsigned dst, const T* src, unsigned nbytes) {
  asm volatile("cp.async.ca.shared.global [%0 + %4], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(sizeof(T)), "r"(nbytes),
               "n"(OFF)
               : "memory");
}
// component plane g of a FAB from the address in plane 0 (one 32 x 32 + 64-bit
// multiply-add; the planes hold fewer than 2^32 cells)
template <typename T> TMK_D T* plane_ptr(T* p0, unsigned plane, int g) {
  return reinterpret_cast<T*>((unsigned long long)p0 + (unsigned long long)plane * (unsigned)(g * sizeof(T)));
}
// the cp.async copies of one lane's column of a ring row, components C...
template <typename T, int G, int C, bool XONLY>
TMK_D void cp_async_column(unsigned dst, const T* src, unsigned plane, unsigned nbytes) {
  if constexpr (C < Grp<G>::N) {
    if constexpr (!XONLY || live<G, 0>(C)) {
      constexpr int off = C * MARCH_RW * 2 * (int)sizeof(T);
      cp_async_elem<T, off>(dst, plane_ptr(src, plane, Grp<G>::glob(C)), nbytes);
      cp_async_elem<T, off + (int)sizeof(T)>(dst, plane_ptr(src, plane, 11 + Grp<G>::glob(C)), nbytes);
    }
    cp_async_column<T, G, C + 1, XONLY>(dst, src, plane, nbytes);
  }
}
TMK_D void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest K groups have landed
template <int K> TMK_D void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(K) : "memory"); }

// The inputs of a cell's plastic return the in-plane group does not hold: the
// antiplane group's updated sxz, syz (stored by the antiplane kernel, which
// has completed) and the plastic strain of the step's input, both sides.
template <typename T>
TMK_D void plastic_inputs(const T* in0, const T* out0, unsigned plane, typename PairOf<T>::P* pin) {
  pin[0] = mk2(*plane_ptr(out0, plane, 7), *plane_ptr(out0, plane, 18));
  pin[1] = mk2(*plane_ptr(out0, plane, 8), *plane_ptr(out0, plane, 19));
  pin[2] = mk2(*plane_ptr(in0, plane, 10), *plane_ptr(in0, plane, 21));
}

// Stores the updated group G of one cell (out0: its address in plane 0).  With
// PL (a plastic level whose return is fused) the in-plane group first takes
// LinElastLevelGodunov::plasticUpdate (PLASTICCORRECTION,
// srcLinElast/PlasticPhysicsF.ChF:30-133, as the reference applies it after
// the level's update, LinElastLevelGodunov.cpp:643-667): the cell's six
// updated stresses and its plastic strain (pin, from plastic_inputs) give the
// return; the antiplane stresses are rewritten where the point yielded, the
// plastic rate and strain always.
template <typename T, int G, bool PL>
TMK_D void store_cell(T* out0, unsigned plane, const MarchConst<T>& mc, typename PairOf<T>::P* u,
                      const typename PairOf<T>::P* pin) {
  constexpr int N = Grp<G>::N;
  if constexpr (G == 0 && PL) {
    T sxz[2] = {pin[0].x, pin[0].y}, syz[2] = {pin[1].x, pin[1].y}, gam[2] = {pin[2].x, pin[2].y};
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      T sxx = sd ? u[2].y : u[2].x, syy = sd ? u[3].y : u[3].x;
      T szz = sd ? u[4].y : u[4].x, sxy = sd ? u[5].y : u[5].x;
      T lam;
      if (plastic_flow_k<T>(mc.pk, sxx, syy, szz, sxy, sxz[sd], syz[sd], lam, gam[sd], mc.pdt)) {
        if (sd) { u[2].y = sxx; u[3].y = syy; u[4].y = szz; u[5].y = sxy; }
        else { u[2].x = sxx; u[3].x = syy; u[4].x = szz; u[5].x = sxy; }
        *plane_ptr(out0, plane, 11 * sd + 7) = sxz[sd];
        *plane_ptr(out0, plane, 11 * sd + 8) = syz[sd];
      }
      *plane_ptr(out0, plane, 11 * sd + 9) = lam;
      *plane_ptr(out0, plane, 11 * sd + 10) = gam[sd];
    }
  }
#pragma unroll
  for (int c = 0; c < N; ++c) {
    const int gg = Grp<G>::glob(c);
    *plane_ptr(out0, plane, gg) = u[c].x;
    *plane_ptr(out0, plane, 11 + gg) = u[c].y;
  }
}

// Fluxes of the coarse-fine faces of row `row` that this item owns, into the
// level's flux-register capture buffer (flux registers of the AMR coupling).
// Entry kinds: 0 the x face below the lane's column, 1 the one above, 2 the
// y face below the row, 3 the one above; entries are sorted by row and the
// loop is uniform over the warp.  flux(kind, F) gives the fluxes of a face.
template <typename T, int G, typename FluxOf>
TMK_D void march_capture(const PatchDev<T>& pp, const MarchItem& it, const MarchConst<T>& mc, int row, int lane,
                         int& cpos, FluxOf flux) {
  using P = typename PairOf<T>::P;
  constexpr int N = Grp<G>::N;
  const int4* caps = mc.caps[G];
  const int cend = it.cap0 + it.ncap;
  while (cpos < cend) {
    const int4 e = caps[cpos];
    if (e.x > row) break;
    ++cpos;
    if (e.x < row || e.z != lane) continue;   // rows left to the fault-row kernel, other lanes
    P F[N];
    flux(e.y, F);
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const int g = Grp<G>::glob(c);
      pp.cap[(size_t)e.w * 22 + g] = (double)F[c].x;
      pp.cap[(size_t)e.w * 22 + 11 + g] = (double)F[c].y;
    }
  }
}

// The predictor scheme of every reference deck (PPM, primitive limiting, no
// characteristic limiting), fixed at compile time: SCH = 1.  SCH = 0 reads the
// scheme flags from the launch constants.
constexpr int MARCH_SCH_RUNTIME = 0, MARCH_SCH_PPM_PRIM = 1;
template <typename T>
TMK_HD bool march_scheme_fixed(const MarchConst<T>& mc) { return mc.ppm && mc.plim && !mc.clim; }

// Fluxes of the patch form (GETFLUXF over all faces of the valid box): a cell
// of row `row` stores its lo faces, the last one of a row or column its hi face
// too; the antiplane group also zeroes the components without a flux (plastic
// rate and strain).
template <typename T, int G, int D>
TMK_D void store_face(const PatchDev<T>& pp, int x, int row, const typename PairOf<T>::P* F) {
  constexpr int N = Grp<G>::N;
  const int nx = pp.vhi0 - pp.vlo0 + (D == 0 ? 2 : 1), ny = pp.vhi1 - pp.vlo1 + (D == 0 ? 1 : 2);
  const unsigned plane = (unsigned)nx * (unsigned)ny;
  T* const f = (D == 0 ? pp.Fx : pp.Fy) + ((long long)(row - pp.vlo1) * nx + (x - pp.vlo0));
#pragma unroll
  for (int c = 0; c < N; ++c) {
    *plane_ptr(f, plane, Grp<G>::glob(c)) = F[c].x;
    *plane_ptr(f, plane, 11 + Grp<G>::glob(c)) = F[c].y;
  }
  if constexpr (G == 1) {
#pragma unroll
    for (int c = 9; c < 11; ++c) { *plane_ptr(f, plane, c) = T(0); *plane_ptr(f, plane, 11 + c) = T(0); }
  }
}

template <typename T, int G>
TMK_D void fault_row_finish(const PatchDev<T>& pp, const MarchItem& it, const MarchConst<T>& mc, int lane,
                            const typename PairOf<T>::P* st, bool faces);

// PL: a plastic level with the fused return (in-plane group only): every
// stored cell takes the plastic return, and the kernel runs after the
// antiplane one.
// FORM: how the items of the fault row end.  MARCH_LEVEL leaves row 0 to
// march_fault_row_kernel.  The other two run when the fault kernel is the launch
// before: an item keeps its row 0, waits for the fault kernel when the rest of
// its rows are done and finishes it, MARCH_OWN on a level (row 0 kept in the
// level's stash), MARCH_PATCH on one patch by itself (patches[0]; row 0 kept in
// shared memory, items by index with the strips of columns fastest and runs of
// mc.patch_run rows, and the fluxes of all faces where the patch has arrays for
// them).
constexpr int MARCH_LEVEL = 0, MARCH_PATCH = 1, MARCH_OWN = 2;
template <typename T, int G, bool PL, int SCH, int FORM>
TMK_D void march_items(const PatchDev<T>* __restrict__ patches, const MarchItem* __restrict__ items, int nitems,
                       const MarchConst<T>& mc, int block) {
  using P = typename PairOf<T>::P;
  constexpr int N = Grp<G>::N, NW = kWaves<G>;
  constexpr bool PATCH = FORM == MARCH_PATCH;
  extern __shared__ __align__(16) unsigned char march_smem[];
  P* const ring = reinterpret_cast<P*>(march_smem) + (size_t)(threadIdx.x >> 5) * march_warp_pairs<T, G>();
  const int wid = block * MARCH_WARPS + __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  // a later kernel of the step may be scheduled now; every warp waits for the
  // kernel before it (the fault kernel or the other component group) before
  // it reads the fault buffers or exits, so kernels still complete in order
  asm volatile("griddepcontrol.launch_dependents;");
  if (wid >= nitems) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  // the fused plastic return reads the antiplane kernel's stresses: wait for it
  if (PL) asm volatile("griddepcontrol.wait;" ::: "memory");
  MarchItem it;
  if constexpr (PATCH) {
    const PatchDev<T>& p0 = patches[0];
    const unsigned ns = (unsigned)(p0.vhi0 - p0.vlo0 + MARCH_COLS) / MARCH_COLS, r = (unsigned)wid / ns;
    it.patch = 0;
    it.x0 = p0.vlo0 + (int)((unsigned)wid - r * ns) * MARCH_COLS;
    it.y0 = p0.vlo1 + (int)r * mc.patch_run;
    it.y1 = min(it.y0 + mc.patch_run - 1, p0.vhi1);
    it.fslot = p0.fault && it.y0 == p0.dlo1 ? 0 : -1;
    it.cap0 = 0;
    it.ncap = 0;
  } else {
    it = items[wid];
  }
  const PatchDev<T>& pp = patches[it.patch];
  const int x = it.x0 - MARCH_HALO + lane;
  const int dlo0 = pp.dlo0, dhi0 = pp.dhi0, dlo1 = pp.dlo1, dhi1 = pp.dhi1;
  const int ahi0 = pp.alo0 + pp.anx - 1;
  const bool lane_in = x >= dlo0 && x <= dhi0 && x >= pp.alo0 && x <= ahi0;
  // lane 0 also stages the column left of it (ring entry 0), lane 31 the one
  // right of it (entry 33), each from its own column's address -1 / +1
  const int dxe = lane == 0 ? -1 : 1;
  const bool ext_in = (lane == 0 || lane == 31) && x + dxe >= dlo0 && x + dxe <= dhi0 && x + dxe >= pp.alo0 &&
                      x + dxe <= ahi0;
  const int ext_pos = lane == 0 ? 0 : 33;
  constexpr bool kFixed = SCH == MARCH_SCH_PPM_PRIM;
  const bool plim = kFixed || mc.plim != 0, clim = !kFixed && mc.clim != 0, lim = kFixed || mc.lim != 0;
  const bool ppm = kFixed || mc.ppm != 0;
  const MK<T>& kx = mc.kx;
  const MK<T>& ky = mc.ky;
  const bool fault = pp.fault != 0;
  const bool defer0 = it.fslot >= 0;      // row 0 is finished by march_fault_row_kernel (PATCH, OWN: at the end)
  // what a fault-row item keeps for its row 0
  P* stash0 = nullptr;
  if constexpr (PATCH)
    stash0 = reinterpret_cast<P*>(march_smem) + (size_t)MARCH_WARPS * march_warp_pairs<T, G>() +
             (size_t)(threadIdx.x >> 5) * MARCH_STASH_VECS * N * 32 + lane;
  else if (defer0)
    stash0 = reinterpret_cast<P*>(mc.stash[G]) + (size_t)it.fslot * MARCH_STASH_VECS * N * 32 + lane;
  const bool col_valid = x >= it.x0 && x < it.x0 + MARCH_COLS && x >= pp.vlo0 && x <= pp.vhi0;
  const int anx = pp.anx;
  const unsigned plane = (unsigned)anx * (unsigned)pp.any;
  // a lane of this warp holds a cell on a domain x edge: every lane takes the
  // interior differences and face values, overwritten there by the edge's;
  // other warps (most) skip the edge code on a uniform branch
  const bool edge_lo = x == dlo0, edge_hi = x == dhi0;
  const bool warp_xedge = __any_sync(0xffffffffu, edge_lo || edge_hi);

  const int q_s = max(it.y0 - 1, dlo1);
  const int q_e = it.y1 + 1;

  // the lane's addresses in plane 0: of the next row to stage, of the row stored next
  const T* lsrc = pp.Uin + ((long long)(q_s - pp.alo1) * anx + (x - pp.alo0));
  T* sdst = pp.Uout + ((long long)(q_s - 1 - pp.alo1) * anx + (x - pp.alo0));
  const T* psrc = PL ? pp.Uin + ((long long)(q_s - 1 - pp.alo1) * anx + (x - pp.alo0)) : nullptr;
  const T* const uin = pp.Uin;
  const unsigned ring32 = (unsigned)__cvta_generic_to_shared(ring);

  auto load_row = [&](int y, P* w) {
    const bool ok = lane_in && y >= dlo1 && y <= dhi1;
    const T* const p0 = ok ? uin + ((long long)(y - pp.alo1) * anx + (x - pp.alo0)) : uin;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      if (!live<G, 1>(c)) { w[c] = mk2(T(0), T(0)); continue; }
      const int g = Grp<G>::glob(c);
      w[c] = ok ? mk2(*plane_ptr(p0, plane, g), *plane_ptr(p0, plane, 11 + g)) : mk2(T(0), T(0));
    }
  };
  // row y (the next one to stage) into its ring slot: cp.async for cells in
  // the domain, zeros elsewhere (and for rows past the last one the item
  // reads); the two outer columns only for the components live in x (the only
  // ones whose neighbours are read)
  // ring slots of rows q-1, q, q+1, q+2 and of the row in flight, handed on each row
  constexpr int RP = march_row_pairs<T, G>();
  int r_m1 = 4 * RP, r_0 = 0, r_1 = RP, r_2 = 2 * RP, r_3 = 3 * RP;
  const int y_last = min(dhi1, q_e + 2);
  auto load_row_async = [&](int y, int slot) {
    const bool ok = lane_in && y <= y_last;       // y >= q_s >= dlo1
    const T* const src = ok ? lsrc : uin;
    const unsigned row32 = ring32 + (unsigned)(slot * (int)sizeof(P));
    cp_async_column<T, G, 0, false>(row32 + (unsigned)((lane + 1) * (int)sizeof(P)), src, plane,
                                    ok ? (unsigned)sizeof(T) : 0u);
    if (lane == 0 || lane == 31) {      // the outer columns: own address -1 / +1 (ext_in and ok: a cell of the FAB)
      const bool oke = ext_in && ok;
      cp_async_column<T, G, 0, true>(row32 + (unsigned)(ext_pos * (int)sizeof(P)), oke ? src + dxe : uin, plane,
                                     oke ? (unsigned)sizeof(T) : 0u);
    }
    cp_async_commit();
    lsrc += anx;
  };

  int cpos = it.cap0;                     // next coarse-fine face to store
  // What a lane carries from row to row: the half slopes and lo deltas of row
  // q, the traced x values of row q-1, the traced and corrected y values of
  // row q-1 (An, Ap) and their jump jp.  Two sets, used in turn by two copies
  // of the row's code: with one set each value would be moved once a row.
  constexpr bool kS = kSlopesInSmem<T, G>;
  P* const slopes = ring + MARCH_RING * RP + lane;     // [2][4][32]
  constexpr bool kD = kDiffsOnce<T>;
  P* const diffs = slopes;                             // [4 or 2][32] (FP64, which keeps no slopes there)
  struct Carry {
    P n4[N], dlo[N];
    P Anx[NW], Apx[NW], Any[NW], Apy[NW], jpy[NW], Bny[NW], Bpy[NW], jpB[NW];
  } c0, c1;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    const P z = mk2(T(0), T(0));
    c0.Anx[w] = z; c0.Apx[w] = z; c0.Any[w] = z; c0.Apy[w] = z; c0.jpy[w] = z;
    c0.Bny[w] = z; c0.Bpy[w] = z; c0.jpB[w] = z;
  }
  {
#pragma unroll
    for (int y = 0; y < MARCH_AHEAD; ++y) load_row_async(q_s + y, y * RP);
    P Wa[N], Wb[N];
    load_row(q_s - 2, Wa);
    load_row(q_s - 1, Wb);
    cp_async_wait<MARCH_AHEAD - 2>();      // rows q_s, q_s + 1 have landed (a lane reads its own columns)
    const bool hl = q_s - 1 >= dlo1, hll = q_s - 2 >= dlo1, hr = q_s + 1 <= dhi1;
    const P* r0 = ring + lane + 1;
    const P* r1 = ring + RP + lane + 1;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      if (!live<G, 1>(c)) continue;
      const P W0 = r0[c * MARCH_RW];
      P nl = psub(Wb[c], W0), nr = psub(W0, r1[c * MARCH_RW]);
      if (kD) diffs[slope_slot<G>(c) * 32] = nr;
      if (!hl) nl = nr;
      if (!hr) nr = nl;
      if (!hl && !hr) { nl = mk2(T(0), T(0)); nr = nl; }
      c0.n4[c] = half_slope(nl, nr, lim);
      if (hl) {
        P na = psub(Wa[c], Wb[c]);
        if (!hll) na = nl;
        c0.dlo[c] = delta_lo<T>(nl, c0.n4[c], half_slope(na, nl, lim));
      } else {
        c0.dlo[c] = edge_delta(c0.n4[c], lim);
      }
      if (kS) { slopes[slope_slot<G>(c) * 32] = c0.n4[c]; slopes[(4 + slope_slot<G>(c)) * 32] = c0.dlo[c]; }
    }
  }

  auto row_step = [&](const int q, Carry& in, Carry& out) {
    load_row_async(q + MARCH_AHEAD, r_3);  // the row in flight while this one is computed
    // fused plastic return: its other inputs for row q-1, stored at the end of
    // this iteration, requested now so that the row's work hides their latency
    P pin[3];
    if constexpr (PL) {
      if (col_valid && q - 1 >= it.y0 && q - 1 <= it.y1) plastic_inputs<T>(psrc, sdst, plane, pin);
      psrc += anx;
    }
    cp_async_wait<MARCH_AHEAD - 2>();     // rows up to q+2 have landed
    __syncwarp();                         // ... every lane's copies, whose neighbours read them
    P Bn_q[NW], Bp_q[NW];
    if (q <= dhi1) {
      const P* const rw = ring + r_0 + lane + 1;
      P W0[N], m[N], p[N], nl[N], nr[N], n4[N], dl[N];
#pragma unroll
      for (int c = 0; c < N; ++c) { W0[c] = rw[c * MARCH_RW]; m[c] = mk2(T(0), T(0)); p[c] = m[c]; }
      // the cell's stresses relative to the background, for its characteristic values
      P Wr[N];
#pragma unroll
      for (int c = 0; c < N; ++c)
        Wr[c] = Grp<G>::glob(c) < 3 ? W0[c] : padd(W0[c], kall(mc.nbg[Grp<G>::glob(c)]));
      if (ppm) {
        // y deltas of row q; slope and lo delta of row q+1
        const P* const r1 = ring + r_1 + lane + 1;
        const P* const r2 = ring + r_2 + lane + 1;
#pragma unroll
        for (int c = 0; c < N; ++c) {
          if (!live<G, 1>(c)) continue;
          const P W1 = r1[c * MARCH_RW];
          nl[c] = kD ? diffs[slope_slot<G>(c) * 32] : psub(W0[c], W1);
          nr[c] = psub(W1, r2[c * MARCH_RW]);
          if (kD) diffs[slope_slot<G>(c) * 32] = nr[c];
        }
        if (q + 2 > dhi1) {
#pragma unroll
          for (int c = 0; c < N; ++c) nr[c] = nl[c];
        }
#pragma unroll
        for (int c = 0; c < N; ++c) {
          if (!live<G, 1>(c)) continue;
          n4[c] = kS ? slopes[slope_slot<G>(c) * 32] : in.n4[c];
          m[c] = kS ? slopes[(4 + slope_slot<G>(c)) * 32] : in.dlo[c];
          const P n1 = half_slope(nl[c], nr[c], lim);
          dl[c] = delta_lo<T>(nl[c], n1, n4[c]);
          p[c] = delta_hi<T>(nl[c], dl[c]);
          if (kS) { slopes[slope_slot<G>(c) * 32] = n1; slopes[(4 + slope_slot<G>(c)) * 32] = dl[c]; }
          else { out.n4[c] = n1; out.dlo[c] = dl[c]; }
        }
        if (q + 1 > dhi1) {
#pragma unroll
          for (int c = 0; c < N; ++c)
            if (live<G, 1>(c)) p[c] = pneg(edge_delta(n4[c], lim));
        }
#pragma unroll
        for (int c = 0; c < N; ++c)
          if (live<G, 1>(c) && plim) limit_mono(m[c], p[c], n4[c]);
        trace<G, 1, T>(ky, kx, Wr, m, p, clim, out.Any, out.Apy);
        // x deltas
        P n[N], d[N];
#pragma unroll
        for (int c = 0; c < N; ++c) {
          if (!live<G, 0>(c)) continue;
          nl[c] = psub(rw[c * MARCH_RW - 1], W0[c]);
          if (!kD) nr[c] = psub(W0[c], rw[c * MARCH_RW + 1]);
        }
        if constexpr (kD) {
          // lane 31's differences to the column right of it, one per lane for
          // all components and sides in one instruction
          constexpr int NX = slope_slot<G, 0>(N);
          int cc = slot_comp<G, 0>(0);
#pragma unroll
          for (int k = 1; k < NX; ++k)
            if ((lane >> 1) == k) cc = slot_comp<G, 0>(k);
          const T* const last = reinterpret_cast<const T*>(ring + r_0 + cc * MARCH_RW + 32) + (lane & 1);
          const T e = last[0] - last[2];
#pragma unroll
          for (int c = 0; c < N; ++c) {
            if (!live<G, 0>(c)) continue;
            const int k = 2 * slope_slot<G, 0>(c);
            const P r = shfl_dn2(nl[c], 1);
            const T ex = __shfl_sync(0xffffffffu, e, k), ey = __shfl_sync(0xffffffffu, e, k + 1);
            nr[c] = lane == 31 ? mk2(ex, ey) : r;
          }
        }
        if (warp_xedge) {
#pragma unroll
          for (int c = 0; c < N; ++c) {
            if (!live<G, 0>(c)) continue;
            const P l = nl[c];
            if (edge_lo) nl[c] = edge_hi ? mk2(T(0), T(0)) : nr[c];
            if (edge_hi) nr[c] = edge_lo ? mk2(T(0), T(0)) : l;
          }
        }
#pragma unroll
        for (int c = 0; c < N; ++c) {
          if (!live<G, 0>(c)) continue;
          n[c] = half_slope(nl[c], nr[c], lim);
          d[c] = delta_lo<T>(nl[c], n[c], shfl_up2(n[c], 1));
        }
        if (warp_xedge && edge_lo) {
#pragma unroll
          for (int c = 0; c < N; ++c)
            if (live<G, 0>(c)) d[c] = edge_delta(n[c], lim);
        }
#pragma unroll
        for (int c = 0; c < N; ++c)
          if (live<G, 0>(c)) p[c] = delta_hi<T>(nr[c], shfl_dn2(d[c], 1));
        if (warp_xedge && edge_hi) {
#pragma unroll
          for (int c = 0; c < N; ++c)
            if (live<G, 0>(c)) p[c] = pneg(edge_delta(n[c], lim));
        }
#pragma unroll
        for (int c = 0; c < N; ++c) {
          if (!live<G, 0>(c)) continue;
          m[c] = d[c];
          if (plim) limit_mono(m[c], p[c], n[c]);
        }
        trace<G, 0, T>(kx, kx, Wr, m, p, clim, out.Anx, out.Apx);
      } else {
        chars<G, 1, T>(ky, Wr, out.Any, out.Apy);
        chars<G, 0, T>(kx, Wr, out.Anx, out.Apx);
      }
      // first-pass x faces of row q, corrected y values
      P AnR[NW], ApL[NW], jn[NW], jp[NW], sum[NW], dif[NW];
#pragma unroll
      for (int w = 0; w < NW; ++w) { AnR[w] = shfl_dn2(out.Anx[w], 1); ApL[w] = shfl_up2(out.Apx[w], 1); }
      if (warp_xedge) {
        if (edge_lo) edge_value<G>(kx, kx.bgp, mc.xout_lo != 0, out.Anx, ApL);
        if (edge_hi) edge_value<G>(kx, kx.bgn, mc.xout_hi != 0, out.Apx, AnR);
      }
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        jn[w] = psub(AnR[w], out.Anx[w]);
        jp[w] = psub(out.Apx[w], ApL[w]);
        Bn_q[w] = out.Any[w];
        Bp_q[w] = out.Apy[w];
      }
      jumps<G>(jn, jp, sum, dif);
      correct<G, 0, T>(kx, sum, dif, Bn_q, Bp_q);
    } else {
      // past the domain's y-hi edge: the values arriving through it
      edge_value<G>(ky, ky.bgn, mc.yout_hi != 0, in.Apy, out.Any);
      edge_value<G>(ky, ky.bgn, mc.yout_hi != 0, in.Bpy, Bn_q);
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const P z = mk2(T(0), T(0));
        out.Apy[w] = z; Bp_q[w] = z; out.Anx[w] = z; out.Apx[w] = z;
      }
    }
    const int yr = q - 1;
    if (defer0 && yr == dlo1) {
      // row 0 of a fault patch: keep what fault_row_finish needs
      P* const st = stash0;
      const P* wo = ring + r_m1 + lane + 1;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        st[(0 * NW + w) * 32] = in.Anx[w]; st[(1 * NW + w) * 32] = in.Apx[w];
        st[(2 * NW + w) * 32] = out.Any[w]; st[(3 * NW + w) * 32] = in.Apy[w];
        st[(4 * NW + w) * 32] = Bn_q[w]; st[(5 * NW + w) * 32] = in.Bpy[w];
      }
#pragma unroll
      for (int c = 0; c < N; ++c) st[(6 * NW + c) * 32] = wo[c * MARCH_RW];
    } else if (yr >= it.y0) {
      // row q-1: transverse correction of its x values, final x faces, update
      P jn[NW], jp[NW], sum[NW], dif[NW], BnR[NW], BpL[NW], du[N], u[N];
#pragma unroll
      for (int w = 0; w < NW; ++w) jn[w] = psub(out.Any[w], in.Any[w]);
      jumps<G>(jn, in.jpy, sum, dif);
      correct<G, 1, T>(kx, sum, dif, in.Anx, in.Apx);
#pragma unroll
      for (int w = 0; w < NW; ++w) { BnR[w] = shfl_dn2(in.Anx[w], 1); BpL[w] = shfl_up2(in.Apx[w], 1); }
      if (warp_xedge) {
        if (edge_lo) edge_value<G>(kx, kx.bgp, mc.xout_lo != 0, in.Anx, BpL);
        if (edge_hi) edge_value<G>(kx, kx.bgn, mc.xout_hi != 0, in.Apx, BnR);
      }
#pragma unroll
      for (int w = 0; w < NW; ++w) { jn[w] = psub(BnR[w], in.Anx[w]); jp[w] = psub(in.Apx[w], BpL[w]); }
      jumps<G>(jn, jp, sum, dif);
      add_update<G, 0, T>(kx, kx, sum, dif, du);
#pragma unroll
      for (int w = 0; w < NW; ++w) jn[w] = psub(Bn_q[w], in.Bny[w]);
      jumps<G>(jn, in.jpB, sum, dif);
      add_update<G, 1, T>(ky, kx, sum, dif, du);
      const P* wo = ring + r_m1 + lane + 1;
#pragma unroll
      for (int c = 0; c < N; ++c) u[c] = padd(wo[c * MARCH_RW], du[c]);
      if (col_valid && yr <= it.y1) store_cell<T, G, PL>(sdst, plane, mc, u, pin);
      if (it.ncap && yr <= it.y1)
        march_capture<T, G>(pp, it, mc, yr, lane, cpos, [&](int kind, P* F) {
          if (kind == 0) face_flux<G, 0, T>(kx, in.Anx, BpL, F);
          else if (kind == 1) face_flux<G, 0, T>(kx, BnR, in.Apx, F);
          else if (kind == 3) face_flux<G, 1, T>(ky, Bn_q, in.Bpy, F);
          else {
            P below[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) below[w] = psub(in.Bpy[w], in.jpB[w]);
            face_flux<G, 1, T>(ky, in.Bny, below, F);
          }
        });
      if constexpr (PATCH) {
        if (col_valid && yr <= it.y1) {
          P F[N];
          if (pp.Fx) {
            face_flux<G, 0, T>(kx, in.Anx, BpL, F);
            store_face<T, G, 0>(pp, x, yr, F);
            if (x == pp.vhi0) { face_flux<G, 0, T>(kx, BnR, in.Apx, F); store_face<T, G, 0>(pp, x + 1, yr, F); }
          }
          if (pp.Fy) {
            P below[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) below[w] = psub(in.Bpy[w], in.jpB[w]);
            face_flux<G, 1, T>(ky, in.Bny, below, F);
            store_face<T, G, 1>(pp, x, yr, F);
            if (yr == pp.vhi1) { face_flux<G, 1, T>(ky, Bn_q, in.Bpy, F); store_face<T, G, 1>(pp, x, yr + 1, F); }
          }
        }
      }
    }
    sdst += anx;
    const int freed = r_m1;
    r_m1 = r_0; r_0 = r_1; r_1 = r_2; r_2 = r_3; r_3 = freed;
    // advance: the jumps over row q of the values from below (at the domain's
    // y-lo edge those arriving through it; a fault patch's row 0 is finished later)
    if (q == dlo1 && !fault) {
      edge_value<G>(ky, ky.bgp, mc.yout_lo != 0, out.Any, in.Apy);
      edge_value<G>(ky, ky.bgp, mc.yout_lo != 0, Bn_q, in.Bpy);
    }
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      out.jpy[w] = psub(out.Apy[w], in.Apy[w]);
      out.jpB[w] = psub(Bp_q[w], in.Bpy[w]);
      out.Bny[w] = Bn_q[w];
      out.Bpy[w] = Bp_q[w];
    }
  };
  for (int q = q_s;; q += 2) {
    row_step(q, c0, c1);
    if (q + 1 > q_e) break;
    row_step(q + 1, c1, c0);
    if (q + 2 > q_e) break;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if constexpr (FORM != MARCH_LEVEL) {
    if (defer0) fault_row_finish<T, G>(pp, it, mc, lane, stash0, PATCH);
  }
}

template <typename T, int G, bool PL = false, int SCH = MARCH_SCH_RUNTIME>
__global__ void __launch_bounds__(32 * MARCH_WARPS, MarchMinBlocks<T, G>::value)
march_kernel(const PatchDev<T>* __restrict__ patches, const MarchItem* __restrict__ items, int nitems,
             const __grid_constant__ MarchConst<T> mc) {
  march_items<T, G, PL, SCH, MARCH_LEVEL>(patches, items, nitems, mc, (int)blockIdx.x);
}

// Both groups in one launch, the in-plane CTAs first, where the launches and
// their order are what a step waits for: after the fault kernel one launch
// finishes the step, and the groups share the SMs that either leaves idle (mixed
// 512x256, slip weakening: 16.5 us a step, 18.8 as separate launches).  The
// patch form, FP64 128x128 with fluxes: 81 us, bound by the FP64 pipe; the tile
// kernel, which forms face states, 557 us.
template <typename T, int SCH, int FORM>
__global__ void __launch_bounds__(32 * MARCH_WARPS, MarchMinBlocks<T, 0>::value)
march_both_kernel(const PatchDev<T>* __restrict__ patches, const MarchItem* __restrict__ items0, int n0,
                  const MarchItem* __restrict__ items1, int n1, const __grid_constant__ MarchConst<T> mc) {
  const int b0 = (n0 + MARCH_WARPS - 1) / MARCH_WARPS;
  if ((int)blockIdx.x < b0) march_items<T, 0, false, SCH, FORM>(patches, items0, n0, mc, (int)blockIdx.x);
  else march_items<T, 1, false, SCH, FORM>(patches, items1, n1, mc, (int)blockIdx.x - b0);
}

// Row 0 of a fault-row strip of group G once the fault kernel has produced the
// first-pass fault states and the fault-face fluxes: the transverse correction
// of the row's x values, its final x faces and its update (the same steps as
// the marching loop, with the stashed row-0 values; st: the lane's).  faces: the
// patch form's fluxes too.
template <typename T, int G>
TMK_D void fault_row_finish(const PatchDev<T>& pp, const MarchItem& it, const MarchConst<T>& mc, int lane,
                            const typename PairOf<T>::P* st, bool faces) {
  using P = typename PairOf<T>::P;
  constexpr int N = Grp<G>::N, NW = kWaves<G>;
  const int x = it.x0 - MARCH_HALO + lane;
  const int dlo0 = pp.dlo0, dhi0 = pp.dhi0, dlo1 = pp.dlo1;
  P Bnx[NW], Bpx[NW], An1[NW], Ap0[NW], Bn1[NW], Bp0[NW], u[N], Fy0[N], Fy1[N];
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    Bnx[w] = st[(0 * NW + w) * 32]; Bpx[w] = st[(1 * NW + w) * 32];
    An1[w] = st[(2 * NW + w) * 32]; Ap0[w] = st[(3 * NW + w) * 32];
    Bn1[w] = st[(4 * NW + w) * 32]; Bp0[w] = st[(5 * NW + w) * 32];
  }
#pragma unroll
  for (int c = 0; c < N; ++c) u[c] = st[(6 * NW + c) * 32];
  const int fi1 = x - (pp.vlo0 - 1);
  const bool ok1 = fi1 >= 0 && fi1 < pp.nfirst && x >= dlo0 && x <= dhi0;
  const int nv = pp.vhi0 - pp.vlo0 + 1, fi2 = x - pp.vlo0;
  const bool ok2 = fi2 >= 0 && fi2 < nv;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    const int g = Grp<G>::glob(c);
    Fy0[c] = ok2 ? mk2((T)pp.ffault[(size_t)g * nv + fi2], (T)pp.ffault[(size_t)(11 + g) * nv + fi2])
                 : mk2(T(0), T(0));
  }
  // y face 1 less the first-pass fault state, as the sums (2 ds) and
  // differences (2 Z dv) of the jumps that the transverse term takes
  P sum[NW], dif[NW], jn[NW], jp[NW], BnR[NW], BpL[NW];
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    const int gv = Grp<G>::glob(wave_v<G, 1>(w)), gs = Grp<G>::glob(wave_s<G, 1>(w));
    P v0 = mk2(T(0), T(0)), s0 = v0;
    if (ok1) {
      const double b = (double)mc.ky.s0[G == 0 ? w : 2];
      v0 = mk2((T)pp.first[(size_t)gv * pp.nfirst + fi1], (T)pp.first[(size_t)(11 + gv) * pp.nfirst + fi1]);
      s0 = mk2((T)(pp.first[(size_t)gs * pp.nfirst + fi1] - b), (T)(pp.first[(size_t)(11 + gs) * pp.nfirst + fi1] - b));
    }
    sum[w] = psub(padd(An1[w], Ap0[w]), padd(s0, s0));
    dif[w] = pfma(pneg(is_p<G>(w) ? mc.ky.Zp : mc.ky.Zs), padd(v0, v0), psub(An1[w], Ap0[w]));
  }
  correct<G, 1, T>(mc.kx, sum, dif, Bnx, Bpx);
#pragma unroll
  for (int w = 0; w < NW; ++w) { BnR[w] = shfl_dn2(Bnx[w], 1); BpL[w] = shfl_up2(Bpx[w], 1); }
  if (x == dlo0) edge_value<G>(mc.kx, mc.kx.bgp, mc.xout_lo != 0, Bnx, BpL);
  if (x == dhi0) edge_value<G>(mc.kx, mc.kx.bgn, mc.xout_hi != 0, Bpx, BnR);
  face_flux<G, 1, T>(mc.ky, Bn1, Bp0, Fy1);
  if (it.ncap) {
    int cpos = it.cap0;
    march_capture<T, G>(pp, it, mc, dlo1, lane, cpos, [&](int kind, P* F) {
      if (kind == 0) face_flux<G, 0, T>(mc.kx, Bnx, BpL, F);
      else if (kind == 1) face_flux<G, 0, T>(mc.kx, BnR, Bpx, F);
      else {
#pragma unroll
        for (int c = 0; c < N; ++c) F[c] = kind == 2 ? Fy0[c] : Fy1[c];
      }
    });
  }
  const bool col_valid = x >= it.x0 && x < it.x0 + MARCH_COLS && x >= pp.vlo0 && x <= pp.vhi0;
  if (faces && col_valid) {
    P F[N];
    if (pp.Fx) {
      face_flux<G, 0, T>(mc.kx, Bnx, BpL, F);
      store_face<T, G, 0>(pp, x, dlo1, F);
      if (x == pp.vhi0) { face_flux<G, 0, T>(mc.kx, BnR, Bpx, F); store_face<T, G, 0>(pp, x + 1, dlo1, F); }
    }
    if (pp.Fy) {
      store_face<T, G, 1>(pp, x, dlo1, Fy0);
      if (pp.vhi1 == dlo1) store_face<T, G, 1>(pp, x, dlo1 + 1, Fy1);
    }
  }
  if (col_valid) {
#pragma unroll
    for (int w = 0; w < NW; ++w) { jn[w] = psub(BnR[w], Bnx[w]); jp[w] = psub(Bpx[w], BpL[w]); }
    jumps<G>(jn, jp, sum, dif);
    P du[N];
    add_update<G, 0, T>(mc.kx, mc.kx, sum, dif, du);
#pragma unroll
    for (int c = 0; c < N; ++c) u[c] = padd(u[c], pfma(psub(Fy1[c], Fy0[c]), mc.sc, du[c]));
    const unsigned plane = (unsigned)pp.anx * (unsigned)pp.any;
    const size_t o = fab_idx(pp, 0, x, dlo1);
    T* const out0 = pp.Uout + o;
    P pin[3];
    if (mc.plastic) {
      plastic_inputs<T>(pp.Uin + o, out0, plane, pin);
      store_cell<T, G, true>(out0, plane, mc, u, pin);
    } else {
      store_cell<T, G, false>(out0, plane, mc, u, pin);
    }
  }
}

// One warp per fault-row strip: rows0 (in-plane) then rows1 (antiplane).  With
// the fused plastic return the antiplane rows are finished by a launch of
// their own before the in-plane ones (whose stores apply the return).
template <typename T>
__global__ void __launch_bounds__(32 * MARCH_WARPS) march_fault_row_kernel(const PatchDev<T>* __restrict__ patches,
                                                                           const MarchItem* __restrict__ rows0, int n0,
                                                                           const MarchItem* __restrict__ rows1, int n1,
                                                                           const __grid_constant__ MarchConst<T> mc) {
  const int wid = blockIdx.x * MARCH_WARPS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  auto stash = [&](const MarchItem& it, int g, int n) {
    return reinterpret_cast<const typename PairOf<T>::P*>(mc.stash[g]) + (size_t)it.fslot * MARCH_STASH_VECS * n * 32 + lane;
  };
  if (wid < n0) {
    const MarchItem it = rows0[wid];
    fault_row_finish<T, 0>(patches[it.patch], it, mc, lane, stash(it, 0, Grp<0>::N), false);
  } else if (wid < n0 + n1) {
    const MarchItem it = rows1[wid - n0];
    fault_row_finish<T, 1>(patches[it.patch], it, mc, lane, stash(it, 1, Grp<1>::N), false);
  }
}


}  // namespace tmk
