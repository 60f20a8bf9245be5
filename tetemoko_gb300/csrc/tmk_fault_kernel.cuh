// tmk_fault_kernel.cuh -- the friction solves of a level's fault faces.
//
// Per face, in the reference's call order at the y-lo face
// (srcLinElast/LinElastPatchGodunov.cpp:289-452 with ibcLinElast/RSIBC.cpp:
// 166-336, SWIBC.cpp:161-331): the first-pass solve with the persistent
// boundary data, the half-step predicted boundary data, the solve of the states
// corrected by the x fluxes of the row, the fault-face fluxes and the
// boundary-data update.
//
// What bounds it: the latency of one face's chain.  On GB300 an FP64
// instruction holds its SM sub-partition's FP64 pipe for 64 cycles whatever
// the number of active lanes, so a warp's time is its count of FP64
// instructions times 31 ns (ncu: an FP64 exp is 17 of them, log 32, a division
// 10), conversions between FP64 and FP32 included.  Hence
//   * the laws read the predicted states only through their left-going
//     characteristic values An (tmk_march.cuh) and, as a first guess, the slip
//     rate, so a state crosses to the solve as two or three numbers a side;
//   * predictors, per-face constants, x corrections and solves sit on different
//     warps, hence sub-partitions, and only the solves' chain is serial;
//   * constants are computed on the host, boundary data are requested first;
//   * the logarithms of the state evolution and of the solve's bracket are
//     evaluated only where a short series or an FP32 test does not decide.
#pragma once
#include "tmk_launch.h"
#include "tmk_march.cuh"

namespace tmk {

template <typename T>
struct FaultConst {
  MK<T> kx, ky;
  T nbg[9];                 // minus the background
  typename PairOf<T>::P lZp, lZs;       // what the impedances lose in T (rv Z in y)
  T sig[9];                 // characteristic Courant numbers (general predictor)
  Consts<T> k;
  int fast;                 // PPM with primitive limiting: the deltas of tmk_march.cuh
  int xout_lo, xout_hi;
  double s0[3];             // background stresses of the y direction (syy, sxy, syz)
  double inv_rho, lam, l2g, G;
  void load(const DevParams& p, double dt, double dx) {
    kx.load(p, 0, dt / dx);
    ky.load(p, 1, dt / dx);
    for (int c = 0; c < 9; ++c) nbg[c] = (T)-p.bg[c];
    const double l[9] = {-p.cp, -p.cs, -p.cs, 0.0, 0.0, 0.0, p.cs, p.cs, p.cp};
    for (int c = 0; c < 9; ++c) sig[c] = (T)(l[c] * (dt / dx));
    k.load(p);
    const T lp = (T)(p.Zp - (double)(T)p.Zp), ls = (T)(p.Zs - (double)(T)p.Zs);
    lZp = mk2(lp, -lp); lZs = mk2(ls, -ls);
    fast = p.order == 2 && p.prim_lim && !p.char_lim;
    xout_lo = p.bc[0] == 0; xout_hi = p.bc[1] == 0;
    s0[0] = p.bg[4]; s0[1] = p.bg[6]; s0[2] = p.bg[8];
    inv_rho = 1.0 / p.rho; lam = p.lam; l2g = p.lam + 2.0 * p.G; G = p.G;
  }
};

// threads: x and y predictors of both sides (4 SEG), the faces (SEG), and the
// two cells or faces beyond either end of the segment (10, rounded to a warp)
constexpr int fault_threads(int seg) { return seg == FAULT_SEG ? 192 : 96; }

// the wave pairs of direction D: P, S of (vx, vy), S of vz
template <int D> TMK_HD constexpr int pair_v(int w) { return w == 0 ? D : w == 1 ? 1 - D : 2; }
template <int D> TMK_HD constexpr int pair_s(int w) { return w == 0 ? 3 + D : w == 1 ? 6 : 7 + D; }
// the half of a pair constant that belongs to side s
template <typename P> TMK_D auto side_of(const P& p, int s) { return s ? p.y : p.x; }

TMK_D float one_slope(float nl, float nr, bool limit) {
  const float q = 0.25f * (nl + nr);
  if (!limit) return q;
  return nl * nr > 0.f ? clip_mag(q, nl, nr) : 0.f;
}
TMK_D double one_slope(double nl, double nr, bool limit) {
  const double q = mul_pow2<-2>(nl + nr);
  if (!limit) return q;
  return same_sign1(nl, nr) ? clip_mag(q, nl, nr) : 0.0;
}

// Traced characteristic values of one side of cell (i, j) in direction D: An,
// Ap (x) or An alone and the velocities of the S pairs of the lo-face state (y,
// where only the states entering the fault are read).
template <int D, typename T>
TMK_D void fault_chars(const PatchDev<T>& p, const FaultConst<T>& fc, const DevParams& P, int s, int i, int j,
                       T* An, T* Ap, T* vlo) {
  bool in[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const int c = (D == 0 ? i : j) - 2 + m;
    in[m] = c >= (D == 0 ? p.dlo0 : p.dlo1) && c <= (D == 0 ? p.dhi0 : p.dhi1);
  }
  const MK<T>& k = D == 0 ? fc.kx : fc.ky;
  if (fc.fast) {
    T w[6][5];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const int g = 11 * s + (c < 3 ? pair_v<D>(c) : pair_s<D>(c - 3));
#pragma unroll
      for (int m = 0; m < 5; ++m)
        w[c][m] = in[m] ? p.Uin[fab_idx(p, g, D == 0 ? i - 2 + m : i, D == 0 ? j : j - 2 + m)] : T(0);
    }
    T dm[6], dp[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      T nl = w[c][1] - w[c][2], nr = w[c][2] - w[c][3];
      T n2l = w[c][0] - w[c][1], n2r = w[c][3] - w[c][4];
      if (!in[1]) nl = in[3] ? nr : T(0);
      if (!in[3]) nr = in[1] ? nl : T(0);
      if (!in[0]) n2l = nl;
      if (!in[4]) n2r = nr;
      const T n = one_slope(nl, nr, true), nm = one_slope(n2l, nl, true), np = one_slope(nr, n2r, true);
      T m = in[1] ? fma(n - nm, T(2.0 / 3.0), nl) : n + n;
      T q = in[3] ? fma(np - n, T(2.0 / 3.0), -nr) : -(n + n);
      const T b = T(8) * n, m2 = m + m, q2 = q + q;
      dm[c] = clip_mag(m, q2, b);
      dp[c] = clip_mag(q, m2, b);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const T Z = side_of(q == 0 ? k.Zp : k.Zs, D == 0 ? 0 : s), a = q == 0 ? k.aP : k.aS, b = q == 0 ? k.bP : k.bS;
      const T v = w[q][2], sr = w[3 + q][2] + fc.nbg[pair_s<D>(q)];
      const T nm = fma(Z, dm[q], dm[3 + q]), np = fma(Z, dp[q], dp[3 + q]);
      const T dn = fma(b, np, a * nm);          // the traced left-going delta at the lo face
      // the friction laws take the unrounded Z: the rest of its product with v
      if constexpr (D == 1 && !kExact<T>) An[q] = fma(Z, v, fma(side_of(q == 0 ? fc.lZp : fc.lZs, s), v, sr + dn));
      else An[q] = fma(Z, v, sr) + dn;
      const T pm = fma(-Z, dm[q], dm[3 + q]);
      if (D == 0) {
        const T pp = fma(-Z, dp[q], dp[3 + q]);
        Ap[q] = fma(-Z, v, sr) + fma(b, pm, a * pp);
      } else if (q > 0) {
        // deltas are doubled: the untraced right-going one is pm / 2
        vlo[q - 1] = v + side_of(k.hZs, s) * (dn - T(0.5) * pm);
      }
    }
  } else {
    T w5[NSIDE][5], WM[NSIDE], WP[NSIDE];
    for (int c = 0; c < NSIDE; ++c)
      for (int m = 0; m < 5; ++m)
        w5[c][m] = in[m] ? p.Uin[fab_idx(p, 11 * s + c, D == 0 ? i - 2 + m : i, D == 0 ? j : j - 2 + m)] : T(0);
    ppm_predict<D, T>(fc.k, (D == 1 && s == 1) ? T(-1) : T(1), w5, in, P.prim_lim != 0, P.char_lim != 0, fc.sig, WM,
                      WP, P.order, P.fourth != 0);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const T Z = side_of(q == 0 ? k.Zp : k.Zs, D == 0 ? 0 : s);
      const T n0 = fc.nbg[pair_s<D>(q)];
      const T v = WM[pair_v<D>(q)], sr = WM[pair_s<D>(q)] + n0;
      if constexpr (D == 1 && !kExact<T>) An[q] = fma(Z, v, fma(side_of(q == 0 ? fc.lZp : fc.lZs, s), v, sr));
      else An[q] = fma(Z, v, sr);
      if (D == 0) Ap[q] = fma(-Z, WP[pair_v<D>(q)], WP[pair_s<D>(q)] + n0);
      else if (q > 0) vlo[q - 1] = WM[pair_v<D>(q)];
    }
  }
}

template <typename Real, int SEG>
__global__ void __launch_bounds__(fault_threads(SEG)) fault_kernel(const PatchDev<Real>* __restrict__ patches,
                                                                   const int* __restrict__ fault_patches,
                                                                   const DevParams* __restrict__ params, double time,
                                                                   DevStatus* st,
                                                                   const __grid_constant__ FaultConst<Real> fc,
                                                                   int after) {
  using T = Real;
  constexpr bool kFp64 = std::is_same<Real, double>::value;
  constexpr int NCELL = SEG + 2;             // cells / faces [s0-1, s0+SEG]
  __shared__ T sXn[2][3][NCELL], sXp[2][3][NCELL];      // x values of the fault-row cells
  __shared__ T sAn[2][3][NCELL], sV[2][2][NCELL];       // y values entering the faces, first pass
  __shared__ T sVc[2][2][SEG];                          // ... velocities corrected by the x fluxes
  __shared__ double sA[2][3][NCELL], sB[2][3][SEG];     // the whole values (with the background) in FP64, both passes
  // The kernel launched after this one may be scheduled now (it reads none of
  // this kernel's outputs before it waits for it).  As a programmatic dependent
  // of the in-plane marching kernel this one reads nothing that kernel writes
  // (the state it reads is the step's input buffer) and waits for it before
  // exiting, so that the step's kernels complete in order.  As the step's first
  // kernel after its ghost cells (`after`) it waits for what is before it, also
  // for the kernel it lets start, which reads those cells.
  if (after) pdl_wait();
  pdl_trigger();
  const PatchDev<Real>& p = patches[fault_patches[blockIdx.y]];
  const DevParams& P = params[p.scen];
  const int s0 = p.vlo0 + blockIdx.x * SEG;
  if (s0 > p.vhi0) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  const int s1 = min(s0 + SEG - 1, p.vhi0), j0 = p.dlo1;
  // faces whose first-pass state this segment produces: its own, plus the
  // ghost faces lo-1 / hi+1 of the patch for the first / last segment
  const int fa = (s0 == p.vlo0) ? max(p.vlo0 - 1, p.dlo0) : s0;
  const int fb = (s1 == p.vhi0) ? min(p.vhi0 + 1, p.dhi0) : s1;
  const int tid = threadIdx.x;
  const double dt = p.dt, dx = p.dx;
  const int bs = p.bnx;

  // roles: x predictor (side, cell), y predictor (side, face), face
  int role = -1, side = 0, ci = 0;
  if (tid < 5 * SEG) {
    role = min(tid / (2 * SEG), 2);
    side = (tid / SEG) & 1;
    ci = 1 + tid % SEG;
  } else if (tid < 5 * SEG + 10) {
    const int e = tid - 5 * SEG;
    role = min(e >> 2, 2);
    side = (e >> 1) & 1;
    ci = (e & 1) ? SEG + 1 : 0;
    if (ci == SEG + 1 && s1 + 1 < s0 + SEG) ci = -1;      // a short segment holds that cell already
  }
  const int i = s0 - 1 + ci;
  const bool face = role == 2 && ci >= 0 && i >= fa && i <= fb;
  const bool own = face && i >= s0 && i <= s1;

  // (A) predictors; on the face threads the face's constants and boundary data
  RSFaceK fk;
  SWFaceK wk;
  double* const Bi = p.B + (i - p.blo0);
  double b_state = 0.0, b_rt = 0.0, b_s0 = 0.0, b_s1 = 0.0, b_s2 = 0.0;
  const bool rs = P.fault_law == 1;
  if (role == 2) {
    if (face) {
      b_state = Bi[(rs ? 10 : 7) * bs];
      if (own) {
        b_rt = Bi[(rs ? 9 : 8) * bs];
        b_s0 = Bi[(rs ? 6 : 5) * bs];
        b_s1 = Bi[(rs ? 7 : 6) * bs];
        if (rs) b_s2 = Bi[8 * bs];
      }
      if (rs) fk = rs_face_k(P, rs_face(P, p.fric, i - p.blo0, bs), p.fric != nullptr, (i + 0.5) * dx - P.rs_x0, b_state);
      else wk = sw_face_k(P, cell_from<!kFp64>(i, dx, P.sw_fbc0));
    }
  } else if (role == 0 && ci >= 0) {
    if (i >= p.dlo0 && i <= p.dhi0 && i <= s1 + 1) {
      T An[3], Ap[3];
      fault_chars<0, T>(p, fc, P, side, i, j0, An, Ap, nullptr);
#pragma unroll
      for (int q = 0; q < 3; ++q) { sXn[side][q][ci] = An[q]; sXp[side][q][ci] = Ap[q]; }
    }
  } else if (role == 1 && ci >= 0) {
    if (i >= fa && i <= fb) {
      T An[3], v[2];
      fault_chars<1, T>(p, fc, P, side, i, j0, An, nullptr, v);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        sAn[side][q][ci] = An[q];
        sA[side][q][ci] = (double)An[q] + fc.s0[q];
      }
      sV[side][0][ci] = v[0];
      sV[side][1][ci] = v[1];
    }
  }
  __syncthreads();

  FaultFace f;
  double half = 0.0;
  if (face) {
    // (B) first-pass friction solve with the persistent boundary data, and the
    //     half-step predicted boundary data (updateBoundary, final=false)
    int it = 0;
    if (rs)
      it = rs_face_solve<kFp64>(P, fk, sA[0][0][ci], sA[1][0][ci], sA[0][1][ci], sA[1][1][ci], b_state,
                                sV[0][0][ci] - sV[1][0][ci], sV[0][1][ci] - sV[1][1][ci], f);
    else
      sw_face_solve(P, wk, sA[0][0][ci], sA[1][0][ci], sA[0][1][ci], sA[1][1][ci], sA[0][2][ci], sA[1][2][ci], b_state,
                    f);
    if (it > RS_IMAX) atomicAdd(&st->newton_maxed, 1ull);
    // the components of the face state that transverse terms read
    double* first = p.first + (i - (p.vlo0 - 1));
    const int nf = p.nfirst;
    first[0] = f.vx1; first[1 * nf] = f.vy; first[2 * nf] = f.vz1;
    first[4 * nf] = f.syy; first[6 * nf] = f.sxy; first[8 * nf] = f.syz;
    first[11 * nf] = f.vx2; first[12 * nf] = f.vy; first[13 * nf] = f.vz2;
    first[15 * nf] = f.syy; first[17 * nf] = f.sxy; first[19 * nf] = f.syz;
    if (own) half = rs ? rs_state_next(P, fk, b_state, f.V, 0.5 * dt) : b_state + (0.5 * dt) * f.V;
  } else if (tid < 2 * SEG) {
    // (C) transverse correction of the entering values by the first-pass x
    //     fluxes of the fault row (the same terms as the marching kernels')
    const int s = side, fi = s0 + ci - 1;
    if (fi <= s1) {
      T sum[3], dif[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const T an = sXn[s][q][ci], ap = sXp[s][q][ci];
        T apl = sXp[s][q][ci - 1], anr = sXn[s][q][ci + 1];
        if (fi == p.dlo0) apl = fc.xout_lo ? side_of(fc.kx.bgp[q], s) : -an - T(2) * fc.kx.s0[q];
        if (fi == p.dhi0) anr = fc.xout_hi ? side_of(fc.kx.bgn[q], s) : -ap - T(2) * fc.kx.s0[q];
        const T jn = anr - an, jp = ap - apl;
        sum[q] = jn + jp;
        dif[q] = jn - jp;
      }
      const T cvP = side_of(fc.kx.cvP, s), cvS = side_of(fc.kx.cvS, s);
      sB[s][0][ci - 1] = (double)(sAn[s][0][ci] + fma(cvP, sum[1], fc.kx.c_lam * dif[0])) + fc.s0[0];
      sB[s][1][ci - 1] = (double)(sAn[s][1][ci] + fma(cvS, sum[0], fc.kx.c_G * dif[1])) + fc.s0[1];
      sB[s][2][ci - 1] = (double)(sAn[s][2][ci] + cvS * sum[2]) + fc.s0[2];
      // the velocities take the velocity part alone: 2 hZs cvS = its factor
      const T cv = T(2) * side_of(fc.ky.hZs, s) * cvS;
      sVc[s][0][ci - 1] = fma(cv, sum[0], sV[s][0][ci]);
      sVc[s][1][ci - 1] = fma(cv, sum[2], sV[s][1][ci]);
    }
  }
  __syncthreads();

  if (own) {
    // (D) final friction solve with the predicted boundary data
    const int c = ci - 1;
    int it = 0;
    if (rs)
      it = rs_face_solve<kFp64>(P, fk, sB[0][0][c], sB[1][0][c], sB[0][1][c], sB[1][1][c], half,
                                sVc[0][0][c] - sVc[1][0][c], sVc[0][1][c] - sVc[1][1][c], f);
    else
      sw_face_solve(P, wk, sB[0][0][c], sB[1][0][c], sB[0][1][c], sB[1][1][c], sB[0][2][c], sB[1][2][c], half, f);
    if (it > RS_IMAX) atomicAdd(&st->newton_maxed, 1ull);
    // (E) y fluxes through the fault face (GETFLUXF)
    double* ff = p.ffault + (i - p.vlo0);
    const int nv = p.vhi0 - p.vlo0 + 1;
    const double fvx = -f.sxy * fc.inv_rho, fvy = -f.syy * fc.inv_rho, fvz = -f.syz * fc.inv_rho;
    const double fl = -f.vy * fc.lam, f2 = -f.vy * fc.l2g;
    ff[0] = fvx; ff[1 * nv] = fvy; ff[2 * nv] = fvz;
    ff[3 * nv] = fl; ff[4 * nv] = f2; ff[5 * nv] = fl;
    ff[6 * nv] = -f.vx1 * fc.G; ff[7 * nv] = 0.0; ff[8 * nv] = -f.vz1 * fc.G;
    ff[11 * nv] = -fvx; ff[12 * nv] = -fvy; ff[13 * nv] = -fvz;
    ff[14 * nv] = -fl; ff[15 * nv] = -f2; ff[16 * nv] = -fl;
    ff[17 * nv] = f.vx2 * fc.G; ff[18 * nv] = 0.0; ff[19 * nv] = f.vz2 * fc.G;
    // (F) boundary-data update with the final fault state (final=true, t+dt):
    //     RSSETBND, SWSETBND
    const double t1 = time + dt;
    if (rs) {
      const double np = rs_state_next(P, fk, b_state, f.V, dt);
      Bi[0] = f.Vx;
      Bi[1 * bs] = f.Vz;
      Bi[2 * bs] = f.V;
      Bi[3 * bs] = f.sxy + fk.tau0;
      Bi[4 * bs] = f.syz;
      Bi[5 * bs] = f.syy;
      Bi[6 * bs] = b_s0 + dt * f.Vx;
      Bi[7 * bs] = b_s1 + dt * f.Vz;
      Bi[8 * bs] = b_s2 + dt * f.V;
      if (b_rt > t1) Bi[9 * bs] = f.V > P.rs_thr ? t1 : 1e10;
      Bi[10 * bs] = np;
      if (isnan(np)) report(st, ST_NAN, (long long)i);
    } else {
      Bi[0] = f.Vx;
      Bi[1 * bs] = f.Vz;
      Bi[2 * bs] = f.sxy;
      Bi[3 * bs] = f.syz;
      Bi[4 * bs] = f.V;
      Bi[5 * bs] = b_s0 + dt * f.Vx;
      Bi[6 * bs] = b_s1 + dt * f.Vz;
      Bi[7 * bs] = b_state + dt * f.V;
      if (b_rt > t1 && f.V > P.sw_thr) Bi[8 * bs] = t1;
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace tmk
