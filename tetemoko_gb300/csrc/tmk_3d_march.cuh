// The 3-D patch step on characteristic values (PPM with primitive limiting),
// both forms: T = float with an FP64 state (mixed), T = double.
//
// Past the limiters the step of a uniform medium is linear with constant
// coefficients, so the values that meet at the faces of a cell (tmk_march.cuh)
// carry everything: for each direction D and wave pair w of D
//   An = s + Z v + traced delta at the cell's lo face, Ap = s - Z v + ... at its
// hi face, w = 0 the P pair (v_D, s_DD), w = 1, 2 the S pairs (v_t, s_Dt) of the
// two other directions t, ascending.  The face states WHalf1[D] are the pairs
// (An of a cell, Ap of the one below); the transverse term of direction E on
// the values of D needs the jumps of E's values over the cell; so WHalf2[D][E]
// are the pairs of A_D + T_E(A_E) with scale 1/3, WHalf[D] those of
// A_D + T_E(WHalf2[E][F]) + T_F(WHalf2[F][E]) with scale 1/2, and the update of
// a cell reads the values of its 27 neighbours
// (srcLinElast/LinElastPatchGodunov.cpp:174-469).  Hence two passes over the
// patch instead of thirteen:
//   values_kernel   the limited predictors of all three directions -> 18 pairs
//                   (n, p) per cell
//   step_kernel     everything else, marching in z over a tile of x and y
// and between them plane_kernel, the friction solves of the fault plane, which
// read the first kernel's values alone: WHalf1[1], WHalf2[1][0], WHalf2[1][2],
// WHalf[1] and the boundary data of one face are one thread's work.
//
// What bounds them, at 192x96x96 mixed (rate and state): the FP32 copy of the
// state (80 us) and the z values (40 us) DRAM; the x and y values (73 us) the
// issue of the limiters; the plane (48 us) the latency of four dependent solves,
// beside which the step's tiles away from the fault run; the step (294 us)
// issue, 48 % of slots, and its last wave of CTAs.  A call 690 us; one pass per
// term, each through memory, took 1383 us.  FP64 (64x48x48): every kernel the
// FP64 pipe; 581 us, was 2703 us.  32-cell boxes of a 96x64x64 level, mixed: 807
// us, was 1097 (520 of either is reading the state back).
#pragma once

#include "tmk_3d.cuh"
#include "tmk_march.cuh"

namespace tmk {
namespace d3 {

// ------------------------------------------------------------ waves
template <int D> constexpr int kTan1 = D == 0 ? 1 : 0;
template <int D> constexpr int kTan2 = D == 2 ? 1 : 2;
template <int D> TMK_HD constexpr int wv(int w) { return w == 0 ? D : w == 1 ? kTan1<D> : kTan2<D>; }
TMK_HD constexpr int shear(int a, int b) { return 5 + a + b; }             // 6 xy, 7 xz, 8 yz
template <int D> TMK_HD constexpr int ws(int w) { return w == 0 ? 3 + D : shear(D, wv<D>(w)); }
template <int D> TMK_HD constexpr int slot(int t) { return t == kTan1<D> ? 1 : 2; }   // the S pair with tangent t

// launch constants (the same products as the 2-D kernels': MK in tmk_march.cuh)
template <typename T>
struct K3 {
  T Zp, Zs, aP, bP, aS, bS;
  T c_lam[2], c_G[2], c_vP[2], c_vS[2];   // transverse terms, scales 1/2 and 1/3
  T e_v, e_l2g, e_lam, e_G;               // update
  T hZp, hZs, irho, l2g, lam, G;          // face states and fluxes
  T nbg[9];                               // minus the background
  float lZs;                              // what Zs loses in T
  double s0[3];                           // background syy, sxy, syz (the fault's tractions)
  int out[6];                             // absorbing edge (else free)
  void load(const DevParams& p, double dt, double dx) {
    const double r = dt / dx, sp = p.cp * r, ss = p.cs * r;
    Zp = (T)p.Zp; Zs = (T)p.Zs;
    const double zp = (double)Zp, zs = (double)Zs;         // the rounded ones (MK)
    lZs = (float)(p.Zs - zs);
    aP = (T)(0.5 * (1.0 - sp) * (1.0 - sp)); bP = (T)(0.5 * (sp * sp - sp));
    aS = (T)(0.5 * (1.0 - ss) * (1.0 - ss)); bS = (T)(0.5 * (ss * ss - ss));
    for (int k = 0; k < 2; ++k) {
      const double sc = k == 0 ? 0.5 : 1.0 / 3.0;
      c_lam[k] = (T)(sc * r * p.lam * (0.5 / zp));
      c_G[k] = (T)(sc * r * p.G * (0.5 / zs));
      c_vP[k] = (T)(zp * (0.5 * sc * r / p.rho));
      c_vS[k] = (T)(zs * (0.5 * sc * r / p.rho));
    }
    const double l = p.lam + 2.0 * p.G;
    e_v = (T)(0.5 * r / p.rho);
    e_l2g = (T)(r * l * (0.5 / zp)); e_lam = (T)(r * p.lam * (0.5 / zp)); e_G = (T)(r * p.G * (0.5 / zs));
    hZp = (T)(0.5 / zp); hZs = (T)(0.5 / zs); irho = (T)(1.0 / p.rho);
    l2g = (T)l; lam = (T)p.lam; G = (T)p.G;
    for (int c = 0; c < 9; ++c) nbg[c] = (T)-p.bg[c];
    s0[0] = p.bg[4]; s0[1] = p.bg[6]; s0[2] = p.bg[8];
    for (int k = 0; k < 6; ++k) out[k] = p.bc[k] == 0;
  }
};

// ------------------------------------------------------------ work of a patch
// the patch and local index of work item t (uniform over the warp or CTA that asks)
template <typename T> TMK_D const Step3<T>* find_item(const One<T>& s, long long t, long long& lt) { lt = t; return &s.g; }
template <typename T> TMK_D const Step3<T>* find_item(const Many<T>& s, long long t, long long& lt) { return s.find(t, lt); }

// values (n, p) of side s, direction D, wave w: one plane over the slope box each
template <typename T> TMK_D typename PairOf<T>::P* val_plane(const Step3<T>& g, int s, int D, int w) {
  using V = typename PairOf<T>::P;
  return reinterpret_cast<V*>(g.AF) + ((s * 3 + D) * 3 + w) * g.S.cells();
}
// the fault faces' states (stress less background, velocity), level l, side s, wave w
template <typename T> TMK_D typename PairOf<T>::P* plane_face(const Step3<T>& g, int l, int s, int w) {
  using V = typename PairOf<T>::P;
  return reinterpret_cast<V*>(g.FA) + ((l * 2 + s) * 3 + w) * g.fplane.cells();
}

// ------------------------------------------------------------ predictors
// Components a marching warp stages: for x and y (DM = 1) all but szz, for z
// (DM = 2) the six live there.
template <int DM> constexpr int kValComps = DM == 1 ? 8 : 6;
template <int DM> TMK_HD constexpr int val_comp(int k) {
  return DM == 1 ? (k < 5 ? k : k + 1) : (k < 3 ? k : k == 3 ? 5 : k + 3);
}
template <int DM> TMK_HD constexpr int val_index(int c) { return DM == 1 ? (c < 5 ? c : c - 1) : (c < 3 ? c : c == 5 ? 3 : c - 3); }
template <int D> TMK_HD constexpr bool wave_comp(int c) {
  return c < 3 || c == 3 + D || c == shear(D, kTan1<D>) || c == shear(D, kTan2<D>);
}

template <int DM, int D, typename T>
TMK_D void trace3(const K3<T>& k, const typename PairOf<T>::P* w, const typename PairOf<T>::P* m,
                  const typename PairOf<T>::P* p, typename PairOf<T>::P* An, typename PairOf<T>::P* Ap) {
  using P = typename PairOf<T>::P;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int v = val_index<DM>(wv<D>(q)), s = val_index<DM>(ws<D>(q));
    const T z = q == 0 ? k.Zp : k.Zs;
    const P Z = mk2(z, D == 1 ? -z : z), nZ = pneg(Z);
    const P a = kall(q == 0 ? k.aP : k.aS), b = kall(q == 0 ? k.bP : k.bS);
    const P nm = pfma(Z, m[v], m[s]), np = pfma(Z, p[v], p[s]);
    const P pm = pfma(nZ, m[v], m[s]), pp = pfma(nZ, p[v], p[s]);
    An[q] = pfma(b, np, pfma(a, nm, pfma(Z, w[v], w[s])));
    Ap[q] = pfma(b, pm, pfma(a, pp, pfma(nZ, w[v], w[s])));
  }
}
// to: the cell's address in plane 0
template <int D, typename V>
TMK_D void store_values(V* to, unsigned plane, const V* An, const V* Ap) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    *plane_ptr(to, plane, 3 * D + q) = mk2(An[q].x, Ap[q].x);
    *plane_ptr(to, plane, 9 + 3 * D + q) = mk2(An[q].y, Ap[q].y);
  }
}

template <typename T, int DM, int K>
TMK_D void stage_column(unsigned dst, const T* src, const T* src2, unsigned plane, unsigned nbytes) {
  if constexpr (K < kValComps<DM>) {
    constexpr int off = K * 32 * 2 * (int)sizeof(T);
    cp_async_elem<T, off>(dst, plane_ptr(src, plane, val_comp<DM>(K)), nbytes);
    cp_async_elem<T, off + (int)sizeof(T)>(dst, plane_ptr(src2, plane, val_comp<DM>(K)), nbytes);
    stage_column<T, DM, K + 1>(dst, src, src2, plane, nbytes);
  }
}

// A warp marches along DM over a run of rows (planes) with x in its lanes: the
// limited deltas of DM from a rolling window of rows in shared memory, and
// (DM = 1) those of x from its neighbour lanes, where a delta reads the slopes
// of both neighbours (two halo lanes on either side of a strip).  For z the
// lanes hold 32 consecutive cells of the plane, across the ends of rows.
template <typename T, int DM, typename Src>
__global__ void __launch_bounds__(32 * VAL_WARPS, sizeof(T) == 4 ? 4 : 2)
values_kernel(const __grid_constant__ Src src, const __grid_constant__ K3<T> k, long long nitems) {
  using P = typename PairOf<T>::P;
  constexpr int NC8 = kValComps<DM>, RP = NC8 * 32;
  constexpr bool X = DM == 1;
  extern __shared__ __align__(16) unsigned char val_smem[];
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const unsigned lane = threadIdx.x & 31u;
  // the z kernel, scheduled beside the x and y one, completes after it
  if constexpr (X) asm volatile("griddepcontrol.launch_dependents;");
  const long long item = (long long)blockIdx.x * VAL_WARPS + warp;
  long long lt = 0;
  const Step3<T>* gp = item < nitems ? find_item<T>(src, item, lt) : nullptr;
  if (!gp) {
    if constexpr (!X) asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  const Step3<T>& g = *gp;
  // item -> cell of the lane, run along DM
  const unsigned u = (unsigned)lt;
  const int run = g.vrun;
  int x, y, z;
  bool own = true;                      // not a halo lane
  if constexpr (X) {
    const Strips st = strips(g.S.n[0], VAL_HALO);
    const unsigned nr = (unsigned)cdiv(g.S.n[1], run), nw = nr * (unsigned)(st.whole * g.S.n[2]);
    const bool rest = u >= nw;
    const unsigned gl = rest ? (unsigned)st.group : 32u, per = 32u / gl, ns = rest ? 1u : (unsigned)st.whole;
    const unsigned v = rest ? u - nw : u, t = v / ns, strip = rest ? (unsigned)st.whole : v - t * ns;
    const unsigned third = t / nr, second = t - third * nr, cx = lane & (gl - 1u);
    x = g.S.lo[0] + (int)(strip * (32 - 2 * VAL_HALO) + cx) - VAL_HALO;
    y = g.S.lo[1] + (int)second * run;
    z = g.S.lo[2] + (int)(third * per + lane / gl);
    own = cx >= VAL_HALO && cx < gl - VAL_HALO && z < g.S.lo[2] + g.S.n[2];
  } else {
    const unsigned ns = (unsigned)cdiv(g.S.n[0] * g.S.n[1], 32), third = u / ns;
    const unsigned cell = (u - third * ns) * 32u + lane, cy = cell / (unsigned)g.S.n[0];
    x = g.S.lo[0] + (int)(cell - cy * (unsigned)g.S.n[0]);
    y = g.S.lo[1] + (int)cy;
    z = g.S.lo[2] + (int)third * run;
    own = (int)cy < g.S.n[1];
  }
  const int q0 = X ? y : z;             // the same for all lanes
  const int q1 = min(q0 + run - 1, g.S.lo[DM] + g.S.n[DM] - 1);
  const int dloq = g.dlo[DM], dhiq = g.dhi[DM];
  const Bx& A = g.Ap;
  const bool lane_in = x >= g.dlo[0] && x <= g.dhi[0] && x >= A.lo[0] && x < A.lo[0] + A.n[0] &&
                       (X ? z < g.S.lo[2] + g.S.n[2] : own);
  const bool store = lane_in && own && x < g.S.lo[0] + g.S.n[0] && x >= g.S.lo[0];
  const long long pcs = A.cells(), dq = X ? A.n[0] : (long long)A.n[0] * A.n[1];
  const T* const safe = g.Up;
  // the lane's address in component 0 of the next row to stage
  const T* lsrc = g.Up + A.at(x, y, z);
  const long long side2 = (long long)g.uside * pcs;
  P* const ring = reinterpret_cast<P*>(val_smem) + warp * 4 * RP;
  const unsigned ring32 = (unsigned)__cvta_generic_to_shared(ring) + lane * (unsigned)sizeof(P);
  const int q_last = min(dhiq, q1 + 2);
  auto stage = [&](int q) {
    const bool ok = lane_in && q <= q_last;
    const T* s = ok ? lsrc : safe;
    stage_column<T, DM, 0>(ring32 + (unsigned)(((q - q0) & 3) * RP * (int)sizeof(P)), s, s + side2, (unsigned)pcs,
                           ok ? (unsigned)sizeof(T) : 0u);
    cp_async_commit();
    lsrc += dq;
  };
  auto row = [&](int q) -> const P* { return ring + ((q - q0) & 3) * RP + lane; };
  stage(q0); stage(q0 + 1); stage(q0 + 2);
  constexpr bool kD = kDiffsOnce<T>;
  P n4[NC8], dlo[NC8], nd[NC8];         // nd (FP64): the difference to the next row
  {
    const bool hl = q0 - 1 >= dloq, hll = q0 - 2 >= dloq, hr = q0 + 1 <= dhiq;
    P Wa[NC8], Wb[NC8];
    const T* const b = g.Up + A.at(x, y, z) - dq;
#pragma unroll
    for (int c = 0; c < NC8; ++c) {
      if (!wave_comp<DM>(val_comp<DM>(c))) continue;
      const long long o = val_comp<DM>(c) * pcs;
      Wb[c] = lane_in && hl ? mk2(b[o], b[o + side2]) : mk2(T(0), T(0));
      Wa[c] = lane_in && hll ? mk2(b[o - dq], b[o - dq + side2]) : mk2(T(0), T(0));
    }
    cp_async_wait<1>();
    const P *r0 = row(q0), *r1 = row(q0 + 1);
#pragma unroll
    for (int c = 0; c < NC8; ++c) {
      n4[c] = mk2(T(0), T(0)); dlo[c] = n4[c];
      if (!wave_comp<DM>(val_comp<DM>(c))) continue;
      P nl = psub(Wb[c], r0[c * 32]), nr2 = psub(r0[c * 32], r1[c * 32]);
      if (kD) nd[c] = nr2;
      if (!hl) nl = nr2;
      if (!hr) nr2 = nl;
      if (!hl && !hr) { nl = mk2(T(0), T(0)); nr2 = nl; }
      n4[c] = half_slope(nl, nr2, true);
      if (hl) {
        P na = psub(Wa[c], Wb[c]);
        if (!hll) na = nl;
        dlo[c] = delta_lo<T>(nl, n4[c], half_slope(na, nl, true));
      } else {
        dlo[c] = twice(n4[c]);
      }
    }
  }
  const bool edge_lo = x == g.dlo[0], edge_hi = x == g.dhi[0];
  const bool warp_xedge = X && __any_sync(0xffffffffu, edge_lo || edge_hi);
  P* to = reinterpret_cast<P*>(g.AF) + (store ? g.S.at(x, y, z) : 0);
  const unsigned scs = (unsigned)g.S.cells();
  const long long dso = X ? g.S.n[0] : (long long)g.S.n[0] * g.S.n[1];
  for (int q = q0; q <= q1; ++q, to += dso) {
    stage(q + 3);
    cp_async_wait<1>();                 // rows up to q+2 have landed
    __syncwarp();
    const P *rw = row(q), *r1 = row(q + 1), *r2 = row(q + 2);
    P W[NC8], Wr[NC8], m[NC8], p[NC8], nl[NC8], nr[NC8];
#pragma unroll
    for (int c = 0; c < NC8; ++c) {
      const int gc = val_comp<DM>(c);
      W[c] = rw[c * 32];
      Wr[c] = gc < 3 ? W[c] : padd(W[c], kall(k.nbg[gc]));
      m[c] = mk2(T(0), T(0)); p[c] = m[c];
    }
#pragma unroll
    for (int c = 0; c < NC8; ++c) {
      if (!wave_comp<DM>(val_comp<DM>(c))) continue;
      const P W1 = r1[c * 32];
      nl[c] = kD ? nd[c] : psub(W[c], W1);
      nr[c] = psub(W1, r2[c * 32]);
      if (kD) nd[c] = nr[c];
    }
    if (q + 2 > dhiq) {
#pragma unroll
      for (int c = 0; c < NC8; ++c) nr[c] = nl[c];
    }
#pragma unroll
    for (int c = 0; c < NC8; ++c) {
      if (!wave_comp<DM>(val_comp<DM>(c))) continue;
      const P n1 = half_slope(nl[c], nr[c], true), d1 = delta_lo<T>(nl[c], n1, n4[c]);
      m[c] = dlo[c];
      p[c] = delta_hi<T>(nl[c], d1);
      if (q + 1 > dhiq) p[c] = pneg(twice(n4[c]));
      limit_mono(m[c], p[c], n4[c]);
      n4[c] = n1;
      dlo[c] = d1;
    }
    P An[3], Ap[3];
    trace3<DM, DM, T>(k, Wr, m, p, An, Ap);
    if (store) store_values<DM>(to, scs, An, Ap);
    if constexpr (X) {
      if (g.fault && q == dloq && store) {
        // the velocities of the S pairs of the state entering the fault (the
        // friction solve's first guess): the untraced right-going delta is pm / 2
        const long long fo = g.fplane.at(x, q, z), fcs = g.fplane.cells();
#pragma unroll
        for (int w = 1; w < 3; ++w) {
          const int v = val_index<DM>(wv<DM>(w)), s = val_index<DM>(ws<DM>(w));
          const P Z = mk2(k.Zs, -k.Zs), pm = pfma(pneg(Z), m[v], m[s]);
          const P dn = psub(An[w], pfma(Z, Wr[v], Wr[s]));
          const P vl = pfma(mk2(k.hZs, -k.hZs), pfma(kall(T(-0.5)), pm, dn), Wr[v]);
          g.FV[(w - 1) * fcs + fo] = vl.x;
          g.FV[(2 + w - 1) * fcs + fo] = vl.y;
        }
      }
      // x: neighbours by lane
      P n[NC8], d[NC8];
#pragma unroll
      for (int c = 0; c < NC8; ++c) {
        if (!wave_comp<0>(val_comp<DM>(c))) continue;
        const P wl = shfl_up2(W[c], 1);
        nl[c] = psub(wl, W[c]);
        nr[c] = shfl_dn2(nl[c], 1);       // the next lane's difference to this one
      }
      if (warp_xedge) {
#pragma unroll
        for (int c = 0; c < NC8; ++c) {
          if (!wave_comp<0>(val_comp<DM>(c))) continue;
          const P l = nl[c];
          if (edge_lo) nl[c] = edge_hi ? mk2(T(0), T(0)) : nr[c];
          if (edge_hi) nr[c] = edge_lo ? mk2(T(0), T(0)) : l;
        }
      }
#pragma unroll
      for (int c = 0; c < NC8; ++c) {
        if (!wave_comp<0>(val_comp<DM>(c))) continue;
        n[c] = half_slope(nl[c], nr[c], true);
        d[c] = delta_lo<T>(nl[c], n[c], shfl_up2(n[c], 1));
      }
      if (warp_xedge && edge_lo) {
#pragma unroll
        for (int c = 0; c < NC8; ++c)
          if (wave_comp<0>(val_comp<DM>(c))) d[c] = twice(n[c]);
      }
#pragma unroll
      for (int c = 0; c < NC8; ++c)
        if (wave_comp<0>(val_comp<DM>(c))) p[c] = delta_hi<T>(nr[c], shfl_dn2(d[c], 1));
      if (warp_xedge && edge_hi) {
#pragma unroll
        for (int c = 0; c < NC8; ++c)
          if (wave_comp<0>(val_comp<DM>(c))) p[c] = pneg(twice(n[c]));
      }
#pragma unroll
      for (int c = 0; c < NC8; ++c) {
        if (!wave_comp<0>(val_comp<DM>(c))) continue;
        m[c] = d[c];
        limit_mono(m[c], p[c], n[c]);
      }
      trace3<DM, 0, T>(k, Wr, m, p, An, Ap);
      if (store) store_values<0>(to, scs, An, Ap);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if constexpr (!X) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ------------------------------------------------------------ linear stages
// Transverse term of direction E on the values of direction D; SC 0: scale
// 1/2, 1: scale 1/3; rv: +-1 where the y direction takes part.
template <int E, int D, int SC, typename T>
TMK_D void correct3(const K3<T>& k, T rv, const T* sum, const T* dif, typename PairOf<T>::P* a) {
  constexpr int F = 3 - D - E;
  const T r = (D == 1 || E == 1) ? rv : T(1);
  const T vP = r * k.c_vP[SC], vS = r * k.c_vS[SC];
  constexpr int sE = slot<D>(E), sF = slot<D>(F);
  const T sd = sum[slot<E>(D)];
  a[0].x = fma(vP, sd, fma(k.c_lam[SC], dif[0], a[0].x));
  a[0].y = fma(-vP, sd, fma(k.c_lam[SC], dif[0], a[0].y));
  const T ds = dif[slot<E>(D)];
  a[sE].x = fma(vS, sum[0], fma(k.c_G[SC], ds, a[sE].x));
  a[sE].y = fma(-vS, sum[0], fma(k.c_G[SC], ds, a[sE].y));
  const T sf = sum[slot<E>(F)];
  a[sF].x = fma(vS, sf, a[sF].x);
  a[sF].y = fma(-vS, sf, a[sF].y);
}
// update increments of direction D (x starts them)
template <int D, typename T>
TMK_D void update3(const K3<T>& k, T rv, const T* sum, const T* dif, T* du) {
  const T ev = (D == 1 ? rv : T(1)) * k.e_v;
#pragma unroll
  for (int w = 0; w < 3; ++w) {
    du[wv<D>(w)] = fma(ev, sum[w], du[wv<D>(w)]);
    du[ws<D>(w)] = fma(w == 0 ? k.e_l2g : k.e_G, dif[w], du[ws<D>(w)]);
  }
  du[3 + kTan1<D>] = fma(k.e_lam, dif[0], du[3 + kTan1<D>]);
  du[3 + kTan2<D>] = fma(k.e_lam, dif[0], du[3 + kTan2<D>]);
}
// the value arriving at a domain edge (the background's velocity is zero)
template <typename T> TMK_D T arriving(bool outflow, T leaving, T nbg) { return outflow ? T(0) : fma(T(2), nbg, -leaving); }

// sums and differences of the jumps between a cell's hi face (hn, hp) and lo face (ln, lp)
template <typename T> TMK_D void jump(T hn, T hp, T ln, T lp, T& sum, T& dif) {
  const T jn = hn - ln, jp = hp - lp;
  sum = jn + jp;
  dif = jn - jp;
}

// float -> double of an increment by its bits (a conversion holds the FP64 pipe
// for 64 cycles a warp), not for denormals: a cell that has one among its nine
// increments takes the conversions (192x96x96 690 us a call,
// 686 with them dropped; a test for each increment 695)
TMK_D double widen(float f) {
  const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
  const unsigned e = a >= 0x7f800000u ? 1792u << 20 : 896u << 20;        // infinities and NaN stay what they are
  const unsigned hi = (u & 0x80000000u) | ((a >> 3) + e);
  return a < 0x00800000u ? 0.0 : __hiloint2double((int)hi, (int)(u << 29));
}
TMK_D double widen(double f) { return f; }
TMK_D bool has_denormal(const float* f) {
  unsigned least = ~0u;
#pragma unroll
  for (int c = 0; c < 9; ++c) least = min(least, (__float_as_uint(f[c]) << 1) - 1u);      // zeros wrap around
  return least < 0x00ffffffu;
}
TMK_D bool has_denormal(const double*) { return false; }

// fluxes of the D face with values (n, p) of one side into the 22-component
// flux array (GETFLUXF; lambda, gamma and the antiplane stress carry none)
template <int D, typename T>
TMK_D void store_flux(const Step3<T>& g, const K3<T>& k, T rvs, int s, int i, int j, int kk, const T* n, const T* p) {
  const Bx& fb = g.flF[D];
  const long long cs = fb.cells();
  double* out = g.F[D] + (long long)(11 * s) * cs + fb.at(i, j, kk);
  const T rv = D == 1 ? rvs : T(1);
  T f[9];
#pragma unroll
  for (int w = 0; w < 3; ++w) {
    const T fs = fma(T(0.5), n[w] + p[w], -k.nbg[ws<D>(w)]);
    const T fv = rv * (w == 0 ? k.hZp : k.hZs) * (n[w] - p[w]);
    f[wv<D>(w)] = -rv * k.irho * fs;
    f[ws<D>(w)] = -rv * (w == 0 ? k.l2g : k.G) * fv;
    if (w == 0) { f[3 + kTan1<D>] = -rv * k.lam * fv; f[3 + kTan2<D>] = f[3 + kTan1<D>]; }
  }
  f[shear(kTan1<D>, kTan2<D>)] = T(0);
#pragma unroll
  for (int c = 0; c < 9; ++c) out[c * cs] = (double)f[c];
  out[9 * cs] = 0.0;
  out[10 * cs] = 0.0;
}

// asynchronous copies of one thread's element of nine planes to shared entries NT apart
template <typename E, int NT, int C>
TMK_D void stage_plane(unsigned dst, const E* src, unsigned plane, unsigned nbytes) {
  if constexpr (C < 9) {
    asm volatile("cp.async.ca.shared.global [%0 + %4], [%1], %2, %3;" ::"r"(dst), "l"(plane_ptr(src, plane, C)),
                 "n"(sizeof(E)), "r"(nbytes), "n"(C * NT * (int)sizeof(E))
                 : "memory");
    stage_plane<E, NT, C + 1>(dst, src, plane, nbytes);
  }
}

// ------------------------------------------------------------ the step
// One CTA per tile of 30 x (NR - 2) cells, run of planes and side; a warp per
// row of y, x in the lanes, marching in z.  (The columns left over by whole
// tiles: 14 x (2 NR - 2), 6 x (4 NR - 2) or 2 x (8 NR - 2) cells, two to eight
// rows to a warp.)  Neighbours: x by lane, y through
// shared memory (two exchanges a plane), z carried from plane to plane.  When
// plane m arrives, the stages that need nothing above it are done for m, then
// plane m - 1 is finished.  8 rows, FP32 at two CTAs per SM (128 registers), FP64
// at one.  What a thread carries of the first values and the z jumps stays in its
// own shared memory slots, where cp.async puts the next plane's values: kept in
// registers they spilled, and the loads of the spills, not those of the values,
// were what warps waited for (192x96x96 mixed 394 us, 294 now).  A call there took
// 738 us with 16 rows, 708 with 14 and 906 with 12 (at one CTA), 694 with 8; a
// 64x48x48 FP64 patch 602 with 10 rows and 582 with 8.
// GL: lanes of a row, 32 or (0) fewer, from the strips; FLUX: a patch has flux
// arrays.  Both fixed at compile time: the common form spills least.
template <typename T, int GL, bool FLUX>
TMK_D void step_tile(const Step3<T>& g, const K3<T>& k, unsigned u) {
  using V = typename PairOf<T>::P;
  constexpr int NR = step_rows<T>;
  // [9] A_y, WHalf2[1][0] of plane m, WHalf2[1][2] of plane m - 1; [3] the final y values of plane m - 1
  extern __shared__ __align__(16) unsigned char step_smem[];
  constexpr int PL = (NR + 2) * 32;       // entries of one value; rows of a lane group each
  constexpr int NT = 32 * NR;
  V* const s1 = reinterpret_cast<V*>(step_smem);
  V* const s2 = s1 + 9 * PL;
  // the thread's values of two planes and the state it updates, copied in by
  // cp.async: the values of plane m + 1 land where those of m - 1 were
  V* const vals = s2 + 3 * PL + threadIdx.x;                                // [2][9][NT]
  double* const unext = reinterpret_cast<double*>(s2 + 3 * PL + 18 * NT) + threadIdx.x;
  // and its p jumps of the z values, kept from plane to plane ([4][3][NT]: of A_z,
  // WHalf2[2][0], WHalf2[2][1], the final values): registers here would spill
  T* const js = reinterpret_cast<T*>(reinterpret_cast<double*>(s2 + 3 * PL + 18 * NT) + 9 * NT) + threadIdx.x;
  const unsigned v32 = (unsigned)__cvta_generic_to_shared(vals), u32 = (unsigned)__cvta_generic_to_shared(unext);
  const unsigned side = u & 1u;
  const Strips st = strips(g.cur.n[0], 1);
  const unsigned nw = (unsigned)st.whole * (unsigned)cdiv(g.cur.n[1], NR - 2);
  const unsigned nt = (unsigned)step_tiles<T>(g.cur.n[0], g.cur.n[1]), tz = (u >> 1) / nt, t1 = (u >> 1) - tz * nt;
  const unsigned gl = GL ? GL : (unsigned)st.group;            // lanes of a group, that is of a row
  const unsigned ty = GL && st.whole ? t1 / (unsigned)st.whole : t1 - nw;
  const unsigned tx = GL && st.whole ? t1 - ty * (unsigned)st.whole : (unsigned)st.whole;
  const int cx = (int)(threadIdx.x & (gl - 1u)), row = (int)(threadIdx.x / gl), rows = (int)(32u * NR / gl);
  const int at = (int)gl + (int)threadIdx.x;                   // the thread's entry: row + 1, column cx
  const int s = (int)side;
  const T rv = s ? T(-1) : T(1);
  const int x = g.cur.lo[0] + (int)tx * 30 - 1 + cx, y = g.cur.lo[1] + (int)ty * (rows - 2) - 1 + row;
  const int z0 = g.cur.lo[2] + (int)tz * g.zrun, z1 = min(z0 + g.zrun, g.cur.lo[2] + g.cur.n[2]) - 1;
  const bool in = x >= g.S.lo[0] && x < g.S.lo[0] + g.S.n[0] && y >= g.S.lo[1] && y < g.S.lo[1] + g.S.n[1];
  const bool upd = cx >= 1 && cx <= (int)gl - 2 && row >= 1 && row <= rows - 2 && x < g.cur.lo[0] + g.cur.n[0] &&
                   y < g.cur.lo[1] + g.cur.n[1];
  const bool xlo = x == g.dlo[0], xhi = x == g.dhi[0];
  const bool warp_x = __any_sync(0xffffffffu, xlo || xhi);
  const bool ylo = y == g.dlo[1], yhi = y == g.dhi[1], yfault = ylo && g.fault != 0;
  // the fault plane's states: the kernel before this one in the stream
  if (__any_sync(0xffffffffu, yfault)) asm volatile("griddepcontrol.wait;" ::: "memory");
  const int zlo = g.dlo[2], zhi = g.dhi[2];
  const unsigned scs = (unsigned)g.S.cells();
  const unsigned dz = (unsigned)g.S.n[0] * (unsigned)g.S.n[1];
  const int ms = max(z0 - 1, zlo);
  const V* vp = reinterpret_cast<const V*>(g.AF) + (unsigned long long)scs * (unsigned)(s * 9) + (in ? g.S.at(x, y, ms) : 0);
  const V zero = mk2(T(0), T(0));
  const unsigned acs = (unsigned)g.A.cells();
  const long long adz = (long long)g.A.n[0] * g.A.n[1];
  double* up = g.U + (unsigned long long)acs * (unsigned)(11 * s) + (upd ? g.A.at(x, y, z0) : 0);

  auto xjump = [&](const V* a, T* sum, T* dif) {
    T hn[3], lp[3];
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      hn[w] = __shfl_down_sync(0xffffffffu, a[w].x, 1);
      lp[w] = __shfl_up_sync(0xffffffffu, a[w].y, 1);
    }
    if (warp_x) {
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        if (xhi) hn[w] = arriving(k.out[1] != 0, a[w].y, k.nbg[ws<0>(w)]);
        if (xlo) lp[w] = arriving(k.out[0] != 0, a[w].x, k.nbg[ws<0>(w)]);
      }
    }
#pragma unroll
    for (int w = 0; w < 3; ++w) jump(hn[w], a[w].y, a[w].x, lp[w], sum[w], dif[w]);
  };
  // the lo face values of a cell in y: the row below, the edge, or the fault's
  // state of level l in plane kz
  const bool on_plane = yfault && in && x >= g.fplane.lo[0] && x < g.fplane.lo[0] + g.fplane.n[0];
  auto ylo_face = [&](const V* sm, const V* a, int l, int kz, T* ln, T* lp) {
#pragma unroll
    for (int w = 0; w < 3; ++w) { ln[w] = a[w].x; lp[w] = sm[w * PL + at - (int)gl].y; }
    if (ylo) {
      if (yfault) {
        const bool have = on_plane && kz >= g.fplane.lo[2] && kz < g.fplane.lo[2] + g.fplane.n[2];
        const long long o = have ? g.fplane.at(x, y, kz) : 0;
#pragma unroll
        for (int w = 0; w < 3; ++w) {
          const V f = have ? plane_face(g, l, s, w)[o] : zero;
          const T Z = rv * (w == 0 ? k.Zp : k.Zs);
          ln[w] = fma(Z, f.y, f.x);
          lp[w] = fma(-Z, f.y, f.x);
        }
      } else {
#pragma unroll
        for (int w = 0; w < 3; ++w) lp[w] = arriving(k.out[2] != 0, a[w].x, k.nbg[ws<1>(w)]);
      }
    }
  };
  auto yjump = [&](const V* sm, const V* a, int l, int kz, T* sum, T* dif) {
    T ln[3], lp[3], hn[3];
    ylo_face(sm, a, l, kz, ln, lp);
#pragma unroll
    for (int w = 0; w < 3; ++w) hn[w] = sm[w * PL + at + (int)gl].x;
    if (yhi) {
#pragma unroll
      for (int w = 0; w < 3; ++w) hn[w] = arriving(k.out[3] != 0, a[w].y, k.nbg[ws<1>(w)]);
    }
#pragma unroll
    for (int w = 0; w < 3; ++w) jump(hn[w], a[w].y, ln[w], lp[w], sum[w], dif[w]);
  };

  // carried from plane to plane (plane k = m - 1): WHalf2[2][0], WHalf2[2][1] and
  // the final z values (their p jumps and the first values are in shared memory)
  V zx[3], zy[3], fz[3];
#pragma unroll
  for (int w = 0; w < 3; ++w) { zx[w] = zero; zy[w] = zero; fz[w] = zero; }
  constexpr unsigned VSLOT = 9 * NT;
  stage_plane<V, NT, 0>(v32 + (ms & 1) * VSLOT * (unsigned)sizeof(V), vp, scs, in ? (unsigned)sizeof(V) : 0u);
  cp_async_commit();
  for (int m = ms; m <= z1 + 1; ++m) {
    const bool have = m <= zhi, fin = m > ms && m - 1 >= z0;      // uniform over the CTA
    V bx[3], by[3], bz[3], nzx[3], nzy[3], nfz[3];
    const V *const vm = vals + (m & 1) * VSLOT, *const vb = vals + ((m + 1) & 1) * VSLOT;      // planes m and m - 1
    cp_async_wait<0>();                   // the thread's values of plane m
    if (have) {
#pragma unroll
      for (int w = 0; w < 3; ++w) { bx[w] = vm[w * NT]; by[w] = vm[(3 + w) * NT]; bz[w] = vm[(6 + w) * NT]; }
    } else {
      // past the domain's z-hi edge: only the values arriving through it
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const bool o = k.out[5] != 0;
        const T b = k.nbg[ws<2>(w)];
        bx[w] = zero; by[w] = zero;
        bz[w] = mk2(arriving(o, vb[(6 + w) * NT].y, b), T(0));
        nzx[w] = mk2(arriving(o, zx[w].y, b), T(0));
        nzy[w] = mk2(arriving(o, zy[w].y, b), T(0));
        nfz[w] = mk2(arriving(o, fz[w].y, b), T(0));
      }
    }
    if (fin && upd) stage_plane<double, NT, 0>(u32, up, acs, 8u);
    cp_async_commit();
    // ---- first exchange: A_y and WHalf2[1][0] of plane m, WHalf2[1][2] of plane m - 1
    V yx[3], yz[3], xz[3];
    T sum[3], dif[3];
    if (have) {
#pragma unroll
      for (int w = 0; w < 3; ++w) { yx[w] = by[w]; nzx[w] = bz[w]; }
      xjump(bx, sum, dif);
      correct3<0, 1, 1, T>(k, rv, sum, dif, yx);
      correct3<0, 2, 1, T>(k, rv, sum, dif, nzx);
#pragma unroll
      for (int w = 0; w < 3; ++w) { s1[w * PL + at] = by[w]; s1[(3 + w) * PL + at] = yx[w]; }
    }
    if (fin) {
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        xz[w] = vb[w * NT]; yz[w] = vb[(3 + w) * NT];
        const T jn = bz[w].x - vb[(6 + w) * NT].x;
        sum[w] = jn + js[w * NT];
        dif[w] = jn - js[w * NT];
      }
      correct3<2, 0, 1, T>(k, rv, sum, dif, xz);
      correct3<2, 1, 1, T>(k, rv, sum, dif, yz);
#pragma unroll
      for (int w = 0; w < 3; ++w) s1[(6 + w) * PL + at] = yz[w];
    }
    // the p jump of A_z over plane m; at the domain's z-lo edge the value from below arrives through it
#pragma unroll
    for (int w = 0; w < 3; ++w)
      js[w * NT] = bz[w].y - (m == zlo ? arriving(k.out[4] != 0, bz[w].x, k.nbg[ws<2>(w)]) : vb[(6 + w) * NT].y);
    __syncthreads();
    V xy[3], fx[3], fy[3];
    if (have) {
#pragma unroll
      for (int w = 0; w < 3; ++w) { xy[w] = bx[w]; nzy[w] = bz[w]; nfz[w] = bz[w]; }
      yjump(s1, by, 0, m, sum, dif);
      correct3<1, 0, 1, T>(k, rv, sum, dif, xy);
      correct3<1, 2, 1, T>(k, rv, sum, dif, nzy);
      // the final z values of plane m: jumps of WHalf2[0][1] in x and WHalf2[1][0] in y
      xjump(xy, sum, dif);
      correct3<0, 2, 0, T>(k, rv, sum, dif, nfz);
      yjump(s1 + 3 * PL, yx, 1, m, sum, dif);
      correct3<1, 2, 0, T>(k, rv, sum, dif, nfz);
    }
    if (fin) {
      // the final x and y values of plane m - 1
#pragma unroll
      for (int w = 0; w < 3; ++w) { fx[w] = vb[w * NT]; fy[w] = vb[(3 + w) * NT]; }
      yjump(s1 + 6 * PL, yz, 2, m - 1, sum, dif);
      correct3<1, 0, 0, T>(k, rv, sum, dif, fx);
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const T jn = nzy[w].x - zy[w].x;
        sum[w] = jn + js[(6 + w) * NT];
        dif[w] = jn - js[(6 + w) * NT];
      }
      correct3<2, 0, 0, T>(k, rv, sum, dif, fx);
      xjump(xz, sum, dif);
      correct3<0, 1, 0, T>(k, rv, sum, dif, fy);
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const T jn = nzx[w].x - zx[w].x;
        sum[w] = jn + js[(3 + w) * NT];
        dif[w] = jn - js[(3 + w) * NT];
      }
      correct3<2, 1, 0, T>(k, rv, sum, dif, fy);
#pragma unroll
      for (int w = 0; w < 3; ++w) s2[w * PL + at] = fy[w];
    }
    __syncthreads();
    // plane m - 1's values have been used: those of plane m + 1 may land
    if (m < zhi && m <= z1) {
      vp += dz;
      stage_plane<V, NT, 0>(v32 + ((m + 1) & 1) * VSLOT * (unsigned)sizeof(V), vp, scs, in ? (unsigned)sizeof(V) : 0u);
    }
    cp_async_commit();
    if (fin) {
      const int kz = m - 1;
      T du[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) du[c] = T(0);
      xjump(fx, sum, dif);
      update3<0, T>(k, rv, sum, dif, du);
      yjump(s2, fy, 3, kz, sum, dif);
      update3<1, T>(k, rv, sum, dif, du);
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const T jn = nfz[w].x - fz[w].x;
        sum[w] = jn + js[(9 + w) * NT];
        dif[w] = jn - js[(9 + w) * NT];
      }
      update3<2, T>(k, rv, sum, dif, du);
      if (FLUX && (g.F[0] || g.F[1] || g.F[2])) {
        // the lo faces of this cell, and the hi face of the last one
        T n[3], p[3], hn[3];
#pragma unroll
        for (int w = 0; w < 3; ++w) {
          hn[w] = __shfl_down_sync(0xffffffffu, fx[w].x, 1);
          p[w] = __shfl_up_sync(0xffffffffu, fx[w].y, 1);
          if (xhi) hn[w] = arriving(k.out[1] != 0, fx[w].y, k.nbg[ws<0>(w)]);
          if (xlo) p[w] = arriving(k.out[0] != 0, fx[w].x, k.nbg[ws<0>(w)]);
          n[w] = fx[w].x;
        }
        if (upd && g.F[0]) {
          store_flux<0, T>(g, k, rv, s, x, y, kz, n, p);
          if (x == g.cur.lo[0] + g.cur.n[0] - 1) {
#pragma unroll
            for (int w = 0; w < 3; ++w) p[w] = fx[w].y;
            store_flux<0, T>(g, k, rv, s, x + 1, y, kz, hn, p);
          }
        }
        if (upd && g.F[1]) {
          ylo_face(s2, fy, 3, kz, n, p);
          store_flux<1, T>(g, k, rv, s, x, y, kz, n, p);
          if (y == g.cur.lo[1] + g.cur.n[1] - 1) {
#pragma unroll
            for (int w = 0; w < 3; ++w) {
              hn[w] = yhi ? arriving(k.out[3] != 0, fy[w].y, k.nbg[ws<1>(w)]) : s2[w * PL + at + (int)gl].x;
              p[w] = fy[w].y;
            }
            store_flux<1, T>(g, k, rv, s, x, y + 1, kz, hn, p);
          }
        }
        if (upd && g.F[2]) {
#pragma unroll
          for (int w = 0; w < 3; ++w) { n[w] = fz[w].x; p[w] = fz[w].y - js[(9 + w) * NT]; }
          store_flux<2, T>(g, k, rv, s, x, y, kz, n, p);
          if (kz == g.cur.lo[2] + g.cur.n[2] - 1) {
#pragma unroll
            for (int w = 0; w < 3; ++w) { hn[w] = nfz[w].x; p[w] = fz[w].y; }
            store_flux<2, T>(g, k, rv, s, x, y, kz + 1, hn, p);
          }
        }
      }
      cp_async_wait<1>();                 // the state; the next plane's values may still be on their way
      if (upd) {
        if (has_denormal(du)) {
#pragma unroll
          for (int c = 0; c < 9; ++c) *plane_ptr(up, acs, c) = unext[c * NT] + (double)du[c];
        } else {
#pragma unroll
          for (int c = 0; c < 9; ++c) *plane_ptr(up, acs, c) = unext[c * NT] + widen(du[c]);
        }
      }
      up += adz;
    }
    // hand plane m on; at the domain's z-lo edge the values from below arrive through it
    if (m == zlo) {
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const bool o = k.out[4] != 0;
        const T b = k.nbg[ws<2>(w)];
        zx[w].y = arriving(o, nzx[w].x, b);
        zy[w].y = arriving(o, nzy[w].x, b);
        fz[w].y = arriving(o, nfz[w].x, b);
      }
    }
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      js[(3 + w) * NT] = nzx[w].y - zx[w].y;
      js[(6 + w) * NT] = nzy[w].y - zy[w].y;
      js[(9 + w) * NT] = nfz[w].y - fz[w].y;
      zx[w] = nzx[w]; zy[w] = nzy[w]; fz[w] = nfz[w];
    }
  }
}

template <typename T, bool FLUX, typename Src>
__global__ void __launch_bounds__(32 * step_rows<T>, step_ctas<T>)
step_kernel(const __grid_constant__ Src src, const __grid_constant__ K3<T> k) {
  long long lt;
  const Step3<T>* gp = find_item<T>(src, blockIdx.x, lt);
  if (!gp) return;
  const Step3<T>& g = *gp;
  // a tile of whole strips or of the columns left over
  const Strips st = strips(g.cur.n[0], 1);
  const unsigned nt = (unsigned)step_tiles<T>(g.cur.n[0], g.cur.n[1]), u = (unsigned)lt;
  const bool whole = (u >> 1) % nt < (unsigned)st.whole * (unsigned)cdiv(g.cur.n[1], step_rows<T> - 2);
  if (whole) step_tile<T, 32, FLUX>(g, k, u);
  else step_tile<T, 0, FLUX>(g, k, u);
}

// ------------------------------------------------------------ the fault plane
// One thread per fault face (x, z) of the first pass: the four friction solves
// of the face from the predictors' values around it, and on valid faces the
// boundary data.  Faces of the grown plane whose transverse term leaves the
// slope box keep the uncorrected values there (no output reads them).
template <typename T, typename Src>
__global__ void __launch_bounds__(64) plane_kernel(const __grid_constant__ Src src, const __grid_constant__ K3<T> k,
                                                   const DevParams* Pp, DevStatus* st) {
  using V = typename PairOf<T>::P;
  // the step's tiles away from the fault may start (the values they read were
  // complete before this kernel started)
  asm volatile("griddepcontrol.launch_dependents;");
  TMK3_FIND(T)
  const Step3<T>& g = *gp;
  const DevParams& P = *Pp;
  if (!g.fault || lt >= g.fplane.cells()) return;
  int i, j, kz;
  g.fplane.cell(lt, i, j, kz);
  const long long fo = lt, fcs = g.fplane.cells();
  const bool rs = P.fault_law == 1;
  double* const Bi = g.B + g.bb.at(i, j, kz);
  const long long bs = g.bb.cells();
  const double b0 = Bi[(rs ? 10 : 7) * bs];
  constexpr bool kFused = !kExact<T> && std::is_same<Src, One<T>>::value;       // cell_from
  RSFaceK fk;
  SWFaceK wk;
  if (rs) fk = rs_face_k(P, rs_face(P, nullptr, 0, 0), false, (i + 0.5) * g.dx - P.rs_x0, b0);
  else wk = sw_face_k<true>(P, cell_from<kFused>(i, g.dx, P.sw_fbc0), cell_from<kFused>(kz, g.dx, P.sw_fbc1));
  auto inS = [&](int a, int c) { return g.S.has(a, j, c); };
  auto val = [&](int s, int D, int w, int a, int c) { return val_plane(g, s, D, w)[g.S.at(a, j, c)]; };
  // jumps of the first-pass values of x (or z) over cell (a, c); false outside ccBox
  auto jump1 = [&](auto dir, int s, int a, int c, T* sum, T* dif) {
    constexpr int D = decltype(dir)::value;
    const int q = D == 0 ? a : c;
    const bool lo = q == g.dlo[D], hi = q == g.dhi[D];
    if (!inS(a, c) || (!lo && !inS(D == 0 ? a - 1 : a, D == 0 ? c : c - 1)) ||
        (!hi && !inS(D == 0 ? a + 1 : a, D == 0 ? c : c + 1)))
      return false;
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      const V v = val(s, D, w, a, c);
      const T hn = hi ? arriving(k.out[2 * D + 1] != 0, v.y, k.nbg[ws<D>(w)])
                      : val(s, D, w, D == 0 ? a + 1 : a, D == 0 ? c : c + 1).x;
      const T lp = lo ? arriving(k.out[2 * D] != 0, v.x, k.nbg[ws<D>(w)])
                      : val(s, D, w, D == 0 ? a - 1 : a, D == 0 ? c : c - 1).y;
      jump(hn, v.y, v.x, lp, sum[w], dif[w]);
    }
    return true;
  };
  // WHalf2[D][E] values of cell (a, c), (D, E) = (0, 2) or (2, 0)
  auto second = [&](auto dir, int s, int a, int c, V* v) {
    constexpr int D = decltype(dir)::value, E = 2 - D;
    T sum[3], dif[3];
#pragma unroll
    for (int w = 0; w < 3; ++w) v[w] = val(s, D, w, a, c);
    const T rv = s ? T(-1) : T(1);
    if (jump1(std::integral_constant<int, E>{}, s, a, c, sum, dif)) correct3<E, D, 1, T>(k, rv, sum, dif, v);
  };
  // jumps of WHalf2[D][E] in D over this face's cell
  auto jump2 = [&](auto dir, int s, T* sum, T* dif) {
    constexpr int D = decltype(dir)::value;
    const int q = D == 0 ? i : kz;
    const bool lo = q == g.dlo[D], hi = q == g.dhi[D];
    V v[3], h[3], l[3];
    second(dir, s, i, kz, v);
    if (!hi) second(dir, s, D == 0 ? i + 1 : i, D == 0 ? kz : kz + 1, h);
    if (!lo) second(dir, s, D == 0 ? i - 1 : i, D == 0 ? kz : kz - 1, l);
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      const T hn = hi ? arriving(k.out[2 * D + 1] != 0, v[w].y, k.nbg[ws<D>(w)]) : h[w].x;
      const T lp = lo ? arriving(k.out[2 * D] != 0, v[w].x, k.nbg[ws<D>(w)]) : l[w].y;
      jump(hn, v[w].y, v[w].x, lp, sum[w], dif[w]);
    }
  };
  using DX = std::integral_constant<int, 0>;
  using DZ = std::integral_constant<int, 2>;
  V ay[2][3];
  T vv[2][2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
#pragma unroll
    for (int w = 0; w < 3; ++w) ay[s][w] = val(s, 1, w, i, kz);
    vv[s][0] = g.FV[(2 * s) * fcs + fo];
    vv[s][1] = g.FV[(2 * s + 1) * fcs + fo];
  }
  FaultFace f;
  auto predicted = [&](double dt) { return rs ? rs_state_next(P, fk, b0, f.V, dt) : b0 + dt * f.V; };
  // the velocities move with the velocity part of the terms: 2 hZs times it
  auto move = [&](auto dir, auto sc, const T* sum, const T* dif, int s, V* a, T* v) {
    constexpr int E = decltype(dir)::value, SC = decltype(sc)::value;
    const T rv = s ? T(-1) : T(1);
    correct3<E, 1, SC, T>(k, rv, sum, dif, a);
    const T c = T(2) * k.hZs * k.c_vS[SC];
    v[0] = fma(c, E == 0 ? sum[0] : sum[slot<2>(0)], v[0]);
    v[1] = fma(c, E == 2 ? sum[0] : sum[slot<0>(2)], v[1]);
  };
  using Half = std::integral_constant<int, 0>;
  using Third = std::integral_constant<int, 1>;
  // the four solves in turn -- WHalf1[1], WHalf2[1][0], WHalf2[1][2] and, on
  // valid faces, WHalf[1] -- through one copy of the solve's code (its size
  // showed as instruction fetch stalls)
  const bool valid = g.cur.has(i, j, kz);
  double bval = b0;
#pragma unroll 1
  for (int l = 0; l < 4; ++l) {
    if (l == 3 && !valid) return;
    V a[2][3];
    T v[2][2], sum[3], dif[3];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
#pragma unroll
      for (int w = 0; w < 3; ++w) a[s][w] = ay[s][w];
      v[s][0] = vv[s][0]; v[s][1] = vv[s][1];
      if (l == 1) {
        if (jump1(DX{}, s, i, kz, sum, dif)) move(DX{}, Third{}, sum, dif, s, a[s], v[s]);
      } else if (l == 2) {
        if (jump1(DZ{}, s, i, kz, sum, dif)) move(DZ{}, Third{}, sum, dif, s, a[s], v[s]);
      } else if (l == 3) {
        jump2(DX{}, s, sum, dif);
        move(DX{}, Half{}, sum, dif, s, a[s], v[s]);
        jump2(DZ{}, s, sum, dif);
        move(DZ{}, Half{}, sum, dif, s, a[s], v[s]);
      }
    }
    int it = 0;
    const double aP1 = (double)a[0][0].x + k.s0[0], aP2 = (double)a[1][0].x + k.s0[0];
    // the laws take the unrounded Zs: the rest of its product with the velocities
    auto whole = [&](int s, int w) {
      const double d = (double)a[s][w].x + k.s0[w];
      if constexpr (kExact<T>) return d;
      else return d + widen((s ? -k.lZs : k.lZs) * v[s][w - 1]);
    };
    const double aS1 = whole(0, 1), aS2 = whole(1, 1);
    if (rs) it = rs_face_solve<kExact<T>>(P, fk, aP1, aP2, aS1, aS2, bval, v[0][0] - v[1][0], v[0][1] - v[1][1], f);
    else sw_face_solve(P, wk, aP1, aP2, aS1, aS2, whole(0, 2), whole(1, 2), bval, f);
    if (it > RS_IMAX) atomicAdd(&st->newton_maxed, 1ull);
    const T sP = (T)(f.syy - k.s0[0]), sS = (T)(f.sxy - k.s0[1]), sz = (T)(f.syz - k.s0[2]), vy = (T)f.vy;
    plane_face(g, l, 0, 0)[fo] = mk2(sP, vy);
    plane_face(g, l, 0, 1)[fo] = mk2(sS, (T)f.vx1);
    plane_face(g, l, 0, 2)[fo] = mk2(sz, (T)f.vz1);
    plane_face(g, l, 1, 0)[fo] = mk2(sP, vy);
    plane_face(g, l, 1, 1)[fo] = mk2(sS, (T)f.vx2);
    plane_face(g, l, 1, 2)[fo] = mk2(sz, (T)f.vz2);
    // the next solve's boundary value: predicted over dt/3 from the first
    // state, over dt/2 from WHalf2[1][2]
    if (l != 1 && l != 3) bval = predicted(l == 0 ? (1.0 / 3.0) * g.dt : 0.5 * g.dt);
  }
  const double next = predicted(g.dt), t1 = g.time + g.dt;
  Bi[0] = f.Vx;
  Bi[bs] = f.Vz;
  if (rs) {
    Bi[2 * bs] = f.V;
    Bi[3 * bs] = f.sxy + fk.tau0;
    Bi[4 * bs] = f.syz;
    Bi[5 * bs] = f.syy;
    Bi[6 * bs] += g.dt * f.Vx;
    Bi[7 * bs] += g.dt * f.Vz;
    Bi[8 * bs] += g.dt * f.V;
    if (Bi[9 * bs] > t1) Bi[9 * bs] = f.V > P.rs_thr ? t1 : 1e10;
    Bi[10 * bs] = next;
    if (isnan(next)) report(st, ST_NAN, g.bb.at(i, j, kz));
  } else {
    Bi[2 * bs] = f.sxy;
    Bi[3 * bs] = f.syz;
    Bi[4 * bs] = f.V;
    Bi[5 * bs] += g.dt * f.Vx;
    Bi[6 * bs] += g.dt * f.Vz;
    Bi[7 * bs] = next;
    if (Bi[8 * bs] > t1 && f.V > P.sw_thr) Bi[8 * bs] = t1;
  }
}

template <typename T, int DM> constexpr size_t val_smem_bytes() {
  return (size_t)VAL_WARPS * 4 * kValComps<DM> * 32 * 2 * sizeof(T);
}
template <typename T> constexpr size_t step_smem_bytes() {
  return (size_t)12 * (step_rows<T> + 2) * 32 * 2 * sizeof(T) + (size_t)step_rows<T> * 32 * (9 * (4 * sizeof(T) + 8) + 12 * sizeof(T));
}

// The whole step on stream s (One: one patch, Many: a batch); hp: the context's
// parameters on the host.
template <typename T, typename Plan>
cudaError_t launch_march3(const Plan& pl, const DevParams& hp, const DevParams* P, DevStatus* st, double dt, double dx,
                          cudaStream_t s) {
  K3<T> k;
  k.load(hp, dt, dx);
  using Src = typename Plan::Src;
  static DeviceOnce once;
  cudaError_t e = once_per_device(once, [] {
    cudaError_t r = allow_smem(values_kernel<T, 1, Src>, val_smem_bytes<T, 1>());
    if (r == cudaSuccess) r = allow_smem(values_kernel<T, 2, Src>, val_smem_bytes<T, 2>());
    if (r == cudaSuccess) r = allow_smem(step_kernel<T, false, Src>, step_smem_bytes<T>());
    if (r == cudaSuccess) r = allow_smem(step_kernel<T, true, Src>, step_smem_bytes<T>());
    return r;
  });
  if (e != cudaSuccess) return e;
  if (pl.copy() && pl.n(K_AP)) to_pred_kernel<T, Src><<<blocks(pl.n(K_AP)), 128, 0, s>>>(pl.src(K_AP));
  // The z predictor does not wait for the x and y one, nor the step's tiles away
  // from the fault for the plane kernel (launch attribute; the kernels still
  // complete in order, since every z warp and the tiles on the fault wait).
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  auto config = [&](long long ctas, int threads, size_t smem, bool beside) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = beside ? attr : nullptr;
    cfg.numAttrs = beside ? 1 : 0;
    return cfg;
  };
  const long long nxy = pl.n(K_VXY), nz = pl.n(K_VZ);
  cudaLaunchConfig_t cfg = config((nxy + VAL_WARPS - 1) / VAL_WARPS, 32 * VAL_WARPS, val_smem_bytes<T, 1>(), false);
  if ((e = cudaLaunchKernelEx(&cfg, values_kernel<T, 1, Src>, pl.src(K_VXY), k, nxy)) != cudaSuccess) return e;
  cfg = config((nz + VAL_WARPS - 1) / VAL_WARPS, 32 * VAL_WARPS, val_smem_bytes<T, 2>(), true);
  if ((e = cudaLaunchKernelEx(&cfg, values_kernel<T, 2, Src>, pl.src(K_VZ), k, nz)) != cudaSuccess) return e;
  if (pl.fault())
    plane_kernel<T, Src><<<(unsigned)((pl.n(K_PL) + 63) / 64), 64, 0, s>>>(pl.src(K_PL), k, P, st);
  cfg = config(pl.n(K_STEP), 32 * step_rows<T>, step_smem_bytes<T>(), pl.fault());
  const bool flux = pl.flux(0) || pl.flux(1) || pl.flux(2);
  e = flux ? cudaLaunchKernelEx(&cfg, step_kernel<T, true, Src>, pl.src(K_STEP), k)
           : cudaLaunchKernelEx(&cfg, step_kernel<T, false, Src>, pl.src(K_STEP), k);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace d3
}  // namespace tmk
