"""Timing cases of the Godunov step through the public entry points.

A case is a dict of plain values; `prepare` builds what a program holds before
the call (contexts, levels, recorded graphs, device arrays), `run` makes one
pass through the public calls and returns the updated state, `work` counts what
a pass cannot do without, and `exact` gives the same pass in plain FP64 torch.

Kinds of case:
  level     a device-resident 2-D level: `steps` steps (one call each, or one
            replay of a recorded graph), then the state read back on the device
  patch     one 2-D patch step on the caller's FP64 arrays, as a Chombo patch
            loop calls it (a patch on the fault, inside a larger domain)
  patch3    one 3-D patch step on the caller's FP64 arrays
  level3    a device-resident 3-D level of several patches, one step
  amr       a subcycled 3-level hierarchy (ratio 2, plasticity), two coarse steps
  ensemble  independent rate-and-state scenarios stepped as one level
The mixed form carries its volume state to FP32 accuracy, so its results are
taken as FP32 arrays; the FP64 form's as FP64.
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from tetemoko_gb300 import _capi as A, scenarios as S
from tetemoko_gb300.amr import AMRHierarchy, refine_domain
from tetemoko_gb300.level import (Context, LinElastEnsemble, LinElastLevelGodunov, LinElastLevelGodunov3D,
                                  LinElastPatchGodunov, LinElastPatchGodunov3D)

G = A.TMK_NGHOST
DX = 0.1


def listed():
    return [
        # the benchmark workload: a long rate-and-state run, steps replayed from a graph, state read every 20 steps
        dict(name="rs_mixed_2048x1024", kind="level", law="rs", mixed=True, plastic=False, nx=2048, ny=1024, box=0,
             steps=20, graph=True),
        # the slip-weakening workload of a single study, small enough that launches and the fault solve show
        dict(name="sw_mixed_512x256", kind="level", law="sw", mixed=True, plastic=False, nx=512, ny=256, box=0,
             steps=20, graph=True),
        # the same workload in the plain FP64 form, called step by step
        dict(name="sw_fp64_512x256", kind="level", law="sw", mixed=False, plastic=False, nx=512, ny=256, box=0,
             steps=4, graph=False),
        # the benchmark workload in the plain FP64 form
        dict(name="rs_fp64_2048x1024", kind="level", law="rs", mixed=False, plastic=False, nx=2048, ny=1024, box=0,
             steps=2, graph=False),
        # a Chombo-laid level (patches of at most 128 cells a side, ragged last ones) with plasticity, step by step
        dict(name="plastic_mixed_1000x500_b128", kind="level", law="sw", mixed=True, plastic=True, nx=1000, ny=500,
             box=128, steps=4, graph=False),
        # the smallest level a test or a tutorial run steps: latency of the calls
        dict(name="rs_mixed_64x32", kind="level", law="rs", mixed=True, plastic=False, nx=64, ny=32, box=0, steps=4,
             graph=False),
        # one patch of a Chombo patch loop, with the face fluxes its flux registers need
        dict(name="patch_fp64_128x128_flux", kind="patch", law="rs", nx=128, ny=128, flux=True),
        # the 3-D patch step at the benchmark's size
        dict(name="patch3_mixed_192x96x96", kind="patch3", law="rs", mixed=True, nx=192, ny=96, nz=96),
        # the 3-D patch step in the plain FP64 form on one Chombo-sized patch
        dict(name="patch3_fp64_64x48x48", kind="patch3", law="rs", mixed=False, nx=64, ny=48, nz=48),
        # a 3-D level of 32-cell patches: ghost exchange and the batched patch loop
        dict(name="level3_mixed_96x64x64_b32", kind="level3", law="sw", mixed=True, nx=96, ny=64, nz=64, box=32),
        # a refined run: three subcycled levels with plasticity, replayed from a graph
        dict(name="amr_mixed_512x256_l3", kind="amr", law="rs", mixed=True, nx=512, ny=256, levels=3),
        # a parameter study: independent scenarios of different grids in one launch
        dict(name="ensemble_mixed_16", kind="ensemble", count=16, steps=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["level", "level", "level", "patch", "patch3", "patch3", "level3", "amr", "ensemble"])
    law = rng.choice(["rs", "sw"])
    if kind == "level":
        nx, ny = _log(rng, 48, 2048), _log(rng, 24, 1024)
        mixed = rng.random() < 0.6
        box = rng.choice([0, 0, 64, 128])
        if box and -(-nx // box) * -(-ny // box) > 32:      # at most 32 patches
            box = 0
        steps = rng.choice([2, 4, 20]) if mixed else rng.choice([1, 2])
        return dict(kind=kind, law=law, mixed=mixed, plastic=rng.random() < 0.3, nx=nx, ny=ny, box=box, steps=steps,
                    graph=steps % 2 == 0 and rng.random() < 0.5)
    if kind == "patch":
        return dict(kind=kind, law=law, nx=_log(rng, 8, 256), ny=_log(rng, 8, 256), flux=rng.random() < 0.5)
    if kind == "patch3":
        mixed = rng.random() < 0.6
        hi = (192, 96, 96) if mixed else (64, 48, 48)
        return dict(kind=kind, law=law, mixed=mixed, nx=_log(rng, 16, hi[0]), ny=_log(rng, 16, hi[1]),
                    nz=_log(rng, 16, hi[2]))
    if kind == "level3":
        return dict(kind=kind, law=law, mixed=True, nx=_log(rng, 32, 96), ny=_log(rng, 32, 64), nz=_log(rng, 32, 64),
                    box=rng.choice([24, 32, 48]))
    if kind == "amr":
        return dict(kind=kind, law=law, mixed=True, nx=64 * rng.randint(2, 8), ny=32 * rng.randint(2, 8),
                    levels=rng.choice([2, 3]))
    return dict(kind=kind, count=rng.randint(2, 16), steps=rng.choice([4, 20]))


# ------------------------------------------------------------------ inputs
def _scenario(case, nx, ny):
    prec = A.TMK_PREC_MIXED if case.get("mixed", case["kind"] == "ensemble") else A.TMK_PREC_FP64
    plastic = bool(case.get("plastic", case["kind"] == "amr"))
    make = S.rate_state if case["law"] == "rs" else S.slip_weakening
    return make(nx=nx, ny=ny, dx=DX, precision=prec, plasticity=plastic)


def _boxes(nx, ny, box):
    if not box:
        return [(0, 0, nx - 1, ny - 1)]
    return [(i, j, min(i + box, nx) - 1, min(j + box, ny) - 1) for j in range(0, ny, box) for i in range(0, nx, box)]


def _boxes3(n, box):
    r = [[(i, min(i + box, m) - 1) for i in range(0, m, box)] for m in n]
    return [((x[0], y[0], z[0]), (x[1], y[1], z[1])) for z in r[2] for y in r[1] for x in r[0]]


def _waves(sc, shape, seed, plastic=False):
    """(22, *shape) FP64 state: the background plus smooth seeded waves (0.2 m/s, 2 MPa; wavelengths of 12 to
    120 cells), and on a plastic level a band of shear above the yield stress."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    U = torch.empty((22,) + tuple(shape), dtype=torch.float64, device="cuda")
    axes = [torch.arange(n, dtype=torch.float64, device="cuda").reshape([-1 if a == k else 1 for a in range(len(shape))])
            for k, n in enumerate(shape)]
    for c, bg in enumerate(sc.background()):
        U[c] = float(bg)
        if c % 11 > 8:
            continue
        amp = 0.1 if c % 11 < 3 else 1.0
        r = torch.rand((2, len(shape) + 2), generator=gen, device="cuda", dtype=torch.float64).tolist()
        for q in r:
            k = 2.0 * math.pi / (12.0 * 10.0 ** q[-1])
            d = [v - 0.5 for v in q[:len(shape)]]
            n = math.sqrt(sum(v * v for v in d)) + 1e-9
            U[c] += amp * torch.sin(sum(a * (k * v / n) for a, v in zip(axes, d)) + 6.2831853 * q[-2])
    if plastic:
        m = shape[-2]
        for side in (0, 11):
            U[side + 6, m // 4:m // 2] += 45.0
    return U


def _fault_data(sc, shape, seed):
    """Fault data (nb, *shape): the scenario's initial values with a seeded state (psi) or slip."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 7)
    b0 = torch.from_numpy(sc.initial_B(xlo=0, xhi=0, ghost=0)).cuda()
    B = b0.reshape((-1,) + (1,) * len(shape)).expand((-1,) + tuple(shape)).clone()
    r = torch.rand(tuple(shape), generator=gen, device="cuda", dtype=torch.float64)
    if sc.scheme.fault_law == A.TMK_FAULT_RS:
        B[10] += 0.01 * (r - 0.5)
    else:
        B[7] = 0.3 * r
    return B


def _cut(a, box, axes=2):
    """The part of a domain-wide (ghost-grown) array over `box` grown by the ghost width."""
    lo, hi = (box[:2], box[2:]) if axes == 2 else box
    s = tuple(slice(lo[d], hi[d] + 1 + 2 * G) for d in reversed(range(axes)))
    return a[(slice(None),) + s].contiguous()


class _State(dict):
    """What `prepare` returns; its library objects are closed, in order, when it goes."""

    def closing(self, *objs):
        weakref.finalize(self, lambda: [o.close() for o in objs])
        return self


def _inputs(case, seed):
    """The case's scenario, domain-wide state and fault data (torch, FP64, on the GPU)."""
    kind = case["kind"]
    if kind == "patch":
        nx, ny = case["nx"], case["ny"]
        sc = _scenario(case, 3 * nx, 2 * ny)
        return sc, _waves(sc, (ny + 2 * G, nx + 2 * G), seed), _fault_data(sc, (nx + 2 * G,), seed)
    if kind in ("patch3", "level3"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        sc = _scenario(case, nx, ny)
        if sc.sw is not None:
            sc.sw.fric_box_center[0] = nx * DX / 2
            sc.sw.zc[0] = nz * DX / 2
        return (sc, _waves(sc, (nz + 2 * G, ny + 2 * G, nx + 2 * G), seed),
                _fault_data(sc, (nz + 2 * G, nx + 2 * G), seed))
    nx, ny = case["nx"], case["ny"]
    sc = _scenario(case, nx, ny)
    return (sc, _waves(sc, (ny + 2 * G, nx + 2 * G), seed, case.get("plastic", False)),
            _fault_data(sc, (nx + 2 * G,), seed))


def _dt(case, sc):
    return sc.dt() / math.sqrt(3.0) if case["kind"] in ("patch3", "level3") else sc.dt()


def _out_arrays(level, n, law):
    """Device arrays that the patches' state and fault data are read into."""
    Us, Bs = [], []
    for p in range(n):
        us, bs = level.patch_shapes(p)
        Us.append(torch.empty(us, dtype=torch.float64, device="cuda"))
        Bs.append(torch.empty(bs, dtype=torch.float64, device="cuda") if level.touches_fault(p) else None)
    return Us, Bs


def _member(case, seed, k):
    """Scenario k of an ensemble: seeded friction, a grid of the repository's ensemble, waves of its own."""
    rng = np.random.default_rng(seed * 1000 + k)
    nx, ny = S.ENSEMBLE_GRIDS[k % len(S.ENSEMBLE_GRIDS)]
    sc = S.rate_state(nx=nx, ny=ny, dx=DX, precision=A.TMK_PREC_MIXED)
    sc.rs.a = float(rng.uniform(0.006, 0.012))
    sc.rs.b = sc.rs.a + float(rng.uniform(0.002, 0.006))
    sc.rs.L = float(rng.uniform(0.01, 0.05))
    sc.rs.psi_init = S.psi_steady(sc.elastic.sxy0, -sc.elastic.syy0, 1e-12, sc.rs.a, sc.rs.V0, sc.constants()["Zs"])
    return sc, _waves(sc, (ny + 2 * G, nx + 2 * G), seed * 1000 + k), _fault_data(sc, (nx + 2 * G,), seed * 1000 + k)


def prepare(case, seed):
    kind = case["kind"]
    st = _State(kind=kind, t=0.0, mixed=bool(case.get("mixed", kind == "ensemble")))
    if kind == "ensemble":
        mem = [_member(case, seed, k) for k in range(case["count"])]
        ctxs = [Context(sc) for sc, _, _ in mem]
        doms = [(0, 0, sc.nx - 1, sc.ny - 1) for sc, _, _ in mem]
        lv = LinElastEnsemble(ctxs, doms, [[d] for d in doms])
        for k, (_, U, B) in enumerate(mem):
            lv.set_patch(k, U, B)
        dt = mem[0][0].dt()
        g = lv.graph(case["steps"], 0.0, dt)
        st.update(level=lv, dt=dt, steps=case["steps"], graph=g, out=_out_arrays(lv, len(mem), "rs"))
        return st.closing(g, lv, *ctxs)
    sc, U, B = _inputs(case, seed)
    dt = _dt(case, sc)
    ctx = Context(sc)
    st.update(dt=dt, U=U, B=B)
    if kind == "patch":
        nx, ny = case["nx"], case["ny"]
        pg = LinElastPatchGodunov(ctx, domain=(0, 0, 3 * nx - 1, 2 * ny - 1))
        pg.set_current_box((nx, 0, 2 * nx - 1, ny - 1))
        st.update(patch=pg, lo=(nx - G, -G), flux=case["flux"])
        return st.closing(ctx)
    if kind == "patch3":
        hi = (case["nx"] - 1, case["ny"] - 1, case["nz"] - 1)
        pg = LinElastPatchGodunov3D(ctx, ((0, 0, 0), hi))
        pg.set_current_box(((0, 0, 0), hi))
        st.update(patch=pg)
        return st.closing(ctx)
    if kind == "level3":
        n = (case["nx"], case["ny"], case["nz"])
        boxes = _boxes3(n, case["box"])
        lv = LinElastLevelGodunov3D(ctx, boxes, ((0, 0, 0), tuple(m - 1 for m in n)))
        for p, b in enumerate(boxes):
            Bp = None
            if lv.touches_fault(p):
                Bp = B[:, b[0][2]:b[1][2] + 1 + 2 * G, b[0][0]:b[1][0] + 1 + 2 * G].contiguous()
            lv.set_patch(p, _cut(U, b, 3), Bp)
        st.update(level=lv, out=_out_arrays(lv, len(boxes), case["law"]))
        return st.closing(lv, ctx)
    if kind == "amr":
        nx, ny, n = case["nx"], case["ny"], case["levels"]
        levels, dom, dx, boxes = [], (0, 0, nx - 1, ny - 1), DX, _boxes(nx, ny, 128)
        for k in range(n):
            if k:
                # the next level: a band on the fault as wide and as high as the base, in its own cells
                dom, dx = refine_domain(dom, 2), dx / 2
                x0 = (dom[2] + 1 - nx) // 2 // 32 * 32
                boxes = [(b[0] + x0, b[1], b[2] + x0, b[3]) for b in _boxes(nx, ny, 128)]
            levels.append(LinElastLevelGodunov(ctx, boxes, domain=dom, dx=dx))
        for p, b in enumerate(levels[0].boxes):
            Bp = B[:, b[0]:b[2] + 1 + 2 * G].contiguous() if levels[0].touches_fault(p) else None
            levels[0].set_patch(p, _cut(U, b), Bp)
        for k in range(1, n):
            levels[k].attach_coarser(levels[k - 1], 2)
            levels[k].interp_from_coarser()
        torch.cuda.synchronize()
        h = AMRHierarchy(levels, [2] * (n - 1))
        g = h.graph(2, dt)
        st.update(levels=levels, graph=g, out=[_out_arrays(lv, len(lv.boxes), case["law"]) for lv in levels])
        return st.closing(g, h, *levels, ctx)
    boxes = _boxes(case["nx"], case["ny"], case["box"])
    lv = LinElastLevelGodunov(ctx, boxes)
    for p, b in enumerate(boxes):
        Bp = B[:, b[0]:b[2] + 1 + 2 * G].contiguous() if lv.touches_fault(p) else None
        lv.set_patch(p, _cut(U, b), Bp)
    g = lv.graph(case["steps"], 0.0, dt) if case["graph"] else None
    st.update(level=lv, steps=case["steps"], graph=g, out=_out_arrays(lv, len(boxes), case["law"]))
    return st.closing(*([g] if g else []), lv, ctx)


# -------------------------------------------------------------------- pass
def _valid(a):
    return a[(slice(None),) + (slice(G, -G),) * (a.dim() - 1)]


def _result(st, a):
    """Valid part of an array, in the type the form carries."""
    return _valid(a).float() if st["mixed"] else _valid(a)


def _read(st, level, out):
    Us, Bs = out
    for p, (U, B) in enumerate(zip(Us, Bs)):
        level.get_patch(p, U, B)
    return [_result(st, U) for U in Us], [_result(st, B) for B in Bs if B is not None]


def run(state):
    st = state
    kind, dt, t = st["kind"], st["dt"], st["t"]
    if kind in ("level", "ensemble"):
        lv = st["level"]
        if st["graph"] is not None:
            st["graph"].launch(t)
        else:
            for k in range(st["steps"]):
                lv.step(t + k * dt, dt)
        st["t"] = t + st["steps"] * dt
        return _read(st, lv, st["out"])
    if kind == "patch":
        pg = st["patch"]
        pg.set_current_time(t)
        st["t"] = t + dt
        _, Fx, Fy = pg.update_state(st["U"], st["lo"], dt, B=st["B"], bxlo=st["lo"][0], with_flux=st["flux"])
        return [st["U"], st["B"]] + ([Fx, Fy] if st["flux"] else [])
    if kind == "patch3":
        pg = st["patch"]
        pg.set_current_time(t)
        st["t"] = t + dt
        pg.update_state(st["U"], (-G, -G, -G), dt, B=st["B"], blo=(-G, -G))
        return [_result(st, st["U"]), _result(st, st["B"])]
    if kind == "level3":
        st["level"].step(t, dt)
        st["t"] = t + dt
        return _read(st, st["level"], st["out"])
    st["graph"].launch(t)
    st["t"] = t + 2 * dt
    return [_read(st, lv, out) for lv, out in zip(st["levels"], st["out"])]


# -------------------------------------------------------------------- work
def work(case):
    """Per step: the 18 evolving components of every valid cell read and written once (a plastic level reads 20 and
    writes 22), in the form's storage type; the 3-D entry points keep an FP64 state in both forms.  A level's state is
    also read back once a pass.  Operations per cell and step: the predictor's slopes, limiters and tracing, the
    Riemann solves, transverse terms and update of both sides, about 900 in 2-D and 2100 in 3-D."""
    kind = case["kind"]
    if kind == "ensemble":
        grids = [S.ENSEMBLE_GRIDS[k % len(S.ENSEMBLE_GRIDS)] for k in range(case["count"])]
        cells, steps = sum(a * b for a, b in grids), case["steps"]
        return dict(bytes=cells * (144.0 * steps + 176.0), flops=900.0 * cells * steps)
    if kind in ("patch3", "level3"):
        cells = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=cells * 288.0, flops=2100.0 * cells)
    cells = case["nx"] * case["ny"]
    if kind == "patch":
        return dict(bytes=cells * (288.0 + (352.0 if case["flux"] else 0.0)), flops=900.0 * cells)
    if kind == "amr":
        n = cells * 2 * (2 ** case["levels"] - 1)
        return dict(bytes=168.0 * n + 176.0 * cells * case["levels"], flops=900.0 * n)
    size = 4.0 if case["mixed"] else 8.0
    return dict(bytes=cells * size * ((42.0 if case["plastic"] else 36.0) * case["steps"] + 44.0),
                flops=900.0 * cells * case["steps"])


# ------------------------------------------------------------------- exact
# The step in plain FP64 torch on arrays [side][component][(z,) y, x] over the domain (or a patch and its
# ghost cells, whose outermost layers no valid cell's update reads).
_ROT = {0: (0, 1, 2, 6, 7), 1: (1, 2, 0, 8, 6), 2: (2, 0, 1, 7, 8)}      # cx, cy, cz, cxy, cxz


def _at(a, axis, s):
    i = [slice(None)] * a.dim()
    i[axis] = s
    return a[tuple(i)]


class _Exact:
    def __init__(self, sc, dim, dt, dx, x_faces, z_faces=None, t0=0.0):
        c = sc.constants()
        e = sc.elastic
        self.sc, self.dim, self.dt, self.dx, self.t = sc, dim, dt, dx, t0
        self.rho, self.lam, self.G, self.Zs, self.Zp, self.K = (c[k] for k in ("rho", "lam", "G", "Zs", "Zp", "K"))
        self.cs, self.cp = e.cs, e.cp
        self.x, self.z = x_faces, z_faces                    # fault faces' coordinates
        self.bg = sc.background()

    def rv(self, D):
        r = torch.ones(2, dtype=torch.float64, device="cuda")
        if D == 1:
            r[1] = -1.0
        return r.reshape((2,) + (1,) * self.dim)

    def pairs(self, D):
        cx, cy, cz, cxy, cxz = _ROT[D]
        return ((cx, cx + 3, self.Zp, self.cp), (cy, cxy, self.Zs, self.cs), (cz, cxz, self.Zs, self.cs))

    def predict(self, W, D):
        """Piecewise-parabolic normal predictor with primitive limiting: cell states at the lo and hi faces."""
        ax = W.dim() - 1 - D
        d = _at(W, ax, slice(1, None)) - _at(W, ax, slice(None, -1))
        dl = torch.cat([_at(d, ax, slice(0, 1)), d], ax)
        dr = torch.cat([d, _at(d, ax, slice(-1, None))], ax)
        dc = 0.5 * (dl + dr)
        s = torch.minimum(dc.abs(), 2 * torch.minimum(dl.abs(), dr.abs())) * torch.sign(dc)
        s = torch.where(dl * dr > 0, s, torch.zeros_like(s))
        del dl, dr, dc
        f = 0.5 * (_at(W, ax, slice(1, None)) + _at(W, ax, slice(None, -1))) - (
            _at(s, ax, slice(1, None)) - _at(s, ax, slice(None, -1))) / 6.0
        lo = torch.cat([_at(W - 0.5 * s, ax, slice(0, 1)), f], ax)
        hi = torch.cat([f, _at(W + 0.5 * s, ax, slice(-1, None))], ax)
        m, p = lo - W, hi - W
        flat = m * p >= 0
        m, p = (torch.where(flat, torch.zeros_like(m), torch.sign(m) * torch.minimum(m.abs(), 2 * p.abs())),
                torch.where(flat, torch.zeros_like(p), torch.sign(p) * torch.minimum(p.abs(), 2 * m.abs())))
        WM, WP, rv = W.clone(), W.clone(), self.rv(D)
        for v, q, Z, c in self.pairs(D):
            sg = c * self.dt / self.dx
            nm, np_ = m[:, q] + rv * Z * m[:, v], p[:, q] + rv * Z * p[:, v]     # left-going
            pm, pp = m[:, q] - rv * Z * m[:, v], p[:, q] - rv * Z * p[:, v]      # right-going
            nm = nm + 0.5 * sg * (np_ - nm) - 3.0 * (nm + np_) * (0.5 * sg - sg * sg / 3.0)
            pp = pp - 0.5 * sg * ((pp - pm) + 3.0 * (1.0 - 2.0 / 3.0 * sg) * (pm + pp))
            WM[:, q] += 0.5 * (nm + pm)
            WM[:, v] += rv * (nm - pm) / (2 * Z)
            WP[:, q] += 0.5 * (np_ + pp)
            WP[:, v] += rv * (np_ - pp) / (2 * Z)
        return WM, WP

    def faces(self, WM, WP, D, fault=None):
        """Face states of direction D (one more than cells along D): Riemann solves, absorbing edges, and on the
        y-lo faces the fault condition `fault` (a function of the states above it)."""
        ax = WM.dim() - 1 - D
        ghost = torch.zeros_like(_at(WM, ax, slice(0, 1)))
        for s in range(2):
            for c in range(9):
                ghost[s, c] = float(self.bg[11 * s + c])
        L, R = torch.cat([ghost, WP], ax), torch.cat([WM, ghost], ax)
        g, rv = torch.zeros_like(L), self.rv(D)
        for v, q, Z, _ in self.pairs(D):
            wp, wn = L[:, q] - rv * Z * L[:, v], R[:, q] + rv * Z * R[:, v]
            g[:, q] = 0.5 * (wn + wp)
            g[:, v] = rv * (wn - wp) / (2 * Z)
        if D == 1 and fault is not None:
            _at(g, ax, 0).copy_(fault(_at(WM, ax, 0)))
        return g

    def jump(self, g, D):
        ax = g.dim() - 1 - D
        return _at(g, ax, slice(1, None)) - _at(g, ax, slice(None, -1))

    def along(self, g, D, scale):
        """scale x (d/dx_D of the fluxes' linear map) applied to the face states g, or their differences."""
        cx, cy, cz, cxy, cxz = _ROT[D]
        a, rv = torch.zeros_like(g), -scale * self.rv(D)
        a[:, cx] = rv * g[:, cx + 3] / self.rho
        a[:, cy] = rv * g[:, cxy] / self.rho
        a[:, cz] = rv * g[:, cxz] / self.rho
        a[:, cx + 3] = rv * g[:, cx] * (self.lam + 2 * self.G)
        a[:, cy + 3] = rv * g[:, cx] * self.lam
        a[:, cz + 3] = rv * g[:, cx] * self.lam
        a[:, cxy] = rv * g[:, cy] * self.G
        a[:, cxz] = rv * g[:, cz] * self.G
        return a

    # ---- fault laws: W, Wg are [2][9][faces]; b is psi (rate and state) or the slip
    def solve(self, W, b):
        Zs, Zp = self.Zs, self.Zp
        px1, px2 = -W[0, 6] - Zs * W[0, 0], W[1, 6] - Zs * W[1, 0]
        py1, py2 = -W[0, 4] - Zp * W[0, 1], W[1, 4] - Zp * W[1, 1]
        g = torch.zeros_like(W)
        syy, vy = -0.5 * (py1 - py2), -0.5 * (py1 + py2) / Zp
        g[0, 4], g[1, 4], g[0, 1], g[1, 1] = syy, syy, vy, vy
        if self.sc.rs is not None:
            r = self.sc.rs
            tau0 = self.tau0()
            phi = 0.5 * (px2 - px1) + tau0
            sgn, ph = torch.sign(phi), phi.abs()
            alpha, eta = -syy * r.a, 0.5 * Zs
            lb = b / r.a - math.log(2 * r.V0)
            vmax = ph / Zs
            zmax = torch.asinh(torch.exp(lb) * vmax)
            lo, hi = torch.zeros_like(zmax), zmax.clone()
            z = torch.minimum(ph / alpha, zmax)
            for _ in range(200):                     # bracketed Newton on z = asinh(beta V)
                ex, em = torch.exp(z - lb), torch.exp(-z - lb)
                f = alpha * z + 0.5 * eta * (ex - em) - ph
                lo, hi = torch.where(f < 0, z, lo), torch.where(f < 0, hi, z)
                n = z - f / (alpha + 0.5 * eta * (ex + em))
                z = torch.where((n >= lo) & (n <= hi), n, 0.5 * (lo + hi))
            V, tau = 0.5 * (torch.exp(z - lb) - torch.exp(-z - lb)), alpha * z
            sxy = sgn * tau - tau0
            vx1 = -(sxy + px1) / Zs
            g[0, 6], g[1, 6], g[0, 0], g[1, 0] = sxy, sxy, vx1, vx1 - sgn * V
            return g
        w = self.sc.sw
        pz1, pz2 = -W[0, 8] - Zs * W[0, 2], W[1, 8] - Zs * W[1, 2]
        tau0 = self.tau0()
        fx, fz = 0.5 * (px2 - px1), 0.5 * (pz2 - pz1)
        lock = torch.sqrt((fx + tau0) ** 2 + fz ** 2)
        inside = ((self.x - w.fric_box_center[0]).abs() < w.fric_box_width[0]).double()
        if self.z is not None:
            inside = inside * ((self.z - w.fric_box_center[1]).abs() < w.fric_box_width[1]).double()
        mu = w.fs * inside + (1 - inside) * w.outside_friction
        mu = mu - (mu - w.fd) * torch.clamp(b / w.dw, max=1.0)
        tau = torch.minimum(lock, -syy * mu) - tau0
        ph = torch.sqrt(fx * fx + fz * fz)
        sxy, syz = fx / ph * tau, fz / ph * tau
        g[0, 6], g[1, 6], g[0, 8], g[1, 8] = sxy, sxy, syz, syz
        g[0, 0], g[0, 2] = -(sxy + px1) / Zs, -(syz + pz1) / Zs
        g[1, 0], g[1, 2] = (sxy - px2) / Zs, (syz - pz2) / Zs
        return g

    def tau0(self):
        if self.sc.rs is not None:
            r = self.sc.rs
            return r.nsig * torch.exp(-0.5 * ((self.x - r.x0) / r.r0) ** 2) + 0.0 * (0.0 if self.z is None else self.z)
        w, x = self.sc.sw, self.x - self.sc.sw.fric_box_center[0]
        t = w.tau[0] * ((x - w.xc[0]).abs() < w.xw[0]).double()
        if self.z is not None:
            t = t * ((self.z - w.fric_box_center[1] - w.zc[0]).abs() < w.zw[0]).double()
        return t

    def evolve(self, g, B, dt, final):
        """The state variable (or slip) after dt at the slip rate of the fault state g; `final` updates B."""
        vx, vz = g[0, 0] - g[1, 0], g[0, 2] - g[1, 2]
        V = torch.sqrt(vx * vx + vz * vz)
        if self.sc.rs is None:
            new = B[7] + dt * V
            if final:
                rt = B[8].clone()
                B[0], B[1], B[2], B[3], B[4], B[7] = vx, vz, g[0, 6], g[0, 8], V, new
                B[5] += dt * vx
                B[6] += dt * vz
                hit = (rt > self.t + dt) & (V > self.sc.sw.rupture_threshold)
                B[8] = torch.where(hit, torch.full_like(rt, self.t + dt), rt)
            return new
        r = self.sc.rs
        xx = V * dt / r.L
        phi1 = torch.where(xx > 1e-12, -torch.expm1(-xx) / xx.clamp(min=1e-300), 1.0 - 0.5 * xx)
        new = r.f0 + r.b * torch.log(torch.exp((B[10] - r.f0) / r.b - xx) + (r.V0 * dt / r.L) * phi1)
        if final:
            rt = B[9].clone()
            B[0], B[1], B[2], B[3], B[4], B[5] = vx, vz, V, g[0, 6] + self.tau0(), g[0, 8], g[0, 4]
            B[6] += dt * vx
            B[7] += dt * vz
            B[8] += dt * V
            hit = (rt > self.t + dt) & (V > r.rupture_threshold)
            late = torch.where(rt > self.t + dt, torch.full_like(rt, 1e10), rt)
            B[9] = torch.where(hit, torch.full_like(rt, self.t + dt), late)
            B[10] = new
        return new

    def step(self, U, B):
        """One step of U [2][11][...] and B [nb][faces] in place; returns the final face states per direction."""
        dim, dt, k = self.dim, self.dt, self.dt / self.dx
        W = U[:, :9]
        pre = [self.predict(W, D) for D in range(dim)]
        key = 10 if self.sc.rs is not None else 7
        seen = {}

        def fault(name, value):
            def solve(Wc):
                seen[name] = self.solve(Wc, value())
                return seen[name]
            return solve

        H1 = [self.faces(*pre[D], D, fault("first", lambda: B[key])) for D in range(dim)]
        final = []
        if dim == 2:
            for D in range(2):
                T = self.along(self.jump(H1[1 - D], 1 - D), 1 - D, -0.5 * k)
                final.append(self.faces(pre[D][0] + T, pre[D][1] + T, D,
                                        fault("final", lambda: self.evolve(seen["first"], B, 0.5 * dt, False))))
        else:
            H2 = {}
            for D in range(3):
                for E in range(3):
                    if E != D:
                        T = self.along(self.jump(H1[E], E), E, -k / 3.0)
                        H2[D, E] = self.faces(pre[D][0] + T, pre[D][1] + T, D,
                                              fault("second%d" % E, lambda: self.evolve(seen["first"], B, dt / 3.0, False)))
            for D in range(3):
                a, b = [E for E in range(3) if E != D]
                T = self.along(self.jump(H2[a, b], a), a, -0.5 * k) + self.along(self.jump(H2[b, a], b), b, -0.5 * k)
                final.append(self.faces(pre[D][0] + T, pre[D][1] + T, D,
                                        fault("final", lambda: self.evolve(seen["second2"], B, 0.5 * dt, False))))
        for D in range(dim):
            U[:, :9] -= k * self.along(self.jump(final[D], D), D, 1.0)
        self.evolve(seen["final"], B, dt, True)
        if self.sc.plastic is not None and self.sc.scheme.plasticity:
            self.plastic(U)
        self.t += dt
        return final

    def plastic(self, U):
        p, dt = self.sc.plastic, self.dt
        s = U[:, 3:9]
        n = (s[:, 0] + s[:, 1] + s[:, 2]) / 3.0
        J2 = ((s[:, 0] - s[:, 1]) ** 2 + (s[:, 1] - s[:, 2]) ** 2 + (s[:, 2] - s[:, 0]) ** 2) / 6.0 + (
            s[:, 3:] ** 2).sum(1)
        tau = torch.sqrt(J2)
        Y = tau - torch.clamp(-p.mu * n + p.b + U[:, 10] * p.h, min=0.0)
        lam = torch.where(Y > 0, Y / (dt * (p.h + self.G + p.mu * p.beta * self.K) + p.eta), torch.zeros_like(Y))
        f = torch.where(Y > 0, 1.0 - dt * lam * self.G / tau.clamp(min=1e-300), torch.ones_like(Y))
        n1 = n - dt * lam * self.K * p.beta
        for c in range(3):
            s[:, c] = n1 + f * (s[:, c] - n)
        s[:, 3:] *= f[:, None]
        U[:, 9] = lam
        U[:, 10] += dt * lam


def _exact_level(sc, U, B, steps, dt):
    x = (torch.arange(sc.nx, dtype=torch.float64, device="cuda") + 0.5) * DX
    e = _Exact(sc, 2, dt, DX, x)
    u = _valid(U).reshape((2, 11) + tuple(n - 2 * G for n in U.shape[1:])).clone()
    b = _valid(B).clone()
    for _ in range(steps):
        e.step(u, b)
    return u.reshape((22,) + tuple(u.shape[2:])), b


def exact(case, seed):
    kind = case["kind"]
    if kind == "amr":
        return None
    if kind == "ensemble":
        res = [_exact_level(sc, U, B, case["steps"], sc.dt())
               for sc, U, B in (_member(case, seed, k) for k in range(case["count"]))]
        return [u for u, _ in res], [b for _, b in res]
    sc, U, B = _inputs(case, seed)
    dt = _dt(case, sc)
    if kind == "level":
        u, b = _exact_level(sc, U, B, case["steps"], dt)
        boxes = _boxes(case["nx"], case["ny"], case["box"])
        return ([u[:, q[1]:q[3] + 1, q[0]:q[2] + 1] for q in boxes],
                [b[:, q[0]:q[2] + 1] for q in boxes if q[1] == 0])
    ar = lambda n, lo=0: (torch.arange(lo, lo + n, dtype=torch.float64, device="cuda") + 0.5) * DX  # noqa: E731
    if kind == "patch":
        nx, ny = case["nx"], case["ny"]
        e = _Exact(sc, 2, dt, DX, ar(nx + 2 * G, nx - G))
        region = U[:, G:]                                   # the rows below y = 0 lie outside the domain
        u = region.reshape((2, 11) + tuple(region.shape[1:])).clone()
        b = B.clone()
        fin = e.step(u, b)
        Uo, Bo = U.clone(), B.clone()
        Uo[:, G:-G, G:-G] = u.reshape(region.shape)[:, :ny, G:-G]
        Bo[:, G:-G] = b[:, G:-G]
        if not case["flux"]:
            return [Uo, Bo]
        F = []
        for D, g in enumerate(fin):
            f = torch.zeros((2, 11) + tuple(g.shape[2:]), dtype=torch.float64, device="cuda")
            f[:, :9] = e.along(g, D, 1.0)
            f = f.reshape((22,) + tuple(g.shape[2:]))
            F.append(f[:, :ny, G:G + nx + 1] if D == 0 else f[:, :ny + 1, G:G + nx])
        return [Uo, Bo] + F
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    e = _Exact(sc, 3, dt, DX, ar(nx)[None, :], ar(nz)[:, None])
    u = _valid(U).reshape((2, 11, nz, ny, nx)).clone()
    b = _valid(B).clone()
    e.step(u, b)
    u = u.reshape(22, nz, ny, nx)
    if kind == "patch3":
        return [u, b]
    boxes = _boxes3((nx, ny, nz), case["box"])
    cut = lambda a, q: a[:, q[0][2]:q[1][2] + 1, q[0][1]:q[1][1] + 1, q[0][0]:q[1][0] + 1]  # noqa: E731
    return ([cut(u, q) for q in boxes],
            [b[:, q[0][2]:q[1][2] + 1, q[0][0]:q[1][0] + 1] for q in boxes if q[0][1] == 0])
