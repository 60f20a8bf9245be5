"""Rate-and-state faces at the ends of what the friction laws meet == the oracle:
slip rates below the last bit of the sides' velocities, faces without traction,
states so low that the aging law's exponential overflows, and the lines between
the forms of the solve and of the state evolution.  Through every form that
solves them: the 2-D patch step, the 2-D level and the 3-D patch step, FP64 and
mixed."""
import numpy as np
import pytest

import oracle as O
from tetemoko_gb300 import _capi as A, scenarios as S
from tests.helpers import perturbed_state

pytestmark = pytest.mark.gpu

G = A.TMK_NGHOST
NY, NZ = 5, 3
FORMS = ["patch_fp64", "level_fp64", "level_mixed", "patch3_fp64", "patch3_mixed"]


def _sc(form, law, nx=37, **rs):
    prec = A.TMK_PREC_MIXED if form.endswith("mixed") else A.TMK_PREC_FP64
    sc = S.rate_state(nx=nx, ny=NY, dx=0.1, precision=prec, state_law=law)
    for k, v in rs.items():
        setattr(sc.rs, k, v)
    return sc


def _step(form, sc, U, B, dt):
    """One step of the 2-D state U, B (uniform in z for the 3-D forms): the GPU's and
    the oracle's (status or None, U, B) with the fault data over the valid faces."""
    import torch
    from tetemoko_gb300.level import Context, LinElastLevelGodunov, LinElastPatchGodunov, LinElastPatchGodunov3D
    ctx = Context(sc)
    Uo, Bo, nx = U.copy(), B.copy(), sc.nx
    v = slice(G, -G)
    if form.startswith("patch3"):
        rep = lambda a: np.ascontiguousarray(np.repeat(a[:, None], NZ + 2 * G, axis=1))
        Uo, Bo = rep(U), rep(B)
        lo, hi = (0, 0, 0), (nx - 1, NY - 1, NZ - 1)
        Ud, Bd = torch.from_numpy(Uo.copy()).cuda(), torch.from_numpy(Bo.copy()).cuda()
        rc, _ = O.patch_update_state_3d(sc, Uo, (-G, -G, -G), lo, hi, lo, hi, Bo, (-G, -G), 0.1, 0.0, dt)
        pg = LinElastPatchGodunov3D(ctx, (lo, hi))
        pg.set_current_box((lo, hi))
        pg.update_state(Ud, (-G, -G, -G), dt, B=Bd, blo=(-G, -G))
        out = None, Ud.cpu().numpy()[:, v, v, v], Bd.cpu().numpy()[:, v, v]
        ref = rc, Uo[:, v, v, v], Bo[:, v, v]
    else:
        rc, _, _ = O.patch_update_state(sc, Uo, (-G, -G), (0, 0), (nx - 1, NY - 1), Bo, -G, 0.0, dt)
        ref = rc, Uo[:, v, v], Bo[:, v]
        if form.startswith("patch"):
            Ud, Bd = torch.from_numpy(U.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
            pg = LinElastPatchGodunov(ctx)
            pg.set_current_box((0, 0, nx - 1, NY - 1))
            pg.update_state(Ud, (-G, -G), dt, B=Bd, bxlo=-G)
            out = None, Ud.cpu().numpy()[:, v, v], Bd.cpu().numpy()[:, v]
        else:
            lv = LinElastLevelGodunov(ctx, [(0, 0, nx - 1, NY - 1)])
            lv.set_level(U, B)
            lv.step(0.0, dt)
            Ug, Bg = U.copy(), B.copy()
            lv.get_level(Ug, Bg)
            out = lv.status()[0], Ug[:, v, v], Bg[:, v]
            lv.close()
    ctx.close()
    return out, ref


@pytest.mark.parametrize("law", [A.TMK_RS_SLIP_LAW, A.TMK_RS_AGING_LAW], ids=["slip", "aging"])
@pytest.mark.parametrize("form", FORMS)
def test_slip_rate_below_the_velocities_last_bit_is_zero(cuda_lib, form, law):
    """psi = 1.5 holds the fault at about 1e-55 m/s while its sides move at 0.1 m/s
    or so: the difference of the sides' velocities is exactly zero, so the slip law's
    logarithm makes the half-step state NaN, the final slip rate with it, and the
    step reports it; the aging law goes on."""
    sc = _sc(form, law)
    U = perturbed_state(sc, np.random.default_rng(2), amp_v=0.5, amp_s=2.0)
    B = sc.initial_B()
    B[10] = 1.5
    (rc, Ug, Bg), (rco, Uo, Bo) = _step(form, sc, U, B, sc.dt() / 2)
    nan = law == A.TMK_RS_SLIP_LAW
    assert np.isnan(Bo[10]).all() == nan and (nan or not Bo[:3].any())
    assert np.array_equal(Bg[:3], Bo[:3], equal_nan=True)
    assert np.array_equal(np.isnan(Bg), np.isnan(Bo))
    if rc is not None:
        assert rc == rco == (2 if nan else 0)
    if not nan:
        assert np.abs(Bg[10] - Bo[10]).max() <= 1e-12 * 1.5


@pytest.mark.parametrize("form", FORMS)
def test_a_face_without_traction_is_reported(cuda_lib, form):
    """No shear on the fault and none to nucleate: the direction of slip is 0/0, the
    slip rate and the state NaN, and the step reports it."""
    sc = _sc(form, A.TMK_RS_AGING_LAW, nsig=0.0)
    sc.elastic.sxy0 = 0.0
    U, B = sc.initial_U(), sc.initial_B()
    B[10] = 0.6
    (rc, Ug, Bg), (rco, Uo, Bo) = _step(form, sc, U, B, sc.dt() / 2)
    assert np.isnan(Bo[[0, 2, 10]]).all()
    assert np.array_equal(np.isnan(Bg), np.isnan(Bo))
    assert rc is None or rc == rco == 2


@pytest.mark.parametrize("form", FORMS)
def test_aging_law_at_rest_far_below_steady_state(cuda_lib, form):
    """b = 5e-5 and psi 0.05 below f0: e^(1000) overflows, on a fault that stands
    still (slip rate exactly zero): the state is f0 + b log(V0 dt / L)."""
    sc = _sc(form, A.TMK_RS_AGING_LAW, a=0.001, b=5e-5)
    sc.elastic.sxy0 = 50.0
    sc.rs.nsig = 0.0
    U = perturbed_state(sc, np.random.default_rng(2), amp_v=0.5, amp_s=2.0)
    B = sc.initial_B()
    B[10] = 0.55
    dt = sc.dt() / 2
    (rc, Ug, Bg), (rco, Uo, Bo) = _step(form, sc, U, B, dt)
    assert rco == 0 and not Bo[:3].any()
    assert rc in (0, None) and not Bg[:3].any()
    known = sc.rs.f0 + sc.rs.b * np.log(sc.rs.V0 * dt / sc.rs.L)
    assert np.abs(Bo[10] - known).max() <= 1e-14
    assert np.abs(Bg[10] - known).max() <= 1e-14


def test_mixed_solve_is_fp64_to_the_last_digits(cuda_lib):
    """600 faces of a uniform state (so that both forms solve the same equations):
    the tractions of the mixed form's solve against the FP64 form's.  Its one FP64
    Newton step leaves 8e-17 of the traction in the median, the rounding of FP64;
    with that step divided by an FP32 derivative the difference was 4e-16.  Bound 3e-16."""
    from tetemoko_gb300.level import Context, LinElastLevelGodunov
    nx, tau = 600, []
    rng = np.random.default_rng(8)
    F = np.stack([rng.uniform(0.006, 0.014, nx + 2 * G), rng.uniform(0.015, 0.02, nx + 2 * G),
                  rng.uniform(0.01, 0.05, nx + 2 * G)])
    psi = rng.uniform(0.62, 0.9, nx + 2 * G)
    for prec in (A.TMK_PREC_FP64, A.TMK_PREC_MIXED):
        sc = S.rate_state(nx=nx, ny=5, dx=0.1, precision=prec)
        sc.rs.nsig = 0.0
        B = sc.initial_B()
        B[10] = psi
        ctx = Context(sc)
        lv = LinElastLevelGodunov(ctx, [(0, 0, nx - 1, 4)])
        lv.set_level(sc.initial_U(), B)
        lv.set_fault_friction(0, F)
        lv.step(0.0, sc.dt())
        lv.get_level(sc.initial_U(), B)
        assert lv.status()[0] == 0
        tau.append(B[3, G:-G].copy())
        lv.close()
        ctx.close()
    assert np.median(np.abs(tau[1] - tau[0]) / tau[0]) <= 3e-16


# (a, b, psi from, psi to, the sides' velocity difference if not 0): what the sweep of
# the state over the faces crosses.  With 70 MPa of shear on 120 MPa, f0 = 0.6, L = 0.02 m, V0 = 1e-6 m/s and dt = 7.5 ms:
SWEEPS = {
    "slip_in_a_step": (0.008, 0.012, 0.40, 0.75),    # V dt / L = 0.01 (psi near 0.50) and r = 1e-3 (psi = 0.505)
    "sum_in_range": (0.010, 4e-4, 0.312, 0.324),     # r = 1e300, where log1p gives way to the sum itself
    "exp_of_minus_z": (0.0305, 0.036, 0.20, 0.90),   # z = 19, past which e^-z is dropped
    "bracket_end": (0.008, 0.012, 0.160, 0.170),     # the root at V = phi / Zs
    "bracket_far": (0.008, 0.012, 0.00, 0.30),
    "tiny_rate": (0.008, 0.012, 0.85, 0.97),         # V = 1e-21 to 1e-27 from rest
    "halvings": (0.008, 0.012, 0.93, 0.99, 1.0),     # 80 halvings from 1 m/s to the root (psi = 0.957)
}
# what RSNEWTON itself does not solve, and FP64 leaves to it:
UNSOLVED = {
    "tiniest_rate": (0.008, 0.012, 0.97, 1.05),      # below the velocities' last bit at RSNEWTON's residual
    "unreached": (0.008, 0.012, 0.99, 1.15, 1.0),    # 100 halvings from 1 m/s end above the root (psi = 1.07)
    "unreached_from_above": (0.008, 0.012, 0.99, 1.15, 40.0),     # ... from the bracket's middle
    "beta_squared": (0.0015, 0.004, 0.40, 0.60),     # beta^2 overflows past psi = 0.513: NaN from V = 0
}
CASES = [(f, n) for n in SWEEPS for f in FORMS] + [(f, n) for n in UNSOLVED for f in FORMS if f.endswith("fp64")]


@pytest.mark.parametrize("law", [A.TMK_RS_SLIP_LAW, A.TMK_RS_AGING_LAW], ids=["slip", "aging"])
@pytest.mark.parametrize("form,name", CASES, ids=["%s-%s" % c for c in CASES])
def test_the_lines_between_the_forms_of_the_solve(cuda_lib, form, name, law):
    """241 faces of a uniform state (which the mixed form holds exactly, but for the FP32
    rounding of a moving fault's shear, 1e-7 of it) whose psi crosses a line.
    RSNEWTON stops at a residual of 2.2e-12 MPa: a relative error of the slip rate of 2.2e-12 / (a sn), or of FP64's rounding of phi where that is more;
    the mixed form's accepted step is at most 1e-8 of the slip rate off.  The slip rate
    is the difference of two velocities of phi / Zs: 1e-14 of that.  Each bound twice,
    for the two or four solves in turn; the state moves by b, or the slip law's
    a + (b - a), times V dt / L for a relative change of V."""
    nx = 241
    a, b, p0, p1, *move = {**SWEEPS, **UNSOLVED}[name]
    sc = _sc(form, law, nx=nx, a=a, b=b, nsig=0.0)
    if law == A.TMK_RS_SLIP_LAW:
        sc.rs.L = 2.0           # the explicit step is stable
    U, B, dt = sc.initial_U(), sc.initial_B(), sc.dt() / 2
    B[10] = np.linspace(p0, p1, nx + 2 * G)
    alpha, phi, Zs = 120.0 * a, 70.0, sc.constants()["Zs"]
    if move:
        U[0], U[11] = 0.5 * move[0], -0.5 * move[0]
        phi += 0.5 * Zs * move[0]
    (rc, Ug, Bg), (rco, Uo, Bo) = _step(form, sc, U, B, dt)
    nan = np.isnan(Bo[10])
    assert np.array_equal(np.isnan(Bg), np.isnan(Bo)) and (rc is None or rc == rco)
    assert name in UNSOLVED or not nan.any()
    V = np.where(nan, 0.0, Bo[2])
    mixed = form.endswith("mixed")
    shear = 1e-7 * phi if mixed and move else 0.0
    rel = max(2.2e-12 / alpha, 1e-15 * phi / alpha) + (1e-8 if mixed else 0.0) + shear / alpha
    dV = 2.0 * (rel * V + 1e-14 * phi / Zs)
    ok = ~nan
    assert (np.abs(Bg[2] - Bo[2])[ok] <= dV[ok]).all()
    # alpha z: z moves by the relative change of V; never less than FP64's rounding
    assert (np.abs(Bg[3] - Bo[3])[ok] <= 2.0 * alpha * rel + 2.0 * shear + 1e-12 * phi).all()
    x = V * dt / sc.rs.L
    dpsi = 1e-13 + 4.0 * (a + b) * (x + 1.0 * (law == A.TMK_RS_SLIP_LAW) * x * 60.0) * rel
    dpsi = dpsi + 4.0 * (a + b) * dt / sc.rs.L * 1e-14 * phi / Zs * 60.0
    assert (np.abs(Bg[10] - Bo[10])[ok] <= dpsi[ok]).all()


@pytest.mark.parametrize("form", ["level", "patch3"])
def test_mixed_shear_holds_the_velocities_by_the_whole_impedance(cuda_lib, form):
    """600 faces whose sides move at +-2 m/s, varying slowly along the fault, weak
    enough to slip: the shear they carry, tau + Zs/2 V, mixed less FP64.  The rounding
    of the entering values (18.5 MPa in FP32) is 4e-7 a face, 1.6e-8 in the mean; the
    impedance rounded to FP32 would shift the mean by 4.2e-8 Zs v = 7.7e-7.  Bound 2e-7."""
    import torch
    from tetemoko_gb300.level import Context, LinElastLevelGodunov, LinElastPatchGodunov3D
    nx, shear = 600, []
    for prec in (A.TMK_PREC_FP64, A.TMK_PREC_MIXED):
        sc = S.rate_state(nx=nx, ny=NY, dx=0.1, precision=prec)
        sc.rs.nsig = 0.0
        U, B, dt = sc.initial_U(), sc.initial_B(), sc.dt() / 2
        v = 2.0 + 0.1 * np.sin(np.arange(nx + 2 * G) * 0.011)
        U[0], U[11] = v, -v
        B[10] = 0.4
        ctx = Context(sc)
        if form == "level":
            lv = LinElastLevelGodunov(ctx, [(0, 0, nx - 1, NY - 1)])
            lv.set_level(U, B)
            lv.step(0.0, dt)
            lv.get_level(U, B)
            lv.close()
            Bv = B[:, G:-G]
        else:
            rep = lambda a: torch.from_numpy(np.repeat(a[:, None], NZ + 2 * G, axis=1).copy()).cuda()
            dom = ((0, 0, 0), (nx - 1, NY - 1, NZ - 1))
            Ud, Bd = rep(U), rep(B)
            pg = LinElastPatchGodunov3D(ctx, dom)
            pg.set_current_box(dom)
            pg.update_state(Ud, (-G,) * 3, dt, B=Bd, blo=(-G, -G))
            Bv = Bd.cpu().numpy()[:, G + 1, G:-G]
        shear.append(Bv[3] + 0.5 * sc.constants()["Zs"] * Bv[2])
        assert (Bv[2] > 0.5).all()
        ctx.close()
    assert abs(np.mean(shear[1] - shear[0])) <= 2e-7
