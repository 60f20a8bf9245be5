"""Fault data held to their own scales: the joint launch of both component groups
leaves the same bits as separate launches, and a 3-D step moves the slips by the
oracle's slip rate times dt."""
import numpy as np
import pytest

import oracle as O
from tetemoko_gb300 import _capi as A, scenarios as S
from tests.helpers import perturbed_state, perturbed_state_3d, random_B_3d

pytestmark = pytest.mark.gpu

G = A.TMK_NGHOST
LEVELS = {"27x3": ((27, 3), None), "29x9": ((29, 9), None), "85x33": ((85, 33), None),
          "patches": ((70, 40), [(0, 0, 30, 12), (31, 0, 69, 12), (0, 13, 69, 39)])}


@pytest.mark.parametrize("prec", [A.TMK_PREC_MIXED, A.TMK_PREC_FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("law", ["rs", "rs_slip", "sw", "sw_ref9", "rs_ctu", "rs_plastic"])
@pytest.mark.parametrize("name", list(LEVELS))
def test_one_launch_leaves_the_bits_of_separate_launches(cuda_lib, name, law, prec):
    """Both forms run the same operations in the same order on every cell and face."""
    from tetemoko_gb300.level import Context, LinElastLevelGodunov
    (nx, ny), boxes = LEVELS[name]
    if law.startswith("sw"):
        layout = A.TMK_SW_LAYOUT_REFERENCE9 if law == "sw_ref9" else A.TMK_SW_LAYOUT_OFFSET11
        sc = S.slip_weakening(nx=nx, ny=ny, dx=0.1, layout=layout, precision=prec)
    else:
        sc = S.rate_state(nx=nx, ny=ny, dx=0.1, precision=prec, plasticity=law == "rs_plastic",
                          state_law=A.TMK_RS_SLIP_LAW if law == "rs_slip" else A.TMK_RS_AGING_LAW)
        sc.rs.L = 0.5
    if law == "rs_ctu":
        sc.scheme.normal_pred_order = 0
    boxes = boxes or [(0, 0, nx - 1, ny - 1)]
    U0 = perturbed_state(sc, np.random.default_rng(5), amp_v=0.2, amp_s=2.0)
    B0 = sc.initial_B()
    out = []
    for first, run in ((1, 4), (0, 16)):
        ctx = Context(sc)
        lv = LinElastLevelGodunov(ctx, boxes)
        t = lv.tuning()
        t.fault_first, t.min_run = first, run
        lv.set_tuning(t)
        lv.set_level(U0, B0)
        for k in range(3):
            lv.step(k * sc.dt(), sc.dt())
        U, B = U0.copy(), B0.copy()
        lv.get_level(U, B)
        assert lv.status()[0] == 0
        out.append((U[:, G:-G, G:-G], B[:, G:-G]))
        lv.close()
        ctx.close()
    (Ua, Ba), (Ub, Bb) = out
    assert np.isfinite(Ub).all() and np.isfinite(Bb).all()
    assert np.abs(Bb - B0[:, G:-G]).max() > 0
    np.testing.assert_array_equal(Ba, Bb)
    np.testing.assert_array_equal(Ua, Ub)


@pytest.mark.parametrize("prec", [A.TMK_PREC_MIXED, A.TMK_PREC_FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("law", ["rs", "sw"])
@pytest.mark.parametrize("n", [(31, 13, 16), (8, 7, 5)], ids=["31x13x16", "8x7x5"])
def test_3d_slips_move_by_the_slip_rate(cuda_lib, n, law, prec):
    """Increments of the slips (rows 6 to 8, slip weakening 5 to 7) in units of dt times
    the largest slip rate, to the slip rates' own bounds (1e-12, mixed 1e-3: the
    fault amplifies the FP32 rounding of its shear), and what adding them to the
    stored slips rounds off: 100 m in the component that the reference starts there."""
    import torch
    from tetemoko_gb300.level import Context, LinElastPatchGodunov3D
    if law == "sw":
        sc = S.slip_weakening(nx=n[0], ny=n[1], dx=0.1, precision=prec)
        sc.sw.fric_box_center[0] += 0.03        # no face on the nucleation patch's rim
        slips, rates = [5, 6, 7], [0, 1, 4]
    else:
        sc = S.rate_state(nx=n[0], ny=n[1], dx=0.1, precision=prec)
        slips, rates = [6, 7, 8], [0, 1, 2]
    rng = np.random.default_rng(31)
    lo, hi = (0, 0, 0), tuple(m - 1 for m in n)
    U0, B0 = perturbed_state_3d(sc, rng, lo, hi), random_B_3d(sc, rng, n[0] + 2 * G, n[2] + 2 * G)
    dt = sc.dt() / 3 ** 0.5
    Ur, Br = U0.copy(), B0.copy()
    rc, _ = O.patch_update_state_3d(sc, Ur, (-G,) * 3, lo, hi, lo, hi, Br, (-G, -G), 0.1, 0.5, dt)
    assert rc == 0
    ctx = Context(sc)
    pg = LinElastPatchGodunov3D(ctx, (lo, hi))
    pg.set_current_box((lo, hi))
    pg.set_current_time(0.5)
    Ud, Bd = torch.from_numpy(U0.copy()).cuda(), torch.from_numpy(B0.copy()).cuda()
    pg.update_state(Ud, (-G,) * 3, dt, B=Bd, blo=(-G, -G))
    v = (slice(None), slice(G, -G), slice(G, -G))
    Bg, Bo, Bi = Bd.cpu().numpy()[v], Br[v], B0[v]
    ctx.close()
    tol = 1e-3 if prec == A.TMK_PREC_MIXED else 1e-12
    rate = np.abs(Bo[rates]).max()
    assert rate > 0.01
    for k in slips:
        bound = tol * dt * rate + 2.0 * np.finfo(float).eps * np.abs(Bi[k]).max()
        assert np.abs(Bg[k] - Bo[k]).max() <= bound, k
        if k != slips[1] or law == "sw":        # the rate-and-state law carries no antiplane slip
            assert np.abs(Bo[k] - Bi[k]).max() > 10.0 * bound, k
