"""A level stepped with the fault kernel first and both component groups in one
launch, whose items finish the fault row, equals the same level stepped with
separate launches: widths around a strip's 28 columns, heights that leave a
last run of one row, one-row runs' neighbours, several patches, every law, with
and without plasticity.  Three steps; the two forms run the same operations, so
1e-12 (FP64) or a few FP32 roundings a step (2e-6) of the largest velocity and
stress."""
import numpy as np
import pytest

from tetemoko_gb300 import _capi as A, scenarios as S
from tests.helpers import perturbed_state

pytestmark = pytest.mark.gpu

G = A.TMK_NGHOST
VEL, STR = [0, 1, 2, 11, 12, 13], [3, 4, 5, 6, 7, 8, 14, 15, 16, 17, 18, 19]
LEVELS = {"27x3": ((27, 3), None), "28x5": ((28, 5), None), "29x9": ((29, 9), None), "85x33": ((85, 33), None),
          "patches": ((70, 40), [(0, 0, 30, 12), (31, 0, 69, 12), (0, 13, 69, 39)])}


@pytest.mark.parametrize("prec", [A.TMK_PREC_MIXED, A.TMK_PREC_FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("law", ["rs", "sw", "sw_ref9", "rs_ctu", "rs_plastic", "none"])
@pytest.mark.parametrize("name", list(LEVELS))
def test_one_launch_equals_two(cuda_lib, name, law, prec):
    from tetemoko_gb300.level import Context, LinElastLevelGodunov
    (nx, ny), boxes = LEVELS[name]
    if law.startswith("sw"):
        layout = A.TMK_SW_LAYOUT_REFERENCE9 if law == "sw_ref9" else A.TMK_SW_LAYOUT_OFFSET11
        sc = S.slip_weakening(nx=nx, ny=ny, dx=0.1, layout=layout, precision=prec)
    else:
        sc = S.rate_state(nx=nx, ny=ny, dx=0.1, precision=prec, plasticity=law == "rs_plastic")
    if law == "rs_ctu":
        sc.scheme.normal_pred_order = 0
    if law == "none":
        sc.scheme.fault_law = A.TMK_FAULT_NONE
    boxes = boxes or [(0, 0, nx - 1, ny - 1)]
    U0 = perturbed_state(sc, np.random.default_rng(5), amp_v=0.2, amp_s=2.0)
    B0 = sc.initial_B() if law != "none" else None
    out = []
    for first, run in ((1, 4), (0, 16)):
        ctx = Context(sc)
        lv = LinElastLevelGodunov(ctx, boxes)
        t = lv.tuning()
        t.fault_first, t.min_run = first, run
        lv.set_tuning(t)
        for p, b in enumerate(boxes):
            Up = U0[:, b[1]:b[3] + 1 + 2 * G, b[0]:b[2] + 1 + 2 * G]
            Bp = B0[:, b[0]:b[2] + 1 + 2 * G] if lv.touches_fault(p) else None
            lv.set_patch(p, np.ascontiguousarray(Up), np.ascontiguousarray(Bp) if Bp is not None else None)
        for k in range(3):
            lv.step(k * sc.dt(), sc.dt())
        out.append(lv.get_patches())
        assert lv.status()[0] == 0
        lv.close()
        ctx.close()
    tol = 1e-12 if prec == A.TMK_PREC_FP64 else 2e-6
    for p in range(len(boxes)):
        a, b = (np.asarray(o[0][p])[:, G:-G, G:-G] for o in out)
        assert np.isfinite(b).all()
        for g in (VEL, STR):
            assert np.abs(a[g] - b[g]).max() <= tol * np.abs(U0[g]).max(), (p, g)
        if out[0][1][p] is not None:
            a, b = (np.asarray(o[1][p])[:, G:-G] for o in out)
            assert np.array_equal(a, b) or np.abs(a - b).max() <= 1e3 * tol * np.abs(b).max()
