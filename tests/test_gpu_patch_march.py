"""The FP64 patch step on the marching kernels == the oracle at the edges of its
work: patches one short of, equal to and one past a strip's 28 columns, runs of
one row and ragged last runs, one-cell patches, patches inside the domain, at
its corners and as large as it, with and without the fault, in every scheme the
marching kernels run.  1e-12 of the largest velocity and stress over the patch
with its halo, for the state, all face fluxes and the fault's data."""
import numpy as np
import pytest

import oracle as O
from tetemoko_gb300 import _capi as A, scenarios as S
from tests.helpers import RTOL_FP64, perturbed_state

pytestmark = pytest.mark.gpu

G = A.TMK_NGHOST
VEL, STR = [0, 1, 2, 11, 12, 13], [3, 4, 5, 6, 7, 8, 14, 15, 16, 17, 18, 19]
NONE = [9, 10, 20, 21]
# (domain, valid box)
SIZES = [((27, 5), (0, 0, 26, 4)), ((28, 1), (0, 0, 27, 0)), ((29, 2), (0, 0, 28, 1)), ((57, 33), (0, 0, 56, 32)),
         ((90, 70), (3, 0, 86, 64)), ((90, 70), (7, 5, 62, 47)), ((90, 70), (89, 69, 89, 69)),
         ((90, 70), (0, 0, 0, 0)), ((1, 1), (0, 0, 0, 0)), ((400, 150), (0, 0, 399, 149))]


def _sc(law, nx, ny):
    if law.startswith("sw"):
        layout = A.TMK_SW_LAYOUT_REFERENCE9 if law == "sw_ref9" else A.TMK_SW_LAYOUT_OFFSET11
        return S.slip_weakening(nx=nx, ny=ny, dx=0.1, layout=layout)
    sc = S.rate_state(nx=nx, ny=ny, dx=0.1)
    if law == "none":
        sc.scheme.fault_law = A.TMK_FAULT_NONE
        for k, v in enumerate((0, 1, 0, 1, 1, 0)):
            sc.scheme.boundary_type[k] = v
    elif law == "rs_charlim":
        sc.scheme.use_prim_limiting, sc.scheme.use_char_limiting = 0, 1
    elif law == "rs_ctu":
        sc.scheme.normal_pred_order = 0
    return sc


def _err(a, b, ref, groups):
    """max over groups of components of |a - b| / the group's largest |ref| or |b|"""
    return max(np.abs(a[g] - b[g]).max() / max(np.abs(ref[g]).max(), np.abs(b[g]).max()) for g in groups)


@pytest.mark.parametrize("law", ["rs", "sw", "sw_ref9", "none", "rs_charlim", "rs_ctu"])
@pytest.mark.parametrize("dom,valid", SIZES, ids=["%dx%d_%d" % (d + (n,)) for n, (d, v) in enumerate(SIZES)])
def test_patch_edges_match_oracle(cuda_lib, dom, valid, law):
    import torch
    from tetemoko_gb300.level import Context, LinElastPatchGodunov
    sc = _sc(law, *dom)
    rng = np.random.default_rng(37)
    U0 = perturbed_state(sc, rng, lo=valid[:2], hi=valid[2:])
    fault = law != "none" and valid[1] == 0
    B0 = sc.initial_B(xlo=valid[0], xhi=valid[2]) if fault else None
    ulo, bxlo, dt, time = (valid[0] - G, valid[1] - G), valid[0] - G, sc.dt(), 0.75
    Ur, Br = U0.copy(), (B0.copy() if fault else None)
    rc, Fxr, Fyr = O.patch_update_state(sc, Ur, ulo, valid[:2], valid[2:], Br, bxlo, time, dt, with_flux=True)
    assert rc == 0
    ctx = Context(sc)
    pg = LinElastPatchGodunov(ctx)
    pg.set_current_box(valid)
    pg.set_current_time(time)
    Ud = torch.from_numpy(U0.copy()).cuda()
    Bd = torch.from_numpy(B0.copy()).cuda() if fault else None
    _, Fx, Fy = pg.update_state(Ud, ulo, dt, B=Bd, bxlo=bxlo, with_flux=True)
    Ug, F = Ud.cpu().numpy(), [Fx.cpu().numpy(), Fy.cpu().numpy()]
    # the same step without fluxes leaves the same state
    Ud2 = torch.from_numpy(U0.copy()).cuda()
    pg.update_state(Ud2, ulo, dt, B=torch.from_numpy(B0.copy()).cuda() if fault else None, bxlo=bxlo)
    assert np.array_equal(Ud2.cpu().numpy(), Ug)
    ctx.close()
    v = (slice(None), slice(G, -G), slice(G, -G))
    inside = np.zeros(U0.shape, bool)
    inside[v] = True
    inside[NONE] = False
    assert np.array_equal(Ug[~inside], U0[~inside])
    assert _err(Ug[v], Ur[v], U0, (VEL, STR)) <= RTOL_FP64
    for f, r in zip(F, (Fxr, Fyr)):
        assert _err(f, r, r, (VEL, STR)) <= RTOL_FP64
        assert not f[NONE].any()
    if fault:
        # slip velocities, tractions, slips (velocity x dt), rupture time, state variable (or total slip)
        rs = law.startswith("rs")
        groups = [[0, 1, 2], [3, 4, 5], [6, 7, 8], [9], [10]] if rs else [[0, 1, 4], [2, 3], [5, 6], [8], [7]]
        vel, stress = np.abs(U0[VEL]).max(), np.abs(U0[STR]).max()
        Bg, Bo = Bd.cpu().numpy()[:, G:-G], Br[:, G:-G]
        for g, scale in zip(groups, (vel, stress, vel * dt, 1e10, max(np.abs(Bo[groups[4]]).max(), vel * dt))):
            assert np.abs(Bg[g] - Bo[g]).max() <= RTOL_FP64 * scale, g
