"""The 3-D step on characteristic values == the oracle at the edges of its work:
patches one short of, equal to and one past a tile's 30 columns and 6 rows, the
predictor's 28 columns and 16 rows or planes, one-cell patches, and patches
whose halo ends at or past the domain's edges.  Bounds as for the patch step:
1e-12 in FP64; in the mixed form the FP32 rounding of one step's increments,
2e-5, and 1e-3 for the fault's boundary data, where slip rates amplify the
rounding of the shear.  Scales: the largest velocity and the largest stress (of the
boundary data also the largest slip) over the whole patch with its halo, since a
patch of one cell has none of its own.  The slip-weakening patch is centred off
the grid: whether a face exactly on its rim lies inside is a matter of rounding,
and fused multiply-adds decide it otherwise in the mixed form than in FP64."""
import numpy as np
import pytest

import oracle as O
from tetemoko_gb300 import _capi as A, scenarios as S
from tests.helpers import RTOL_FP64, perturbed_state_3d, random_B_3d

pytestmark = pytest.mark.gpu

G = A.TMK_NGHOST
# (domain, valid box)
SIZES = [((29, 7, 3), ((0, 0, 0), (28, 6, 2))), ((30, 6, 17), ((0, 0, 0), (29, 5, 16))),
         ((31, 13, 16), ((0, 0, 0), (30, 12, 15))), ((61, 12, 5), ((0, 0, 0), (60, 11, 4))),
         ((40, 20, 20), ((1, 0, 1), (28, 15, 16))), ((40, 20, 20), ((3, 2, 3), (32, 17, 18))),
         ((40, 20, 20), ((39, 19, 19), (39, 19, 19))), ((40, 20, 20), ((0, 0, 0), (0, 0, 0))),
         ((1, 1, 1), ((0, 0, 0), (0, 0, 0))), ((2, 3, 2), ((0, 0, 0), (1, 2, 1)))]


def _sc(law, nx, ny):
    if law == "sw":
        sc = S.slip_weakening(nx=nx, ny=ny, dx=0.1, layout=A.TMK_SW_LAYOUT_OFFSET11)
        sc.sw.fric_box_center[0] += 0.03
    else:
        sc = S.rate_state(nx=nx, ny=ny, dx=0.1)
    if law == "none":
        sc.scheme.fault_law = A.TMK_FAULT_NONE
        for k, v in enumerate((0, 1, 0, 1, 1, 0)):
            sc.scheme.boundary_type[k] = v
    return sc


def _err(a, b, ref, groups):
    """max over groups of components of |a - b| / the group's largest |ref| or |b|"""
    return max(np.abs(a[g] - b[g]).max() / max(np.abs(ref[g]).max(), np.abs(b[g]).max()) for g in groups)


VEL, STR = [0, 1, 2, 11, 12, 13], [3, 4, 5, 6, 7, 8, 14, 15, 16, 17, 18, 19]


@pytest.mark.parametrize("prec", [A.TMK_PREC_MIXED, A.TMK_PREC_FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("law", ["rs", "sw", "none"])
@pytest.mark.parametrize("dom,valid", SIZES, ids=["x".join(map(str, d)) + "_" + str(n) for n, (d, v) in enumerate(SIZES)])
def test_tile_edges_match_oracle(cuda_lib, dom, valid, law, prec):
    import torch
    from tetemoko_gb300.level import Context, LinElastPatchGodunov3D
    sc = _sc(law, dom[0], dom[1])
    dlo, dhi = (0, 0, 0), tuple(n - 1 for n in dom)
    lo, hi = valid
    rng = np.random.default_rng(911)
    U0 = perturbed_state_3d(sc, rng, lo, hi)
    fault = law != "none" and lo[1] == 0
    ulo, blo = tuple(a - G for a in lo), (lo[0] - G, lo[2] - G)
    B0 = random_B_3d(sc, rng, hi[0] - lo[0] + 1 + 2 * G, hi[2] - lo[2] + 1 + 2 * G) if fault else None
    dt, time = sc.dt(), 0.5
    Ur, Br = U0.copy(), (B0.copy() if fault else None)
    rc, Fr = O.patch_update_state_3d(sc, Ur, ulo, lo, hi, dlo, dhi, Br, blo, 0.1, time, dt, with_flux=True)
    assert rc == 0
    sc.scheme.precision = prec
    ctx = Context(sc)
    pg = LinElastPatchGodunov3D(ctx, (dlo, dhi))
    pg.set_current_box(valid)
    pg.set_current_time(time)
    Ud = torch.from_numpy(U0.copy()).cuda()
    Bd = torch.from_numpy(B0.copy()).cuda() if fault else None
    _, F = pg.update_state(Ud, ulo, dt, B=Bd, blo=blo, with_flux=True)
    torch.cuda.synchronize()
    Ug, Fg = Ud.cpu().numpy(), [f.cpu().numpy() for f in F]
    Bg = Bd.cpu().numpy() if fault else None
    # the same step without fluxes leaves the same state
    Ud2 = torch.from_numpy(U0.copy()).cuda()
    pg.update_state(Ud2, ulo, dt, B=torch.from_numpy(B0.copy()).cuda() if fault else None, blo=blo)
    assert np.array_equal(Ud2.cpu().numpy(), Ug)
    ctx.close()
    tol = RTOL_FP64 if prec == A.TMK_PREC_FP64 else 2e-5
    v = (slice(None), slice(G, -G), slice(G, -G), slice(G, -G))
    inside = np.zeros(U0.shape, bool)
    inside[v] = True
    inside[[9, 10, 20, 21]] = False
    assert np.array_equal(Ug[~inside], U0[~inside])
    assert _err(Ug[v], Ur[v], U0, (VEL, STR)) <= tol
    for d in range(3):
        assert _err(Fg[d], Fr[d], Fr[d], (VEL, STR)) <= tol, d
    if fault:
        bv = (slice(None), slice(G, -G), slice(G, -G))
        groups = [[0, 1, 2], [3, 4, 5], [6, 7, 8], [9], [10]] if law == "rs" else [[0, 1, 4], [2, 3], [5, 6, 7], [8]]
        assert _err(Bg[bv], Br[bv], B0, groups) <= (RTOL_FP64 if prec == A.TMK_PREC_FP64 else 1e-3)
