"""Faces exactly on the rim of a slip-weakening nucleation patch, in every form
that solves them.  An odd number of cells with the patch in the grid's middle
puts a face's centre 1.5 km from the patch's to the last bit of the arithmetic,
so its side is that of the rounding: once in the 2-D mixed form and in a mixed
3-D patch by itself, product first in the FP64 forms (as the oracle) and in a
mixed 3-D batch.  Inside, a uniform state at 70 + 11.6 MPa slips against a
strength of 81.24 MPa; outside it is locked."""
from fractions import Fraction

import numpy as np
import pytest

import oracle as O
from tetemoko_gb300 import _capi as A, scenarios as S

pytestmark = pytest.mark.gpu

G = A.TMK_NGHOST
NY, NZ = 5, 4
FORMS = [("patch", A.TMK_PREC_FP64, False), ("level", A.TMK_PREC_FP64, False), ("level", A.TMK_PREC_MIXED, True),
         ("patch3", A.TMK_PREC_FP64, False), ("patch3", A.TMK_PREC_MIXED, True), ("batch3", A.TMK_PREC_FP64, False),
         ("batch3", A.TMK_PREC_MIXED, False)]


def _sc(nx, prec):
    sc = S.slip_weakening(nx=nx, ny=NY, dx=0.1, precision=prec)
    sc.sw.zw[0] = 1e3
    return sc


def _inside(sc, nx, fused):
    """Faces inside the patch with the position rounded once (fused) or product first."""
    c, xc, xw = sc.sw.fric_box_center[0], sc.sw.xc[0], sc.sw.xw[0]
    out = []
    for i in range(nx):
        x = float(Fraction(i + 0.5) * Fraction(sc.dx) - Fraction(c)) if fused else (i + 0.5) * sc.dx - c
        out.append(not abs(x - xc) - xw >= 0.0)
    return np.array(out)


def _slip_rate(form, sc, nx):
    """Slip rates (faces, or planes x faces) after one step of a uniform state."""
    import torch
    from tetemoko_gb300.level import Context, LinElastLevelGodunov, LinElastPatchGodunov, LinElastPatchGodunov3D
    U, B, dt = sc.initial_U(), sc.initial_B(), sc.dt() / 2
    ctx = Context(sc)
    if form == "level":
        lv = LinElastLevelGodunov(ctx, [(0, 0, nx - 1, NY - 1)])
        lv.set_level(U, B)
        lv.step(0.0, dt)
        lv.get_level(U, B)
        lv.close()
        V = B[4, G:-G]
    elif form == "patch":
        Ud, Bd = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
        pg = LinElastPatchGodunov(ctx)
        pg.set_current_box((0, 0, nx - 1, NY - 1))
        pg.update_state(Ud, (-G, -G), dt, B=Bd, bxlo=-G)
        V = Bd.cpu().numpy()[4, G:-G]
    else:
        rep = lambda a: torch.from_numpy(np.repeat(a[:, None], NZ + 2 * G, axis=1).copy()).cuda()
        dom = ((0, 0, 0), (nx - 1, NY - 1, NZ - 1))
        Ud, Bd = rep(U), rep(B)
        pg = LinElastPatchGodunov3D(ctx, dom)
        pg.set_current_box(dom)
        if form == "patch3":
            pg.update_state(Ud, (-G,) * 3, dt, B=Bd, blo=(-G, -G))
        else:
            pg.update_states([(dom, Ud, (-G,) * 3, Bd, (-G, -G))], dt)
        V = Bd.cpu().numpy()[4, G:-G, G:-G]
    ctx.close()
    return V


@pytest.mark.parametrize("nx", [33, 61, 101, 127])
@pytest.mark.parametrize("form,prec,fused", FORMS, ids=["%s_%s" % (f, "mixed" if p else "fp64") for f, p, _ in FORMS])
def test_rim_faces_keep_their_side(cuda_lib, form, prec, fused, nx):
    sc = _sc(nx, prec)
    want = _inside(sc, nx, fused)
    V = np.atleast_2d(_slip_rate(form, sc, nx))
    assert (np.abs(V) < 0.5).all() and ((V > 1e-3) == want).all()
    if not fused:       # the oracle's rounding
        U, B = sc.initial_U(), sc.initial_B()
        rc, _, _ = O.patch_update_state(sc, U, (-G, -G), (0, 0), (nx - 1, NY - 1), B, -G, 0.0, sc.dt() / 2)
        assert rc == 0 and ((B[4, G:-G] > 1e-3) == want).all()


def test_the_two_roundings_differ_at_these_sizes():
    assert any((_inside(_sc(nx, 0), nx, True) != _inside(_sc(nx, 0), nx, False)).any() for nx in (33, 61, 101, 127))
