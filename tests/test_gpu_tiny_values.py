"""Steps of values at the small end of their type == the oracle: FP64 slopes
without limiting where a quarter by the exponent bits would leave the normal
numbers, and mixed 3-D increments that are FP32 denormals.  No background and no
fault, so that the step is linear and scales with its state."""
import numpy as np
import pytest

import oracle as O
from tetemoko_gb300 import _capi as A, scenarios as S
from tests.helpers import perturbed_state

pytestmark = pytest.mark.gpu

G = A.TMK_NGHOST


def _sc(nx, ny, prec):
    sc = S.rate_state(nx=nx, ny=ny, dx=0.1, precision=prec)
    sc.scheme.fault_law = A.TMK_FAULT_NONE
    for k in range(6):
        sc.scheme.boundary_type[k] = 0
    sc.elastic.sxy0 = sc.elastic.syy0 = 0.0
    return sc


@pytest.mark.parametrize("amp", [1e-307, 1e-300], ids=["below", "above"])
def test_unlimited_fp64_slopes_of_the_smallest_numbers(cuda_lib, amp):
    """Amplitudes on either side of 2^-1020; 1e-12 of the largest value (a last
    place of a denormal is 5e-17 of 1e-307)."""
    import torch
    from tetemoko_gb300.level import Context, LinElastPatchGodunov
    nx, ny = 31, 9
    sc = _sc(nx, ny, A.TMK_PREC_FP64)
    sc.scheme.use_prim_limiting = 0
    U0 = perturbed_state(sc, np.random.default_rng(4), amp_v=0.1, amp_s=1.0) * amp
    Ur = U0.copy()
    rc, _, _ = O.patch_update_state(sc, Ur, (-G, -G), (0, 0), (nx - 1, ny - 1), None, -G, 0.0, sc.dt())
    assert rc == 0
    ctx = Context(sc)
    pg = LinElastPatchGodunov(ctx)
    pg.set_current_box((0, 0, nx - 1, ny - 1))
    Ud = torch.from_numpy(U0.copy()).cuda()
    pg.update_state(Ud, (-G, -G), sc.dt())
    Ug = Ud.cpu().numpy()
    ctx.close()
    assert np.abs(Ug - Ur).max() <= 1e-12 * np.abs(Ur).max()


@pytest.mark.parametrize("amp", [3e-39, 3e-30], ids=["denormal", "normal"])
def test_mixed_3d_increments_that_are_denormals(cuda_lib, amp):
    """One cell's velocities set in a medium at rest, where every slope is zero and
    the step is first order; 1e-5 of the amplitude (a denormal last place is 5e-7)."""
    import torch
    from tetemoko_gb300.level import Context, LinElastPatchGodunov3D
    n = (9, 8, 7)
    sc = _sc(n[0], n[1], A.TMK_PREC_MIXED)
    U0 = np.zeros((22,) + tuple(m + 2 * G for m in n[::-1]))
    for c, f in ((0, 1.0), (1, -0.7), (2, 0.4), (11, 0.6), (12, 0.9), (13, -0.5)):
        U0[c, G + 3, G + 4, G + 4] = f * amp
    lo, hi = (0, 0, 0), tuple(m - 1 for m in n)
    Ur, dt = U0.copy(), sc.dt() / 2
    rc, _ = O.patch_update_state_3d(sc, Ur, (-G,) * 3, lo, hi, lo, hi, None, (0, 0), 0.1, 0.0, dt)
    assert rc == 0
    ctx = Context(sc)
    pg = LinElastPatchGodunov3D(ctx, (lo, hi))
    pg.set_current_box((lo, hi))
    Ud = torch.from_numpy(U0.copy()).cuda()
    pg.update_state(Ud, (-G,) * 3, dt)
    Ug = Ud.cpu().numpy()
    ctx.close()
    for k in range(22):
        scale = amp * (1.0 if k % 11 < 3 else 16.0)           # stresses of a velocity: impedance times it
        assert np.abs(Ug[k] - Ur[k]).max() <= 1e-5 * scale, k
