"""Steps of values at the small end of their type == the oracle: FP64 slopes
without limiting where a quarter by the exponent bits would leave the normal
numbers.  No background and no
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
