"""The squared gradient at points where it is far below the largest of its row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 16, 16), (48, 24, 24), (64, 64, 64), (128, 128, 128)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_pressure_where_the_gradient_vanishes(n, axis):
    """phi = 1 + 1e-3 wave in a box of 1e-9: |grad phi|^2 / 6 is 10^12 of m^2 phi^2 / 2
    and more, but on the crests it vanishes with the square of the derivatives'
    own errors (2^-50 of the largest, 2^-100 squared: 1e-18 of the potential).
    There p = -m^2 phi^2 / 2 within a few roundings: 1e-14."""
    from instaheat_gb300 import gpu
    box = 1e-9
    ctx = gpu.Context(n=n, L=(box,) * 3)
    shape = [1, 1, 1]
    shape[axis] = -1
    phi = 1.0 + 1e-3 * np.cos(4 * np.pi * np.arange(n[axis]) / n[axis])
    crest = np.arange(n[axis]) % (n[axis] // 4) == 0
    f = np.zeros(ctx.Ntot)
    f[:ctx.N] = (phi.reshape(shape) + np.zeros(n)).ravel()
    f[-1] = 1.0
    ctx.mk_rhs(f)
    p = np.moveaxis(ctx.field("pressure").reshape(n), axis, -1)
    ctx.close()
    assert np.abs(p).max() >= 1e12
    want = -phi[crest] ** 2 / 2
    assert np.abs(p[..., crest] / want - 1).max() <= 1e-14
