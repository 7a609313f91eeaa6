"""Ensemble members of one grid whose boxes differ in what they can run: the
fixed-point passes need wave numbers within their exponent range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_autotune_keeps_members_to_their_own_passes(order):
    """A member in a box of 1e-70 has no fixed-point passes (and no tables for
    them): it does not take a twin's, nor a twin its."""
    from instaheat_gb300 import gpu
    n = (16, 16, 16)
    boxes = [(20.0,) * 3, (1e-70,) * 3]
    ens = gpu.Ensemble([dict(n=n, L=boxes[i], precision=gpu.PREC_F64) for i in order])
    can = [m.L_.ih_fft_get_engine(m.h, 9) for m in ens.members]
    assert sorted(can) == [0, gpu.FFT_FIXED_ALL]
    ens.autotune()
    on = [m.L_.ih_fft_get_engine(m.h, 9) for m in ens.members]
    assert all(o & ~c == 0 for o, c in zip(on, can))
    x = np.random.default_rng(1).standard_normal(n)
    for m in ens.members:
        X = np.fft.rfftn(x)
        assert np.abs(m.fft(x) - X).max() <= 1e-13 * np.abs(X).max()
    ens.close()
