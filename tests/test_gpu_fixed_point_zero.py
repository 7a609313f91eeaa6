"""A product with zero is zero in the fixed-point passes: what cancels exactly in
FP64 transforms cancels in them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 8, 8), (24, 18, 12), (32, 32, 32), (72, 48, 24), (144, 96, 48),
                               (256, 128, 64), (288, 24, 24), (512, 16, 8)])
def test_fields_of_one_coordinate(n):
    """The transform of a field of x, of y or of z alone vanishes off its axis (on
    axes of 2^a points it does on the FP64 engines too)."""
    from instaheat_gb300 import gpu
    ctx = gpu.Context(n=n)
    rng = np.random.default_rng(sum(n))
    assert ctx.L_.ih_fft_get_engine(ctx.h, 9) == gpu.FFT_FIXED_ALL
    for axis in range(3):
        shape = [1, 1, 1]
        shape[axis] = -1
        phi = rng.standard_normal(n[axis]).reshape(shape) + np.zeros(n)
        X = ctx.fft(phi)
        X[tuple(slice(None) if a == axis else 0 for a in range(3))] = 0.0
        assert not X.any()
    ctx.close()
