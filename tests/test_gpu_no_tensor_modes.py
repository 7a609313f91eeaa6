"""FP64 contexts without tensor modes hold no projection table and run
everything else, tuned and untuned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 12, 8), (32, 32, 32)])
def test_no_projection_table_without_gw(n):
    from instaheat_gb300 import gpu
    nx, ny, nz = n
    octant = (nx // 2 + 1) * (ny // 2 + 1) * (nz // 2 + 1)
    with_gw, without = gpu.Context(n=n), gpu.Context(n=n, gw=False)
    # 12 coefficients, |k|^2 and the exponents: 14 words per octant mode
    assert with_gw.device_bytes - without.device_bytes == 14 * 8 * octant
    with_gw.close()
    without.ic(seed=4)
    f = without.get_state()
    a, _ = without.mk_rhs(f, filter=1)
    without.autotune()
    b, _ = without.mk_rhs(f, filter=1)
    real = 4 * nx * ny * nz
    assert np.abs(a[:real] - b[:real]).max() <= 1e-11 * np.abs(a[:real]).max()
    without.set_state(f)
    without.dopri_init(gpu.dopri_cfg(1e-8, 1e-8), 0.0, 1e-3)
    without.dopri_step(1e-3)
    without.rk4_step(1e-3)
    assert np.isfinite(without.get_state()[:real]).all()
    without.close()
