"""FP64 stage sums and final combination in integers (FxPoint, ih_fix.cuh):
numbers of terms, zeros, values that leave its exponent range and those that
meet others of a very different size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


def homogeneous(ctx, h, dh):
    """phi, dphi constant: no tensor source, so h and dh obey a linear equation
    mode by mode."""
    f = np.zeros(ctx.Ntot)
    f[:ctx.N], f[ctx.N:2 * ctx.N], f[-1] = 0.2, -0.8, 1.0
    f[4 * ctx.N:4 * ctx.N + 4 * ctx.M] = h
    f[4 * ctx.N + 4 * ctx.M:-1] = dh
    return f


@pytest.mark.parametrize("n", [(16, 16, 16), (24, 18, 12)])
def test_rk4_combination_of_any_size(gpu_mod, n):
    """One RK4 step against the same combination of the library's right-hand
    sides in extended precision, mode by mode: 1e-14 of the largest of y, dt k
    (ten roundings of 1e-16 on the way to k4 and in the sum)."""
    ctx = gpu_mod.Context(n=n, filter=False)
    rng = np.random.default_rng(1)
    size = rng.choice([0.0, 1e-300, 1e-290, 1e-200, 1e-30, 1.0, 1e30, 1e250, 1e270, 1e290],
                      size=2 * ctx.M).repeat(2)
    f = homogeneous(ctx, size * rng.standard_normal(4 * ctx.M), size * rng.standard_normal(4 * ctx.M))
    dt, LD = 3e-3, np.longdouble

    def k(y):
        return ctx.mk_rhs(y)[0]

    def comb(cs, ks):
        return f.astype(LD) + LD(dt) * sum(LD(c) * x.astype(LD) for c, x in zip(cs, ks))

    k1 = k(f)
    k2 = k(comb([0.5], [k1]).astype(float))
    k3 = k(comb([0.5], [k2]).astype(float))
    k4 = k(comb([1.0], [k3]).astype(float))
    want = comb([1 / 6, 1 / 3, 1 / 3, 1 / 6], [k1, k2, k3, k4])
    ctx.set_state(f)
    ctx.rk4_step(dt)
    got = ctx.get_state()
    scale = np.abs(f) + dt * np.max(np.abs([k1, k2, k3, k4]), axis=0)
    t = slice(4 * ctx.N, -1)
    assert np.isfinite(got).all()
    assert np.all(np.abs(got[t] - want[t]) <= 1e-14 * scale[t] + 1e-320)
    ctx.close()


@pytest.mark.parametrize("n", [(16, 16, 16), (24, 18, 12), (64, 32, 32)])
def test_dopri_step_in_and_out_of_the_range(gpu_mod, n):
    """The tensor modes scaled by 2^-900 (FP64 sums) and not (integers): the same
    step, 2^-900 apart to 1e-14 of each segment's norm."""
    rng = np.random.default_rng(2)
    runs = []
    for s in (0, -900):
        ctx = gpu_mod.Context(n=n, filter=False)
        rng = np.random.default_rng(2)
        h, dh = rng.standard_normal((2, 4 * ctx.M))
        ctx.set_state(homogeneous(ctx, np.ldexp(h, s), np.ldexp(dh, s)))
        ctx.dopri_init(gpu_mod.dopri_cfg(1e-2, 1e-2), 0.0, 5e-3)
        info = ctx.dopri_step(5e-3)
        assert info.dt_did == 5e-3 and info.tries == 1
        y = ctx.get_state()[4 * ctx.N:-1]
        runs.append(np.ldexp(y, -s).reshape(2, -1))
        ctx.close()
    a, b = runs
    assert (np.linalg.norm(a - b, axis=1) <= 1e-14 * np.linalg.norm(a, axis=1)).all()
