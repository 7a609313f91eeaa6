"""The FP64 form's update_h from the octant table of projection coefficients:
every sign of kx and ky, the planes kx = 0, ky = 0, kz = 0, Nyquist and the
zero mode, odd thread counts, against the oracle's mode-by-mode formula."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


# a few modes only, non-cubic, radix 3, one octant entry per thread and four
@pytest.mark.parametrize("n", [(8, 8, 8), (16, 12, 8), (48, 18, 12), (32, 32, 32), (128, 96, 64)])
def test_projection_of_every_mode(gpu_mod, n):
    """dh' with h = dh = 0 is the projected source alone; the oracle's numpy
    form projects the same S_ij.  1e-11 of the largest, the bound of the FP64
    right-hand side against the oracle."""
    from oracle.rhs_numpy import NumpyRHS
    L = (20.0, 17.0, 13.0)
    ctx, o = gpu_mod.Context(n=n, L=L), NumpyRHS(n, L)
    rng = np.random.default_rng(sum(n))
    f = np.zeros(ctx.Ntot)
    f[:4 * ctx.N] = 1e-2 * rng.standard_normal(4 * ctx.N)
    f[ctx.N:2 * ctx.N] -= 0.8
    f[-1] = 1.3
    r, _ = ctx.mk_rhs(f)
    ref, _, _ = o.rhs(f)
    a, X = 4 * ctx.N + 4 * ctx.M, 2 * ctx.M
    for s in (slice(a, a + X), slice(a + X, a + 2 * X)):
        assert np.abs(r[s] - ref[s]).max() <= 1e-11 * np.abs(ref[s]).max()
    # the planes of the special cases by themselves
    for s in (slice(a, a + X), slice(a + X, a + 2 * X)):
        got = r[s].view(np.complex128).reshape(n[0], n[1], -1)
        want = ref[s].view(np.complex128).reshape(n[0], n[1], -1)
        for p in ((0,), (n[0] // 2,), (slice(None), 0), (slice(None), n[1] // 2),
                  (slice(None), slice(None), 0), (slice(None), slice(None), -1), (0, 0),
                  (slice(None), 0, 0)):
            assert np.abs(got[p] - want[p]).max() <= 1e-11 * np.abs(want).max()
        assert got[0, 0, 0] == 0.0
    ctx.close()


def test_stage_fusion_is_identical_at_odd_sizes(gpu_mod):
    """The form that also writes the next stage's input takes the same table."""
    runs = []
    for fuse in (False, True):
        ctx = gpu_mod.Context(n=(24, 18, 12))
        ctx.stage_fusion(fuse)
        ctx.ic(seed=3)
        ctx.dopri_init(gpu_mod.dopri_cfg(1e-8, 1e-8), 0.0, 1e-2)
        for _ in range(2):
            ctx.dopri_step(1e-2)
        runs.append(ctx.get_state())
        ctx.close()
    assert np.array_equal(*runs)


@pytest.mark.parametrize("n", [(16, 12, 8), (32, 32, 32)])
def test_sources_outside_the_integer_range(gpu_mod, n):
    """The projection of sources of 2^-960 the size (summed in FP64): the same
    values but for the scale, to 1e-13 of the norm."""
    rng = np.random.default_rng(5)
    x = None
    runs = []
    for s in (0, -480):
        ctx = gpu_mod.Context(n=n)
        x = rng.standard_normal(ctx.N) if x is None else x
        f = np.zeros(ctx.Ntot)
        f[:ctx.N] = np.ldexp(1e-2 * x, s)
        f[ctx.N:2 * ctx.N] = -0.8
        f[-1] = 1.3
        r, _ = ctx.mk_rhs(f)
        runs.append(np.ldexp(r[4 * ctx.N + 4 * ctx.M:-1], -2 * s))
        ctx.close()
    a, b = runs
    assert np.linalg.norm(a) > 0
    assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(a)
