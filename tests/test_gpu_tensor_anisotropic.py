"""Tensor sources of a field that varies mostly along z: S_zz exceeds the other
S_ij by orders of magnitude, and the modes along kz, whose n1 is S_xy alone, keep
their own precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 16, 16), (24, 24, 24), (32, 32, 32), (64, 32, 16)])
@pytest.mark.parametrize("noise", [1e-3, 1e-6])
def test_modes_along_the_dominant_axis(n, noise):
    """n1 of the modes kx = ky = 0 is the transform of d_x phi d_y phi: with
    white noise of `noise` times the wave, the field's own rounding (2^-53 of the
    wave) limits it to about 2^-53 / noise times a few, 1e-10 and better for
    1e-6; with the factor two of the sum over points and the transforms, 2e-9.
    In units of S_zz, which is 1 / noise^2 larger, that is 2e-21."""
    from instaheat_gb300 import gpu
    ctx = gpu.Context(n=n)
    N, M = ctx.N, ctx.M
    rng = np.random.default_rng(2)
    k = np.arange(n[2])
    phi = 1e-2 * (np.cos(6 * np.pi * k / n[2]).reshape(1, 1, -1) + noise * rng.standard_normal(n))
    f = np.zeros(ctx.Ntot)
    f[:N], f[N:2 * N], f[-1] = phi.ravel(), -0.8, 1.0
    r, _ = ctx.mk_rhs(f)
    ctx.close()
    X = np.fft.rfftn(phi.astype(np.longdouble))
    u = 2 * np.pi / 20.0
    d = []
    for axis in (0, 1):
        i = np.arange(n[axis])
        q = np.where(2 * i == n[axis], 0, np.where(i > n[axis] // 2, i - n[axis], i)) * u
        shape = [1, 1, 1]
        shape[axis] = -1
        d.append(np.fft.irfftn(1j * q.reshape(shape) * X, s=n, axes=(0, 1, 2)))
    want = 2 * np.fft.rfftn(d[0] * d[1])[0, 0, 1:]
    a = 4 * N + 4 * M + 2 * M  # dh2
    got = r[a:a + 2 * M].view(complex).reshape(n[0], n[1], -1)[0, 0, 1:]
    assert np.sqrt((np.abs(got - want) ** 2).sum() / (np.abs(want) ** 2).sum()) <= 2e-15 / noise


def test_small_coefficients_count_in_full():
    """A flat box: kz exceeds kx and ky by 10^4, so the coefficient of S_zz in n1 is
    10^-8 of that of S_xy, but S_zz is as much larger and both terms count.  phi =
    wave(z) (1 + 1e-2 noise(x, y)); its rounding limits the derivatives along x and y
    to 2^-53 / 1e-2 = 1e-14 of themselves, the sources to some ten times that:
    1e-12 leaves another factor.  (n0 has 1 - kz^2 / k^2 times S_zz in it, which the
    reference's own formula resolves to 1e-8 here.)"""
    from instaheat_gb300 import gpu
    from oracle.rhs_numpy import NumpyRHS
    n, L = (16, 16, 16), (20.0, 20.0, 0.002)

    class Extended(NumpyRHS):
        def fft(self, x):
            return np.fft.rfftn(np.asarray(x).reshape(self.n).astype(np.longdouble))

        def ifft(self, c):
            return np.fft.irfftn(c, s=self.n, axes=(0, 1, 2)) * np.longdouble(self.N)

    ctx, o = gpu.Context(n=n, L=L), Extended(n, L)
    N, M = ctx.N, ctx.M
    rng = np.random.default_rng(4)
    wave = np.cos(6 * np.pi * np.arange(n[2]) / n[2]).reshape(1, 1, -1)
    phi = 1e-2 * wave * (1.0 + 1e-2 * rng.standard_normal(n[:2] + (1,)))
    f = np.zeros(ctx.Ntot)
    f[:N], f[N:2 * N], f[-1] = phi.ravel(), -0.8, 1.0
    r, _ = ctx.mk_rhs(f)
    ctx.close()
    X = o.fft(phi) / N
    d = [o.ifft(X * 1j * o.g[a].astype(np.longdouble)).ravel() for a in "xyz"]
    o.g = {k: v.astype(np.longdouble) for k, v in o.g.items()}
    a = 4 * N + 4 * M
    want = 2 * o.tt_sources(*d)[1][1:, 1:, 1:]
    got = r[a + 2 * M:a + 4 * M].view(complex).reshape(n[0], n[1], -1)[1:, 1:, 1:]
    assert np.sqrt((np.abs(got - want) ** 2).sum() / (np.abs(want) ** 2).sum()) <= 1e-12
