"""The fixed-point transforms of pencils with one dominant value (a mean in the
spectrum, a spike in the field) or a falling spectrum: no further from extended
precision than the FP64 engines (pass 9 = 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


def norm(a):
    return float(np.sqrt((np.abs(a) ** 2).sum()))


def fields(n, rng):
    """(name, spectrum to invert, or None, and field to transform)."""
    k = np.minimum(np.arange(n[0]), n[0] - np.arange(n[0])).reshape(-1, 1, 1)
    noise = np.fft.rfftn(rng.standard_normal(n))
    mean = noise.copy()
    mean[0, 0, 0] = 1e6 * np.abs(noise).max()
    spike = rng.standard_normal(n)
    spike[n[0] // 3, 1, 2] = 1e6
    return [("mean", mean, None), ("falling", noise * (1.0 + k) ** -3.0, None),
            ("spike", None, spike),
            ("steep", None, np.fft.irfftn(noise, s=n, axes=(0, 1, 2)) * (1.0 + k) ** -3.0)]


@pytest.mark.parametrize("n", [(256, 8, 8), (256, 256, 8), (288, 12, 12), (512, 8, 8),
                               (32, 32, 32), (64, 64, 64)])
def test_transforms(gpu_mod, n):
    ctx = gpu_mod.Context(n=n)
    full = ctx.L_.ih_fft_get_engine(ctx.h, 9)
    assert full == gpu_mod.FFT_FIXED_ALL
    for name, X, x in fields(n, np.random.default_rng(sum(n))):
        if X is not None:
            exact = np.fft.irfftn(X.astype(np.clongdouble), s=n, axes=(0, 1, 2)) * np.prod(n)
            run = lambda: ctx.ifft(X)
        else:
            exact = np.fft.rfftn(x.astype(np.longdouble))
            run = lambda: ctx.fft(x)
        ctx.set_engine(9, full)
        fixed = norm(run() - exact) / norm(exact)
        ctx.set_engine(9, 0)
        fp64 = norm(run() - exact) / norm(exact)
        assert fixed <= max(fp64, 2.0 ** -53)
    ctx.close()


@pytest.mark.parametrize("nz", [64, 128, 256])
@pytest.mark.parametrize("kind", ["wave", "falling"])
def test_rows(gpu_mod, nz, kind):
    """z rows alone (the x and y axes hold copies): a single wave and a falling
    spectrum, forward and back."""
    n = (nz, nz, nz)
    ctx = gpu_mod.Context(n=n)
    rng = np.random.default_rng(nz)
    k = np.arange(nz // 2 + 1)
    z = (rng.standard_normal(k.size) + 1j * rng.standard_normal(k.size)) * (k > 0)
    z *= (k == 3) if kind == "wave" else (1.0 + k) ** -3.0
    z[-1] = z[-1].real
    X = np.zeros(n[:2] + (k.size,), complex)
    X[0, 0] = z
    row = np.fft.irfft(z.astype(np.clongdouble), n=nz) * nz
    err = {}
    for mask in (ctx.L_.ih_fft_get_engine(ctx.h, 9), 0):
        ctx.set_engine(9, mask)
        back = ctx.ifft(X)[0, 0]
        x = np.zeros(n)
        x[0, 0] = row.astype(float)
        exact = np.fft.rfft(row.astype(float).astype(np.longdouble))
        out = ctx.fft(x)[0, 0]
        err[mask] = (norm(back - row) / norm(row), norm(out - exact) / norm(exact))
    ctx.close()
    fixed, fp64 = err.values()
    for a, b in zip(fixed, fp64):
        assert a <= max(b, 2.0 ** -53)
