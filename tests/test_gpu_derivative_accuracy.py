"""Derivatives of the FP64 form against extended precision: the fixed-point
round trips and d/dz are no further off than the FP64 engines (pass 9 = 0),
whatever the spectrum of the field along an axis.

The fields are f(i_axis) p(k) with p = 1 or the wave (1, 0, -1, 0, ...) along z, so
products are exact and the exact derivatives are one-dimensional transforms,
taken in extended precision.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
TWO_PI = np.float64(6.283185307179586)


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


def norm(a):
    return float(np.sqrt((np.abs(a) ** 2).sum()))


def spectrum(kind, L, rng):
    """Half spectrum of a real pencil with no constant part."""
    k = np.arange(L // 2 + 1)
    z = rng.standard_normal(k.size) + 1j * rng.standard_normal(k.size)
    w = {"white": 1.0 + 0.0 * k, "low": 1.0 * (k <= 3), "k^-2": (1.0 + k) ** -2.0,
         "wave": 1.0 * (k == 3)}[kind] * (k > 0)
    return z * w


def exact(f, length, lead):
    """f'' and f' of f (zero mean not needed) in extended precision, with the
    wave numbers that the code has in double."""
    L = f.size
    F = np.fft.rfft(f.astype(LD))
    k = np.arange(F.size)
    q = LD(TWO_PI * TWO_PI / (length * length))
    d2 = -np.fft.irfft(F * (k * k * q), n=L)
    d1 = np.fft.irfft(F * (1j * np.where(2 * k == L, LD(0), k * LD(TWO_PI / length))), n=L)
    shape = [1, 1, 1]
    shape[lead] = -1
    return d2.reshape(shape), d1.reshape(shape)


def errors(ctx, axis, f, wave):
    """Relative errors of the laplacian and, of phi = f alone, of the pressure
    (the squared gradient for the most part) of one right-hand side."""
    n, L = ctx.n, ctx.box
    shape = [1, 1, 1]
    shape[axis] = -1
    p = np.ones(n[2])
    if wave:
        p = np.tile([1.0, 0.0, -1.0, 0.0], n[2] // 4)
    phi = f.reshape(shape) * p.reshape(1, 1, -1) + np.zeros(n)
    y = np.zeros(ctx.Ntot)
    y[:ctx.N] = phi.ravel()
    y[-1] = 1.0
    ctx.mk_rhs(y)
    d2, d1 = exact(f, L[axis], axis)
    kz = (n[2] // 4) if wave else 0
    lap = (d2 - kz * kz * LD(TWO_PI * TWO_PI / (L[2] * L[2])) * f.reshape(shape)) * p + np.zeros(n)
    out = [norm(ctx.field("lap").reshape(n) - lap) / norm(lap)]
    if not wave:
        p = -d1 * d1 / 6 - phi.astype(LD) ** 2 / 2
        out.append(norm(ctx.field("pressure").reshape(n) - p) / norm(p))
    return out


def compare(gpu_mod, n, axis, kind, L=(1.0, 1.0, 1.0)):
    ctx = gpu_mod.Context(n=n, L=L)
    ctx.n, ctx.box = n, L
    assert ctx.L_.ih_fft_get_engine(ctx.h, 9) == gpu_mod.FFT_FIXED_ALL
    rng = np.random.default_rng(n[axis] + axis)
    f = np.fft.irfft(spectrum(kind, n[axis], rng), n=n[axis])
    for wave in ((False, True) if axis < 2 else (False,)):
        ctx.set_engine(9, gpu_mod.FFT_FIXED_ALL)
        fixed = errors(ctx, axis, f, wave)
        ctx.set_engine(9, 0)
        fp64 = errors(ctx, axis, f, wave)
        # a rounding of the laplacian; of the pressure four: its squares' sum, the
        # two products of m^2 phi^2 / 2 and the sum
        for a, b, roundings in zip(fixed, fp64, (1, 4)):
            assert a <= max(b, roundings * 2.0 ** -53)
    ctx.close()


@pytest.mark.parametrize("n", [(72, 24, 24), (72, 72, 24), (144, 48, 48), (96, 96, 96)])
@pytest.mark.parametrize("axis", [0, 1])
def test_white_noise_on_radix_3_axes(gpu_mod, n, axis):
    """The odd parts of the transforms' 1 / N factors sit in the derivative
    coefficients, which have to fill their words all the same."""
    compare(gpu_mod, n, axis, "white")


@pytest.mark.parametrize("kind", ["low", "k^-2", "wave"])
@pytest.mark.parametrize("n,axis", [((256, 8, 8), 0), ((256, 256, 8), 1), ((512, 8, 8), 0),
                                    ((512, 512, 8), 1), ((144, 48, 48), 0), ((144, 144, 48), 1),
                                    ((288, 24, 24), 0), ((288, 288, 24), 1), ((96, 96, 96), 2),
                                    ((128, 128, 128), 2), ((192, 192, 192), 2)])
def test_power_at_small_wave_numbers(gpu_mod, n, axis, kind):
    """Pencils whose derivatives come from a few small k: the products k X are
    small beside the spectrum's and the coefficients' largest values."""
    compare(gpu_mod, n, axis, kind)


@pytest.mark.parametrize("n", [(72, 24, 24), (72, 72, 24), (96, 96, 96), (256, 8, 8), (64, 64, 64)])
def test_fields_of_z_alone(gpu_mod, n):
    """k_x = k_y = 0: one product in a pencil, far below the largest coefficient."""
    compare(gpu_mod, n, 2, "white")


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("L", [(1.0, 100.0, 0.01), (1.0, 1.0, 0.001)])
def test_elongated_boxes(gpu_mod, L, axis):
    """k_z beyond k_y by orders of magnitude: the columns of small k_z keep
    their own exponent."""
    compare(gpu_mod, (64, 64, 64), axis, "low", L)
