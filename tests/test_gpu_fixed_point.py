"""The FP64 form's transforms in 64-bit block fixed point (ih_fix.cu): every
pencil length, the ends of the exponent range, constants, zeros and non-finite
values, against numpy's FP64 transforms and the FP64-pipe engines."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# every pencil length 8..512 along x and y, every row length along z
GRIDS = [(12, 12, 12), (24, 18, 12), (48, 36, 24), (72, 72, 48), (96, 64, 48), (144, 96, 96),
         (192, 192, 192), (288, 24, 24), (384, 384, 8), (384, 12, 12),
         (8, 8, 8), (16, 8, 8), (32, 16, 16), (64, 32, 32), (128, 128, 64), (256, 64, 8),
         (512, 8, 8), (512, 512, 16), (128, 128, 128), (256, 256, 256), (512, 512, 512)]


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


def norm(a):
    return np.sqrt((np.abs(a) ** 2).sum())


def over(a, scale):
    """a / scale, component by component (scale may have no finite inverse)."""
    a = np.ascontiguousarray(a)
    return (a.view(np.float64) / scale).view(a.dtype)


@pytest.mark.parametrize("n", GRIDS[:-1])
def test_transforms(gpu_mod, n):
    """Within 2e-15 in the 2-norm: numpy's own FP64 transform of 2^24 points is
    off by about eps sqrt(log2 N) = 1.1e-16 * 4.9 = 5.4e-16, the fixed-point one
    by less; 2e-15 is twice their sum."""
    ctx = gpu_mod.Context(n=n)
    assert ctx.L_.ih_fft_get_engine(ctx.h, 9) == gpu_mod.FFT_FIXED_ALL, "all passes"
    x = np.random.default_rng(sum(n)).standard_normal(n)
    X = np.fft.rfftn(x)
    assert norm(ctx.fft(x) - X) <= 2e-15 * norm(X)
    y = np.fft.irfftn(X, s=n, axes=(0, 1, 2)) * x.size
    assert norm(ctx.ifft(X) - y) <= 2e-15 * norm(y)
    # a large constant plus fluctuations: the spectrum without its mean is off
    # by the rounding of the constant, 2^-53 per value at least, in both
    G, Y = ctx.fft(1.0 + 1e-3 * x), np.fft.rfftn(1.0 + 1e-3 * x)
    G[0, 0, 0] = Y[0, 0, 0] = 0.0
    assert norm(G - Y) <= 2e-12 * norm(Y)
    ctx.close()


def test_transforms_512_cubed_plane_wave(gpu_mod):
    """The longest rows and pencils together: one real mode and its spectrum."""
    n = GRIDS[-1]
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs about 70 GB of device memory")
    ctx = gpu_mod.Context(n=n)
    i, j, k = np.ogrid[:n[0], :n[1], :n[2]]
    x = np.cos(2 * np.pi * ((3 * i) % n[0] / n[0] + (5 * j) % n[1] / n[1] + (7 * k) % n[2] / n[2]))
    X = ctx.fft(x)
    N = x.size
    assert abs(X[3, 5, 7] - N / 2) <= 1e-15 * N
    X[3, 5, 7] = 0.0
    assert np.abs(X).max() <= 1e-13 * N
    ctx.close()


@pytest.mark.parametrize("scale", [2.0 ** -1040, 1e-300, 2.0 ** -324, 2.0 ** -322, 2.0 ** 36,
                                   2.0 ** 38, 1e300])
def test_exponent_range(gpu_mod, scale):
    """Linear in the data over the whole range of FP64 (subnormals to the
    quantum): powers of two and other scales on both sides of the limits of
    the common case."""
    n = (32, 16, 8)
    ctx = gpu_mod.Context(n=n)
    x = np.random.default_rng(3).uniform(-1, 1, n) * scale
    X = np.fft.rfftn(x / scale)
    got = ctx.fft(x)
    quantum = 2.0 ** -1074
    assert norm(over(got, scale) - X) <= 2e-15 * norm(X) + 64 * quantum / scale * np.sqrt(X.size)
    back = ctx.ifft(got / x.size)
    assert norm(back / scale - x / scale) <= 4e-15 * norm(x / scale) + \
        256 * quantum / scale * np.sqrt(x.size)
    ctx.close()


def test_scales_of_single_rows(gpu_mod):
    """Rows have exponents of their own: a field that is one row of 1e-200 or
    of 1e+8 in a grid of zeros."""
    n = (64, 64, 64)
    ctx = gpu_mod.Context(n=n)
    rng = np.random.default_rng(4)
    for scale in (1e-200, 1e8):
        x = np.zeros(n)
        x[5, 3] = rng.standard_normal(n[2])
        X = np.fft.rfftn(x)
        assert norm(over(ctx.fft(x * scale), scale) - X) <= 2e-15 * norm(X)
    ctx.close()


def test_zeros_and_non_finite(gpu_mod):
    n = (16, 16, 8)
    ctx = gpu_mod.Context(n=n)
    assert np.array_equal(ctx.fft(np.zeros(n)), np.zeros((16, 16, 5)))
    assert np.array_equal(ctx.ifft(np.zeros((16, 16, 5), complex)), np.zeros(n))
    assert np.array_equal(ctx.fft(np.full(n, -2.5))[0, 0, 0], -2.5 * 2048)
    for bad in (np.nan, np.inf, -np.inf):
        x = np.random.default_rng(1).standard_normal(n)
        x[3, 2, 1] = bad
        assert np.isnan(ctx.fft(x)).all()
        x = np.random.default_rng(1).standard_normal(n)
        x[0, 0, 0] = bad
        assert np.isnan(ctx.fft(x)).all()
    ctx.close()


def state(gpu_mod, ctx, seed, amp=1e-3):
    ctx.ic(seed=seed, amp=amp)
    f = ctx.get_state()
    rng = np.random.default_rng(seed)
    f[4 * ctx.N:-1] = 1e-4 * np.sqrt(ctx.N) * rng.standard_normal(8 * ctx.M)
    return f


@pytest.mark.parametrize("n", [(8, 8, 8), (16, 16, 8), (64, 32, 16), (32, 32, 32), (128, 64, 64),
                               (512, 16, 8), (256, 256, 256), (24, 18, 12), (96, 64, 48),
                               (144, 72, 48), (384, 12, 12), (54, 48, 24), (48, 48, 36)])
@pytest.mark.parametrize("flag", [0, 1])
def test_rhs_agrees_with_the_fp64_engines(gpu_mod, n, flag):
    """One right-hand side on the fixed-point passes and on the FP64 engines:
    their fluctuation parts agree to 1e-11 of each segment, the bound of both
    against the oracle; single passes pinned to an FP64 engine in between."""
    ctx = gpu_mod.Context(n=n, L=(20.0, 17.0, 13.0))
    f = state(gpu_mod, ctx, 5)
    passes = ctx.L_.ih_fft_get_engine(ctx.h, 9)
    ctx.set_engine(9, 0)
    ref, _ = ctx.mk_rhs(f, filter=flag, output=flag)
    ctx.set_engine(9, passes)
    runs = [ctx.mk_rhs(f, filter=flag, output=flag)[0]]
    for p, e in ((0, 1), (1, 2), (3, 2), (4, 1), (6, 1)):
        ctx.set_engine(9, passes)
        ctx.set_engine(p, e)
        runs.append(ctx.mk_rhs(f, filter=flag, output=flag)[0])
    N, X = ctx.N, 2 * ctx.M
    edges = [0, N, 2 * N, 3 * N, 4 * N] + [4 * N + i * X for i in range(1, 5)]
    for r in runs:
        for a, b in zip(edges[:-1], edges[1:]):
            w = ref[a:b] - ref[a:b].mean()
            assert norm(r[a:b] - ref[a:b]) <= 1e-11 * norm(w)
        assert abs(r[-1] / ref[-1] - 1) <= 1e-14
    ctx.close()


def test_rhs_of_waves_along_one_axis_and_at_rest(gpu_mod):
    """Derivative rows that are exactly zero beside others that are not (a wave
    along x, y or z), and a homogeneous state."""
    n = (32, 32, 16)
    ctx = gpu_mod.Context(n=n)
    i, j, k = np.meshgrid(*(np.arange(m) for m in n), indexing="ij")
    f = np.zeros(ctx.Ntot)
    f[-1] = 1.0
    f[ctx.N:2 * ctx.N] = -0.8
    for w in (0.0, np.cos(2 * np.pi * i / n[0]), np.cos(4 * np.pi * j / n[1]),
              np.cos(2 * np.pi * k / n[2])):
        f[:ctx.N] = (1.0 + 1e-3 * w + np.zeros(n)).ravel()
        ctx.set_engine(9, gpu_mod.FFT_FIXED_ALL)
        a, _ = ctx.mk_rhs(f)
        ctx.set_engine(9, 0)
        b, _ = ctx.mk_rhs(f)
        assert np.isfinite(a).all()
        N = ctx.N
        # in units of the wave's own derivatives, 1e-3 k^2 and their square
        assert np.abs(a[:4 * N] - b[:4 * N]).max() <= 1e-13
        assert np.abs(a[4 * N:-1] - b[4 * N:-1]).max() <= 1e-13 * N * 1e-3
    ctx.close()


def test_pass_9_is_refused_where_it_does_not_apply(gpu_mod):
    """The mixed form; an axis of 54 points (27 x 2), a row of 36 (18 complex
    values): the passes that remain are offered, the others refused."""
    for kw, can in ((dict(n=(32, 32, 32), precision=gpu_mod.PREC_MIXED), 0),
                    (dict(n=(54, 48, 24)), 2 | 64), (dict(n=(48, 48, 36)), 1 | 2),
                    (dict(n=(48, 32, 32)), gpu_mod.FFT_FIXED_ALL)):
        ctx = gpu_mod.Context(**kw)
        assert ctx.L_.ih_fft_get_engine(ctx.h, 9) == can
        if can != gpu_mod.FFT_FIXED_ALL:
            with pytest.raises(gpu_mod.IHError):
                ctx.set_engine(9, gpu_mod.FFT_FIXED_ALL)
        ctx.set_engine(9, 0)
        ctx.close()
