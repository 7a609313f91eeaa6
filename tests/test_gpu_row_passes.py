"""The FP32 transforms of every row and pencil length against numpy, and the
mixed right-hand side against the FP64 form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


def norm(a):
    return np.sqrt((np.abs(a) ** 2).sum())


# every row length 8..512 and every x, y length with a factor 3 or 9
GRIDS = [(8, 8, 8), (12, 12, 12), (18, 16, 16), (24, 24, 24), (36, 32, 32), (48, 48, 48),
         (72, 64, 64), (96, 96, 96), (144, 128, 128), (192, 192, 192), (288, 24, 24),
         (384, 384, 24), (384, 384, 384), (512, 512, 512)]


@pytest.mark.parametrize("n", GRIDS[:-2])
def test_transforms(gpu_mod, n):
    """Within 1e-6 in the 2-norm: FP32 transforms of up to 2^24 points err by
    about eps sqrt(log2 N) = 6e-8 * 4.9 = 3e-7."""
    ctx = gpu_mod.Context(n=n, precision=gpu_mod.PREC_MIXED)
    x = np.random.default_rng(sum(n)).standard_normal(n)
    X = np.fft.rfftn(x)
    assert norm(ctx.fft(x) - X) <= 1e-6 * norm(X)
    assert norm(ctx.ifft(X) - x * x.size) <= 1e-6 * norm(x * x.size)
    ctx.close()


@pytest.mark.parametrize("n", GRIDS[-2:])
def test_longest_rows(gpu_mod, n):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs about 40 GB of device memory")
    ctx = gpu_mod.Context(n=n, precision=gpu_mod.PREC_MIXED)
    i, j, k = np.ogrid[:n[0], :n[1], :n[2]]
    x = np.cos(2 * np.pi * ((3 * i) % n[0] / n[0] + (5 * j) % n[1] / n[1] + (7 * k) % n[2] / n[2]))
    X = ctx.fft(x)
    assert abs(X[3, 5, 7] - x.size / 2) <= 1e-6 * x.size
    X[3, 5, 7] = 0.0
    assert norm(X) <= 1e-6 * x.size
    ctx.close()


@pytest.mark.parametrize("n", [(8, 8, 8), (24, 18, 12), (32, 32, 32), (48, 36, 24), (64, 64, 64),
                               (96, 64, 48), (144, 72, 48), (128, 128, 128), (192, 96, 96),
                               (54, 48, 24), (48, 48, 36), (384, 12, 12)])
@pytest.mark.parametrize("flag", [0, 1])
def test_rhs_against_fp64(gpu_mod, n, flag):
    """One right-hand side of the mixed form with either z engine against the
    FP64 form: the fluctuation part of each real segment within 1e-5 of its
    magnitude, the tensor segments within 1e-4, the bounds of the other engines."""
    ref = gpu_mod.Context(n=n)
    ref.ic(seed=5, amp=1e-3)
    f = ref.get_state()
    f[4 * ref.N:-1] = 1e-4 * np.sqrt(ref.N) * np.random.default_rng(1).standard_normal(8 * ref.M)
    r, _ = ref.mk_rhs(f, filter=flag, output=flag)
    ctx = gpu_mod.Context(n=n, precision=gpu_mod.PREC_MIXED)
    N, X = ctx.N, 2 * ctx.M
    for engine in (1, 0):
        ctx.set_engine(6, engine)
        got, _ = ctx.mk_rhs(f, filter=flag, output=flag)
        for s in range(4):
            a, b = r[s * N:(s + 1) * N], got[s * N:(s + 1) * N]
            w = a - a.mean()
            assert np.abs(b - b.mean() - w).max() <= 1e-5 * np.abs(w).max() + 1e-12, (engine, s)
        for s in range(4):
            a = r[4 * N + s * X:4 * N + (s + 1) * X]
            b = got[4 * N + s * X:4 * N + (s + 1) * X]
            assert np.abs(b - a).max() <= 1e-4 * np.abs(a).max(), (engine, s)
        assert abs(got[-1] / r[-1] - 1) <= 5e-9
    ref.close()
    ctx.close()
