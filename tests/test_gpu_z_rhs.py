"""The two kernels of the fused FP64 z pass (ih_fixz.cu): eight warps per group
of rows up to 8 groups an SM, one warp above; every row length on both, groups
and blocks that are partly filled, with and without the tensor sources."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# few groups of rows
FEW = [(8, 8, 8), (36, 18, 8), (18, 18, 12), (18, 18, 16), (54, 24, 24), (36, 36, 32), (48, 48, 48),
       (72, 64, 64), (96, 96, 96)]
# many; the last two rows of blocks of (486, 54, 8) and (162, 162, 12) are short
MANY = [(486, 54, 8), (256, 256, 12), (162, 162, 16), (256, 128, 24), (162, 108, 32), (192, 144, 48),
        (162, 96, 64), (144, 128, 96), (128, 128, 128), (192, 192, 192), (256, 256, 256),
        (384, 384, 384)]


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


@pytest.mark.parametrize("n", FEW + MANY)
@pytest.mark.parametrize("gw", [1, 0])
def test_against_the_fp64_engines(gpu_mod, n, gw):
    """Each segment's fluctuations to 1e-11, the bound of both against the
    oracle; derivatives from round trips and from the full spectrum."""
    torch = pytest.importorskip("torch")
    if n[0] * n[1] * n[2] > 2 ** 25 and torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs about 40 GB of device memory")
    ctx = gpu_mod.Context(n=n, L=(20.0, 17.0, 13.0), gw=bool(gw))
    rng = np.random.default_rng(sum(n))
    f = np.zeros(ctx.Ntot)
    f[:4 * ctx.N] = 1e-3 * rng.standard_normal(4 * ctx.N)
    f[:ctx.N] += 0.2
    f[ctx.N:2 * ctx.N] -= 0.8
    f[-1] = 1.3
    passes = ctx.L_.ih_fft_get_engine(ctx.h, 9)
    assert passes & 64, "the z passes"
    ctx.set_engine(9, passes & ~64)
    ref, _ = ctx.mk_rhs(f)
    N, X = ctx.N, 2 * ctx.M
    edges = [0, N, 2 * N, 3 * N, 4 * N] + [4 * N + i * X for i in range(1, 5)]
    for mask in (passes, passes & ~24):
        ctx.set_engine(9, mask)
        r, _ = ctx.mk_rhs(f)
        for a, b in zip(edges[:-1], edges[1:]):
            w = ref[a:b] - ref[a:b].mean()
            assert np.linalg.norm(r[a:b] - ref[a:b]) <= 1e-11 * np.linalg.norm(w)
        assert abs(r[-1] / ref[-1] - 1) <= 1e-14
    ctx.close()
