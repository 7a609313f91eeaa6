"""The z part of the mixed form's RHS in one kernel (rows of 3 2^a and 9 2^a
values) against the FP64 form: every row length, blocks partly filled, with and
without the tensor sources and the output flag."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


GRIDS = [(24, 24, 24), (54, 54, 24), (48, 48, 48), (162, 54, 48), (72, 72, 72), (96, 96, 96),
         (144, 144, 144), (192, 192, 192)]


@pytest.mark.parametrize("n,gw,flag", [(n, *o) for n in GRIDS for o in ((1, 0), (1, 1), (0, 0))] +
                         [((288, 288, 288), 1, 0), ((384, 384, 384), 1, 0)])
def test_against_fp64(gpu_mod, n, gw, flag):
    """The fluctuation part of each real segment within 1e-5 of its magnitude,
    the tensor segments within 1e-4, the bounds of the other engines."""
    torch = pytest.importorskip("torch")
    if n[0] > 200 and torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs about 50 GB of device memory")
    ref = gpu_mod.Context(n=n, gw=bool(gw))
    ref.ic(seed=5, amp=1e-3)
    f = ref.get_state()
    N, X = ref.N, 2 * ref.M
    r, _ = ref.mk_rhs(f, output=flag)
    ref.close()
    ctx = gpu_mod.Context(n=n, precision=gpu_mod.PREC_MIXED, gw=bool(gw))
    got, _ = ctx.mk_rhs(f, output=flag)
    ctx.close()
    for s in range(4):
        a, b = r[s * N:(s + 1) * N], got[s * N:(s + 1) * N]
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(a - a.mean())
    for s in range(4):
        a, b = (v[4 * N + s * X:4 * N + (s + 1) * X] for v in (r, got))
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(a)
