"""The diagnostics' spectra bin by bin and the six summaries against the oracle:
octant table of shells, sums over runs of equal shells within a warp, modes
that fill the last warp of a block partly, boxes with unequal sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_mod():
    from instaheat_gb300 import gpu
    return gpu


@pytest.mark.parametrize("n,L", [((8, 8, 8), (20.0, 20.0, 20.0)), ((18, 12, 8), (14.0, 9.0, 20.0)),
                                 ((54, 36, 24), (20.0, 20.0, 20.0)),
                                 ((128, 16, 8), (40.0, 20.0, 5.0)),
                                 ((64, 48, 32), (11.0, 20.0, 17.0))])
@pytest.mark.parametrize("prec", [0, 1])
def test_every_bin(gpu_mod, oracle_mod, n, L, prec):
    """White spectra, so that every shell has content: each bin within 1e-10 of
    itself or of 1e-3 of the largest (FP64), the summaries within 1e-9.  Mixed
    form: what is transformed in FP32 within 1e-5."""
    ctx = gpu_mod.Context(n=n, L=L, precision=prec)
    o = oracle_mod.Oracle(n=n, L=L)
    rng = np.random.default_rng(sum(n))
    f = o.ic(seed=2, amp=1e-3)
    f[:4 * o.N] += 1e-4 * rng.standard_normal(4 * o.N)
    f[4 * o.N:-1] = 1e-6 * rng.standard_normal(4 * o.Next)
    d = oracle_mod.DiagOutput(o.bins)
    o.rhs(f, filter=0, output=1, diag=d)
    # without the filter the oracle leaves the psi spectrum out: it is that of
    # phi in a state whose phi is this psi
    swapped, ds = f.copy(), oracle_mod.DiagOutput(o.bins)
    swapped[:o.N] = f[2 * o.N:3 * o.N]
    o.rhs(swapped, filter=0, output=1, diag=ds)
    d.psi_ps[:] = ds.phi_ps
    ctx.mk_rhs(f, filter=0, output=1)
    g = ctx.output()
    tol = 1e-5 if prec else 1e-10
    for k in ("phi_ps", "psi_ps", "rho_ps", "gw"):
        ref = getattr(d, k)
        assert np.all(np.abs(g[k] - ref) <= tol * np.maximum(np.abs(ref), 1e-3 * np.abs(ref).max())), k
    np.testing.assert_allclose(g["smry"], d.smry, rtol=1e-5 if prec else 1e-9, atol=1e-9 if prec else 1e-14)
    ctx.close()
    o.close()
