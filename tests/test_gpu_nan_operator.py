"""An operator whose products are NaN (a bad coefficient, or a product that a
timed-out wait poisoned) must not send the Rayleigh-Ritz kernels out of range:
NaN eigenvalues all rank first, so a permutation built from ranks alone has
entries that nothing wrote.  The solve may end as it likes, but without a CUDA
error, and the context stays usable.
"""
import numpy as np
import pytest

from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [0, 1, 2])
@pytest.mark.parametrize("k", [3, 16, 40])
def test_nan_products_leave_the_context_usable(method, k):
    n = 4000
    d = np.arange(1.0, n + 1.0)
    bad = d.copy()
    bad[n // 2] = np.nan
    ctx = S.Context(0)
    try:
        ctx.set_options(rr_method=method)
        X = S.MultiVector(ctx, n, k)
        X.set_random(1)
        S.lobpcg_solve_double(X, S.Diagonal(ctx, bad), atol=1e-6, rtol=1e-50, maxit=3)
        assert "CUDA error" not in ctx.last_error()
        ctx.set_options(rr_method=0)
        Y = S.MultiVector(ctx, n, k)
        Y.set_random(1)
        r = S.lobpcg_solve_double(Y, S.Diagonal(ctx, d), T=S.Diagonal(ctx, 1.0 / d), atol=1e-6, rtol=1e-50,
                                  maxit=200)
        assert r.flag == 0, ctx.last_error()
        # |lambda - nearest eigenvalue| <= residual; distinct integers otherwise
        np.testing.assert_allclose(np.sort(r.lam), np.arange(1.0, k + 1.0), atol=1e-5)
    finally:
        ctx.close()
