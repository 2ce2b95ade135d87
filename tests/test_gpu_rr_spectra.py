"""Rayleigh-Ritz on spectra that the tridiagonal path's shortcuts could get wrong:
equal eigenvalues, clusters, gaps over many orders, both signs, an operator that
decouples, orders of one to several hundred.  However far the solve has got, its X is
orthonormal, X'AX = diag(lambda) and lambda ascends (not for equal eigenvalues, whose
residuals are rounding noise that the solve then orthonormalises against)."""
import numpy as np
import pytest

from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu

N = 3000


def _spectrum(kind):
    i = np.arange(N, dtype=np.float64)
    return {"linear": 1.0 + i, "equal": np.full(N, 2.0), "pairs": 1.0 + np.floor(i / 2),
            "clusters": 1.0 + np.floor(i / 7) + 1e-9 * (i % 7), "graded": 10.0 ** (-6.0 + 8.0 * i / N),
            "signs": (i - N / 2) / 10.0, "big": 1e100 * (1.0 + i), "small": 1e-100 * (1.0 + i)}[kind]


@pytest.mark.parametrize("kind", ["linear", "equal", "pairs", "clusters", "graded", "signs", "big", "small"])
@pytest.mark.parametrize("k", [1, 2, 11, 40, 113])
@pytest.mark.parametrize("method", [0, 2])
def test_ritz_pairs(kind, k, method):
    d = _spectrum(kind)
    ctx = S.Context(0)
    try:
        ctx.set_options(rr_method=method)
        X = S.MultiVector(ctx, N, k)
        X.set_random(5)
        r = S.lobpcg_solve_double(X, S.Diagonal(ctx, d), atol=0.0, rtol=0.0, maxit=4)
        assert "CUDA error" not in ctx.last_error()
        if kind == "equal":
            return
        x, lam = X.to_host(), np.asarray(r.lam)
    finally:
        ctx.close()
    scale = np.abs(d).max()
    # n eps a product summed, times the number of products an iteration chains (about ten)
    tol = 10 * N * 2.0 ** -53
    assert np.abs(x.T @ x - np.eye(k)).max() <= tol * 10
    assert np.abs(x.T @ (d[:, None] * x) - np.diag(lam)).max() <= tol * 10 * scale
    assert np.all(np.diff(lam) >= -tol * scale)
