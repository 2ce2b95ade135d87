"""The inner CG on its fused kernels at the edges of their grids: one element,
fewer rows than a block, a tail of n % 4 rows, one CTA a column and many, one
column and many, one step (no residual update), a zero column (its coefficients
are 0), and a block that FP32 cannot read four at a time."""
import numpy as np
import pytest

from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu


def _cg(a, m, x, steps):
    """CG on diag(a) y = x, all columns, in FP64."""
    with np.errstate(invalid="ignore", divide="ignore"):
        div = lambda u, v: np.where((u != 0) & (v != 0), u / v, 0.0)
        r, y = x.copy(), np.zeros_like(x)
        p = m[:, None] * r
        rho = (r * p).sum(0)
        for _ in range(steps):
            q = a[:, None] * p
            al = div(rho, (p * q).sum(0))
            y += al * p
            r -= al * q
            z = m[:, None] * r
            rho, old = (r * z).sum(0), rho
            p = z + div(rho, old) * p
    return y


@pytest.mark.parametrize("dtype", [S.FLOAT32, S.FLOAT64])
@pytest.mark.parametrize("n,w,steps,jacobi", [(1, 1, 1, True), (2, 3, 1, False), (255, 2, 3, True),
                                              (257, 17, 2, False), (1030, 256, 3, True), (40961, 1, 3, True),
                                              (300007, 9, 2, True), (2097152 + 5, 2, 3, False)])
def test_fused_cg(dtype, n, w, steps, jacobi):
    rng = np.random.default_rng(n)
    a = 1.0 + 3.0 * rng.random(n)  # condition number at most 4
    m = 1.0 / (a * (0.9 + 0.2 * rng.random(n))) if jacobi else np.ones(n)
    x = rng.standard_normal((n, w))
    if w > 1:
        x[:, w // 2] = 0.0
    if dtype == S.FLOAT32:
        a, m, x = (v.astype(np.float32).astype(np.float64) for v in (a, m, x))
    ctx = S.Context(0)
    try:
        T = S.PCGPreconditioner(ctx, S.Diagonal(ctx, a), S.Diagonal(ctx, m) if jacobi else None, steps)
        X, Y = S.MultiVector.from_host(ctx, x, dtype), S.MultiVector(ctx, n, w, dtype)
        T.apply(X, Y)
        y = Y.to_host()
        T.apply(X, Y)  # the counters of the first application were left at zero
        assert np.array_equal(y, Y.to_host())
        ref = _cg(a, m, x, steps)
        # a step rounds its updates of y, r and p (a few eps each, carried on by factors
        # of at most the condition number); once a column has converged both sides hold
        # rounding noise, still relative to y
        eps = 2.0 ** -24 if dtype == S.FLOAT32 else 2.0 ** -53
        bound = 16 * 4 * (steps + 1) * eps * np.linalg.norm(ref, axis=0)
        assert np.all(np.linalg.norm(y - ref, axis=0) <= bound)
    finally:
        ctx.close()
