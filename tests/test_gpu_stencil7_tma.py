"""The FP32 7-point stencil's TMA kernels at the edges of their dispatch: one and
two planes a CTA (odd numbers of planes included), tiles that stick out of the
grid, a last strip with fewer tile rows, columns dealt to several CTAs, and an
output that cannot be written four values at a time; and the inner product that
the inner CG takes in the same pass."""
import numpy as np
import pytest
import scipy.sparse as sp

from blopex_gb300 import problems as P
from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _problem(nx, ny, nz):
    cx, cy, cz = P.stencil7_coefficients(nx, ny, nz, seed=nx + nz)
    rp, ci, va = P.stencil7_to_csr(cx, cy, cz)
    n = nx * ny * nz
    return (cx, cy, cz), sp.csr_matrix((va, ci, rp), shape=(n, n)), n


# two planes a CTA from 6 CTAs an SM on (912 of 152): the tall and the last two grids
GRIDS = [(4, 1, 1), (8, 5, 3), (32, 32, 9), (100, 33, 17), (4, 4, 1851), (36, 40, 601), (68, 600, 49)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("w", [1, 3, 9, 70])
@pytest.mark.parametrize("shift", [0, 1])  # floats the output starts off a 16-byte boundary
def test_apply(grid, w, shift):
    torch = pytest.importorskip("torch")
    coef, A, n = _problem(*grid)
    if n * w > 2e7:
        w = 2
    rng = np.random.default_rng(n + w)
    x = rng.standard_normal((n, w)).astype(np.float32).astype(np.float64)
    ctx = S.Context(0)
    try:
        op = S.Stencil7(ctx, *coef)
        X = S.MultiVector.from_host(ctx, x, S.FLOAT32)
        pad = 4 * n + 4
        buf = torch.full((w * pad + 8,), 7.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        Y = S.MultiVector.wrap_device(ctx, buf.data_ptr() + 4 * shift, n, pad, w, S.FLOAT32)
        op.apply(X, Y)
        y = Y.to_host()
        torch.cuda.synchronize()
        out = buf.cpu().numpy()
    finally:
        ctx.close()
    # coefficients rounded (1), the diagonal's six sums (6), seven products and sums (8)
    bound = 16 * EPS * (abs(A) @ np.abs(x)) + 1e-30
    assert np.all(np.abs(y - A @ x) <= bound)
    used = np.zeros(out.shape, bool)
    for c in range(w):
        used[shift + c * pad:shift + c * pad + n] = True
    assert np.all(out[~used] == 7.0)  # nothing written beside the columns


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("w", [1, 12])
def test_inner_product(grid, w):
    coef, A, n = _problem(*grid)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, w)).astype(np.float32).astype(np.float64)
    ctx = S.Context(0)
    try:
        T = S.PCGPreconditioner(ctx, S.Stencil7(ctx, *coef), None, 1)
        X, Y = S.MultiVector.from_host(ctx, x, S.FLOAT32), S.MultiVector(ctx, n, w, S.FLOAT32)
        T.apply(X, Y)  # one step: y = (x'x / x'Ax) x
        y = Y.to_host()
    finally:
        ctx.close()
    q = A @ x
    xq = (x * q).sum(0)
    alpha = (x * x).sum(0) / xq
    # x'(computed A x) off by 16 eps |x|'|A||x|; alpha and the product rounded to FP32
    rel = 16 * EPS * (np.abs(x) * (abs(A) @ np.abs(x))).sum(0) / xq + 3 * EPS
    assert np.all(np.abs(y - alpha * x) <= rel * np.abs(alpha * x) + 1e-30)
