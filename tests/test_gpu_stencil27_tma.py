"""The FP32 27-point stencil's TMA kernel against the general kernel, which takes
over when the input's columns are off a 16-byte boundary: the same terms in the same
order, so the same bits.  Tiles that stick out, an odd number of planes, one to
several steps of four columns, columns dealt to several CTAs, and a wait that runs
out."""
import numpy as np
import pytest

from blopex_gb300 import problems as P
from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _block(ctx, n, w, shift, fill=None):
    ld = (n + 7) // 4 * 4
    buf = torch.full((w * ld + 4,), float("nan"), dtype=torch.float32, device="cuda")
    if fill is not None:
        for c in range(w):
            buf[shift + c * ld:shift + c * ld + n] = fill[c]
    torch.cuda.synchronize()
    return buf, S.MultiVector.wrap_device(ctx, buf.data_ptr() + 4 * shift, n, ld, w, S.FLOAT32)


def _apply(ctx, op, n, w, x, shift):
    xb, X = _block(ctx, n, w, shift, x)
    yb, Y = _block(ctx, n, w, 0)
    op.apply(X, Y)
    return Y.to_host()


@pytest.mark.parametrize("grid", [(4, 1, 1), (8, 5, 3), (32, 4, 2), (36, 33, 7), (100, 21, 12), (64, 64, 40)])
@pytest.mark.parametrize("w", [1, 4, 6, 9, 70])
def test_same_bits_as_the_general_kernel(grid, w):
    nx, ny, nz = grid
    n = nx * ny * nz
    x = torch.randn(w, n, generator=torch.Generator().manual_seed(n + w)).cuda()
    ctx = S.Context(0)
    try:
        op = S.Stencil27(ctx, nx, ny, nz, P.stencil27_weights(nx, ny, nz, seed=3), 0.25)
        a, b = _apply(ctx, op, n, w, x, 0), _apply(ctx, op, n, w, x, 1)
        assert np.isfinite(a).all() and np.array_equal(a, b)
    finally:
        ctx.close()


def test_gives_up_cleanly():
    nx, ny, nz, w = 96, 96, 96, 16
    n = nx * ny * nz
    x = torch.randn(w, n, generator=torch.Generator().manual_seed(1)).cuda()
    ctx = S.Context(0)
    try:
        op = S.Stencil27(ctx, nx, ny, nz, P.stencil27_weights(nx, ny, nz, seed=3), 0.25)
        ref = _apply(ctx, op, n, w, x, 1)
        ctx.set_options(wait_polls=1)
        y = _apply(ctx, op, n, w, x, 0)
        assert ctx.device_error() != 0
        written = ~np.isnan(y)
        assert not written.all() and np.array_equal(y[written], ref[written])
        ctx.set_options(wait_polls=0)
        assert np.array_equal(_apply(ctx, op, n, w, x, 0), ref) and ctx.device_error() == 0
    finally:
        ctx.set_options(wait_polls=0)
        ctx.close()
