"""FP64 Gram products of narrow blocks (the packed kernel of blockops.cu: at
most 512 entries) against extended precision."""
import numpy as np
import pytest

from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = S.Context(0)
    yield c
    c.close()


def _gram(ctx, mx, my):
    h, w = mx.shape[1], my.shape[1]
    interp = S._Interp(ctx.lib)
    xx = ctx.lib.mv_MultiVectorWrap(interp.ptr, mx.handle, 0)
    yy = ctx.lib.mv_MultiVectorWrap(interp.ptr, my.handle, 0)
    G = np.empty((h, w), order="F")
    ctx.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    assert ctx.last_error() == ""
    return G


# one chunk of 32 rows and its neighbours, one entry, whole and partly empty
# warps, one to sixteen thread groups, several CTAs a split and one
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (31, 3, 5), (32, 16, 16), (33, 1, 64), (65, 30, 17), (8000, 10, 10),
                                   (100003, 8, 8), (4097, 32, 8), (60001, 22, 22), (300007, 31, 2)])
def test_narrow_gram(ctx, n, h, w):
    rng = np.random.default_rng(n + h)
    X, Y = rng.standard_normal((n, h)), rng.standard_normal((n, w))
    mx, my = S.MultiVector.from_host(ctx, X), S.MultiVector.from_host(ctx, Y)
    L = np.longdouble
    # FP64 roundings: 32 in a chunk, the chunks of a split, at most 304 splits
    for a, b, ma, mb in ((X, Y, mx, my), (X, X, mx, mx)):
        G = _gram(ctx, ma, mb)
        ref = a.astype(L).T @ b.astype(L)
        assert np.all(np.abs(G - ref) <= 2.0 ** -53 * (32 + n / 32 / 304 + 310) * (np.abs(a).T @ np.abs(b)))
    assert np.array_equal(G, G.T)
