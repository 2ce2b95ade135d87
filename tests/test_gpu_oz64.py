"""FP64 block updates and Gram products on the tensor cores (oz_xc.cu,
oz_gram64.cu), as the interpreter's mv_MultiVectorByMatrix / Xapy /
ByMultiVector route large FP64 blocks to them, against extended precision.

Bounds.  A value is cut to 55 fraction bits below its group's scale s (a row of
X or a column of C; a column over a group of at most 256 rows), s at most twice
the group's largest magnitude: each factor is off by at most 2^-54 of that
maximum, a product of two by 2^-53 of the maxima's product; the digit products
left out (5 of level 8 and below) by 2^-59; a group's recombined sum is rounded
at 2^-54 s s' <= 2^-52 of it, and once more to FP64.  FP64 additions follow (Z;
over the groups and CTAs of a Gram)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from blopex_gb300 import solver as S  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = S.Context(0)
    yield c
    assert c.device_error() == 0
    c.close()


def _device(ctx, a, shift=0):
    """a (n x k) on the device, its columns `shift` elements off the alignment
    of the allocation and with an odd leading dimension when shifted."""
    n, k = a.shape
    ld = n + 5 if shift else n
    t = torch.zeros(k * ld + 8, dtype=torch.float64, device="cuda")
    v = t[shift:shift + k * ld].view(k, ld)
    v[:, :n] = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    torch.cuda.synchronize()
    mv = S.MultiVector.wrap_device(ctx, v.data_ptr(), n, ld, k)
    mv.keep = (t, v)
    return mv


def _update(ctx, X, C, Y0=None, shift=0):
    """X C, or Y0 + X C in place."""
    h, w = C.shape
    mx = _device(ctx, X, shift)
    my = _device(ctx, Y0 if Y0 is not None else np.full((X.shape[0], w), 7.0), shift)
    Cf = np.asfortranarray(C)
    interp = S._Interp(ctx.lib)
    xx = ctx.lib.mv_MultiVectorWrap(interp.ptr, mx.handle, 0)
    yy = ctx.lib.mv_MultiVectorWrap(interp.ptr, my.handle, 0)
    f = ctx.lib.mv_MultiVectorXapy if Y0 is not None else ctx.lib.mv_MultiVectorByMatrix
    f(xx, h, h, w, Cf.ctypes.data, yy)
    assert ctx.last_error() == ""
    return my.to_host()


def _gram(ctx, mx, my):
    h, w = mx.shape[1], my.shape[1]
    interp = S._Interp(ctx.lib)
    xx = ctx.lib.mv_MultiVectorWrap(interp.ptr, mx.handle, 0)
    yy = ctx.lib.mv_MultiVectorWrap(interp.ptr, my.handle, 0)
    G = np.empty((h, w), order="F")
    ctx.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    assert ctx.last_error() == ""
    return G


def _check_update(X, C, Y0, Y):
    L = np.longdouble
    ref = X.astype(L) @ C.astype(L)
    b = (X.shape[1] * (2.0 ** -53 + 2.0 ** -58) + 2.0 ** -52 * -(-X.shape[1] // 64)) * np.outer(
        np.abs(X).max(1), np.abs(C).max(0))
    if Y0 is not None:
        ref = ref + Y0
        b = b + 2.0 ** -52 * np.abs(Y0)
    # one rounding per block of 64 input columns, of a partial sum
    b = b + 2.0 ** -52 * (np.abs(ref) + (np.abs(X) @ np.abs(C) if X.shape[1] > 64 else 0.0))
    assert np.all(np.abs(Y - ref) <= b), float((np.abs(Y - ref) / b).max())


# one and several tiles of 128 rows with ragged ends, one and two units of 32
# columns, K steps of 16 partly empty, more than 64 columns on either side
@pytest.mark.parametrize("n,h,w,add,shift", [
    (200001, 10, 10, False, 0), (79001, 64, 4, True, 1), (5209, 64, 64, False, 0), (20483, 31, 33, True, 0),
    (41000, 17, 32, False, 1), (4999, 65, 63, True, 0), (2503, 130, 67, True, 1), (1250129, 16, 1, False, 0),
    (650000, 1, 33, False, 0)])
def test_update_on_tensor_cores(ctx, n, h, w, add, shift):
    rng = np.random.default_rng(n + h + w)
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
    Y0 = rng.standard_normal((n, w)) if add else None
    _check_update(X, C, Y0, _update(ctx, X, C, Y0, shift))


def test_update_scales_zeros_and_subnormals(ctx):
    """Rows over 600 decades, zero rows and columns, subnormal rows and
    columns, a cancelling pair of columns."""
    rng = np.random.default_rng(3)
    n, h, w = 40000, 32, 20
    X = rng.standard_normal((n, h)) * 10.0 ** rng.uniform(-290, 140, size=(n, 1))
    X[::97] = 0.0
    X[5::89] = rng.standard_normal((X[5::89].shape[0], h)) * 1e-310
    X[:, 1] = X[:, 0]
    C = rng.standard_normal((h, w)) * 10.0 ** rng.uniform(-5, 5, size=(1, w))
    C[:, 4] = 0.0
    C[:, 9] *= 1e-312
    C[2:, 11] = 0.0
    C[1, 11] = -C[0, 11]
    Y = _update(ctx, X, C)
    L = np.longdouble
    ref = X.astype(L) @ C.astype(L)
    b = (h + 2) * 2.0 ** -52 * np.outer(np.abs(X).max(1), np.abs(C).max(0)).astype(L) + (h + 1) * L(2) ** -1074
    assert np.all(np.abs(Y - ref) <= b + 2.0 ** -52 * np.abs(ref))
    assert np.all(Y[~X.any(1)] == 0) and np.all(Y[:, 4] == 0)  # (some rows of the first stride hold subnormals)


def test_update_nonfinite(ctx):
    """Infinities and NaN reach the rows and columns they reach in FP64, and
    no others."""
    rng = np.random.default_rng(4)
    n, h, w = 30000, 30, 25
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
    X[100, 3], X[128, 0], X[29999, 29], X[777, 7] = np.inf, np.nan, -np.inf, 1e308
    C[4, 5], C[6, 8] = np.inf, np.nan
    Y = _update(ctx, X, C)
    with np.errstate(invalid="ignore", over="ignore"):
        ref = X @ C
    assert np.array_equal(np.isnan(Y), np.isnan(ref))
    assert np.array_equal(np.isinf(Y), np.isinf(ref)) and np.array_equal(Y[np.isinf(Y)], ref[np.isinf(ref)])
    rows, cols = np.setdiff1d(np.arange(n), [100, 128, 29999]), np.setdiff1d(np.arange(w), [5, 8])
    _check_update(X[rows], C[:, cols], None, Y[np.ix_(rows, cols)])


def _check_gram(X, Y, G):
    L = np.longdouble
    ref = np.zeros((X.shape[1], Y.shape[1]), dtype=L)
    b = np.zeros(ref.shape)
    # (the groups of the kernel are of 128 or 256 rows: bounds over 256)
    for r in range(0, X.shape[0], 256):
        x, y = X[r:r + 256], Y[r:r + 256]
        ref += x.astype(L).T @ y.astype(L)
        b += (len(x) * (2.0 ** -53 + 2.0 ** -58) + 2 * 2.0 ** -52) * np.outer(np.abs(x).max(0), np.abs(y).max(0))
    # FP64 additions: over a CTA's groups (up to 8 sums by weight), then the CTAs
    b += 2.0 ** -53 * (X.shape[0] / 128 / 152 + 8 + 64) * (np.abs(X).T @ np.abs(Y))
    assert np.all(np.abs(G - ref) <= b), float((np.abs(G - ref) / b).max())


# 2, 4 and 8 stacked slices (w > 32, > 16, <= 16), tiles of 64, units of 8
# columns partly empty, a short last group
@pytest.mark.parametrize("n,h,w,shift", [
    (400003, 17, 15, 0), (25000, 64, 64, 0), (76001, 40, 33, 1), (98500, 33, 31, 0), (15001, 100, 70, 1),
    (280001, 8, 45, 0), (1000003, 4, 26, 0), (30011, 65, 129, 0), (500000, 64, 4, 1)])
def test_gram_on_tensor_cores(ctx, n, h, w, shift):
    rng = np.random.default_rng(n + h + w)
    X, Y = rng.standard_normal((n, h)) * np.exp(rng.standard_normal((1, h))), rng.standard_normal((n, w))
    mx, my = _device(ctx, X, shift), _device(ctx, Y, shift)
    _check_gram(X, Y, _gram(ctx, mx, my))


@pytest.mark.parametrize("n,h", [(1000003, 11), (250000, 30), (40000, 64), (12001, 97)])
def test_gram_of_one_block_is_symmetric(ctx, n, h):
    rng = np.random.default_rng(n + h)
    X = rng.standard_normal((n, h))
    mx = _device(ctx, X)
    G = _gram(ctx, mx, mx)
    assert np.array_equal(G, G.T)
    _check_gram(X, X, G)


def test_gram_scales_and_nonfinite(ctx):
    """Columns over 200 decades, zero and subnormal columns, a zero stretch;
    then an infinity and a NaN, which reach their columns' entries only."""
    rng = np.random.default_rng(8)
    n, h, w = 120001, 30, 40
    X = rng.standard_normal((n, h)) * 10.0 ** rng.uniform(-120, 80, size=(1, h))
    Y = rng.standard_normal((n, w)) * 10.0 ** rng.uniform(-80, 60, size=(1, w))
    X[:, 3] = 0.0
    X[:, 4] = rng.standard_normal(n) * 1e-311
    X[1000:9000] = 0.0
    Y[:, 6] = 0.0
    mx, my = _device(ctx, X), _device(ctx, Y)
    G = _gram(ctx, mx, my)
    assert np.all(G[3] == 0) and np.all(G[:, 6] == 0)
    s = np.outer(np.linalg.norm(X, axis=0), np.linalg.norm(Y, axis=0))  # (of columns that keep off underflow)
    keep = np.arange(h) != 4
    ref = X.T.astype(np.longdouble) @ Y.astype(np.longdouble)
    assert np.all(np.abs(G - ref)[keep] <= 1e-14 * s[keep])
    assert np.all(np.abs(G[4] - ref[4]) <= 1e-14 * (np.abs(X[:, 4]).astype(np.longdouble) @ np.abs(Y))
                  + n * 2.0 ** -1074)
    X[7, 5], Y[n - 1, 2], Y[5000, 9] = np.inf, np.nan, np.inf
    Y[7, :] = np.abs(Y[7, :])
    G = _gram(ctx, _device(ctx, X), _device(ctx, Y))
    with np.errstate(invalid="ignore"):
        r = X.T @ Y
    assert np.array_equal(np.isnan(G), np.isnan(r)) and np.array_equal(np.isinf(G), np.isinf(r))
