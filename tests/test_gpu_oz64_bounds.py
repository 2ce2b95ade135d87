"""FP64 block updates and Gram products of large blocks against the bounds that
FP64 multiply-adds keep, entry by entry: (h + 2) 2^-53 sum |x_i c_ij| for an
update, (32 + n / 32 / 304 + 310) 2^-53 sum |x_ri y_rj| for a Gram product (32
roundings in a chunk, the chunks of a split, at most 304 splits).  The blocks
are graded, localised and extreme ones, which a scale shared by a group of
values does not absorb."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from blopex_gb300 import solver as S  # noqa: E402

pytestmark = pytest.mark.gpu

L = np.longdouble
EPS = L(2) ** -53


@pytest.fixture(scope="module")
def ctx():
    c = S.Context(0)
    yield c
    assert c.device_error() == 0
    c.close()


def _wrap(ctx, mv):
    interp = S._Interp(ctx.lib)
    return interp, ctx.lib.mv_MultiVectorWrap(interp.ptr, mv.handle, 0)


def _gram(ctx, X, Y):
    h, w = X.shape[1], Y.shape[1]
    mx = S.MultiVector.from_host(ctx, X)
    my = mx if Y is X else S.MultiVector.from_host(ctx, Y)
    (i, xx), (j, yy) = _wrap(ctx, mx), _wrap(ctx, my)
    G = np.full((h, w), 7.0, order="F")
    ctx.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    assert ctx.last_error() == ""
    return G


def _products(X, Y):
    """X' Y to 16 roundings of sum |x_ri y_rj| (16 rows at a time in FP64, these in
    extended precision)."""
    n = X.shape[0] // 16 * 16
    p = np.matmul(X[:n].reshape(-1, 16, X.shape[1]).transpose(0, 2, 1), Y[:n].reshape(-1, 16, Y.shape[1]))
    return p.astype(L).sum(0) + X[n:].T.astype(L) @ Y[n:]


def _check_gram(X, Y, G):
    n = X.shape[0]
    mag = _products(np.abs(X), np.abs(Y))
    err = np.abs(G - _products(X, Y))
    b = (32 + L(n) / 32 / 304 + 310 + 16) * EPS * mag
    assert np.all(err <= b), (float((err[mag > 0] / b[mag > 0]).max()), np.argwhere(err > b)[:3])


# columns of constants next to a power of two: the largest sums that a group of
# rows can hold (w in 17 .. 32 stacks two slices on a row block of 256 rows)
@pytest.mark.parametrize("n,h,w", [(300001, 16, 24), (200003, 20, 32), (400000, 33, 16), (60001, 40, 50)])
def test_gram_of_constant_columns(ctx, n, h, w):
    consts = [1 - 2.0 ** -53, 0.997, 1 - 1e-12, 0.99609375, 1.998, 0.999]
    X = np.empty((n, h))
    Y = np.empty((n, w))
    for c in range(h):
        X[:, c] = consts[c % 6] * (-1 if c // 6 % 2 else 1)
    for c in range(w):
        Y[:, c] = consts[(c + c // 6) % 6] * (-1 if c // 3 % 2 else 1)
    _check_gram(X, Y, _gram(ctx, X, Y))


def _update(ctx, X, C, Y0=None):
    """X C, or Y0 + X C in place."""
    h, w = C.shape
    mx = S.MultiVector.from_host(ctx, X)
    my = S.MultiVector.from_host(ctx, Y0 if Y0 is not None else np.full((X.shape[0], w), 7.0))
    Cf = np.asfortranarray(C)
    (i, xx), (j, yy) = _wrap(ctx, mx), _wrap(ctx, my)
    f = ctx.lib.mv_MultiVectorXapy if Y0 is not None else ctx.lib.mv_MultiVectorByMatrix
    f(xx, h, h, w, Cf.ctypes.data, yy)
    assert ctx.last_error() == ""
    return my.to_host()


TINY = L(2) ** -1074


# products whose scale is below or near FP64's smallest normal numbers, and above
# its largest, of factors that are themselves well inside the range
def test_update_products_out_of_range(ctx):
    rng = np.random.default_rng(21)
    n, h, w = 40000, 32, 20
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
    X *= 10.0 ** rng.uniform(-200, 150, size=(n, 1))
    C *= 10.0 ** rng.choice([-200, -150, -130, -110, -104, 0, 100, 150, 160, 200], size=(1, w))
    Y = _update(ctx, X, C)
    ref, mag = X.astype(L) @ C.astype(L), np.abs(X).astype(L) @ np.abs(C)
    big = mag > 1.7e308
    assert np.all(np.isinf(Y[np.abs(ref) > 1.8e308]))
    err = np.abs(Y - ref)[~big]
    b = ((h + 2) * EPS * mag + (h + 1) * TINY)[~big]
    assert np.all(err <= b), float((err / b).max())


def test_gram_products_out_of_range(ctx):
    rng = np.random.default_rng(22)
    n, h, w = 120001, 24, 36
    X = rng.standard_normal((n, h)) * 10.0 ** rng.choice([-200, -160, -120, 0, 120, 150], size=(1, h))
    Y = rng.standard_normal((n, w)) * 10.0 ** rng.choice([-200, -148, -105, 0, 100, 151], size=(1, w))
    G = _gram(ctx, X, Y)
    xs, ys = np.abs(X).max(0), np.abs(Y).max(0)
    with np.errstate(under="ignore", over="ignore"):
        norm = np.outer(xs.astype(L), ys.astype(L))
        mag = _products(np.abs(X) / xs, np.abs(Y) / ys) * norm
        ref = _products(X / xs, Y / ys) * norm
    fits = mag < 1.7e308
    err = np.abs(G - ref)[fits]
    # (the divisions by the largest values: two roundings of each product)
    b = ((32 + L(n) / 32 / 304 + 310 + 20) * EPS * mag + n * TINY)[fits]
    assert np.all(err <= b), float((err / b).max())
    assert np.all(np.isinf(G[np.abs(ref) > 1.8e308]))


# single rows and columns that leave the common path among ordinary ones: lanes of a
# warp part ways in every tile and group, and meet again before the next load of
# accumulators
def test_gram_mixed_lanes(ctx):
    rng = np.random.default_rng(24)
    n, h, w = 150001, 26, 30
    X, Y = rng.standard_normal((n, h)), rng.standard_normal((n, w))
    X[:, 2::5] *= 1e-300
    Y[:, 1::4] *= 1e-305
    X[256:512, ::3] = 0.0
    xs, ys = np.abs(X).max(0), np.abs(Y).max(0)
    G = _gram(ctx, X, Y)
    with np.errstate(under="ignore"):
        norm = np.outer(xs.astype(L), ys.astype(L))
        mag, ref = _products(np.abs(X) / xs, np.abs(Y) / ys) * norm, _products(X / xs, Y / ys) * norm
    assert np.all(np.abs(G - ref) <= (32 + L(n) / 32 / 304 + 310 + 20) * EPS * mag + n * TINY)


def test_update_mixed_lanes(ctx):
    rng = np.random.default_rng(23)
    n, h, w = 30001, 40, 41
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
    X[::7] *= 1e-305
    X[3::11] = 0.0
    X[5::13, 1:] = 0.0
    C[:, 3::5] *= 1e-170
    Y0 = rng.standard_normal((n, w)) * 1e-150
    Y = _update(ctx, X, C, Y0)
    ref = X.astype(L) @ C + Y0
    mag = np.abs(X).astype(L) @ np.abs(C)
    assert np.all(np.abs(Y - ref) <= (h + 2) * EPS * mag + EPS * (mag + np.abs(Y0)) + (h + 1) * TINY)


class _Cols(ctypes.Structure):
    """blk_cols of internal.h."""
    _fields_ = [("col", ctypes.c_void_p * 384)]


def _columns(t):
    c = _Cols()
    for i in range(t.shape[0]):
        c.col[i] = t[i].data_ptr()
    return c


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a.T)).cuda()


def _tensor_update(ctx, X, C, Z=None):
    """The tensor-core kernel of the callers' products, whatever the size."""
    n, (h, w) = X.shape[0], C.shape
    x, c, y = _dev(X), _dev(C), torch.full((w, n), 7.0, dtype=torch.float64, device="cuda")
    if Z is not None:
        y.copy_(_dev(Z))
    torch.cuda.synchronize()
    cy = _columns(y)
    rc = ctx.lib.gb_oz_bymat64(ctypes.c_void_p(ctx.handle), ctypes.c_long(n), ctypes.byref(_columns(x)), h,
                               ctypes.c_void_p(c.data_ptr()), h, ctypes.byref(cy), w,
                               ctypes.byref(cy) if Z is not None else None)
    assert rc == 0, ctx.last_error()
    assert ctx.device_error() == 0
    return y.cpu().numpy().T


def _check_update(X, C, Z, Y):
    h = X.shape[1]
    ref, mag = X.astype(L) @ C, np.abs(X).astype(L) @ np.abs(C)
    b = (h + 2) * EPS * mag + (h + 1) * TINY
    if Z is not None:
        ref = ref + Z
        b = b + EPS * (np.abs(ref) + b)
    err = np.abs(Y - ref)
    assert np.all(err <= b), (float((err / b).max()), np.argwhere(err > b)[:3])


def _grade(kind, n, h, rng):
    """Factors for the columns (or entries) of X, of very different size."""
    if kind == "even":
        return np.ones(h)
    if kind == "columns":  # columns that have converged to different degrees
        return 10.0 ** -rng.uniform(0, 20, size=h)
    if kind == "steps":
        return np.array([1.0, 1e-3, 1e-9, 1e-13, 1e-17, 1e-30])[np.arange(h) % 6]
    return 10.0 ** -rng.uniform(0, 25, size=(n, h))  # every entry its own


def _coordinates(kind, h, w, rng):
    C = rng.standard_normal((h, w))
    if kind == "identity":
        return np.eye(h, w)
    if kind == "permutation":
        return np.eye(h)[rng.permutation(h)][:, :w] * 3.0
    if kind == "diagonal":
        return np.eye(h, w) * 10.0 ** rng.uniform(-12, 12, size=(h, 1))
    if kind == "triangular":
        return np.triu(C)
    if kind == "rows":  # graded the other way
        return C * 10.0 ** rng.uniform(0, 20, size=(h, 1))
    return C


# shapes: one column, units of 16 columns partly empty, one to four units, K steps
# partly empty, one to several tiles
@pytest.mark.parametrize("n,h,w", [(700, 1, 1), (300, 5, 16), (4001, 16, 17), (2500, 33, 40), (1999, 64, 64)])
@pytest.mark.parametrize("grade", ["even", "columns", "steps", "entries"])
@pytest.mark.parametrize("coords", ["full", "identity", "permutation", "diagonal", "triangular", "rows"])
def test_update_of_graded_blocks(ctx, n, h, w, grade, coords):
    rng = np.random.default_rng(n + len(grade) + 7 * len(coords))
    X = rng.standard_normal((n, h)) * _grade(grade, n, h, rng)
    C = _coordinates(coords, h, w, rng)
    Z = rng.standard_normal((n, C.shape[1])) * 1e-9 if coords == "full" else None
    _check_update(X, C, Z, _tensor_update(ctx, X, C, Z))


# the interpreter's entry, more than 64 input columns (the parts keep the bound of the whole)
@pytest.mark.parametrize("n,h,w,grade,coords,add", [
    (120001, 12, 12, "columns", "identity", False), (50001, 20, 17, "steps", "full", True),
    (20003, 32, 32, "entries", "triangular", False), (5003, 70, 64, "columns", "full", True),
    (2101, 130, 70, "steps", "rows", False), (2503, 129, 65, "entries", "identity", True)])
def test_update_of_large_graded_blocks(ctx, n, h, w, grade, coords, add):
    rng = np.random.default_rng(n + h)
    X = rng.standard_normal((n, h)) * _grade(grade, n, h, rng)
    C = _coordinates(coords, h, w, rng)
    Y0 = rng.standard_normal((n, w)) * 1e-12 if add else None
    _check_update(X, C, Y0, _update(ctx, X, C, Y0))


def test_update_copies_columns_exactly(ctx):
    """C = I: every output column is an input column, to the last bit."""
    rng = np.random.default_rng(31)
    n, h = 60000, 24
    X = rng.standard_normal((n, h)) * 10.0 ** -rng.uniform(0, 40, size=h)
    assert np.array_equal(_update(ctx, X, np.eye(h)), X)


def test_update_of_random_blocks_is_no_further_off_than_multiply_adds(ctx):
    rng = np.random.default_rng(32)
    for n, h, w in ((20000, 8, 16), (20000, 16, 16), (20000, 32, 32), (10000, 64, 64)):
        X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
        ref = X.astype(L) @ C
        mx, my = S.MultiVector.from_host(ctx, X), S.MultiVector(ctx, n, w)
        Cf = np.asfortranarray(C)
        assert ctx.lib.gpu_BlockUpdate(mx.handle, Cf.ctypes.data, h, my.handle, None, 0) == 0
        err = []
        for Y in (my.to_host(), _tensor_update(ctx, X, C)):
            d = (Y - ref).astype(np.float64)
            err.append((np.abs(d).max(), np.sqrt(np.mean(d * d))))
        assert err[1][0] <= err[0][0] and err[1][1] <= err[0][1], (h, w, err)


def _in_place(ctx, X, C, add):
    """Y = X C (+ Y) with Y on the first columns of X."""
    n, (h, w) = X.shape[0], C.shape
    t = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    torch.cuda.synchronize()
    mx = S.MultiVector.wrap_device(ctx, t.data_ptr(), n, n, h)
    my = S.MultiVector.wrap_device(ctx, t.data_ptr(), n, n, w)
    Cf = np.asfortranarray(C)
    (i, xx), (j, yy) = _wrap(ctx, mx), _wrap(ctx, my)
    f = ctx.lib.mv_MultiVectorXapy if add else ctx.lib.mv_MultiVectorByMatrix
    f(xx, h, h, w, Cf.ctypes.data, yy)
    assert ctx.last_error() == ""
    return t.cpu().numpy()[:w].T


# as always right in place: up to 32 output columns, any number of input columns
@pytest.mark.parametrize("n,h,w,add", [(20001, 32, 32, False), (30001, 33, 32, True), (9001, 96, 32, False),
                                       (5003, 130, 25, True)])
def test_update_in_place(ctx, n, h, w, add):
    rng = np.random.default_rng(n)
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w)) / 8
    X[::9] *= 1e-300
    ref = X.astype(L) @ C + (X[:, :w] if add else 0)
    mag = np.abs(X).astype(L) @ np.abs(C) + (np.abs(X[:, :w]) if add else 0)
    Y = _in_place(ctx, X, C, add)
    assert np.all(np.abs(Y - ref) <= (h + 3) * EPS * mag + (h + 1) * TINY)


def test_split_update_in_place(ctx):
    """gpu_BlockUpdate mode 2 with Y = X, to the bound of its splitting."""
    rng = np.random.default_rng(41)
    n, h = 30000, 64
    X, C = rng.standard_normal((n, h)), np.asfortranarray(rng.standard_normal((h, h)))
    X[::9] *= 1e-300
    mx = S.MultiVector.from_host(ctx, X)
    assert ctx.lib.gpu_BlockUpdate(mx.handle, C.ctypes.data, h, mx.handle, None, 2) == 0, ctx.last_error()
    b = h * 2.0 ** -38 * np.outer(np.abs(X).max(1), np.abs(C).max(0))
    assert np.all(np.abs(mx.to_host() - X @ C) <= b + 2.0 ** -45 * (np.abs(X) @ np.abs(C)))


def _gram_blocks(kind, n, h, w, rng):
    X, Y = rng.standard_normal((n, h)), rng.standard_normal((n, w))
    r = np.arange(n)[:, None]
    if kind == "localised":  # columns that are large in different rows of every group
        X *= 10.0 ** -(3.0 * ((r + np.arange(h)) % 7))
        Y *= 10.0 ** -(3.0 * ((r + 3 + np.arange(w)) % 7))
    elif kind == "disjoint":  # large where the other is zero
        X[::2] *= 1e-18
        Y[1::2] = 0.0
    elif kind == "dominant":  # one entry a column, where the other block vanishes
        X[rng.integers(0, n, h), np.arange(h)] = 1e12
        big = np.abs(X).max(1) >= 1e12
        Y[big] = 0.0
    elif kind == "entries":
        X *= 10.0 ** -rng.uniform(0, 25, size=X.shape)
        Y *= 10.0 ** -rng.uniform(0, 25, size=Y.shape)
    elif kind == "rows":  # an amplitude that falls over the domain, in both
        X *= np.exp(-40.0 * r / n)
        Y *= np.exp(-40.0 * r / n)
    elif kind == "opposite":
        X *= np.exp(-40.0 * r / n)
        Y *= np.exp(-40.0 * (n - r) / n)
    elif kind == "sparse":
        X *= rng.random(X.shape) < 0.02
        Y *= rng.random(Y.shape) < 0.02
    elif kind == "heavy":
        X = np.exp(3 * X)
        Y = np.exp(3 * Y)
    return X, Y


# each variant of the kernel (w <= 16, <= 32, more), more than a tile, X'X
@pytest.mark.parametrize("n,h,w", [(500001, 17, 12), (200003, 20, 30), (60001, 40, 45), (30001, 70, 65), (150001, 27, 0)])
@pytest.mark.parametrize("kind", ["even", "localised", "disjoint", "dominant", "entries", "rows", "opposite", "sparse",
                                  "heavy"])
def test_gram_of_graded_blocks(ctx, n, h, w, kind):
    rng = np.random.default_rng(n + len(kind))
    X, Y = _gram_blocks(kind, n, h, w if w else h, rng)
    if w == 0:
        Y = X
    _check_gram(X, Y, _gram(ctx, X, Y))


def _modes(n_grid, k):
    """Orthonormal eigenvectors of the Laplacian on a square."""
    s = np.sin(np.pi * np.outer(np.arange(1, n_grid + 1), np.arange(1, 9)) / (n_grid + 1))
    return np.stack([np.outer(s[:, a % 8], s[:, (a * 3 + 1) % 8]).ravel() for a in range(k)], axis=1)


# what users' blocks look like passes the check: the tensor cores' three launches and
# no second product
@pytest.mark.parametrize("kind", ["normal", "scaled", "uniform", "laplace", "modes"])
def test_gram_of_ordinary_blocks_needs_no_second_product(ctx, kind):
    rng = np.random.default_rng(51)
    n, h, w = 512 * 512, 20, 24
    X, Y = rng.standard_normal((n, h)), rng.standard_normal((n, w))
    if kind == "scaled":
        X, Y = X * 10.0 ** rng.uniform(-30, 30, size=h), Y * n ** -0.5
    elif kind == "uniform":
        X, Y = rng.random((n, h)), rng.random((n, w)) - 0.5
    elif kind == "laplace":
        X, Y = rng.laplace(size=(n, h)), rng.laplace(size=(n, w))
    elif kind == "modes":
        X, Y = _modes(512, h), _modes(512, w)
    mx, my = S.MultiVector.from_host(ctx, X), S.MultiVector.from_host(ctx, Y)
    (i, xx), (j, yy) = _wrap(ctx, mx), _wrap(ctx, my)
    G = np.empty((h, w), order="F")
    ctx.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    before = ctx.lib.gpu_KernelLaunchCount()
    ctx.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    assert ctx.lib.gpu_KernelLaunchCount() - before == 3
    _check_gram(X, Y, G)


def test_gram_of_random_blocks_is_no_further_off_than_multiply_adds(ctx):
    rng = np.random.default_rng(52)
    for n, h, w in ((400000, 20, 15), (300000, 16, 32), (40000, 64, 64), (25000, 64, 64)):
        X, Y = rng.standard_normal((n, h)), rng.standard_normal((n, w))
        ref = _products(X, Y)
        # (parts below the tensor cores' size, by multiply-adds)
        fma = np.hstack([np.vstack([_gram(ctx, X[:, a:a + 8], Y[:, b:b + 8]) for a in range(0, h, 8)])
                         for b in range(0, w, 8)])
        err = [float(np.sqrt(np.mean((g - ref).astype(np.float64) ** 2))) for g in (fma, _gram(ctx, X, Y))]
        assert err[1] <= err[0], (h, w, err)


# (a poll a wait: the kernels give up on the first copy or product that is not there yet)
def test_update_gives_up_cleanly():
    c = S.Context(0)
    rng = np.random.default_rng(61)
    n, h, w = 300000, 32, 24
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
    ref, mag = X @ C, np.abs(X) @ np.abs(C)
    mx, my = S.MultiVector.from_host(c, X), S.MultiVector(c, n, w)
    Cf = np.asfortranarray(C)
    (i, xx), (j, yy) = _wrap(c, mx), _wrap(c, my)

    def call():
        my.upload(np.full((n, w), 3e33))
        c.lib.mv_MultiVectorByMatrix(xx, h, h, w, Cf.ctypes.data, yy)
        return my.to_host()

    c.set_options(wait_polls=1)
    Y = call()
    c.set_options(wait_polls=0)
    assert "timed out" in c.last_error()
    assert c.device_error() == 0  # read and cleared by the call that failed
    done = ~np.isnan(Y)
    assert not done.all()
    assert np.all(np.abs(Y - ref)[done] <= 80 * 2.0 ** -53 * mag[done])
    assert np.all(np.abs(call() - ref) <= 80 * 2.0 ** -53 * mag)
    assert c.device_error() == 0
    c.close()


def test_gram_gives_up_cleanly():
    c = S.Context(0)
    rng = np.random.default_rng(62)
    n, h, w = 300000, 24, 30
    X, Y = rng.standard_normal((n, h)), rng.standard_normal((n, w))
    mx, my = S.MultiVector.from_host(c, X), S.MultiVector.from_host(c, Y)
    (i, xx), (j, yy) = _wrap(c, mx), _wrap(c, my)
    G = np.zeros((h, w), order="F")
    c.set_options(wait_polls=1)
    c.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    c.set_options(wait_polls=0)
    assert "timed out" in c.last_error()
    assert np.isnan(G).all()
    assert c.device_error() == 0
    c.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    _check_gram(X, Y, G)
    c.close()


# with a poll a wait the tensor cores give up, multiply-adds do not: which took the
# product.  (narrow blocks of many rows, for which these are faster, and C of few values)
@pytest.mark.parametrize("n,h,w,coords,tensor", [
    (4000000, 2, 2, "full", False), (262144, 8, 8, "full", False), (1 << 21, 11, 2, "full", False),
    (700, 200, 200, "full", False), (1500, 384, 384, "full", False), (4000, 96, 70, "full", False),
    (1 << 20, 12, 12, "full", True), (200000, 32, 32, "full", True), (30000, 96, 40, "full", True),
    (200000, 32, 32, "identity", False), (200000, 32, 32, "triangular", False), (200000, 32, 32, "diagonal", False),
    (200000, 32, 32, "rows", False)])
def test_updates_that_the_tensor_cores_take(n, h, w, coords, tensor):
    c = S.Context(0)
    rng = np.random.default_rng(71)
    mx, my = S.MultiVector(c, n, h), S.MultiVector(c, n, w)
    mx.set_random(1)
    Cf = np.asfortranarray(_coordinates(coords, h, w, rng))
    (i, xx), (j, yy) = _wrap(c, mx), _wrap(c, my)
    c.set_options(wait_polls=1)
    c.lib.mv_MultiVectorByMatrix(xx, h, h, w, Cf.ctypes.data, yy)
    c.set_options(wait_polls=0)
    assert ("timed out" in c.last_error()) == tensor
    c.close()


@pytest.mark.parametrize("n,h,w,tensor", [
    (1 << 21, 8, 8, False), (1 << 21, 16, 8, False), (1 << 21, 32, 4, False), (1 << 19, 64, 4, False),
    (1 << 21, 15, 0, False), (1 << 20, 16, 0, True), (1 << 20, 12, 12, True), (1 << 19, 64, 8, True),
    (30000, 64, 64, True), (40000, 70, 65, True)])
def test_gram_products_that_the_tensor_cores_take(ctx, n, h, w, tensor):
    mx = S.MultiVector(ctx, n, h)
    mx.set_random(1)
    my = mx
    if w:
        my = S.MultiVector(ctx, n, w)
        my.set_random(2)
    w = w or h
    (i, xx), (j, yy) = _wrap(ctx, mx), _wrap(ctx, my)
    G = np.empty((h, w), order="F")
    before = ctx.lib.gpu_KernelLaunchCount()
    ctx.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
    assert ctx.lib.gpu_KernelLaunchCount() - before == (3 if tensor else 2)


# more than 64 columns on either side, by the tensor-core kernel itself: parts of equal width
@pytest.mark.parametrize("n,h,w", [(2101, 130, 70), (1503, 129, 65), (999, 65, 64), (700, 64, 129)])
@pytest.mark.parametrize("grade,coords,add", [("even", "full", True), ("columns", "rows", False),
                                              ("entries", "triangular", True)])
def test_update_in_parts(ctx, n, h, w, grade, coords, add):
    rng = np.random.default_rng(n + w)
    X = rng.standard_normal((n, h)) * _grade(grade, n, h, rng)
    C = _coordinates(coords, h, w, rng)
    Z = rng.standard_normal((n, w)) * 1e-10 if add else None
    _check_update(X, C, Z, _tensor_update(ctx, X, C, Z))
