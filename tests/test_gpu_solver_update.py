"""The block update of the mixed mode's solver (gb_oz_xc of oz_xc.cu: 42 fraction
bits), called as the solver calls it: an FP64 X, an FP32 or FP64 correction Z, the
result in FP64 and, where asked for, its FP32 copy.

The bounds are those of its splitting: h 2^-38 max |row of X| max |column of C|,
and the rounding of the FP64 result; integers come out exact."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from blopex_gb300 import solver as S  # noqa: E402

pytestmark = pytest.mark.gpu


class _Cols(ctypes.Structure):
    """blk_cols of internal.h."""
    _fields_ = [("col", ctypes.c_void_p * 384)]


@pytest.fixture
def ctx():
    c = S.Context(0)
    yield c
    c.set_options(wait_polls=0)
    c.close()


def _block(a, dtype=torch.float64):
    """Columns on 16-byte boundaries, rows padded as the framework's are."""
    n, k = a.shape
    t = torch.zeros(k, (n + 31) // 32 * 32, dtype=dtype, device="cuda")
    t[:, :n] = torch.from_numpy(np.ascontiguousarray(a.T)).to("cuda", dtype)
    c = _Cols()
    for i in range(k):
        c.col[i] = t[i].data_ptr()
    return t, c


def _update(ctx, X, C, Z=None, z32=False, copy32=False):
    n, (h, w) = X.shape[0], C.shape
    x, cx = _block(X)
    y, cy = _block(np.full((n, w), 7.0))
    y32, c32 = _block(np.full((n, w), 7.0), torch.float32)
    c = torch.from_numpy(np.ascontiguousarray(C.T)).cuda()
    cz = None
    if Z is not None:
        z, cz = _block(Z, torch.float32 if z32 else torch.float64)
    torch.cuda.synchronize()
    rc = ctx.lib.gb_oz_xc(ctypes.c_void_p(ctx.handle), ctypes.c_long(n), ctypes.byref(cx), h,
                          ctypes.c_void_p(c.data_ptr()), h, ctypes.byref(cy), w,
                          ctypes.byref(cz) if cz is not None else None, int(z32),
                          ctypes.byref(c32) if copy32 else None)
    assert rc == 0, ctx.last_error()
    code = ctx.device_error()
    Y = y[:, :n].cpu().numpy().T
    return (Y, y32[:, :n].cpu().numpy().T, code) if copy32 else (Y, code)


def _bound(X, C, Z):
    h = X.shape[1]
    b = h * 2.0 ** -38 * np.outer(np.abs(X).max(1), np.abs(C).max(0))
    ref = X @ C + (Z if Z is not None else 0.0)
    return ref, b + 2.0 ** -52 * (np.abs(X) @ np.abs(C) * (h + 1) + (np.abs(Z) if Z is not None else 0.0))


@pytest.mark.parametrize("n,h,w,z", [(1, 1, 1, None), (129, 17, 33, "f64"), (1000, 64, 64, "f32"),
                                     (100003, 64, 64, "f64"), (70000, 16, 32, None), (4097, 64, 1, "f32"),
                                     (300001, 33, 64, "f32")])
def test_matches_fp64(ctx, n, h, w, z):
    rng = np.random.default_rng(7 * n + h + w)
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
    Z = None if z is None else rng.standard_normal((n, w))
    if z == "f32":
        Z = Z.astype(np.float32).astype(np.float64)
    Y, y32, code = _update(ctx, X, C, Z, z == "f32", copy32=True)
    ref, b = _bound(X, C, Z)
    assert code == 0
    assert np.all(np.abs(Y - ref) <= b), float((np.abs(Y - ref) / b).max())
    assert np.array_equal(y32, Y.astype(np.float32))


def test_wide_ranges_and_zeros(ctx):
    rng = np.random.default_rng(11)
    n, h, w = 20000, 64, 48
    X = rng.standard_normal((n, h)) * 10.0 ** rng.uniform(-20, 20, size=(n, 1))
    X[::97] = 0.0
    X[:, 5] *= 1e-12
    C = rng.standard_normal((h, w)) * 10.0 ** rng.uniform(-10, 10, size=(1, w))
    C[:, 7] = 0.0
    for z32, decades in ((False, 30), (True, 20)):
        Z = rng.standard_normal((n, w)) * 10.0 ** rng.uniform(-decades, decades, size=(n, 1))
        if z32:
            Z = Z.astype(np.float32).astype(np.float64)
        Y, code = _update(ctx, X, C, Z, z32)
        ref, b = _bound(X, C, Z)
        assert code == 0 and np.all(np.abs(Y - ref) <= b), float((np.abs(Y - ref) / b).max())
        assert np.array_equal(Y[::97], Z[::97]) and np.array_equal(Y[:, 7], Z[:, 7])


def test_exact_on_integers(ctx):
    rng = np.random.default_rng(5)
    n, h, w = 50000, 64, 64
    X = rng.integers(-1000, 1001, size=(n, h)).astype(np.float64)
    C = rng.integers(-1000, 1001, size=(h, w)).astype(np.float64)
    Z = rng.integers(-10 ** 6, 10 ** 6, size=(n, w)).astype(np.float64)
    Y, code = _update(ctx, X, C, Z)
    assert code == 0 and np.array_equal(Y, X @ C + Z)


def test_gives_up_cleanly(ctx):
    """One poll a wait: the kernel ends, raises the error word, and has written right
    values or none."""
    rng = np.random.default_rng(1)
    n, h, w = 1 << 20, 64, 64
    X, C = rng.standard_normal((n, h)), rng.standard_normal((h, w))
    ref, b = _bound(X, C, None)
    ctx.set_options(wait_polls=1)
    Y, code = _update(ctx, X, C)
    ctx.set_options(wait_polls=0)
    assert code != 0
    written = Y != 7.0
    assert not written.all()
    assert np.all((np.abs(Y - ref) <= b)[written & ~np.isnan(Y)])
    Y, code = _update(ctx, X, C)
    assert code == 0 and np.all(np.abs(Y - ref) <= b)
