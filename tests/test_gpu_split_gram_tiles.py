"""The split Gram kernel at the edges of its tiles and roles: groups of eight columns
cut short, chunks of 64 rows cut short, one chunk and several a CTA, two, three and
four raw buffers (by the widths and types), columns copied as one tile and one by
one.  Integers of 15 bits times a power of two a column (two digits, products exact in
FP64); the bound is that of the kernel's four digits and double-float sums."""
import ctypes

import numpy as np
import pytest

from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu


def _block(rng, n, w, scaled):
    v = rng.integers(-2 ** 14, 2 ** 14 + 1, size=(n, w)).astype(np.float64)
    return v * 2.0 ** rng.integers(-40, 41, size=(1, w)) if scaled else v


def _bound(L, R):
    """Digits of 32 bits a 64-row chunk (half a unit a factor), levels below them left
    out, FP32 rounding of the combined lower levels, FP64 sums."""
    b = np.zeros((L.shape[1], R.shape[1]))
    c = np.zeros_like(b)
    for r in range(0, L.shape[0], 64):
        x, y = L[r:r + 64], R[r:r + 64]
        b += 64.0 * np.outer(np.abs(x).max(axis=0), np.abs(y).max(axis=0))
        c += np.abs(x.T @ y)
    return 2.0 ** -29 * b + 2.0 ** -30 * c + 2.0 ** -50 * (np.abs(L).T @ np.abs(R))


@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("n", [1, 31, 64, 65, 127, 9728, 19457])
@pytest.mark.parametrize("h,ldt,widths", [(1, "f64", []), (7, "f64", [(1, "f32")]), (8, "f32", [(9, "f64")]),
                                          (33, "f64", [(64, "f64")]), (64, "f64", [(64, "f64"), (5, "f32")]),
                                          (64, "f64", [(33, "f32"), (33, "f32")]), (64, "f32", [(63, "f32")])])
def test_edges(n, h, ldt, widths, scaled):
    rng = np.random.default_rng(n + h)
    dt = {"f32": S.FLOAT32, "f64": S.FLOAT64}
    L, Qs = _block(rng, n, h, scaled), [(_block(rng, n, w, scaled), d) for w, d in widths]
    ctx = S.Context(0)
    try:
        ml = S.MultiVector.from_host(ctx, L, dt[ldt])
        mq = [S.MultiVector.from_host(ctx, q, dt[d]) for q, d in Qs]
        arr = (ctypes.c_void_p * max(1, len(mq)))(*[m.handle for m in mq])
        R = np.hstack([L] + [q for q, _ in Qs])
        G = np.zeros((h, R.shape[1]), order="F")
        assert ctx.lib.gpu_SplitGram(ml.handle, arr, len(mq), G.ctypes.data, h) == 0, ctx.last_error()
        assert np.all(np.abs(G - L.T @ R) <= _bound(L, R))
    finally:
        ctx.close()
