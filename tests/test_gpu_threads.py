"""Host threads with a context each, calling kernels whose shared memory depends
on the call's sizes.  The limit of a kernel's dynamic shared memory belongs to the
function, not to a context: a thread that set it to its own call's size could have
another thread's larger launch refused."""
import threading

import numpy as np
import pytest

from blopex_gb300 import problems as P
from blopex_gb300 import solver as S

pytestmark = pytest.mark.gpu


def _gram_loop(h, w, n, times, out, seed):
    ctx = S.Context(0)
    rng = np.random.default_rng(seed)
    X, Y = rng.standard_normal((n, h)), rng.standard_normal((n, w))
    mx, my = S.MultiVector.from_host(ctx, X), S.MultiVector.from_host(ctx, Y)
    interp = S._Interp(ctx.lib)
    xx = ctx.lib.mv_MultiVectorWrap(interp.ptr, mx.handle, 0)
    yy = ctx.lib.mv_MultiVectorWrap(interp.ptr, my.handle, 0)
    ref, bad = X.T @ Y, 0
    for _ in range(times):
        G = np.full((h, w), 7.0, order="F")
        ctx.lib.mv_MultiVectorByMultiVector(xx, yy, h, h, w, G.ctypes.data)
        bad += not np.allclose(G, ref, rtol=0, atol=1e-11 * n)
    out.append((bad, ctx.last_error()))
    ctx.close()


def _run(jobs):
    threads = [threading.Thread(target=f, args=a) for f, a in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()


# the staged rows of the packed kernel from 17 to 66 KB, and the tensor-core
# kernel's ring for narrow and wide blocks
@pytest.mark.parametrize("sizes,n,times", [([(2, 2), (50, 8), (3, 60), (30, 16)], 6000, 400),
                                           ([(16, 16), (64, 64), (20, 40), (64, 10)], 400000, 30)])
def test_gram_products_of_several_threads(sizes, n, times):
    out = []
    _run([(_gram_loop, (h, w, n, times, out, i)) for i, (h, w) in enumerate(sizes)])
    assert len(out) == len(sizes)
    assert all(bad == 0 and err == "" for bad, err in out), out


def test_solves_of_several_threads():
    """Orders 9 to 120 of the projected problem: Cholesky, tridiagonal reduction,
    bisection and Cholesky-QR kernels."""
    out = []

    def solve(k, seed):
        ctx = S.Context(0)
        rp, ci, va = P.laplacian3d_csr(14, 13, 12)
        A = S.CSRMatrix(ctx, rp, ci, va)
        for i in range(4):
            X = S.MultiVector(ctx, 14 * 13 * 12, k)
            X.set_random(seed + i)
            r = S.lobpcg_solve_double(X, A, atol=1e-4, rtol=1e-50, maxit=300, history=False)
            out.append((k, r.flag, ctx.last_error(), r.lam))
        ctx.close()

    _run([(solve, (k, 10 * k)) for k in (3, 12, 25, 40)])
    assert len(out) == 16
    for k, flag, err, lam in out:
        assert flag == 0 and err == "", (k, flag, err)
    first = {k: min(lam[0] for kk, _, _, lam in out if kk == k) for k in (3, 12, 25, 40)}
    assert np.ptp(list(first.values())) <= 1e-6 * max(first.values())


def test_wait_limit_of_another_threads_context():
    """A context's wait_polls (a poll a wait, so that its kernels give up) is its own:
    the 27-point stencil of another thread's context runs with the default limit."""
    nx = ny = nz = 40
    w = P.stencil27_weights(nx, ny, nz, 1)
    codes, bad = [], []

    def apply(polls, times, out):
        ctx = S.Context(0)
        A = S.Stencil27(ctx, nx, ny, nz, w, 0.5)
        X = S.MultiVector.from_host(ctx, np.random.default_rng(1).standard_normal((nx * ny * nz, 16)), S.FLOAT32)
        Y = S.MultiVector(ctx, nx * ny * nz, 16, S.FLOAT32)
        ctx.set_options(wait_polls=polls)
        for _ in range(times):
            A.apply(X, Y)
            out.append(ctx.device_error())
        ctx.set_options(wait_polls=0)
        ctx.close()

    _run([(apply, (1, 1500, codes)), (apply, (0, 1500, bad))])
    assert any(codes) and not any(bad), (sum(map(bool, codes)), sum(map(bool, bad)))
