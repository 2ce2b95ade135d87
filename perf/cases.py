"""The work that users of this framework have it do, as cases to be timed.

A case is a dict of plain values.  `prepare` builds what a program has in hand
before the call (device blocks, operators, the preconditioner), `run` makes
one pass through the public entry points, `exact` is the same result in plain
FP64 torch, `work` the bytes and operations that the result cannot do without.

Families (the `what` of a case):
  solve         lobpcg_solve_double for a fixed, small number of iterations from
                a given block: one outer step of a continuation or
                self-consistent loop, which restarts LOBPCG from the last
                block, and the unit of which a full solve is made;
  apply         one operator application Y = A X (the block SpMM);
  pcg           the inner-CG preconditioner T X that a preconditioned solve
                applies once per iteration;
  gram, update  mv_MultiVectorByMultiVector and mv_MultiVectorByMatrix, which
                a caller's own block algorithm uses;
  split_gram, split_update
                the FP64-accurate tensor-core products of the mixed mode;
  adjoint       the backward pass: eigenvector adjoint and coefficient
                gradients.

Grids, block widths, options and distributions are those of bench.py and of
the tests: Laplacians and face coefficients exp(N(0,1)), 27-point weights and
masses U[0.5, 1.5], blocks of random columns.
"""
import ctypes
import math

import numpy as np
import torch

from blopex_gb300 import adjoint as AD
from blopex_gb300 import problems as P
from blopex_gb300 import solver as S


def listed():
    return [
        # a small eigenproblem in the default mode: the 20^3 configuration
        # (k = 10, FP64, no preconditioner); launches and latency count
        dict(name="solve_fp64_20", what="solve", kind="csr", nx=20, ny=20, nz=20, k=10, mode="fp64",
             inner=0, its=12),
        # the headline configuration at 128^3: mixed precision, k = 64, 20
        # inner CG steps on the variable-coefficient stencil
        dict(name="solve_mixed_128", what="solve", kind="st7", nx=128, ny=128, nz=128, k=64,
             mode="mixed", inner=20, its=6),
        # T R of that solve once most columns have converged (about 17 of 64
        # columns are active on average)
        dict(name="pcg_fp32_128", what="pcg", kind="st7", nx=128, ny=128, nz=128, w=17, dtype="f32",
             steps=20),
        # the preconditioner of the 2D differentiation configuration (512^2,
        # k = 8), all FP64
        dict(name="pcg_fp64_512x512", what="pcg", kind="st5", nx=512, ny=512, nz=1, w=8, dtype="f64",
             steps=20),
        # the block SpMM of the largest configuration (256^3, k = 64), FP32
        dict(name="apply_st7_fp32_256", what="apply", kind="st7", nx=256, ny=256, nz=256, w=64,
             dtype="f32"),
        # the CSR SpMM of the plain FP64 configuration (128^3, k = 32)
        dict(name="apply_csr_fp64_128", what="apply", kind="csr", nx=128, ny=128, nz=128, w=32,
             dtype="f64"),
        # A R of the generalized 27-point configuration (100^3, k = 128)
        # in the mixed mode's FP32 blocks
        dict(name="apply_st27_fp32_100", what="apply", kind="st27", nx=100, ny=100, nz=100, w=128,
             dtype="f32"),
        # Gram block and block update of the plain FP64 configuration
        dict(name="gram_fp64_32x32", what="gram", n=2097152, h=32, w=32, dtype="f64", same=False),
        dict(name="update_fp64_32x32", what="update", n=2097152, h=32, w=32, dtype="f64"),
        # one Gram of the mixed mode's pencil, X'[X R P] with part of the
        # columns converged, and its X update
        dict(name="split_gram_64_33_33", what="split_gram", n=2097152, h=64, q=33, p=33, ldt="f64"),
        dict(name="split_update_64", what="split_update", n=2097152, h=64, w=64, z="f32"),
        # the backward pass of the 2D differentiation configuration
        dict(name="adjoint_512x512", what="adjoint", nx=512, ny=512, k=8, inner=20, its=5),
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], uniform in its logarithm."""
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def _grid(rng, lo, hi):
    """Dimensions of one scale between lo and hi, mostly unequal and odd."""
    g = _log(rng, lo, hi)
    d = [max(2, min(hi, int(g * rng.uniform(0.8, 1.25)))) for _ in range(3)]
    if rng.random() < 0.4:
        d[0] = max(4, d[0] // 4 * 4)  # rows of whole 16-byte groups
    return d


def draw(rng):
    what = rng.choice(["solve", "solve", "apply", "apply", "pcg", "pcg", "gram", "update",
                       "split_gram", "split_update", "adjoint"])
    if what == "solve":
        mode = rng.choice(["fp64", "mixed"])
        nx, ny, nz = _grid(rng, 10, 72)
        return dict(what=what, kind=rng.choice(["csr", "st7"]), nx=nx, ny=ny, nz=nz,
                    k=_log(rng, 3, 40), mode=mode, inner=rng.choice([0, 5, 20]),
                    its=rng.randint(3, 8))
    if what == "apply":
        kind, dtype = rng.choice(["csr", "st7", "st5", "st27"]), rng.choice(["f32", "f64"])
        if kind == "st5":
            nx, ny, nz = _log(rng, 20, 1500), _log(rng, 20, 1500), 1
        else:
            nx, ny, nz = _grid(rng, 10, 90 if kind == "st27" else 160)
        return dict(what=what, kind=kind, nx=nx, ny=ny, nz=nz, w=_log(rng, 1, 96), dtype=dtype)
    if what == "pcg":
        kind, dtype = rng.choice(["st7", "st7", "st5", "csr"]), rng.choice(["f32", "f64"])
        if kind == "st5":
            nx, ny, nz = _log(rng, 30, 700), _log(rng, 30, 700), 1
        else:
            nx, ny, nz = _grid(rng, 10, 140 if dtype == "f32" else 96)
        return dict(what=what, kind=kind, nx=nx, ny=ny, nz=nz, w=_log(rng, 1, 40), dtype=dtype,
                    steps=rng.choice([5, 10, 20]))
    if what in ("gram", "update"):
        d = dict(what=what, n=_log(rng, 1000, 3000000), h=_log(rng, 2, 96), w=_log(rng, 2, 96),
                 dtype=rng.choice(["f64", "f64", "f32"]))
        if what == "gram":
            d["same"] = rng.random() < 0.3
            if d["same"]:
                d["w"] = d["h"]
        return d
    if what == "split_gram":
        return dict(what=what, n=_log(rng, 5000, 3000000), h=_log(rng, 4, 64), q=_log(rng, 2, 64),
                    p=_log(rng, 2, 64), ldt=rng.choice(["f64", "f32"]))
    if what == "split_update":
        return dict(what=what, n=_log(rng, 5000, 3000000), h=_log(rng, 4, 64), w=_log(rng, 4, 64),
                    z=rng.choice(["f32", "f64", "none"]))
    return dict(what="adjoint", nx=_log(rng, 24, 512), ny=_log(rng, 24, 512), k=rng.randint(2, 10),
                inner=rng.choice([0, 5, 20]), its=rng.randint(2, 6))


# ------------------------------------------------------------------- inputs
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _block(gen, n, k, dtype, scale=1.0):
    """A k x n tensor whose rows are the columns of an n x k block, rows padded
    to a multiple of 32 as the framework's own blocks are."""
    t = torch.zeros(k, (n + 31) // 32 * 32, device="cuda", dtype=dtype)
    for c in range(k):
        t[c, :n] = torch.randn(n, device="cuda", dtype=torch.float32, generator=gen)
        if dtype == torch.float64:  # all 53 bits of the significand in use
            t[c, :n] += torch.randn(n, device="cuda", dtype=torch.float32, generator=gen) * 2.0 ** -26
        t[c, :n] *= scale
    return t


def _wrap(ctx, t, n):
    return S.MultiVector.wrap_device(ctx, t.data_ptr(), n, t.shape[1], t.shape[0],
                                     S.FLOAT64 if t.dtype == torch.float64 else S.FLOAT32)


def _dtype(name):
    return torch.float64 if name == "f64" else torch.float32


def _coefficients(case, seed):
    """Operator coefficients on the device, FP64."""
    g = _gen(seed, 7)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]

    def lognormal(*shape):
        return torch.randn(*shape, device="cuda", dtype=torch.float64, generator=g).exp_()

    if case["kind"] in ("st7", "csr"):
        return [lognormal(nz, ny, nx + 1), lognormal(nz, ny + 1, nx), lognormal(nz + 1, ny, nx)]
    if case["kind"] == "st5":
        return [lognormal(ny, nx + 1), lognormal(ny + 1, nx)]
    return [torch.rand(nx * ny * nz, 13, device="cuda", dtype=torch.float64, generator=g) + 0.5]


def _csr(c):
    """CSR arrays (host) of the 7-point operator with face coefficients c."""
    cx, cy, cz = c
    nz, ny, nx = cy.shape[0], cy.shape[1] - 1, cy.shape[2]
    idx = torch.arange(nx * ny * nz, device="cuda").reshape(nz, ny, nx)
    cols = torch.full((nz, ny, nx, 7), -1, dtype=torch.int64, device="cuda")
    vals = torch.zeros((nz, ny, nx, 7), dtype=torch.float64, device="cuda")
    cols[1:, :, :, 0], vals[1:, :, :, 0] = idx[:-1], -cz[1:-1]
    cols[:, 1:, :, 1], vals[:, 1:, :, 1] = idx[:, :-1], -cy[:, 1:-1]
    cols[:, :, 1:, 2], vals[:, :, 1:, 2] = idx[:, :, :-1], -cx[:, :, 1:-1]
    cols[..., 3], vals[..., 3] = idx, _diagonal(c).reshape(nz, ny, nx)
    cols[:, :, :-1, 4], vals[:, :, :-1, 4] = idx[:, :, 1:], -cx[:, :, 1:-1]
    cols[:, :-1, :, 5], vals[:, :-1, :, 5] = idx[:, 1:], -cy[:, 1:-1]
    cols[:-1, :, :, 6], vals[:-1, :, :, 6] = idx[1:], -cz[1:-1]
    ok = cols >= 0
    rowptr = torch.zeros(idx.numel() + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = ok.reshape(-1, 7).sum(1).cumsum(0)
    return rowptr.int().cpu().numpy(), cols[ok].int().cpu().numpy(), vals[ok].cpu().numpy()


def _diagonal(c):
    if len(c) == 3:
        cx, cy, cz = c
        return (cx[:, :, :-1] + cx[:, :, 1:] + cy[:, :-1] + cy[:, 1:] + cz[:-1] + cz[1:]).reshape(-1)
    cx, cy = c
    return (cx[:, :-1] + cx[:, 1:] + cy[:-1] + cy[1:]).reshape(-1)


SHIFT27 = 0.5


def _operator(ctx, case, c):
    if case["kind"] == "csr":
        return S.CSRMatrix(ctx, *_csr(c))
    h = [x.cpu().numpy() for x in c]
    if case["kind"] == "st7":
        return S.Stencil7(ctx, *h)
    if case["kind"] == "st5":
        return S.Stencil5(ctx, *h)
    return S.Stencil27(ctx, case["nx"], case["ny"], case["nz"], h[0], SHIFT27)


def _rows(case):
    return case["n"] if "n" in case else case["nx"] * case["ny"] * case.get("nz", 1)


class _State:
    pass


_streams = []


def _stream():
    """One stream for all states: a program solves one problem after another."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0].cuda_stream


def prepare(case, seed):
    s = _State()
    s.case, what = case, case["what"]
    s.n = n = _rows(case)
    s.ctx = ctx = S.Context(0, _stream(),
                            precision=S.MIXED if case.get("mode") == "mixed" else S.FP64)
    s.lib = ctx.lib
    g = _gen(seed, 1)
    if what in ("solve", "apply", "pcg"):
        c = _coefficients(case, seed)
        s.A = _operator(ctx, case, c)
    if what == "solve":
        s.T = None
        jac = S.Diagonal(ctx, (1.0 / _diagonal(c)).cpu().numpy())
        if case["inner"]:
            s.T = S.PCGPreconditioner(ctx, s.A, jac, case["inner"])
        elif case["mode"] == "mixed":
            s.T = jac
        s.x0 = _block(g, n, case["k"], torch.float64)
        s.x = torch.zeros_like(s.x0)
        s.X0, s.X = _wrap(ctx, s.x0, n), _wrap(ctx, s.x, n)
    elif what in ("apply", "pcg"):
        s.op = s.A
        if what == "pcg":
            jac = S.Diagonal(ctx, (1.0 / _diagonal(c)).cpu().numpy())
            s.op = S.PCGPreconditioner(ctx, s.A, jac, case["steps"])
        s.x = _block(g, n, case["w"], _dtype(case["dtype"]))
        s.y = torch.zeros_like(s.x)
        s.X, s.Y = _wrap(ctx, s.x, n), _wrap(ctx, s.y, n)
    elif what == "gram":
        s.x = _block(g, n, case["h"], _dtype(case["dtype"]), n ** -0.5)
        s.y = s.x if case["same"] else _block(g, n, case["w"], _dtype(case["dtype"]), n ** -0.5)
        s.X = _wrap(ctx, s.x, n)
        s.Y = s.X if case["same"] else _wrap(ctx, s.y, n)
        s.interp = S._Interp(ctx.lib)
        s.xx = s.lib.mv_MultiVectorWrap(s.interp.ptr, s.X.handle, 0)
        s.yy = s.lib.mv_MultiVectorWrap(s.interp.ptr, s.Y.handle, 0)
    elif what == "update":
        s.x = _block(g, n, case["h"], _dtype(case["dtype"]))
        s.y = torch.zeros(case["w"], s.x.shape[1], device="cuda", dtype=s.x.dtype)
        s.X, s.Y = _wrap(ctx, s.x, n), _wrap(ctx, s.y, n)
        s.c = _matrix(case, seed)
        s.interp = S._Interp(ctx.lib)
        s.xx = s.lib.mv_MultiVectorWrap(s.interp.ptr, s.X.handle, 0)
        s.yy = s.lib.mv_MultiVectorWrap(s.interp.ptr, s.Y.handle, 0)
    elif what == "split_gram":
        s.l = _block(g, n, case["h"], _dtype(case["ldt"]), n ** -0.5)
        s.q = _block(g, n, case["q"], torch.float32, n ** -0.5)
        s.p = _block(g, n, case["p"], torch.float32, n ** -0.5)
        s.L, s.Q, s.P = _wrap(ctx, s.l, n), _wrap(ctx, s.q, n), _wrap(ctx, s.p, n)
        s.blocks = (ctypes.c_void_p * 2)(s.Q.handle, s.P.handle)
    elif what == "split_update":
        s.x = _block(g, n, case["h"], torch.float64)
        s.y = torch.zeros(case["w"], s.x.shape[1], device="cuda", dtype=torch.float64)
        s.X, s.Y, s.Z = _wrap(ctx, s.x, n), _wrap(ctx, s.y, n), None
        if case["z"] != "none":
            s.z = _block(g, n, case["w"], _dtype(case["z"]))
            s.Z = _wrap(ctx, s.z, n)
        s.c = _matrix(case, seed)
    else:
        # eigenpairs in hand: those of a constant-coefficient operator are known
        nx, ny, k = case["nx"], case["ny"], case["k"]
        a, b = (0.6 + torch.rand(2, generator=torch.Generator().manual_seed(int(seed)))).tolist()
        s.A = S.Stencil5(ctx, np.full((ny, nx + 1), a), np.full((ny + 1, nx), b))
        jac = S.Diagonal(ctx, np.full(n, 0.5 / (a + b)))
        s.T = S.PCGPreconditioner(ctx, s.A, jac, case["inner"]) if case["inner"] else jac
        lx = 4 * a * np.sin(np.pi * np.arange(1, k + 1) / (2 * (nx + 1))) ** 2
        ly = 4 * b * np.sin(np.pi * np.arange(1, k + 1) / (2 * (ny + 1))) ** 2
        both = np.add.outer(ly, lx).ravel()
        order = np.argsort(both)[:k]
        s.lam = both[order]
        s.x = torch.zeros(k, (n + 31) // 32 * 32, device="cuda", dtype=torch.float64)
        i = torch.arange(1, nx + 1, device="cuda", dtype=torch.float64) * (math.pi / (nx + 1))
        j = torch.arange(1, ny + 1, device="cuda", dtype=torch.float64) * (math.pi / (ny + 1))
        for c, o in enumerate(order):
            v = torch.outer(torch.sin(j * (int(o) // k + 1)), torch.sin(i * (int(o) % k + 1))).reshape(-1)
            s.x[c, :n] = v / v.norm()
        s.X = _wrap(ctx, s.x, n)
        r = np.random.default_rng(seed)
        s.G = np.asfortranarray(r.standard_normal((n, k)))
        s.glam = r.standard_normal(k)
    torch.cuda.synchronize()
    return s


def _matrix(case, seed):
    """The host coordinate matrix C of an update, column-major."""
    r = np.random.default_rng(seed)
    return np.asfortranarray(r.standard_normal((case["h"], case["w"])) / math.sqrt(case["h"]))


# ------------------------------------------------------------------ a pass
def run(s):
    case, what = s.case, s.case["what"]
    if what == "solve":
        s.X.copy_from(s.X0)
        r = S.lobpcg_solve_double(s.X, s.A, T=s.T, atol=1e-8, rtol=1e-50, maxit=case["its"],
                                  history=False)
        return {"lam": r.lam, "res": r.res, "x": s.x[:, :s.n]}
    if what in ("apply", "pcg"):
        s.op.apply(s.X, s.Y)
        return s.y[:, :s.n]
    if what == "gram":
        out = np.empty((case["h"], case["w"]), order="F")
        s.lib.mv_MultiVectorByMultiVector(s.xx, s.yy, case["h"], case["h"], case["w"], out.ctypes.data)
        return out
    if what == "update":
        s.lib.mv_MultiVectorByMatrix(s.xx, case["h"], case["h"], case["w"], s.c.ctypes.data, s.yy)
        return s.y[:, :s.n]
    if what == "split_gram":
        out = np.empty((case["h"], case["h"] + case["q"] + case["p"]), order="F")
        if s.lib.gpu_SplitGram(s.L.handle, s.blocks, 2, out.ctypes.data, case["h"]):
            raise S.GpuError(s.ctx.last_error())
        return out
    if what == "split_update":
        if s.lib.gpu_BlockUpdate(s.X.handle, s.c.ctypes.data, case["h"], s.Y.handle,
                                 s.Z.handle if s.Z is not None else None, 2):
            raise S.GpuError(s.ctx.last_error())
        return s.y[:, :s.n]
    adj = AD.eigenvector_adjoint(s.X, s.lam, s.A, G=s.G, glam=s.glam, T=s.T, tol=1e-8,
                                 maxit=case["its"])
    return {"w": adj.W.to_host(), "xg": adj.xg, "grad": AD.operator_gradient(s.A, s.X, adj.W)}


# ----------------------------------------------------------------- FP64 truth
def _apply64(kind, case, c, x):
    """The operator on a block x (columns as rows), FP64 torch."""
    if kind == "st5":
        cx, cy = c
        v = torch.nn.functional.pad(x.reshape(-1, case["ny"], case["nx"]), (1, 1, 1, 1))
        m = v[:, 1:-1, 1:-1]
        y = (cx[:, :-1] * (m - v[:, 1:-1, :-2]) + cx[:, 1:] * (m - v[:, 1:-1, 2:])
             + cy[:-1] * (m - v[:, :-2, 1:-1]) + cy[1:] * (m - v[:, 2:, 1:-1]))
        return y.reshape(x.shape)
    v = torch.nn.functional.pad(x.reshape(-1, case["nz"], case["ny"], case["nx"]), (1,) * 6)
    m = v[:, 1:-1, 1:-1, 1:-1]
    if kind != "st27":
        cx, cy, cz = c
        y = (cx[:, :, :-1] * (m - v[:, 1:-1, 1:-1, :-2]) + cx[:, :, 1:] * (m - v[:, 1:-1, 1:-1, 2:])
             + cy[:, :-1] * (m - v[:, 1:-1, :-2, 1:-1]) + cy[:, 1:] * (m - v[:, 1:-1, 2:, 1:-1])
             + cz[:-1] * (m - v[:, :-2, 1:-1, 1:-1]) + cz[1:] * (m - v[:, 2:, 1:-1, 1:-1]))
        return y.reshape(x.shape)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    y = SHIFT27 * m
    w = c[0].reshape(nz, ny, nx, 13)
    for e, (di, dj, dk) in enumerate(P.STENCIL27_OFFSETS.tolist()):
        def cut(d, size):  # cells whose neighbour at offset d is on the grid, and those neighbours
            return slice(max(0, -d), size - max(0, d)), slice(max(0, d), size + min(0, d))
        (a0, b0), (a1, b1), (a2, b2) = cut(dk, nz), cut(dj, ny), cut(di, nx)
        f = w[a0, a1, a2, e] * (m[:, a0, a1, a2] - m[:, b0, b1, b2])
        y[:, a0, a1, a2] += f
        y[:, b0, b1, b2] -= f
    return y.reshape(x.shape)


def _columns(case, seed):
    """The block X of an apply or pcg case, a few columns at a time in FP64."""
    n, w = _rows(case), case["w"]
    x = _block(_gen(seed, 1), n, w, _dtype(case["dtype"]))
    step = max(1, (1 << 26) // n)
    for c0 in range(0, w, step):
        yield slice(c0, min(w, c0 + step)), x[c0:c0 + step, :n].double()


def exact(case, seed):
    what, n = case["what"], _rows(case)
    if what in ("apply", "pcg"):
        c = _coefficients(case, seed)
        out = torch.empty(case["w"], n, device="cuda", dtype=torch.float64)
        for cols, x in _columns(case, seed):
            out[cols] = (_apply64(case["kind"], case, c, x) if what == "apply"
                         else _pcg64(case, c, x))
        return out
    g = _gen(seed, 1)
    if what == "gram":
        x = _block(g, n, case["h"], _dtype(case["dtype"]), n ** -0.5)
        y = x if case["same"] else _block(g, n, case["w"], _dtype(case["dtype"]), n ** -0.5)
        return _gram64(x, y).cpu().numpy()
    if what == "update":
        x = _block(g, n, case["h"], _dtype(case["dtype"]))[:, :n]
        return _update64(x, _matrix(case, seed), None)
    if what == "split_gram":
        l = _block(g, n, case["h"], _dtype(case["ldt"]), n ** -0.5)
        q = _block(g, n, case["q"], torch.float32, n ** -0.5)
        p = _block(g, n, case["p"], torch.float32, n ** -0.5)
        return torch.cat([_gram64(l, l), _gram64(l, q), _gram64(l, p)], dim=1).cpu().numpy()
    if what == "split_update":
        x = _block(g, n, case["h"], torch.float64)[:, :n]
        z = None
        if case["z"] != "none":
            z = _block(g, n, case["w"], _dtype(case["z"]))[:, :n].double()
        return _update64(x, _matrix(case, seed), z)
    return None  # iterates of a solve stopped early have no closed form


def _gram64(x, y):
    """x y' by blocks of 32 rows of the block vectors, so that the roundings of
    one long running sum do not enter (the padding is zero)."""
    out = []
    for z in (x, y):
        out.append(z.double().reshape(z.shape[0], -1, 32).transpose(0, 1))
    return torch.bmm(out[0], out[1].transpose(1, 2)).sum(0)


def _halves(a):
    """a = hi + lo with 26-bit halves (Dekker)."""
    t = a * 134217729.0
    hi = t - (t - a)
    return hi, a - hi


def _update64(x, c, z):
    """C' x + z with exact products and compensated sums, so that the result
    carries one rounding and not the h roundings of a running sum."""
    c = torch.from_numpy(c).cuda()
    hi = torch.zeros(c.shape[1], x.shape[1], device="cuda", dtype=torch.float64)
    lo = torch.zeros_like(hi)

    def add(p):
        nonlocal hi, lo
        t = hi + p
        b = t - hi
        lo += (hi - (t - b)) + (p - b)
        hi = t

    for i in range(x.shape[0]):
        xi, ci = x[i].double()[None], c[i][:, None]
        (xh, xl), (ch, cl) = _halves(xi), _halves(ci)
        p = ci * xi
        lo += ((ch * xh - p) + ch * xl + cl * xh) + cl * xl
        add(p)
    if z is not None:
        add(z)
    return hi + lo


def _pcg64(case, c, x):
    m = 1.0 / _diagonal(c)
    r, y = x.clone(), torch.zeros_like(x)
    z = m * r
    p, rho = z.clone(), (r * z).sum(1, keepdim=True)
    for it in range(case["steps"]):
        q = _apply64(case["kind"], case, c, p)
        alpha = rho / (p * q).sum(1, keepdim=True)
        y += alpha * p
        r -= alpha * q
        if it + 1 < case["steps"]:
            z = m * r
            new = (r * z).sum(1, keepdim=True)
            p = z + (new / rho) * p
            rho = new
    return y


# ---------------------------------------------------------------- the floor
def _op_work(case, es):
    """Coefficient bytes and flops per column of one operator application."""
    n, kind = _rows(case), case["kind"]
    if kind == "csr":
        return 7 * n * (es + 4) + 4 * n, 14.0 * n
    return {"st7": (3 * n * es, 13.0 * n), "st5": (2 * n * es, 9.0 * n),
            "st27": (13 * n * es, 53.0 * n)}[kind]


def work(case):
    what, n = case["what"], _rows(case)
    es = 8 if case.get("dtype", "f64") == "f64" else 4
    if what == "apply":
        cb, cf = _op_work(case, es)
        return {"bytes": 2.0 * es * n * case["w"] + cb, "flops": cf * case["w"]}
    if what == "pcg":
        cb, cf = _op_work(case, es)
        return {"bytes": 2.0 * es * n * case["w"] + cb + es * n,
                "flops": case["steps"] * (cf + 11.0 * n) * case["w"]}
    if what == "gram":
        h, w = case["h"], case["w"]
        return {"bytes": 1.0 * es * n * (h if case["same"] else h + w),
                "flops": 1.0 * n * h * (h + 1) if case["same"] else 2.0 * n * h * w}
    if what == "update":
        return {"bytes": 1.0 * es * n * (case["h"] + case["w"]), "flops": 2.0 * n * case["h"] * case["w"]}
    if what == "split_gram":
        h, w = case["h"], case["q"] + case["p"]
        return {"bytes": n * ((8.0 if case["ldt"] == "f64" else 4.0) * h + 4.0 * w),
                "flops": 2.0 * n * h * w + 1.0 * n * h * (h + 1)}
    if what == "split_update":
        z = {"f32": 4.0, "f64": 8.0, "none": 0.0}[case["z"]]
        return {"bytes": n * (8.0 * case["h"] + (8.0 + z) * case["w"]),
                "flops": 2.0 * n * case["h"] * case["w"]}
    k, its = case["k"], case["its"]
    if what == "solve":
        # per iteration A R, T R, the Gram blocks of [X R P] and the updates
        # of X, P and their images
        cb, cf = _op_work(case, 8)
        return {"bytes": 16.0 * n * k + cb,
                "flops": its * ((1 + case["inner"]) * cf * k + 11.0 * n * k * case["inner"]
                                + 2.0 * n * (9 + 10) * k * k)}
    # adjoint: G and X in, W and the gradient out; per step A, T, two
    # projections and the column updates
    return {"bytes": 8.0 * n * (3 * k + 2),
            "flops": its * n * k * (9.0 * (1 + case["inner"]) + 11.0 * case["inner"] + 8.0 * k + 16.0)}
