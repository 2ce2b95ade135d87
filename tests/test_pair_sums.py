"""The inner product that the FP32 7-point stencil folds in, restated on the CPU.

Each thread sums exact products of its cells in compensated FP32 pairs, a plane at a
time; one warp merges the CTA's pairs with a third word (acc_triple32 of blas32.cuh)
and the CTAs' sums are added in FP64.  Its error is compared with that of pairs of
four products, merged over a warp in two words and summed in FP64 from there."""
import numpy as np
import pytest

f = np.float32


def _two_sum(a, b):
    s = (a + b).astype(f)
    bp = (s - a).astype(f)
    return s, ((a - (s - bp).astype(f)).astype(f) + (b - bp).astype(f)).astype(f)


def _prod(s, c, a, b):
    p = (a * b).astype(f)
    e = (a.astype(np.float64) * b.astype(np.float64) - p.astype(np.float64)).astype(f)
    t, err = _two_sum(s, p)
    return t, (c + (err + e).astype(f)).astype(f)


def _pair(s, c, s2, c2):
    t, e = _two_sum(s, s2)
    return t, ((c + c2).astype(f) + e).astype(f)


def _triple(s, c, d, s2, c2, d2):
    t, e = _two_sum(s, s2)
    u, g = _two_sum(c, c2)
    v, h = _two_sum(u, e)
    return t, v, ((d + d2).astype(f) + (g + h).astype(f)).astype(f)


def _quads(a, b):
    """Pairs of four products each."""
    s = np.zeros(a.shape[:-1], f)
    c = s.copy()
    for k in range(4):
        s, c = _prod(s, c, a[..., k], b[..., k])
    return s, c


def _warps_in_fp64(a, b):
    s, c = _quads(a.reshape(-1, 32, 4), b.reshape(-1, 32, 4))
    for o in (16, 8, 4, 2, 1):
        i = np.arange(32) ^ o
        s, c = _pair(s, c, s[:, i], c[:, i])
    return np.sum((s[:, 0].astype(float) + c[:, 0].astype(float)).astype(np.longdouble))


def _ctas(a, b):
    """CTAs of two planes: 8 warps of 32 lanes, four cells of each plane a lane."""
    s, c = _quads(a.reshape(-1, 8, 32, 2, 4), b.reshape(-1, 8, 32, 2, 4))
    s, c = _pair(s[..., 0], c[..., 0], s[..., 1], c[..., 1])
    S = np.zeros((s.shape[0], 32), f)
    C, D, Z = S.copy(), S.copy(), S.copy()
    for w in range(8):
        S, C, D = _triple(S, C, D, s[:, w], c[:, w], Z)
    for o in (16, 8, 4, 2, 1):
        i = np.arange(32) ^ o
        S, C, D = _triple(S, C, D, S[:, i], C[:, i], D[:, i])
    return np.sum((S[:, 0].astype(float) + (C[:, 0].astype(float) + D[:, 0].astype(float))).astype(np.longdouble))


@pytest.mark.parametrize("kind", ["positive", "energy", "signed"])
def test_folded_inner_product_is_as_accurate_as_fp64_sums(kind):
    rng = np.random.default_rng(3)
    err = [[], []]
    for _ in range(16):
        a = rng.standard_normal(1 << 19).astype(f)
        b = {"positive": lambda: a, "signed": lambda: rng.standard_normal(a.size).astype(f),
             "energy": lambda: (a * np.exp(rng.standard_normal(a.size)) + 0.5 * rng.standard_normal(a.size)).astype(f)}[kind]()
        exact = np.sum(a.astype(np.longdouble) * b.astype(np.longdouble))
        mag = float(np.sum(np.abs(a.astype(float) * b.astype(float))))
        for e, g in zip(err, (_warps_in_fp64, _ctas)):
            e.append(float(g(a, b) - exact) / mag)
    rms = [np.sqrt(np.mean(np.square(e))) for e in err]
    assert rms[1] <= 1.05 * rms[0], rms
