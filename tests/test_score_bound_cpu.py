"""The one-sided error of the K2 score bound, on the CPU in double precision.

The counting kernel bounds ln v! by z ln z - z + ln(2 pi) / 2 at z = v + 1/2
(Burnside).  Its error e(v) is positive and decreasing, so that a cell's bound,
ln n! + ln m! - ln (n + m + 1)!, errs by e(n) + e(m) - e(n + m + 1), which must lie
in (0, 0.1176]: the score is never below the bound and at most 0.1176 a cell above.
"""
import numpy as np
import pytest

CELL = 0.1176


def error(v):
    lgamma = np.vectorize(__import__("math").lgamma)
    z = v + 0.5
    return z * np.log(z) - z + 0.5 * np.log(2 * np.pi) - lgamma(v + 1.0)


@pytest.mark.parametrize("lo,hi,step", [(0, 40, 1), (0, 3000, 61)])
def test_cells_err_to_one_side(lo, hi, step):
    v = np.arange(lo, hi, step, dtype=np.float64)
    e = error(v)
    assert (e > 0).all() and (np.diff(e) < 0).all()
    n, m = np.meshgrid(v, v)
    d = error(n) + error(m) - error(n + m + 1.0)
    assert d.min() > 0 and d.max() <= CELL


# ------------------------------------------------- the kernel's coefficients
F32, F64 = np.float32, np.float64


def _fma(a, b, c):
    return (F64(a) * F64(b) + F64(c)).astype(F32)


def _lg2(x, err):
    """A logarithm as far off as lg2.approx may be: 2^-22, absolutely in (1/2, 2)
    and relatively outside."""
    v = np.log2(x.astype(F64))
    return (v + err * 2.0**-22 * np.where((x > 0.5) & (x < 2), 1.0, np.abs(v))).astype(F32)


def _bound(score, cs, cn, err):
    """L of tables [t][cells] in FP32, in the kernel's operations."""
    acc = [np.zeros(len(cs), F32), np.zeros(len(cs), F32)]
    tsum = np.zeros(len(cs), F32)
    for c in range(cs.shape[1]):
        z = [v[:, c].astype(F32) + F32(0.5 if score == "k2" else 1e-30) for v in (cs, cn)]
        t = z[0] + z[1]
        if score == "k2":
            t = t + F32(0.5)
        lt = _lg2(t, -err)
        for i in range(2):
            acc[i] = _fma(z[i], _lg2(z[i], err) - lt, acc[i])
        tsum = tsum + lt
    total = acc[0] + acc[1]
    return _fma(F32(-0.5), tsum, total) if score == "k2" else total


def _scores(score, cs, cn, nc, nn):
    """The FP32 score as the search evaluates it, and the FP64 one."""
    import math

    n = nc + nn
    vals = np.unique(np.concatenate([cs.ravel(), cn.ravel(), (cs + cn).ravel(), (cs + cn).ravel() + 1, [nc, nn]]))
    inv32 = F32(1.0 / n)
    if score == "k2":
        t64 = np.array([math.lgamma(v + 1.0) for v in vals])
        t32 = t64.astype(F32)
    else:
        t64 = np.array([math.log2(v / n) if v else 0.0 for v in vals])
        t32 = np.array([math.log2(v * float(inv32)) if v else 0.0 for v in vals]).astype(F32)
    at = lambda t, v: t[np.searchsorted(vals, v)]  # noqa: E731
    s32, s64 = np.zeros(len(cs), F32), np.zeros(len(cs))
    if score == "k2":
        for c in range(cs.shape[1]):
            a, b, t = cn[:, c], cs[:, c], cn[:, c] + cs[:, c] + 1
            s32 = s32 + ((at(t32, a) + at(t32, b)) - at(t32, t))
            s64 = s64 + ((at(t64, a) + at(t64, b)) - at(t64, t))
        return np.abs(s32), np.abs(s64)
    ha, hx = np.zeros(len(cs), F32), np.zeros(len(cs), F32)
    p = nc / n
    hy64 = -p * math.log2(p) - (1 - p) * math.log2(1 - p)
    hy = F32(-(float(F32(nc) * inv32) * float(at(t32, nc))))
    hy = F32(float(hy) - float(F32(nn) * inv32) * float(at(t32, nn)))
    for c in range(cs.shape[1]):
        pc, pn = cs[:, c].astype(F32) * inv32, cn[:, c].astype(F32) * inv32
        ha = _fma(-pc, at(t32, cs[:, c]), ha)
        ha = _fma(-pn, at(t32, cn[:, c]), ha)
        hx = _fma(-(pc + pn), at(t32, cs[:, c] + cn[:, c]), hx)
        for v, sign in ((cs[:, c], 1), (cn[:, c], 1), (cs[:, c] + cn[:, c], -1)):
            s64 = s64 + sign * v / n * at(t64, v)
    return (hx + hy) - ha, s64 + hy64


def _tables(rng, cells, nc, nn, count):
    """Random tables: even ones, skewed ones, empty cells, a class in one cell."""
    out = []
    for n in (nc, nn):
        alpha = 10.0 ** rng.uniform(-2, 2, (count, 1)) * np.ones(cells)
        w = rng.gamma(alpha) + 1e-300
        w *= rng.random((count, cells)) < rng.choice([0.3, 1.0], (count, 1))
        w[w.sum(1) == 0, 0] = 1.0
        out.append(rng.multinomial(n, w / w.sum(1, keepdims=True)))
    # Half of them with the classes alike (small effects), as most sets are.
    alike = out[0][: count // 2] + 1e-9
    out[1][: count // 2] = rng.multinomial(nn, alike / alike.sum(1, keepdims=True))
    return out


@pytest.mark.parametrize("score", ["k2", "mi"])
@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("nc,nn", [(1, 1), (1, 9), (31, 1025), (2048, 2048), (5, 400000), (131072, 131072),
                                   (1 << 22, 1 << 22)])
def test_coefficients_bound_the_scores(episdet, order, score, nc, nn):
    """No set scoring s is ruled out at a threshold of s (or worse), and none scores
    worse than its seed key says, whatever the logarithms' errors."""
    import ctypes

    co = (ctypes.c_double * 4)()
    episdet.lib().episdet_test_bound_coefficients(order, int(score == "mi"), nc, nn, co)
    cut_mul, cut_add, seed_mul, seed_add = co
    rng = np.random.default_rng(nc + 7 * order)
    cs, cn = _tables(rng, 9 if order == 2 else 27, nc, nn, 600)
    s32, s64 = _scores(score, cs, cn, nc, nn)
    for err in (-1.0, 0.0, 1.0):
        low = _bound(score, cs, cn, err)
        assert np.isfinite(low).all()
        for s in (s32, s64):
            cut = s * cut_mul + cut_add
            assert (low >= cut - np.spacing(np.abs(cut).astype(F32))).all()
        assert (low >= s32 * cut_mul + cut_add).all()
        seed = ((low.astype(F64) + seed_add) * seed_mul).astype(F32)
        assert ((s32 <= seed) if score == "k2" else (s32 >= seed)).all()
