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
