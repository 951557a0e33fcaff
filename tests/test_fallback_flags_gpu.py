"""What fallback_out (factor_corr) and fallback_count (stock_corr) report: the
pairs that fail the cancellation gate, and not those that are recomputed for
another reason (a factor that another one misses, a column whose mean on the
joint dates is far from its own)."""
import ctypes as C

import numpy as np
import pytest

from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu


def gate(X, valid):
    return np.triu(O._gram_corr(X.astype(np.float64), valid)[1], 1)


# means are 0 or at least 5 standard deviations: no pair is near the gate's ratio
@pytest.mark.parametrize("F", [2, 5, 12, 13])
@pytest.mark.parametrize("R", [(10, 100), (60, 400)])
def test_factor_corr_flags_are_the_gate(F, R):
    from fcb200 import _native as nat
    r = np.random.default_rng(F)
    X = r.standard_normal((*R, F))
    X[..., F // 2][r.random(R) < 0.5] = np.nan
    X[: R[0] // 2, :, 0] = np.nan
    if F > 4:
        X[..., 3] += 8.0
    out, fb = np.empty((F, F)), np.zeros((F, F), np.uint8)
    nat.check(nat.lib().fcb_factor_corr(nat.ptr(X), 1, None, *R, F, nat.ptr(out), nat.ptr(fb)), "factor_corr")
    P = X.reshape(-1, F)
    assert np.array_equal(np.triu(fb, 1) != 0, gate(P, np.isfinite(P)))


def test_stock_corr_count_is_the_gate():
    from fcb200 import _native as nat
    r = np.random.default_rng(3)
    T, N = 400, 12
    X = r.standard_normal((T, N))
    m = np.ones((T, N), np.uint8)
    m[: T // 2, :4] = 0
    X[: T // 2, 4:8] += 10.0      # on the dates that columns 0..3 miss
    X[:, 8] += 8.0
    out, n = np.empty((N, N)), C.c_int()
    nat.check(nat.lib().fcb_stock_corr(nat.ptr(X), 1, nat.ptr(m), T, N, nat.ptr(out), None, C.byref(n)), "stock_corr")
    assert n.value == gate(X, m != 0).sum()
