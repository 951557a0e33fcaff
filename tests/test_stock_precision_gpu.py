"""stock_corr against 80-bit sums where the way its moments are formed could
show: columns that lose much of their squares to dates another column misses,
long panels, means far from zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ULP = 1.11e-16  # of a correlation between 0.5 and 1


def exact(X, m):
    P, N = X.astype(np.longdouble), X.shape[1]
    out = np.ones((N, N), np.longdouble)
    for i in range(N):
        for j in range(i + 1, N):
            o = m[:, i] & m[:, j]
            x, y = P[o, i] - P[o, i].mean(), P[o, j] - P[o, j].mean()
            out[i, j] = (x * y).sum() / np.sqrt((x * x).sum()) / np.sqrt((y * y).sum())
    return out


def rms_error(X, m):
    import torch

    import fcb200
    got = fcb200.stock_corr(torch.from_numpy(X).cuda(), torch.from_numpy(m).cuda()).cpu().numpy()
    err = (got.astype(np.longdouble) - exact(X, m))[np.triu_indices(X.shape[1], 1)]
    return float(np.sqrt(np.mean(err * err)))


def common(T, N, seed):
    r = np.random.default_rng(seed)
    return r, 0.02 * (np.sqrt(0.9) * r.standard_normal((T, 1)) + np.sqrt(0.1) * r.standard_normal((T, N)))


# A sum is formed of chains of 32 dates and T / 32 of those: 0.29 ulps rms a step, growing as the sum does, 1.0 ulp at
# T = 1218 and 1.3 at 2040.  Three of them and the correlation's own roundings: 1.0 * sqrt(1.5) + 0.65 = 1.9 ulps and
# 2.2.  A third is left for the subtraction of up to a quarter of the squares.
@pytest.mark.parametrize("share", [0.2, 0.5, 0.7, 0.9])
@pytest.mark.parametrize("T,ulps", [(120, 2.0), (1218, 2.5), (2040, 2.9)])
def test_an_outlier_that_others_miss(T, ulps, share):
    N = 48
    r, X = common(T, N, T)
    m = r.random((T, N)) < 0.93
    amp = 0.02 * np.sqrt(share / (1 - share) * T)
    for q in range(7):  # on date q + 3 every seventh column has an outlier, and the others miss the date
        cols = np.arange(N) % 7 == q
        X[q + 3, cols] = amp * np.sign(r.standard_normal(cols.sum()))
        m[q + 3] = cols
    # (the pairs of one group share their outlier: its product alone makes their correlation)
    assert rms_error(X, m) < ulps * ULP


# Above 2048 dates the sums that a cancelling pair takes were compensated: their own error a third of an ulp, three of
# them and the correlation's roundings sqrt(1.5) * 0.45 + 0.65 = 1.2 ulps; a tenth for the number of pairs.
@pytest.mark.parametrize("miss", [0.0, 0.05, 0.2])
@pytest.mark.parametrize("T", [2500, 4500])
def test_means_far_from_zero_in_long_panels(T, miss):
    N = 32
    r, X = common(T, N, T)
    assert rms_error(X + 1.0, r.random((T, N)) >= miss) < 1.3 * ULP


def test_more_direct_sums_than_the_list_holds():
    """Five of six pairs lose most of a column's squares: 640000 ordered pairs, more than twice the list of those that
    are summed apart."""
    import torch

    import fcb200
    from conftest import corr_match
    from oracle import fc_oracle as O
    r = np.random.default_rng(2)
    T, N = 60, 800
    X = 0.02 * r.standard_normal((T, N))
    m = np.ones((T, N), bool)
    d = np.arange(N) % 6
    m[:6] = np.arange(6)[:, None] == d[None, :]     # of the first six dates a column has one, with an outlier
    X[d, np.arange(N)] = 0.2 * np.sign(r.standard_normal(N))
    got = fcb200.stock_corr(torch.from_numpy(X).cuda(), torch.from_numpy(m).cuda()).cpu().numpy()
    assert corr_match(got, O.stock_corr(X, m))
