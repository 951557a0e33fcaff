"""stock_corr's list-sum moments against the oracle: tile edges, chunked
dates (T above one chunk and above the compensated second pass), columns that
miss few, most and whole groups of dates, outliers that only some pairs see,
constant columns and a panel with no missing cell.  The bound is the reference
suite's 1e-12; outlier rows amplify the one-pass sums' rounding by at most
(outlier / spread)^2 = 1e4 here, 1e-16 * 1e4."""
import numpy as np
import pytest

from conftest import corr_match
from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu


def panel(T, N, seed):
    r = np.random.default_rng(seed)
    X = 0.02 * r.standard_t(4, (T, N)) + 0.01 * r.standard_normal((T, 1))
    m = r.random((T, N)) < 0.98
    start = r.integers(0, max(1, T // 8), N)
    m &= np.arange(T)[:, None] >= start[None, :]
    kind = r.integers(0, 8, N)
    for j in range(N):
        if kind[j] == 1:
            m[r.integers(0, T):, j] = False           # delisted: most dates may be missing
        elif kind[j] == 2:
            m[:, j] &= r.random(T) < 0.5              # half missing
        elif kind[j] == 3:
            X[r.integers(0, T), j] += 2.0             # an outlier that pairs see or miss
        elif kind[j] == 4:
            X[:, j] = 0.25                            # constant
        elif kind[j] == 5:
            X[r.random(T) < 0.02, j] = np.nan
    return X, m


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("T,N", [(1, 5), (2, 33), (31, 64), (32, 65), (33, 31), (257, 129), (1536, 40), (1537, 97),
                                 (2049, 63), (3100, 34)])
def test_masked_pairs(T, N, dt):
    import torch

    import fcb200
    X, m = panel(T, N, 1000 * T + N)
    X = X.astype(dt)
    for mask in (m, None):
        got = fcb200.stock_corr(torch.from_numpy(X).cuda(), None if mask is None else torch.from_numpy(mask).cuda())
        assert corr_match(got.cpu().numpy(), O.stock_corr(X, mask)), (T, N, dt, mask is None)


def test_full_panel_and_several_blocks_of_pair_sums():
    """No missing cell (the path without lists), and N above one block of pair
    sums: a few columns of it against the same columns alone."""
    import torch

    import fcb200
    r = np.random.default_rng(5)
    X = r.standard_normal((40, 5200)).astype(np.float32)
    m = r.random(X.shape) < 0.9
    dX, dm = torch.from_numpy(X).cuda(), torch.from_numpy(m).cuda()
    assert corr_match(fcb200.stock_corr(dX[:, :300].contiguous()).cpu().numpy(), O.stock_corr(X[:, :300]))
    got = fcb200.stock_corr(dX, dm)
    pick = np.sort(r.choice(5200, 150, replace=False))
    part = got[torch.from_numpy(pick).cuda()][:, torch.from_numpy(pick).cuda()].cpu().numpy()
    assert corr_match(part, O.stock_corr(X[:, pick], m[:, pick]))
    assert torch.equal(torch.nan_to_num(got, nan=9.0), torch.nan_to_num(got.T, nan=9.0))
