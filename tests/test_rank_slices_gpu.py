"""cs_rank of rows too wide for one CTA, by slices of their value range, against
the oracle, bit for bit: smooth, tied and clustered rows, rows whose evenly
spaced sample does not show them, widths at the ends of the form's range."""
import numpy as np
import pytest

from conftest import bitwise_f32
from oracle import fc_oracle as O
from test_section_rank_gpu import stress_rows

pytestmark = pytest.mark.gpu


def misleading_rows(N, seed):
    """Rows whose 512 evenly spaced cells are all alike, invalid or outliers; and one value in every other cell."""
    r = np.random.default_rng(seed)
    at = np.arange(512) * N // 512
    z = r.standard_normal(N)
    alike, absent, outliers = z.copy(), z.copy(), 1.0 + 1e-5 * z
    alike[at] = 0.25
    absent[at] = np.nan
    outliers[at] = 1e6 * r.standard_normal(512)
    half = np.where(np.arange(N) % 2 == 0, 0.5, z)
    two = np.where(z > 0, 3.0, -3.0)
    return np.array([alike, absent, outliers, half, two, np.sort(z)]).astype(np.float32)


@pytest.mark.parametrize("N", [16385, 16387, 20000, 40001, 65536, 65537])
def test_cs_rank_wide_rows(N):
    import torch

    import fcb200
    X = np.concatenate([stress_rows(N, N), misleading_rows(N, N + 1)])
    mask = np.random.default_rng(N + 2).random(X.shape) < 0.9
    mask[3] = False
    mask[20] = True
    for T in (1, len(X)):
        dX, dm = torch.from_numpy(X[-T:]).cuda(), torch.from_numpy(mask[-T:]).cuda()
        for m, dmm in ((mask[-T:], dm), (None, None)):
            for desc in (False, True):
                got = fcb200.cross_sectional_rank(dX, dmm, descending=desc).cpu().numpy()
                assert bitwise_f32(got, O.cs_rank(X[-T:], m, desc)), (N, T, m is None, desc)


def repeated_rows(N, seed):
    """Rows in which values fill slices: few values, one value with little beside it, few valid cells, and both sides
    of each; the sample sees the value but not the cells around it, or does not see it."""
    r = np.random.default_rng(seed)
    z = r.standard_normal(N)
    at = np.arange(512) * N // 512
    rows = [np.full(N, 3.0), np.where(r.random(N) < 1e-3, z, 3.0), np.where(np.arange(N) < 5, -1.0, 3.0),
            np.where(np.arange(N) > N - 6, 9.0, 3.0), r.integers(0, 7, N), (r.random(N) < 0.3).astype(float),
            r.integers(0, 30, N), np.where(r.random(N) < 0.9, 0.0, z), np.where(r.random(N) < 0.2, 0.5, z),
            np.where(r.random(N) < 0.98, np.nan, z), np.where(r.random(N) < 0.98, np.nan, 1.0), np.full(N, np.nan)]
    hidden = np.full(N, np.nan)
    hidden[at] = 1.0
    rest = z.copy()
    rest[at] = np.nan
    one_seen = rest.copy()
    one_seen[at[::100]] = 0.0
    below = np.full(N, 2.0)
    below[1::2] = -1.0
    below[at] = 2.0
    return np.array(rows + [hidden, rest, one_seen, below]).astype(np.float32)


# each side of the lines at which the global sort takes over
@pytest.mark.parametrize("N,T", [(16385, 16), (18432, 160), (18433, 160), (40960, 64), (40961, 64), (65535, 32)])
def test_cs_rank_of_repeated_values(N, T):
    import torch

    import fcb200
    X = np.tile(repeated_rows(N, N), (-(-T // 16), 1))[:T]
    mask = np.random.default_rng(N + 2).random(X.shape) < 0.97
    dX, dm = torch.from_numpy(X).cuda(), torch.from_numpy(mask).cuda()
    for m, dmm in ((mask, dm), (None, None)):
        for desc in (False, True):
            got = fcb200.cross_sectional_rank(dX, dmm, descending=desc).cpu().numpy()
            assert bitwise_f32(got, O.cs_rank(X, m, desc)), (N, T, m is None, desc)
