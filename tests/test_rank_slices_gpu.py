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
