"""Section ranks by value-spread buckets (and their radix form for crowded
sections) against the oracle, bit for bit, at the widths where the kernel
variants begin and end and on rows that stress the bucket map."""
import numpy as np
import pytest

from conftest import bitwise_f32
from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu


def stress_rows(N, seed=0):
    """Rows of one width: smooth, heavy-tailed, tied (few to all), clustered, extreme and empty ones."""
    r = np.random.default_rng(seed)
    z = r.standard_normal(N)
    cluster = 1000.0 + 1e-3 * z
    cluster[r.random(N) < 0.01] = 0.0
    ladder = np.exp2(r.integers(-149, 127, N).astype(np.float64)) * np.where(r.random(N) < 0.5, -1, 1)
    inf = z.copy()
    inf[r.random(N) < 0.1] = np.inf
    inf[r.random(N) < 0.1] = -np.inf
    zeros = np.where(r.random(N) < 0.6, np.where(r.random(N) < 0.5, 0.0, -0.0), z)
    few_zeros = np.where(r.random(N) < 0.02, 0.0, z)
    one = np.full(N, np.nan)
    one[N // 2] = -1.5
    rows = [z, few_zeros, np.exp(3 * z), r.standard_t(2, N), np.round(z, 2), np.round(z, 1), np.round(z, 3) * (r.random(N) < 0.99), r.integers(0, 7, N), np.full(N, 0.1),
            cluster, ladder, inf, zeros, one, np.full(N, np.nan), np.full(N, -np.finfo(np.float32).max),
            np.where(z > 0, np.finfo(np.float32).max, -np.finfo(np.float32).max), np.arange(N), -np.arange(N) * 1e-40]
    X = np.array(rows, np.float64).astype(np.float32)
    X[:, r.random(N) < 0.05] = np.nan
    return X


# T <= 148 takes the wide CTAs, T > 148 the narrow ones; each width is an edge of a variant or of a quad
@pytest.mark.parametrize("T", [19, 152])
@pytest.mark.parametrize("N", [1, 3, 33, 1023, 1024, 1025, 2047, 2049, 4095, 4097, 5000, 6144, 6145, 8191, 8193, 16384])
def test_cs_rank_and_scan_stress_rows(N, T):
    import torch

    import fcb200
    X = np.tile(stress_rows(N, N), (-(-T // 19), 1))[:T]
    mask = np.random.default_rng(N + 1).random((T, N)) < 0.9
    mask[3] = False
    dX, dm = torch.from_numpy(X).cuda(), torch.from_numpy(mask).cuda()
    for m, dmm in ((mask, dm), (None, None)):
        for desc in (False, True):
            got = fcb200.cross_sectional_rank(dX, dmm, descending=desc).cpu().numpy()
            assert bitwise_f32(got, O.cs_rank(X, m, desc)), (N, T, m is None, desc)
    got = fcb200.parameter_scan([("direction", ["ascending", "descending"]), ("mask_mode", ["masked", "unmasked"])], dX, dm)
    for g, exp in zip(got["groups"], O.parameter_scan(X, mask)):
        assert bitwise_f32(g["result"], exp), (N, T, g["axis_values"])
    fcb200.check_device()
