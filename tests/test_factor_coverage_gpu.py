"""factor_corr of factors that cover different shares of the rows, up to 12
factors: each side of the shares at which the Gram pass changes its form (two
thirds for one factor, nine tenths for all), alone and mixed, against the
oracle, against 80-bit sums and, in a batch, against the single calls."""
import numpy as np
import pytest

from conftest import corr_match
from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu


def run(X, mask, planes):
    import torch
    from fcb200 import _native as nat
    T, N, F = X.shape
    ws = nat.lib().fcb_workspace_create()
    try:
        d = torch.from_numpy(np.ascontiguousarray(np.moveaxis(X, -1, 0) if planes else X)).cuda()
        dm = None if mask is None else torch.from_numpy(mask.astype(np.uint8)).cuda()
        out = torch.empty((F, F), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        nat.check(nat.lib().fcb_dev_factor_corr(d.data_ptr(), 0 if X.dtype == np.float32 else 1,
                                                None if dm is None else dm.data_ptr(), T, N, F, planes, out.data_ptr(), ws,
                                                None), "factor_corr")
        torch.cuda.synchronize()
        return out.cpu().numpy()
    finally:
        nat.lib().fcb_workspace_destroy(ws)


def panel(T, N, F, kind, seed):
    r = np.random.default_rng(seed)
    X = r.standard_normal((T, N, F)) + 0.5 * r.standard_normal((T, N, 1))
    share = {"mixed": r.choice([0.1, 0.4, 0.6, 0.65, 0.68, 0.75, 0.95, 1.0], F), "low": np.full(F, 0.3),
             "high": np.full(F, 0.8), "full": np.full(F, 0.97), "one": np.where(np.arange(F) == F // 2, 0.5, 1.0)}[kind]
    X[r.random(X.shape) >= share] = np.nan
    if kind == "mixed" and F > 3:
        X[: T // 2, :, 0] = np.nan             # listed late
        X[T // 3:, :, 1] = np.nan              # dropped early: few rows in common with the first
        X[r.random((T, N)) < 0.2] = np.nan     # rows with no factor
        X[0, 0, 2] = 1e6                       # an outlier that others miss
        X[0, 0, 3] = np.nan
    return X, r.random((T, N)) < 0.9


@pytest.mark.parametrize("F", [2, 3, 4, 5, 6, 8, 9, 10, 11, 12])
def test_coverage(F):
    for kind in ("mixed", "low", "high", "full", "one"):
        for T, N in ((3, 7), (20, 100), (40, 701)):
            X, m = panel(T, N, F, kind, 17 * F + T)
            for dt in (np.float32, np.float64):
                for mask in (m, None):
                    got = [run(X.astype(dt), mask, p) for p in (0, 1)]
                    assert corr_match(got[0], O.factor_corr(X.astype(dt), mask)), (kind, T, dt, mask is None)
                    assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64))


def exact(X):
    P = X.reshape(-1, X.shape[-1]).astype(np.longdouble)
    F = P.shape[1]
    out = np.ones((F, F), np.longdouble)
    for i in range(F):
        for j in range(F):
            if i != j:
                o = np.isfinite(P[:, i]) & np.isfinite(P[:, j])
                x, y = P[o, i] - P[o, i].mean(), P[o, j] - P[o, j].mean()
                out[i, j] = (x * y).sum() / np.sqrt((x * x).sum()) / np.sqrt((y * y).sum())
    return out


# A sum of 2000 rows takes about 75 roundings (up to 63 four-row steps and the merges), 0.29 ulps rms each of a sum
# that grows as they go (1 / sqrt(3)): 1.5 ulps.  Three such sums in a correlation near 0.9 and its own five
# roundings make 1.5 * sqrt(1.5) + 0.6 = 2.5 ulps of 1.1e-16, 2.8e-16 rms.  Half as much again for 15 pairs.
@pytest.mark.parametrize("share", [0.3, 0.6, 0.7])
def test_precision_of_small_pools(share):
    r = np.random.default_rng(5)
    T, N, F = 40, 50, 6
    X = np.sqrt(0.9) * r.standard_normal((T, N, 1)) + np.sqrt(0.1) * r.standard_normal((T, N, F))
    X[r.random(X.shape) >= share] = np.nan
    err = (run(X, None, 0).astype(np.longdouble) - exact(X))[np.triu_indices(F, 1)]
    assert np.sqrt(np.mean(err * err)) < 4.2e-16


def test_batch_mixes_the_forms():
    import torch

    import fcb200
    r = np.random.default_rng(9)
    panels = []
    for k, (F, kind) in enumerate(((12, "high"), (5, "low"), (4, "full"), (14, "low"), (8, "mixed"), (10, "full"))):
        X, m = panel(20, 200 + 31 * k, F, kind, k)
        X = np.ascontiguousarray(np.moveaxis(X, -1, 0)).astype(np.float32)
        p = {"X": X, "R": r.standard_normal(X.shape[1:]).astype(np.float32), "fmask": m.astype(np.uint8)}
        p = {n: torch.from_numpy(v).cuda() for n, v in p.items()}
        p["ic"] = torch.empty(X.shape[:2], dtype=torch.float64, device="cuda")
        p["corr"] = torch.empty((F, F), dtype=torch.float64, device="cuda")
        panels.append(p)
    fcb200.Batch(panels, min_valid=2).run()
    torch.cuda.synchronize()
    for k, p in enumerate(panels):
        X, m = np.moveaxis(p["X"].cpu().numpy(), 0, -1), p["fmask"].cpu().numpy() != 0
        one = run(X, m, 1)
        assert np.array_equal(p["corr"].cpu().numpy().view(np.uint64), one.view(np.uint64)), k
        assert corr_match(one, O.factor_corr(X, m)), k


# A correlation near 0.9 takes five roundings of its own, 0.29 ulps rms each; each of its three sums is exact to its
# last rounding and a third of one for the additions in the blocks: 0.65 and sqrt(1.5) * 0.39 = 0.48 ulps, 0.8 of
# 1.1e-16 in all.  A tenth is left for the mean and the 264 pairs.
@pytest.mark.parametrize("mean", [0.0, 5.0, 1000.0])
def test_precision_of_larger_pools(mean):
    sq = []
    for seed in range(4):
        r = np.random.default_rng(seed)
        T, N, F = 200, 1000, 12
        X = mean + np.sqrt(0.9) * r.standard_normal((T, N, 1)) + np.sqrt(0.1) * r.standard_normal((T, N, F))
        err = (run(X, None, 0).astype(np.longdouble) - exact(X))[np.triu_indices(F, 1)]
        sq.append(np.mean(err * err))
    assert np.sqrt(np.mean(sq)) < 1e-16


# 140000 rows of 16 independent f32 factors, correlations near 3e-3.  A staged chain of up to 158 rows is 9 on average
# and its additions are off by 0.29 ulps of that: 0.29 * 1.1e-16 * 9 / sqrt(140000) = 0.8e-18; twice that for the
# matrix instruction's own additions, and a tenth for the 480 pairs.
def test_precision_of_f32_staged_sums():
    sq = []
    for seed in range(4):
        X = np.random.default_rng(seed).standard_normal((200, 700, 16)).astype(np.float32)
        err = (run(X, None, 0).astype(np.longdouble) - exact(X))[np.triu_indices(16, 1)]
        sq.append(np.mean(err * err))
    assert np.sqrt(np.mean(sq)) < 1.75e-18
