"""The learned entry point's two routes -- value-spread buckets without
statistics, the learned buckets with them -- and a batch whose panels carry a
model: ranks and IC are the oracle's in each, and only the learned buckets
write statistics."""
import numpy as np
import pytest

from conftest import bitwise_f32
from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu


def panel(T, N, F, seed):
    r = np.random.default_rng(seed)
    X = r.standard_normal((F, T, N)).astype(np.float32)
    X[0] = np.exp(X[0])
    X[r.random(X.shape) < 0.02] = np.nan
    k = r.random(X.shape) < 0.05
    X[k] = np.round(X[k], 2)
    X[-1, 1] = 0.5                                  # a constant section
    R = (0.1 * np.nan_to_num(X[0]) + r.standard_normal((T, N))).astype(np.float32)
    return X, R, r.random((T, N)) < 0.95, r.random((T, N)) < 0.97


def fitted(X, fm):
    import torch

    import fcb200
    F, T, N = X.shape
    ranks = torch.from_numpy(np.stack([O.cs_rank(x, fm, False) for x in X])).cuda()
    model = fcb200.CdfModel(F, seed=3)
    model.fit(torch.from_numpy(X).cuda(), ranks, T, N, 0, T, steps=200, lr=3e-3)
    torch.cuda.synchronize()
    return model


def matches(X, R, fm, rm, ranks, ic):
    for f in range(len(X)):
        assert bitwise_f32(ranks[f], O.cs_rank(X[f], fm, False)), (X.shape, f)
        assert np.array_equal(ic[f], O.rolling_ic(X[f], R, fm, rm, 2), equal_nan=True), (X.shape, f)


# widths on each side of the one-factor learned kernel's and of a section's largest block
@pytest.mark.parametrize("F,N", [(1, 700), (1, 5000), (1, 12000), (3, 700), (3, 5000), (3, 12000), (2, 17000)])
@pytest.mark.parametrize("with_stats", [False, True])
def test_entry_point(F, N, with_stats):
    import torch
    from fcb200 import _native as nat
    T = 6
    X, R, fm, rm = panel(T, N, F, N + F)
    model = fitted(X, fm)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (X, R, fm.astype(np.uint8), rm.astype(np.uint8))]
    ranks, ic = torch.full((F, T, N), -1.0, device="cuda"), torch.full((F, T), -1.0, dtype=torch.float64, device="cuda")
    stats = torch.full((F, T, 4), -7, dtype=torch.int32, device="cuda")
    nat.check(nat.lib().fcb_dev_rank_ic_panel_learned(
        *[a.data_ptr() for a in d], F, T, N, 2, ranks.data_ptr(), ic.data_ptr(), model.handle, 0,
        stats.data_ptr() if with_stats else None, torch.cuda.current_stream().cuda_stream), "learned")
    matches(X, R, fm, rm, ranks.cpu().numpy(), ic.cpu().numpy())
    assert bool((stats == -7).all()) is not with_stats


def test_batch_with_models():
    import torch

    import fcb200
    panels, host = [], []
    for N, F in ((700, 3), (5000, 2), (900, 1)):
        X, R, fm, rm = panel(6, N, F, N)
        p = {"X": X, "R": R, "fmask": fm.astype(np.uint8), "rmask": rm.astype(np.uint8)}
        p = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in p.items()}
        p["model"] = fitted(X, fm)
        p["ranks"] = torch.empty_like(p["X"])
        p["ic"] = torch.empty((F, 6), dtype=torch.float64, device="cuda")
        panels.append(p)
        host.append((X, R, fm, rm))
    b = fcb200.Batch(panels, min_valid=2)
    for run in (b.run, b.run_per_panel):
        for p in panels:
            p["ranks"].zero_(), p["ic"].zero_()
        run()
        torch.cuda.synchronize()
        for p, h in zip(panels, host):
            matches(*h, p["ranks"].cpu().numpy(), p["ic"].cpu().numpy())
