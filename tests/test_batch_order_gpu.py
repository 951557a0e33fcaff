"""The batch's two orders, one kernel variant after another and side by side,
with panels in every variant (two of them in some): ranks, IC and factor
correlations are those of the oracle, run after run."""
import numpy as np
import pytest

from conftest import bitwise_f32, corr_match
from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu

WIDTHS = (60, 300, 512, 700, 1000, 1400, 2000, 3000, 5000, 7000, 9000, 250)


@pytest.mark.parametrize("concurrent", [0, 1])
def test_every_variant(concurrent):
    import torch

    import fcb200
    r = np.random.default_rng(concurrent)
    panels = []
    for N in WIDTHS:
        X = r.standard_normal((3, 7, N)).astype(np.float32)
        X[r.random(X.shape) < 0.03] = np.nan
        p = {"X": X, "R": r.standard_normal((7, N)).astype(np.float32), "fmask": (r.random((7, N)) < 0.95).astype(np.uint8)}
        p = {k: torch.from_numpy(v).cuda() for k, v in p.items()}
        p["ranks"] = torch.empty_like(p["X"])
        p["ic"] = torch.empty((3, 7), dtype=torch.float64, device="cuda")
        p["corr"] = torch.empty((3, 3), dtype=torch.float64, device="cuda")
        panels.append(p)
    b = fcb200.Batch(panels, min_valid=2, config={"concurrent": concurrent})
    for _ in range(3):
        for p in panels:
            p["ranks"].zero_(), p["ic"].zero_(), p["corr"].zero_()
        b.run()
        torch.cuda.synchronize()
        for p in panels:
            X, R, m = (p[k].cpu().numpy() for k in ("X", "R", "fmask"))
            m = m != 0
            for f in range(3):
                assert bitwise_f32(p["ranks"][f].cpu().numpy(), O.cs_rank(X[f], m, False)), X.shape
                assert np.array_equal(p["ic"][f].cpu().numpy(), O.rolling_ic(X[f], R, m, None, 2), equal_nan=True), X.shape
            assert corr_match(p["corr"].cpu().numpy(), O.factor_corr(np.moveaxis(X, 0, -1), m)), X.shape
