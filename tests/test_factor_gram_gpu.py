"""factor_corr at the widths of the register Gram pass and just above, in both
layouts and both input types, against the oracle: few and many rows, partial
rows from none to most, constant and empty factors, offsets."""
import numpy as np
import pytest

from conftest import corr_match
from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu


def panel(T, N, F, miss, seed):
    r = np.random.default_rng(seed)
    X = r.standard_normal((T, N, F)).astype(np.float32)
    X[..., F // 2] += 0.5 * X[..., 0]
    if F > 2:
        X[..., 1] = np.exp(X[..., 1]) + 3.0
    if F > 4:
        X[..., 2] = 7.0
        X[..., 3] = 1000.0 + X[..., 3]
    X[r.random(X.shape) < miss] = np.nan
    if F > 6:
        X[..., 5] = np.inf
        X[..., 6][r.random((T, N)) < 0.9] = np.nan
    return X, r.random((T, N)) < 0.95


# a block takes rows in steps of 128 and its warps in steps of 32; the queue of partial rows is flushed from 65 on
@pytest.mark.parametrize("F", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12, 13])
def test_factor_corr_register_widths(F):
    from fcb200 import _native as nat
    import torch
    lib = nat.lib()
    ws = lib.fcb_workspace_create()
    try:
        for T, N, miss in ((1, 1, 0.0), (1, 33, 0.1), (3, 43, 0.5), (40, 700, 0.0), (41, 701, 0.01), (30, 1000, 0.3)):
            X, m = panel(T, N, F, miss, 100 * F + T)
            for dtype in (np.float32, np.float64):
                for mask in (m, None):
                    exp = O.factor_corr(X.astype(dtype), mask)
                    rows = X.astype(dtype)
                    dM = None if mask is None else torch.from_numpy(mask.astype(np.uint8)).cuda()
                    got = []
                    for planes, arr in ((0, rows), (1, np.ascontiguousarray(np.moveaxis(rows, -1, 0)))):
                        dX = torch.from_numpy(arr).cuda()
                        dO = torch.empty((F, F), dtype=torch.float64, device="cuda")
                        torch.cuda.synchronize()
                        nat.check(lib.fcb_dev_factor_corr(dX.data_ptr(), 0 if dtype == np.float32 else 1,
                                                          None if dM is None else dM.data_ptr(), T, N, F, planes,
                                                          dO.data_ptr(), ws, None), "factor_corr")
                        torch.cuda.synchronize()
                        got.append(dO.cpu().numpy())
                    assert corr_match(got[0], exp), (T, N, F, miss, dtype, mask is None)
                    assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64)) or F == 1
    finally:
        lib.fcb_workspace_destroy(ws)
