"""Device entry points whose output is written over their input of the same
type and shape: the results are those of separate buffers."""
import numpy as np
import pytest

from conftest import bitwise_f32
from oracle import fc_oracle as O
from test_section_rank_gpu import stress_rows

pytestmark = pytest.mark.gpu


# one CTA a row, slices of a row (and what takes their place in place), the global sort
@pytest.mark.parametrize("N", [5000, 16384, 16385, 20000, 40001, 65537])
def test_cs_rank_in_place(N):
    import torch
    from fcb200 import _native as nat
    X = stress_rows(N, N)
    mask = np.random.default_rng(N).random(X.shape) < 0.9
    for m in (mask, None):
        for desc in (0, 1):
            d = torch.from_numpy(X).cuda()
            dm = None if m is None else torch.from_numpy(m.astype(np.uint8)).cuda()
            nat.check(nat.lib().fcb_dev_cs_rank_f32(d.data_ptr(), None if dm is None else dm.data_ptr(), len(X), N, desc,
                                                    d.data_ptr(), torch.cuda.current_stream().cuda_stream), "cs_rank")
            assert bitwise_f32(d.cpu().numpy(), O.cs_rank(X, m, bool(desc))), (N, m is None, desc)


def tied(N, dt):
    """Factors that are constant on the joint cells only, tied, smooth; and a returns row each."""
    r = np.random.default_rng(N)
    z = r.standard_normal((6, N))
    f = np.where(r.random((6, N)) < 0.5, 2.5, z)
    f[1] = np.round(z[1], 1)
    f[2] = z[2]
    ret = 0.02 * r.standard_t(3, (6, N))
    ret[:4][(f != 2.5)[:4]] = np.nan           # dates 0 and 3: one factor value where returns are
    ret[1:3] = 0.02 * r.standard_t(3, (2, N))
    ret[4] = np.where(f[4] == 2.5, 0.01, np.nan)  # the returns are constant too
    return f.astype(dt), ret.astype(dt)


@pytest.mark.parametrize("N", [60, 1000, 5000, 9000])
def test_rolling_ic_in_place(N):
    import torch
    from fcb200 import _native as nat
    f, r = tied(N, np.float64)
    ic, rf, rr = O.rolling_ic(f, r, None, None, 2, return_ranks=True)
    df, dr = torch.from_numpy(f).cuda(), torch.from_numpy(r).cuda()
    dic = torch.empty(len(f), dtype=torch.float64, device="cuda")
    nat.check(nat.lib().fcb_dev_rolling_ic(df.data_ptr(), 1, dr.data_ptr(), 1, None, None, len(f), N, 2, dic.data_ptr(),
                                           df.data_ptr(), dr.data_ptr(), torch.cuda.current_stream().cuda_stream), "ic")
    assert np.isnan(ic[[0, 3, 4]]).all() and np.isfinite(ic[[1, 2, 5]]).all()
    assert np.array_equal(dic.cpu().numpy(), ic, equal_nan=True), N
    assert np.array_equal(df.cpu().numpy(), rf) and np.array_equal(dr.cpu().numpy(), rr), N


# one factor, several factors
@pytest.mark.parametrize("F", [1, 3])
@pytest.mark.parametrize("N", [60, 1000, 5000, 16384])
def test_panel_in_place(N, F):
    import torch
    from fcb200 import _native as nat
    f, r = tied(N, np.float32)
    X = np.stack([f] * F)
    dX, dr = torch.from_numpy(X).cuda(), torch.from_numpy(r).cuda()
    dic = torch.empty((F, len(f)), dtype=torch.float64, device="cuda")
    nat.check(nat.lib().fcb_dev_rank_ic_panel(dX.data_ptr(), dr.data_ptr(), None, None, F, len(f), N, 2, dX.data_ptr(),
                                              dic.data_ptr(), 0, torch.cuda.current_stream().cuda_stream), "panel")
    ic = O.rolling_ic(f, r, None, None, 2)
    for k in range(F):
        assert bitwise_f32(dX[k].cpu().numpy(), O.cs_rank(f, None, False)), (N, k)
        assert np.array_equal(dic[k].cpu().numpy(), ic, equal_nan=True), (N, k)
