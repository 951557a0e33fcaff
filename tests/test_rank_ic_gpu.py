"""Rank + IC of one factor row against one returns row (f32 and f64), and of
several factors per date, against the oracle, bit for bit: at the widths where
the kernel variants begin and end and on rows that stress the bucket map."""
import numpy as np
import pytest

from conftest import bitwise_f32
from oracle import fc_oracle as O
from test_section_rank_gpu import stress_rows

pytestmark = pytest.mark.gpu


def wide_rows(N, seed):
    """f64 rows whose order f32 keys do not settle: near ties (few to all), values beyond the f32 range."""
    r = np.random.default_rng(seed)
    z = r.standard_normal(N)
    some = z.copy()
    some[r.random(N) < 0.02] = 0.1
    k = r.random(N) < 0.02
    some[k] = 0.1 + 1e-12 * z[k]
    big = z * 1e300
    big[:: 3] = z[:: 3]
    tiny = z * 1e-300
    tiny[:: 2] = z[:: 2]
    rows = [z, some, 1.0 + 1e-12 * z, np.round(z, 2) + 1e-13 * r.integers(0, 3, N), big, tiny, z * 1e-60, z * 1e-310]
    X = np.array(rows)
    X[:, r.random(N) < 0.05] = np.nan
    return X


def same_ic(a, b):
    return np.array_equal(a, b, equal_nan=True)


def pair(T, N, fdt, rdt):
    """Each date a factor row and a returns row of different kinds, masks with an empty and a full date."""
    rng = np.random.default_rng(T * 131 + N)
    rows = np.concatenate([stress_rows(N, N).astype(np.float64), wide_rows(N, N + 7)])
    f = rows[np.arange(T) % len(rows)].copy()
    r = rows[(np.arange(T) * 5 + 3 + np.arange(T) // len(rows)) % len(rows)].copy()
    r[1::4] = 0.02 * rng.standard_t(3, r[1::4].shape)
    fm, rm = rng.random((T, N)) < 0.9, rng.random((T, N)) < 0.97
    fm[2], rm[4] = False, True
    with np.errstate(over="ignore"):
        return f.astype(fdt), r.astype(rdt), fm, rm


# the two block-shape rules part at 148 sections; each width is an edge of a variant or of a quad
@pytest.mark.parametrize("T", [54, 152])
@pytest.mark.parametrize("N", [1, 3, 33, 1024, 1025, 2048, 4097, 5000, 5377, 8193])
def test_rolling_ic_stress_rows(N, T):
    from fcb200 import _native
    fcb = _native.fcb()
    for fdt, rdt in (("f4", "f4"), ("f8", "f8"), ("f4", "f8"), ("f8", "f4")):
        f, r, fm, rm = pair(T, N, fdt, rdt)
        for masks in ((fm, rm), (None, None)):
            ic, rf, rr = fcb.rolling_ic_f64(f, r, *masks, 2, return_ranks=True)
            ic_e, rf_e, rr_e = O.rolling_ic(f, r, *masks, 2, return_ranks=True)
            assert same_ic(ic, ic_e), (N, T, fdt, rdt, masks[0] is None)
            assert np.array_equal(rf, rf_e) and np.array_equal(rr, rr_e)


@pytest.mark.parametrize("N", [3, 1024, 1025, 3073, 5000, 8192, 16384])
def test_panel_stress_rows(N):
    import fcb200
    T = 27
    f0, r, fm, rm = pair(T, N, "f4", "f4")
    for F in (1, 3):
        X = np.stack([np.roll(f0, k, axis=0) for k in range(F)])
        for masks in ((fm, rm), (None, None)):
            ranks, ic = fcb200.rank_ic_panel(X, r, *masks, min_valid=2)
            for k in range(F):
                assert bitwise_f32(ranks[k], O.cs_rank(X[k], masks[0], False)), (N, F, k)
                assert same_ic(ic[k], O.rolling_ic(X[k], r, *masks, 2)), (N, F, k)
