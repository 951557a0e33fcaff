"""Device memory that the host cs_rank of wide rows holds: no sort scratch where
the rows are ranked by slices, and what the budget says in both forms."""
import ctypes as C

import numpy as np
import pytest

CS_RANK = 1


@pytest.fixture(scope="module")
def nat():
    import fcb_build
    fcb_build.build()
    from fcb200 import _native
    return _native


def budget(nat, T, N):
    out = C.c_uint64()
    assert nat.lib().fcb_memory_budget(CS_RANK, 0, T, N, 1, 0, C.byref(out)) == 0
    return out.value


def test_slices_need_no_scratch(nat):
    assert budget(nat, 5, 20000) == 2 * 4 * 5 * 20000 + 64
    assert budget(nat, 5, 100000) > 2 * 4 * 5 * 100000 + 64  # the global sort's pairs


@pytest.mark.gpu
@pytest.mark.parametrize("N", [16385, 20000, 100000])
def test_workspace_peak_is_the_budget(nat, N):
    T = 5
    x = np.random.default_rng(N).standard_normal((T, N)).astype(np.float32)
    out = np.empty_like(x)
    ws = nat.lib().fcb_workspace_create()
    try:
        nat.check(nat.lib().fcb_cs_rank_f32(nat.ptr(x), None, T, N, 0, nat.ptr(out), ws), "cs_rank")
        peak = C.c_uint64()
        nat.lib().fcb_workspace_stats(ws, C.byref(C.c_uint64()), C.byref(peak), C.byref(C.c_uint64()))
        assert peak.value == budget(nat, T, N)
    finally:
        nat.lib().fcb_workspace_destroy(ws)
