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
