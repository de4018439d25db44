"""A backprojection tile one of whose copies never arrives (GPU, no GPU fault).

ctb_selftest_bounded_wait runs one tile whose fourth stage of angles is left out.
The warps give up at different times and places, and the block has barriers of its
own behind that stage, so it ends only if no warp decides from the stage's stale
data which barriers come next. The call reports the tile's timeout beside the plain
barrier's (codes 1 and 16) within a few limits, and the context computes as before.
"""
import time

import numpy as np
import pytest

import oracle as O
import qtctreconstruction_b200 as ctb
from qtctreconstruction_b200 import FilterType

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit_us", [1, 50, 20000])
def test_lost_copy_ends_the_block(backend, limit_us):
    import torch
    n, depth, na = 96, 8, 90
    sinos = np.random.default_rng(1).uniform(0.0, 1.0, (depth, na, ctb.odd_detector_count(n))).astype(np.float32)
    for _ in range(3):
        t0 = time.perf_counter()
        assert backend.selftest_bounded_wait(limit_us) == ctb.STATUS_TIMEOUT
        assert time.perf_counter() - t0 < 2.0
        assert "(code 17)" in backend._lib.ctb_last_error(backend.handle).decode()
    d_s = torch.from_numpy(sinos).cuda()
    d_o = torch.full((depth, n, n), float("nan"), device="cuda")
    backend.fbp_d(d_s.data_ptr(), *sinos.shape, n, int(FilterType.Ramp), d_o.data_ptr())
    backend.synchronize()
    for z in (0, depth - 1):
        ref = O.reconstruct_slice_f64(sinos[z], O.uniform_angles_deg(na), n, int(FilterType.Ramp))
        assert O.rel_l2(d_o[z].cpu().numpy(), ref) <= 1e-5
