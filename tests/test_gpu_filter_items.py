"""The packed filter's items per CTA on the GPU.

Below length 512 several (slice group, angle) items share a warp; item counts
that leave a CTA part empty, slice counts that leave a group part empty and the
smallest rows of every length must meet the parity bar against the FP64 oracle.
"""
import numpy as np
import pytest

import oracle as O
from qtctreconstruction_b200 import FilterType

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,na", [(1, 1), (2, 3), (5, 7), (9, 5)])
@pytest.mark.parametrize("bins,length", [(3, 64), (26, 64), (28, 128), (53, 128), (54, 256), (106, 256), (107, 512)])
def test_items_meet_parity(backend, bins, length, depth, na):
    import torch
    sq = O.pad_geometry(bins)[0]
    assert max(64, 1 << (sq + bins - 2).bit_length()) == length
    n = max(2, bins // 2)
    rng = np.random.default_rng(bins + depth)
    sinos = rng.uniform(0.0, 1.0, (depth, na, bins)).astype(np.float32)
    ang = O.uniform_angles_deg(na)
    d_s = torch.from_numpy(sinos).cuda()
    d_o = torch.full((depth, n, n), float("nan"), device="cuda")
    backend.fbp_d(d_s.data_ptr(), depth, na, bins, n, int(FilterType.Hann), d_o.data_ptr())
    backend.synchronize()
    got = d_o.cpu().numpy()
    for z in range(depth):
        ref = O.reconstruct_slice_f64(sinos[z], ang, n, int(FilterType.Hann))
        assert O.rel_l2(got[z], ref) <= 1e-5
        assert O.max_abs_rel(got[z], ref) <= 1e-4
