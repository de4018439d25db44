"""Device memory of a host-buffer volume with very many angles (GPU).

A slice of 16^2 pixels with 20000 angles of 1001 bins takes 0.28 GB of sinogram and
filtered rows: the call holds slabs of a sixteenth of the 256 slices, not of a third.
"""
import numpy as np
import pytest

import qtctreconstruction_b200 as ctb
from qtctreconstruction_b200 import FilterType

pytestmark = pytest.mark.gpu


def test_scratch_of_many_angles():
    import torch
    n, depth, na, bins = 16, 256, 20000, 1001
    vol = torch.from_numpy(np.random.default_rng(0).uniform(0.0, 1.0, (depth, n, n)).astype(np.float32)).pin_memory()
    out = torch.full_like(vol, float("nan")).pin_memory()
    with ctb.B200Backend(0) as be:
        be.synchronize()
        before = torch.cuda.mem_get_info()[0]
        be.reconstruct_volume_host(vol.data_ptr(), n, depth, na, bins, int(FilterType.Ramp), out.data_ptr())
        used = before - torch.cuda.mem_get_info()[0]
    assert np.all(np.isfinite(out.numpy()))
    # two sinogram buffers and the filtered rows (at most 2 bins + 120 each) of 16 slices, and 1 GB for the rest
    assert used <= 16 * 4 * na * (2 * bins + 2 * bins + 120) + 2 ** 30
