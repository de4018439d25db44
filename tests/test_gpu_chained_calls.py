"""Calls queued back to back without a wait between them (GPU).

The kernels of a call start while the kernel before them, often the last one of the
call before, is still running, and wait inside for its results. Forward projections,
volumes and pairs of calls where one reads what the other wrote, with inputs that
change from call to call, must give the bits of calls that are waited for.
"""
import numpy as np
import pytest

import qtctreconstruction_b200 as ctb
from qtctreconstruction_b200 import FilterType

pytestmark = pytest.mark.gpu

KIND = int(FilterType.SheppLogan)


def _vols(n, depth, count):
    import torch
    r = np.random.default_rng(n + depth)
    out = []
    for k in range(count):
        v = r.uniform(-1.0, 1.0, (depth, n, n)).astype(np.float32)
        v[:, : (k + 1) * n // 8] = 0.0  # other non-zero bounds each time
        out.append(torch.from_numpy(v).cuda())
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("n,depth,na", [(64, 1, 45), (64, 9, 90), (160, 1, 180), (192, 16, 120)])
def test_forward(backend, n, depth, na):
    import torch
    nd = ctb.odd_detector_count(n)
    vols = _vols(n, depth, 4)

    def run(wait):
        outs = []
        for k in range(12):
            s = torch.full((depth, na, nd), float("nan"), device="cuda")
            st = torch.full((depth, 4), float("nan"), device="cuda")
            outs.append((s, st))
        torch.cuda.synchronize()
        for k, (s, st) in enumerate(outs):
            backend.forward_d(vols[k % 4].data_ptr(), n, depth, na, nd, s.data_ptr(), st.data_ptr())
            if wait:
                backend.synchronize()
        backend.synchronize()
        return [(s.cpu().numpy(), st.cpu().numpy()) for s, st in outs]

    for (s, st), (s1, st1) in zip(run(False), run(True)):
        np.testing.assert_array_equal(s, s1)
        np.testing.assert_array_equal(st, st1)


@pytest.mark.parametrize("n,depth,na", [(64, 1, 45), (64, 16, 90), (160, 5, 180)])
def test_volumes(backend, n, depth, na):
    import torch
    nd = ctb.odd_detector_count(n)
    vols = _vols(n, depth, 4)

    def run(wait):
        outs = [torch.full((depth, n, n), float("nan"), device="cuda") for _ in range(12)]
        torch.cuda.synchronize()
        for k, o in enumerate(outs):
            backend.reconstruct_volume_d(vols[k % 4].data_ptr(), n, depth, na, nd, KIND, o.data_ptr())
            if wait:
                backend.synchronize()
        backend.synchronize()
        return [o.cpu().numpy() for o in outs]

    for o, o1 in zip(run(False), run(True)):
        np.testing.assert_array_equal(o, o1)


@pytest.mark.parametrize("n,depth,na", [(64, 1, 45), (64, 16, 90), (128, 8, 100), (48, 9, 20)])
def test_a_call_reads_what_the_call_before_wrote(backend, n, depth, na):
    """Project, reconstruct, project the reconstruction ...: one buffer each way."""
    import torch
    nd = ctb.odd_detector_count(n)
    vol = _vols(n, depth, 1)[0]

    def run(wait):
        v, s = vol.clone(), torch.full((depth, na, nd), float("nan"), device="cuda")
        st = torch.full((depth, 4), float("nan"), device="cuda")
        torch.cuda.synchronize()
        for _ in range(6):
            backend.forward_d(v.data_ptr(), n, depth, na, nd, s.data_ptr(), st.data_ptr())
            if wait:
                backend.synchronize()
            backend.fbp_d(s.data_ptr(), depth, na, nd, n, KIND, v.data_ptr())
            if wait:
                backend.synchronize()
        backend.synchronize()
        return s.cpu().numpy(), v.cpu().numpy()

    for got, ref in zip(run(False), run(True)):
        assert np.all(np.isfinite(got))
        np.testing.assert_array_equal(got, ref)
