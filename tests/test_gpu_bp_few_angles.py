"""Backprojection of few angles on the GPU: a kernel without the columns.

Angle counts around its chunks of 32 and around the limits of its rule (24, 40 and
64, by how far the tiles fill the SMs), tiles that leave a part empty, outputs past
the detector and batches that mix both kernels, at the parity bar of the
backprojector against the oracle (its float path where the output reaches past the
detector: which taps exist at a detector edge is decided in float); and that the rule takes the faster kernel where few angles
are spread over all the columns' groups.
"""
import numpy as np
import pytest

import oracle as O
import qtctreconstruction_b200 as ctb
from qtctreconstruction_b200 import FilterType

pytestmark = pytest.mark.gpu

ANGLES = [1, 2, 24, 25, 31, 33, 40, 41, 64, 65]


def _check(got, sinos, n):
    ang = O.uniform_angles_deg(sinos.shape[1])
    assert np.all(np.isfinite(got))
    oracle = O.reconstruct_slice_f32 if n > 2 * sinos.shape[2] else O.reconstruct_slice_f64
    for z in {0, len(sinos) - 1}:
        ref = oracle(sinos[z], ang, n, int(FilterType.SheppLogan))
        assert O.rel_l2(got[z], ref) <= 1e-5
        assert O.max_abs_rel(got[z], ref) <= 1e-4


@pytest.mark.parametrize("na", ANGLES)
@pytest.mark.parametrize("n,bins,depth", [(7, 11, 1), (33, 49, 5), (97, 41, 4), (130, 185, 47), (200, 285, 64)])
def test_parity(backend, n, bins, depth, na):
    import torch
    sinos = np.random.default_rng(n + na).uniform(0.0, 1.0, (depth, na, bins)).astype(np.float32)
    d_s = torch.from_numpy(sinos).cuda()
    d_o = torch.full((depth, n, n), float("nan"), device="cuda")
    backend.fbp_d(d_s.data_ptr(), depth, na, bins, n, int(FilterType.SheppLogan), d_o.data_ptr())
    backend.synchronize()
    _check(d_o.cpu().numpy(), sinos, n)


@pytest.mark.parametrize("flags", [0, ctb.BATCH_GRAPH, ctb.BATCH_PERSISTENT, ctb.BATCH_PER_JOB])
def test_batches_equal_single_calls(backend, flags):
    import torch
    jobs, args = [], []
    for n, depth, na in ((64, 5, 16), (64, 5, 120), (128, 16, 60), (128, 16, 150), (160, 33, 24), (160, 33, 130), (40, 9, 1),
                         (300, 64, 24)):
        bins = ctb.odd_detector_count(n)
        s = torch.from_numpy(np.random.default_rng(n + na).uniform(0.0, 1.0, (depth, na, bins)).astype(np.float32)).cuda()
        o, alone = (torch.full((depth, n, n), float("nan"), device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        backend.fbp_d(s.data_ptr(), depth, na, bins, n, int(FilterType.Ramp), alone.data_ptr())
        jobs.append((s, o, alone))
        args.append(dict(sino=s.data_ptr(), depth=depth, num_angles=na, bins=bins, output_size=n,
                         filter=int(FilterType.Ramp), out=o.data_ptr()))
    with backend.batch(args, flags) as b:
        for _ in range(2):
            b.run()
        backend.synchronize()
    for _, o, alone in jobs:
        np.testing.assert_array_equal(o.cpu().numpy(), alone.cpu().numpy())


def test_denormalised_volume_meets_parity(backend):
    import torch
    n, depth, na = 64, 6, 20
    nd = ctb.odd_detector_count(n)
    vol = backend.phantom(ctb.phantom_params(9, 6), n, n, depth)
    d_v = torch.from_numpy(vol).cuda()
    d_o = torch.full_like(d_v, float("nan"))
    backend.reconstruct_volume_d(d_v.data_ptr(), n, depth, na, nd, int(FilterType.Ramp), d_o.data_ptr())
    backend.synchronize()
    ref = O.reconstruct_volume_f32(vol, na, nd, O.RAMP)
    assert O.rel_l2(d_o.cpu().numpy(), ref) <= 1e-5


@pytest.mark.parametrize("convention", [ctb.CONVENTION_SERIAL, ctb.CONVENTION_CUDA])
@pytest.mark.parametrize("n,bins,na", [(64, 91, 20), (90, 40, 33)])
def test_conventions_equal_the_columns(backend, convention, n, bins, na):
    """Both conventions' grids and tap rules, against the columns (shape 3)."""
    import torch
    sinos = torch.from_numpy(np.random.default_rng(na).uniform(0.0, 1.0, (5, na, bins)).astype(np.float32)).cuda()
    outs = []
    backend.set_convention(convention)
    try:
        for shape in (-1, 3):
            backend.set_bp_shape(shape)
            o = torch.full((5, n, n), float("nan"), device="cuda")
            torch.cuda.synchronize()
            backend.fbp_d(sinos.data_ptr(), 5, na, bins, n, int(FilterType.Hann), o.data_ptr())
            backend.synchronize()
            outs.append(o.cpu().numpy())
    finally:
        backend.set_bp_shape(-1)
        backend.set_convention(ctb.CONVENTION_SERIAL)
    assert np.all(np.isfinite(outs[0]))
    assert O.rel_l2(outs[0], outs[1]) <= 1e-5
    assert O.max_abs_rel(outs[0], outs[1]) <= 1e-4


def test_few_angles_are_not_slower_than_the_columns(backend):
    """8 angles over 512^2 x 4 are 8 of the columns' groups: 15 us a call in columns, 12
    without. The automatic choice, timed in turn with the forced shapes, is at least a
    tenth faster than each."""
    import torch
    n, depth, na = 512, 4, 8
    bins = ctb.odd_detector_count(n)
    s, o = torch.rand(depth, na, bins, device="cuda"), torch.empty(depth, n, n, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    best = {}
    backend.set_stream(stream.cuda_stream)
    try:
        for _ in range(100):  # the first rounds also bring the clocks up
            for shape in (-1, 0, 2, 3):
                backend.set_bp_shape(shape)
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record(stream)
                for _ in range(20):
                    backend.fbp_d(s.data_ptr(), depth, na, bins, n, int(FilterType.Ramp), o.data_ptr())
                b.record(stream)
                b.synchronize()
                best[shape] = min(best.get(shape, 1e9), a.elapsed_time(b))
    finally:
        backend.set_bp_shape(-1)
        backend.synchronize()
        backend.set_stream(0)
    assert best[-1] <= 0.9 * min(best[shape] for shape in (0, 2, 3)), best
