"""The backprojector's angle groups, column patterns and slice pairs on the GPU.

A tile walks the angles grouped by the axis along which the detector
coordinate changes least, that coefficient's sign and its size, in columns of
four voxels; angle lists that leave groups empty, lie on the groups' limits or
repeat must meet the parity bar against the oracle, also where the output
reaches past the detector (there against its float path: which taps exist at a
detector edge is decided by SerialBackend's own float coordinate). Two slice groups share an item's weights where the
launch is large enough; a slice's bits must not depend on it.
"""
import numpy as np
import pytest

import oracle as O
import qtctreconstruction_b200 as ctb
from qtctreconstruction_b200 import FilterType

pytestmark = pytest.mark.gpu

ANGLES = {
    "one": [33.0],
    "axes": [0.0, 90.0, 180.0, 270.0],
    "along_x_only": np.linspace(50.0, 130.0, 37),
    "along_y_only": np.linspace(-40.0, 40.0, 41),
    "limits": [45.0, 135.0, 225.0, -45.0, 30.0, 150.0, 60.0, 120.0, 19.4712206, 70.5287794, 41.8103149, 48.1896851],
    "unordered": (np.arange(97) * 111.246117975) % 360.0,
}


def _fbp(backend, sinos, angles, n, shape=-1):
    import torch
    d_s = torch.from_numpy(sinos).cuda()
    d_o = torch.full((sinos.shape[0], n, n), float("nan"), dtype=torch.float32, device="cuda")
    backend.set_bp_shape(shape)
    try:
        backend.fbp_d(d_s.data_ptr(), *sinos.shape, n, int(FilterType.SheppLogan), d_o.data_ptr(), angles_deg=angles)
        backend.synchronize()
    finally:
        backend.set_bp_shape(-1)
    return d_o.cpu().numpy()


@pytest.mark.parametrize("shape", [0, 1, 2, 3])
@pytest.mark.parametrize("n,bins", [(33, 49), (64, 64), (97, 41)])
@pytest.mark.parametrize("name", sorted(ANGLES))
def test_angle_groups_meet_parity(backend, name, n, bins, shape):
    ang = np.asarray(ANGLES[name], np.float32)
    rng = np.random.default_rng(n + bins)
    sinos = rng.uniform(0.0, 1.0, (2, len(ang), bins)).astype(np.float32)
    got = _fbp(backend, sinos, ang, n, shape)
    oracle = O.reconstruct_slice_f32 if n > 2 * bins else O.reconstruct_slice_f64
    for z in range(2):
        ref = oracle(sinos[z], ang, n, int(FilterType.SheppLogan))
        assert O.rel_l2(got[z], ref) <= 1e-5
        assert O.max_abs_rel(got[z], ref) <= 1e-4


@pytest.mark.parametrize("shape", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("depth", [5, 8, 13])
def test_slice_pairs_do_not_change_bits(backend, depth, shape):
    """A deep stack (items of two slice groups, with and without a remainder)
    equals its last slices reconstructed in stacks of one group (the filter
    transforms the slices of a group in pairs, so groups stay whole)."""
    n, na = 500, 61
    rng = np.random.default_rng(depth)
    sinos = rng.uniform(0.0, 1.0, (depth, na, n)).astype(np.float32)
    ang = O.uniform_angles_deg(na)
    deep = _fbp(backend, np.concatenate([sinos[:4]] * 8 + [sinos]), ang, n, shape)[32:]
    for z in range(0, depth, 4):
        np.testing.assert_array_equal(deep[z:min(z + 4, depth)], _fbp(backend, sinos[z:z + 4], ang, n, shape))


@pytest.mark.parametrize("shape", [0, 2, 3])
@pytest.mark.parametrize("n,depth", [(387, 1), (387, 8), (387, 16), (200, 8)])
def test_fewer_ctas_per_sm_than_fit(backend, n, depth, shape):
    """Launches whose tiles inside the circle need one or two CTAs per SM while there
    are more tiles than that: every tile, inside or outside, is still written."""
    na, bins = 7, ctb.odd_detector_count(n)
    rng = np.random.default_rng(n + depth)
    sinos = rng.uniform(0.0, 1.0, (depth, na, bins)).astype(np.float32)
    ang = O.uniform_angles_deg(na)
    got = _fbp(backend, sinos, ang, n, shape)
    assert np.all(np.isfinite(got))
    for z in {0, depth - 1}:
        ref = O.reconstruct_slice_f64(sinos[z], ang, n, int(FilterType.SheppLogan))
        assert O.rel_l2(got[z], ref) <= 1e-5
        assert O.max_abs_rel(got[z], ref) <= 1e-4


@pytest.mark.parametrize("n,depth,na", [(64, 16, 101), (128, 32, 45), (387, 8, 13)])
def test_queued_calls_equal_calls_alone(backend, n, depth, na):
    """Small launches start in the tail of the filter: calls queued back to back, which
    share the filtered rows, give the bits of calls that are waited for."""
    import torch
    bins, ang = ctb.odd_detector_count(n), O.uniform_angles_deg(na)
    rng = np.random.default_rng(n)
    sinos = [rng.uniform(0.0, 1.0, (depth, na, bins)).astype(np.float32) for _ in range(4)]
    alone = [_fbp(backend, s, ang, n) for s in sinos]
    d_s = [torch.from_numpy(s).cuda() for s in sinos]
    d_o = [torch.full((depth, n, n), float("nan"), device="cuda") for _ in range(12)]
    torch.cuda.synchronize()
    for k, o in enumerate(d_o):
        backend.fbp_d(d_s[k % 4].data_ptr(), depth, na, bins, n, int(FilterType.SheppLogan), o.data_ptr(), angles_deg=ang)
    backend.synchronize()
    for k, o in enumerate(d_o):
        np.testing.assert_array_equal(o.cpu().numpy(), alone[k % 4])
