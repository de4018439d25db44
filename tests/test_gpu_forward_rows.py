"""The forward projector's blocks of 32 prepared rows on the GPU.

Image heights around the blocks' and the 8-row groups' ends, non-zero regions
that leave rows, groups and whole blocks out, and slice counts around the 8
slices a warp holds, with the non-zero bounds on and off, against the FP64
oracle at the projector's parity bar.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bounds", [True, False])
@pytest.mark.parametrize("n,depth", [(7, 1), (31, 9), (33, 2), (64, 8), (71, 17)])
@pytest.mark.parametrize("region", ["full", "one_pixel", "corner", "two_bands"])
def test_rows_meet_parity(backend, region, n, depth, bounds):
    import torch
    rng = np.random.default_rng(n + depth)
    vol = rng.uniform(0.5, 1.5, (depth, n, n)).astype(np.float32)
    keep = np.zeros((n, n), bool)
    if region == "full":
        keep[:] = True
    elif region == "one_pixel":
        keep[n // 2, n // 3] = True
    elif region == "corner":
        keep[: max(1, n // 8), n - max(1, n // 8):] = True
    else:
        keep[n // 9, :] = keep[n - 1 - n // 7, n // 2:] = True
    vol[:, ~keep] = 0.0
    na, nd = 23, (3 * n) // 2 + 1
    ang = (np.arange(na) * 111.246117975 % 180.0).astype(np.float32)
    d_v = torch.from_numpy(vol).cuda()
    d_s = torch.full((depth, na, nd), float("nan"), device="cuda")
    d_st = torch.empty(depth, 4, device="cuda")
    backend.set_forward_bounds(bounds)
    try:
        backend.forward_d(d_v.data_ptr(), n, depth, na, nd, d_s.data_ptr(), d_st.data_ptr(), ang)
        backend.synchronize()
    finally:
        backend.set_forward_bounds(True)
    got = d_s.cpu().numpy()
    for z in range(depth):
        ref = O.sinogram_f64(vol[z], na, nd, ang)[0]
        assert np.all(np.isfinite(got[z]))
        assert np.linalg.norm(got[z] - ref) <= 1e-5 * max(np.linalg.norm(ref), 1e-30) + 1e-12


@pytest.mark.parametrize("w,h", [(1, 1), (5, 40), (64, 33), (97, 70)])
@pytest.mark.parametrize("nd_of", ["width", "two", "wide"])
def test_single_slice_meets_parity(backend, w, h, nd_of):
    """A call's only slice has planes and a walk of its own: rectangular images,
    detectors that cut the image and that reach past it, and a call of another
    size in between (the planes' zero borders)."""
    rng = np.random.default_rng(w * h)
    img = rng.uniform(-1.0, 1.0, (h, w)).astype(np.float32)
    img[rng.uniform(size=(h, w)) < 0.3] = 0.0
    nd = {"width": max(w, 2), "two": 2, "wide": 2 * max(w, h) + 3}[nd_of]
    na = 31
    first = backend.computeSinogram(img, na, nd)
    backend.computeSinogram(np.ones((h + 3, w + 2), np.float32), na, nd + 1)
    again = backend.computeSinogram(img, na, nd)
    np.testing.assert_array_equal(first.data, again.data)
    ref = O.sinogram_f32(img, na, nd)[0]
    assert np.linalg.norm(first.data - ref) <= 1e-5 * max(np.linalg.norm(ref), 1e-30) + 1e-12


@pytest.mark.parametrize("nd", [640, 1283])
@pytest.mark.parametrize("depth", [1, 3])
def test_angles_next_to_an_axis(backend, depth, nd):
    """Angles a float step (and much less) away from an axis: the rows where a strip
    meets a column far away do not fit an int. At an even n and these angles s lies
    half way between bins, so the float rules of the outer bins are not at an edge."""
    import torch
    n = 640
    rng = np.random.default_rng(depth)
    vol = rng.uniform(0.5, 1.5, (depth, n, n)).astype(np.float32)
    near = np.float32(90.0)
    ang = np.array([np.nextafter(near, np.float32(0)), near, np.nextafter(near, np.float32(180)), 1e-30, 1e-5,
                    np.nextafter(np.float32(180), np.float32(0)), 37.0], np.float32)
    d_v = torch.from_numpy(vol).cuda()
    d_s = torch.full((depth, len(ang), nd), float("nan"), device="cuda")
    d_st = torch.empty(depth, 4, device="cuda")
    backend.forward_d(d_v.data_ptr(), n, depth, len(ang), nd, d_s.data_ptr(), d_st.data_ptr(), ang)
    backend.synchronize()
    got = d_s.cpu().numpy()
    for z in range(depth):
        ref = O.sinogram_f64(vol[z], len(ang), nd, ang)[0]
        for k in range(len(ang)):
            assert np.linalg.norm(got[z, k] - ref[k]) <= 1e-5 * np.linalg.norm(ref[k]), (z, ang[k])
