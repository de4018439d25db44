"""A slice's bits do not depend on how its call was grouped (GPU).

The backprojector takes the angles of a tile in stages, one or two slice groups
at a time; which angles share a stage follows from the tile shape's ring and
from the pairing, which a launch chooses from all its work. Where the detector
does not cover a tile, some angles of a stage follow the reference's rule for
taps at the detector's ends and the others do not: their sums must not depend
on the company they are in. Sizes with such tiles (as many bins as pixels, or
fewer): deep stacks against their slice groups alone, the shapes that differ in
the ring only, host pipelines against one pass, batches and the server against
single calls.
"""
import numpy as np
import pytest

import qtctreconstruction_b200 as ctb
from qtctreconstruction_b200 import FilterType

pytestmark = pytest.mark.gpu

# output size, bins, angles
SIZES = [(128, 128, 180), (160, 160, 250), (100, 64, 400), (64, 64, 1000)]


def _sinos(n, depth, na, bins):
    return np.random.default_rng(n + depth).uniform(0.0, 1.0, (depth, na, bins)).astype(np.float32)


def _fbp(backend, sinos, n, shape=-1):
    import torch
    d_s = torch.from_numpy(sinos).cuda()
    d_o = torch.full((sinos.shape[0], n, n), float("nan"), dtype=torch.float32, device="cuda")
    backend.set_bp_shape(shape)
    try:
        backend.fbp_d(d_s.data_ptr(), *sinos.shape, n, int(FilterType.SheppLogan), d_o.data_ptr())
        backend.synchronize()
    finally:
        backend.set_bp_shape(-1)
    return d_o.cpu().numpy()


@pytest.mark.parametrize("shape", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("n,bins,na", SIZES)
def test_deep_stack_equals_its_groups(backend, n, bins, na, shape):
    """256 slices, which fill the SMs, against stacks of four, which do not."""
    sinos = _sinos(n, 8, na, bins)
    deep = _fbp(backend, np.concatenate([sinos] * 32), n, shape)
    for z in (0, 4):
        alone = _fbp(backend, sinos[z:z + 4], n, shape)
        for k in (0, 31):
            np.testing.assert_array_equal(deep[8 * k + z:8 * k + z + 4], alone)


@pytest.mark.parametrize("n,bins,na", SIZES)
def test_rings_do_not_change_bits(backend, n, bins, na):
    """Shapes 4 and 5 are shape 0 with other rings of stages."""
    sinos = _sinos(n, 5, na, bins)
    base = _fbp(backend, sinos, n, 0)
    for shape in (4, 5):
        np.testing.assert_array_equal(_fbp(backend, sinos, n, shape), base)


@pytest.mark.parametrize("n,bins,na,depth", [(128, 128, 180, 256), (160, 160, 250, 128), (100, 64, 400, 96)])
def test_host_pipeline_equals_one_pass(backend, n, bins, na, depth):
    sinos = _sinos(n, depth, na, bins)
    got = backend.fbp(sinos, n, int(FilterType.SheppLogan))
    np.testing.assert_array_equal(got, _fbp(backend, sinos, n))


def test_volume_pipeline_equals_one_pass(backend):
    import torch
    n, na, depth = 128, 180, 256
    vol = np.random.default_rng(5).uniform(0.0, 1.0, (depth, n, n)).astype(np.float32)
    d_v = torch.from_numpy(vol).cuda()
    d_o = torch.full_like(d_v, float("nan"))
    backend.reconstruct_volume_d(d_v.data_ptr(), n, depth, na, n, int(FilterType.Ramp), d_o.data_ptr())
    backend.synchronize()
    h_v = torch.from_numpy(vol).pin_memory()
    h_o = torch.full_like(h_v, float("nan")).pin_memory()
    backend.reconstruct_volume_host(h_v.data_ptr(), n, depth, na, n, int(FilterType.Ramp), h_o.data_ptr())
    np.testing.assert_array_equal(h_o.numpy(), d_o.cpu().numpy())


# (output size, bins, angles, depth): alone each takes one slice group per item, together two
MIX = [(160, 160, 250, 64), (160, 128, 180, 64), (160, 100, 300, 60), (144, 144, 226, 64)]


def test_batch_and_server_equal_single_calls(backend):
    import torch
    jobs = []
    for n, bins, na, depth in MIX:
        sinos = _sinos(n, depth, na, bins)
        jobs.append((torch.from_numpy(sinos).cuda(), torch.full((depth, n, n), float("nan"), device="cuda"),
                     n, _fbp(backend, sinos, n)))
    torch.cuda.synchronize()
    args = [dict(sino=s.data_ptr(), depth=s.shape[0], num_angles=s.shape[1], bins=s.shape[2], output_size=n,
                 filter=int(FilterType.SheppLogan), out=o.data_ptr()) for s, o, n, _ in jobs]
    for flags in (0, ctb.BATCH_GRAPH):
        with backend.batch(args, flags) as b:
            b.run()
            backend.synchronize()
        for _, o, _, ref in jobs:
            np.testing.assert_array_equal(o.cpu().numpy(), ref)
            o.fill_(float("nan"))
        torch.cuda.synchronize()
    with ctb.Server(0, memory_budget=4 << 30, copy_threads=1) as srv:
        ids = [srv.submit_device(a["sino"], a["depth"], a["num_angles"], a["bins"], a["output_size"], a["filter"],
                                 a["out"]) for a in args]
        for rid in ids:
            assert srv.wait(rid) == 0
    for _, o, _, ref in jobs:
        np.testing.assert_array_equal(o.cpu().numpy(), ref)
