"""Performance cases: the work a program has this framework do, through its public entry points.

A case is a dict of plain values. `prepare` makes what the program has in hand before the call
(volumes, sinograms, output buffers, a planned batch, a running server), `run` is one pass through
the public API, `exact` the same result in 64 bits by plain torch, `work` the bytes and operations
the pass cannot do without.

The kinds of work ("op"):
  sinogram  computeSinogram: one host slice -> its sinogram (a viewer's or controller's call per slice)
  slice     reconstructSlice: one host sinogram -> its slice
  volume    reconstruct_volume_d: forward projection + FBP of a device-resident volume
  host      reconstruct_volume_host: the same from and to page-locked host memory
  forward   forward_d: forward projection of a device volume at an explicit angle list
  fbp       fbp_d: filtering + backprojection of a device sinogram stack
  stack     reconstructVolumeFromSinograms: a sinogram stack in host arrays (as read from a file)
  batch     a planned batch of uneven FBP jobs, replayed
  serve     uneven device-resident FBP requests submitted to a running server

Input data: "phantom" volumes are sums of random ellipsoids that are exactly zero outside (the
benchmark phantom); "ct" volumes are whole numbers of Hounsfield units with noise everywhere, air
included, as scanners deliver them. Sinograms are exact line integrals of random ellipses plus 0.5 %
noise.
"""
import math
import random

import numpy as np
import torch

import qtctreconstruction_b200 as ctb

RAMP, SHEPP, HANN = int(ctb.FilterType.Ramp), int(ctb.FilterType.SheppLogan), int(ctb.FilterType.Hann)
FILTERS = (RAMP, SHEPP, HANN)

# the largest pass: the voxel-angle updates of a 512^3 volume at 720 angles
MOST_UPDATES = 512 ** 3 * 720


def _odd_bins(n):
    """The detector of a full acquisition of n pixels: ceil(sqrt(2) n), made odd."""
    return math.ceil(math.sqrt(2.0) * n) | 1


def listed():
    return [
        # one slice of a viewer: the smallest call, host memory to host memory
        {"name": "sinogram_slice", "op": "sinogram", "w": 160, "h": 128, "angles": 180, "bins": 160, "data": "ct"},
        # one sinogram reconstructed for display
        {"name": "recon_slice", "op": "slice", "n": 256, "angles": 360, "bins": 363, "filter": SHEPP},
        # the small benchmark volume: many short launches
        {"name": "volume_small", "op": "volume", "n": 128, "depth": 128, "angles": 180, "bins": 183, "filter": RAMP,
         "data": "phantom"},
        # the headline volume, and the largest pass
        {"name": "volume_large", "op": "volume", "n": 512, "depth": 512, "angles": 720, "bins": 725, "filter": SHEPP,
         "data": "phantom"},
        # a scanner's series: odd size, air that is not exactly zero, the detector as wide as the slice
        {"name": "volume_ct", "op": "volume", "n": 387, "depth": 50, "angles": 580, "bins": 387, "filter": HANN,
         "data": "ct"},
        # a whole call on page-locked host memory, copies included
        {"name": "volume_host", "op": "host", "n": 256, "depth": 256, "angles": 360, "bins": 363, "filter": SHEPP,
         "data": "phantom"},
        # forward projection alone, at angles that are neither uniform nor in order
        {"name": "forward_angles", "op": "forward", "n": 300, "depth": 37, "angles": 450, "bins": 425, "data": "ct"},
        # the smallest device-resident FBP
        {"name": "fbp_small", "op": "fbp", "n": 64, "depth": 16, "angles": 101, "bins": 91, "filter": SHEPP},
        # the large request of a serving mix
        {"name": "fbp_large", "op": "fbp", "n": 1024, "depth": 64, "angles": 1440, "bins": 1449, "filter": HANN},
        # a sinogram stack read from a file: pageable arrays in, a new array out, denormalised
        {"name": "stack_file", "op": "stack", "depth": 48, "angles": 402, "bins": 257, "filter": RAMP},
        # the uneven batch: many sizes in one replayed plan
        {"name": "batch_mixed", "op": "batch", "jobs": 12, "n_lo": 64, "n_hi": 384, "depth_hi": 96, "mix": 1},
        # the same kind of requests through the serving loop
        {"name": "serve_mixed", "op": "serve", "jobs": 10, "n_lo": 64, "n_hi": 256, "depth_hi": 64, "mix": 2},
    ]


def draw(rng):
    """One more case of the ranges above."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["sinogram", "slice", "volume", "volume", "volume", "host", "forward", "forward", "fbp", "fbp",
                     "fbp", "stack", "batch", "serve"])
    filt = rng.choice(FILTERS)
    data = rng.choice(["phantom", "ct"])
    if op == "sinogram":
        w, h = log(64, 512), log(64, 512)
        return {"op": op, "w": w, "h": h, "angles": log(90, 720), "bins": rng.choice([w, _odd_bins(max(w, h))]),
                "data": data}
    if op == "slice":
        n = log(64, 512)
        return {"op": op, "n": n, "angles": log(90, 720), "bins": _odd_bins(n), "filter": filt}
    if op in ("batch", "serve"):
        lo = log(64, 96)
        return {"op": op, "jobs": rng.randint(4, 12), "n_lo": lo, "n_hi": log(128, 384), "depth_hi": log(16, 96),
                "mix": rng.randint(3, 1 << 20)}
    if op == "stack":
        return {"op": op, "depth": log(8, 64), "angles": log(90, 480), "bins": log(64, 320), "filter": filt}
    n = log(64, 256 if op == "host" else 1024)
    angles = log(max(60, n // 2), 2 * n)
    most = min(256 if op == "host" else 512, MOST_UPDATES // (n * n * angles))
    depth = log(1, max(1, most))
    bins = rng.choice([_odd_bins(n), _odd_bins(n), n])
    case = {"op": op, "n": n, "depth": depth, "angles": angles, "bins": bins}
    if op != "forward":
        case["filter"] = filt
    if op != "fbp":
        case["data"] = data
    return case


# ------------------------------------------------------------------ programs' long-lived handles
_handles = {}


def _backend():
    """The program's one backend (its context keeps workspaces and tables between calls)."""
    if "backend" not in _handles:
        _handles["backend"] = ctb.B200Backend(0)
    return _handles["backend"]


def _server():
    if "server" not in _handles:
        _handles["server"] = ctb.Server(0, memory_budget=8 << 30, copy_threads=2)
    return _handles["server"]


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ellipsoids(r, count):
    """(centre, semi-axes, rotation, density) with the benchmark phantom's distributions."""
    q = r.normal(size=(count, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, x, y, z = q.T
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y),
                    2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x),
                    2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], 1).reshape(count, 3, 3)
    return r.uniform(-0.6, 0.6, (count, 3)), r.uniform(0.05, 0.4, (count, 3)), rot, r.uniform(-0.3, 1.0, count)


def _volume(data, depth, h, w, seed):
    """A float32 volume [depth][h][w] on the GPU."""
    r = np.random.default_rng(seed)
    centre, semi, rot, dens = _ellipsoids(r, max(10, min(32, w // 12)))

    def axis(n):
        return (2 * torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1)) / max(n, 2)

    zz, yy, xx = axis(depth), axis(h), axis(w)
    vol = torch.zeros(depth, h, w, device="cuda")
    step = max(1, (1 << 24) // (h * w))
    for z0 in range(0, depth, step):
        z1 = min(depth, z0 + step)
        part = vol[z0:z1]
        Z, Y, X = zz[z0:z1, None, None], yy[None, :, None], xx[None, None, :]
        inside = X * X + Y * Y + Z * Z <= 1.0
        for k in range(len(dens)):
            d = [X - float(centre[k, 0]), Y - float(centre[k, 1]), Z - float(centre[k, 2])]
            q = 0.0
            for i in range(3):
                b = sum(float(rot[k, i, j]) * d[j] for j in range(3))
                q = q + (b / float(semi[k, i])) ** 2
            part += torch.where(inside & (q <= 1.0), float(dens[k]), 0.0)
    if data == "phantom":
        return vol
    # a body of water in air, the ellipsoids as tissue and bone, noise everywhere
    body = ((xx[None, :] / 0.85) ** 2 + (yy[:, None] / 0.75) ** 2 <= 1.0).float()
    vol.mul_(300.0).mul_(body).add_(1000.0 * body - 1000.0)
    vol.add_(torch.empty_like(vol).normal_(0.0, 20.0, generator=_gen(seed)))
    return vol.clamp_(-1024.0, 3071.0).round_()


def _angles(count, seed, uniform=True):
    """Degrees: uniform over 180, or a golden-angle order with jitter."""
    if uniform:
        return ctb.uniform_angles_deg(count)
    r = np.random.default_rng(seed + 5)
    return ((np.arange(count) * 111.246117975 + r.uniform(-0.1, 0.1, count)) % 180.0).astype(np.float32)


def _sinograms(depth, angles_deg, bins, n, seed):
    """Sinograms [depth][angles][bins] of random ellipses in a slice of n pixels, on the GPU."""
    r = np.random.default_rng(seed)
    th = torch.from_numpy(np.deg2rad(angles_deg.astype(np.float64))).cuda().float()
    t = torch.arange(bins, device="cuda", dtype=torch.float32) - bins // 2
    z = torch.linspace(-1, 1, depth, device="cuda")[:, None]
    out = torch.zeros(depth, len(angles_deg), bins, device="cuda")
    step = max(1, (1 << 25) // (len(angles_deg) * bins))
    for _ in range(8):
        cx, cy, cz = r.uniform(-0.4, 0.4, 3)
        a, b, e = r.uniform(0.1, 0.45, 3)
        phi, dens = r.uniform(0, math.pi), r.uniform(0.1, 1.0)
        shrink = (1.0 - ((z - cz) / (2 * e)) ** 2).clamp_min(0.0) * (n / 2) ** 2
        A2 = (a * a * torch.cos(th - phi) ** 2 + b * b * torch.sin(th - phi) ** 2)[None, :, None]
        off = (t[None, :] - ((cx * torch.cos(th) + cy * torch.sin(th)) * (n / 2))[:, None])[None] ** 2
        for z0 in range(0, depth, step):
            s = shrink[z0:z0 + step, :, None]
            out[z0:z0 + step] += (2 * dens * a * b) * (A2 * s - off).clamp_min_(0.0).sqrt_() / A2
    top = float(out.max())
    return out.add_(torch.empty_like(out).normal_(0.0, 0.005 * max(top, 1e-3), generator=_gen(seed)))


def _mix(case):
    """The jobs of a batch or of a request stream: sizes drawn from the case alone."""
    r = random.Random(case["mix"])
    jobs = []
    for _ in range(case["jobs"]):
        n = r.randrange(case["n_lo"], case["n_hi"] + 1)
        jobs.append({"n": n, "depth": r.randint(max(1, min(16, case["depth_hi"] // 2)), case["depth_hi"]),
                     "angles": round(math.pi / 2 * n), "bins": _odd_bins(n), "filter": r.choice(FILTERS)})
    return jobs


def _pinned(t):
    return t.cpu().pin_memory()


def prepare(case, seed):
    op = case["op"]
    be = _backend()
    s = {"case": case, "be": be}
    if op == "sinogram":
        s["slice"] = _volume(case["data"], 1, case["h"], case["w"], seed)[0].cpu().numpy()
    elif op == "slice":
        ang = _angles(case["angles"], seed)
        data = _sinograms(1, ang, case["bins"], case["n"], seed)[0].cpu().numpy()
        s["sino"] = ctb.Sinogram(data, ang, 1.0, float(data.min()), float(data.max()))
        s["params"] = ctb.ReconstructionParams(ctb.FilterType(case["filter"]), case["angles"])
    elif op in ("volume", "host", "forward"):
        n, depth = case["n"], case["depth"]
        s["vol"] = _volume(case["data"], depth, n, n, seed)
        if op == "host":
            s["vol"] = _pinned(s["vol"])
            s["out"] = torch.empty(depth, n, n).pin_memory()
        elif op == "volume":
            s["out"] = torch.empty_like(s["vol"])
        else:
            s["angles"] = _angles(case["angles"], 0, uniform=False)
            s["sino"] = torch.empty(depth, case["angles"], case["bins"], device="cuda")
            s["stats"] = torch.empty(depth, 4, device="cuda")
    elif op == "fbp":
        s["sino"] = _sinograms(case["depth"], _angles(case["angles"], seed), case["bins"], case["n"], seed)
        s["out"] = torch.empty(case["depth"], case["n"], case["n"], device="cuda")
    elif op == "stack":
        s["angles"] = _angles(case["angles"], seed)
        s["sino"] = _sinograms(case["depth"], s["angles"], case["bins"], int(case["bins"] / 1.5), seed).cpu().numpy()
        s["params"] = ctb.ReconstructionParams(ctb.FilterType(case["filter"]), case["angles"])
    else:
        s["jobs"] = []
        for k, j in enumerate(_mix(case)):
            sino = _sinograms(j["depth"], _angles(j["angles"], seed), j["bins"], j["n"], seed + 101 * k)
            s["jobs"].append((j, sino, torch.empty(j["depth"], j["n"], j["n"], device="cuda")))
        if op == "batch":
            s["batch"] = be.batch([dict(sino=sino.data_ptr(), depth=j["depth"], num_angles=j["angles"], bins=j["bins"],
                                        output_size=j["n"], filter=j["filter"], out=out.data_ptr())
                                   for j, sino, out in s["jobs"]], ctb.BATCH_GRAPH)
        else:
            s["server"] = _server()
    torch.cuda.synchronize()  # the framework's streams are its own: the inputs are there before a call
    return s


def run(s):
    c, be, op = s["case"], s["be"], s["case"]["op"]
    if op == "sinogram":
        r = be.computeSinogram(s["slice"], c["angles"], c["bins"])
        return r.data, r.angles_deg, r.original_min_hu, r.original_max_hu
    if op == "slice":
        return be.reconstructSlice(s["sino"], c["n"], s["params"])
    if op == "volume":
        be.reconstruct_volume_d(s["vol"].data_ptr(), c["n"], c["depth"], c["angles"], c["bins"], c["filter"],
                                s["out"].data_ptr())
        return s["out"]
    if op == "host":
        be.reconstruct_volume_host(s["vol"].data_ptr(), c["n"], c["depth"], c["angles"], c["bins"], c["filter"],
                                   s["out"].data_ptr())
        return s["out"]
    if op == "forward":
        be.forward_d(s["vol"].data_ptr(), c["n"], c["depth"], c["angles"], c["bins"], s["sino"].data_ptr(),
                     s["stats"].data_ptr(), s["angles"])
        return s["sino"], s["stats"]
    if op == "fbp":
        be.fbp_d(s["sino"].data_ptr(), c["depth"], c["angles"], c["bins"], c["n"], c["filter"], s["out"].data_ptr())
        return s["out"]
    if op == "stack":
        return be.reconstructVolumeFromSinograms(s["sino"], s["angles"], s["params"], denorm=ctb.Denorm.SERIAL)
    if op == "batch":
        s["batch"].run()
        return [out for _, _, out in s["jobs"]]
    srv = s["server"]
    ids = [srv.submit_device(sino.data_ptr(), j["depth"], j["angles"], j["bins"], j["n"], j["filter"], out.data_ptr())
           for j, sino, out in s["jobs"]]
    for rid in ids:
        if srv.wait(rid):
            raise RuntimeError("request failed")
        srv.release(rid)
    return [out for _, _, out in s["jobs"]]


# ------------------------------------------------------------------ work
def _forward_flops(h, w, depth, angles):
    return 4.0 * h * w * depth * angles  # two weighted adds per pixel and angle


def _fbp_flops(n, depth, angles, bins):
    sq = math.ceil(math.sqrt(2.0) * bins)
    length = max(64, 1 << (sq + bins - 2).bit_length())
    rows = depth * angles
    fft = rows / 2 * (2 * 5 * length * math.log2(length) + 6 * length)  # two real rows per complex transform
    return fft + 4.0 * (math.pi / 4) * n * n * depth * angles           # two taps per voxel of the circle and angle


def work(case):
    op = case["op"]
    if op == "sinogram":
        return {"bytes": 4.0 * (case["w"] * case["h"] + case["angles"] * case["bins"]),
                "flops": _forward_flops(case["h"], case["w"], 1, case["angles"])}
    if op == "forward":
        n, d = case["n"], case["depth"]
        return {"bytes": 4.0 * d * (n * n + case["angles"] * case["bins"]),
                "flops": _forward_flops(n, n, d, case["angles"])}
    if op in ("volume", "host"):
        n, d = case["n"], case["depth"]
        return {"bytes": 8.0 * d * n * n,
                "flops": _forward_flops(n, n, d, case["angles"]) + _fbp_flops(n, d, case["angles"], case["bins"])}
    if op in ("batch", "serve"):
        jobs = _mix(case)
    elif op == "stack":
        jobs = [dict(case, n=case["bins"])]
    else:
        jobs = [dict(case, depth=case.get("depth", 1))]
    return {"bytes": sum(4.0 * j["depth"] * (j["n"] ** 2 + j["angles"] * j["bins"]) for j in jobs),
            "flops": sum(_fbp_flops(j["n"], j["depth"], j["angles"], j["bins"]) for j in jobs)}


# ------------------------------------------------------------------ 64-bit results
def _cos_sin(angles_deg):
    th = np.asarray(angles_deg, np.float64) * (math.pi / 180.0)
    c, s = np.cos(th), np.sin(th)
    c[np.asarray(angles_deg) == 90.0] = 0.0
    return c, s


def _exact_forward(vol, angles_deg, bins):
    """Normalised splat projection: sinograms [depth][angles][bins] (float64), per-slice min and max."""
    depth, h, w = vol.shape
    flat = vol.reshape(depth, -1).double()
    lo, hi = flat.amin(1), flat.amax(1)
    span = torch.where(hi - lo < 1e-6, torch.ones_like(lo), hi - lo)
    used = torch.nonzero((flat != 0).any(0))[:, 0]  # zero pixels add nothing
    part = flat[:, used]
    v = torch.where(part != 0, (part - lo[:, None]) / span[:, None], torch.zeros_like(part)).t().contiguous()
    x, y = (used % w).double() - (w - 1) * 0.5, (used // w).double() - (h - 1) * 0.5
    sino = torch.zeros(len(angles_deg), bins, depth, dtype=torch.float64, device=vol.device)
    for a, (c, s) in enumerate(zip(*_cos_sin(angles_deg))):
        pos = x * float(c) + y * float(s) + bins // 2
        i0 = torch.floor(pos)
        frac = pos - i0
        i0 = i0.long()
        ok, last = (i0 >= 0) & (i0 < bins - 1), i0 == bins - 1
        w0 = torch.where(ok, 1.0 - frac, last.double())
        w1 = torch.where(ok, frac, torch.zeros_like(frac))
        row = sino[a]
        row.index_add_(0, i0.clamp(0, bins - 1), v * w0[:, None])
        row.index_add_(0, (i0 + 1).clamp(0, bins - 1), v * w1[:, None])
    return sino.permute(2, 0, 1).contiguous(), lo, hi


def _response(length, kind):
    """The ramp filter and its windows: length / 2 + 1 values, bins 0 and length / 2 left out."""
    h = torch.zeros(length, dtype=torch.float64)
    h[0] = 0.25
    i = torch.arange(1, length, 2)
    m = torch.where(i < length // 2, i, length - i).double()
    h[i] = -1.0 / (math.pi * m) ** 2
    H = 2.0 * torch.fft.rfft(h).real
    f = torch.arange(length // 2 + 1, dtype=torch.float64) / length
    if kind == SHEPP:
        H[1:] *= torch.sin(math.pi * f[1:]) / (math.pi * f[1:])
    elif kind == HANN:
        H *= 0.5 + 0.5 * torch.cos(2 * math.pi * f)
    H[0] = H[-1] = 0.0
    return H


def _exact_fbp(sino, angles_deg, n, kind):
    """Filtered backprojection in normalised units, [depth][n][n] float64."""
    depth, angles, bins = sino.shape
    sq = math.ceil(math.sqrt(2.0) * bins)
    pad = sq // 2 - bins // 2
    length = max(64, 1 << (2 * sq - 1).bit_length())
    H = _response(length, kind).to(sino.device)
    r = n // 2
    g = torch.arange(n, device=sino.device, dtype=torch.float64) - r
    X, Y = g[None, :].expand(n, n), g[:, None].expand(n, n)
    inside = torch.nonzero((X * X + Y * Y <= r * r).reshape(-1))[:, 0]
    X, Y = X.reshape(-1)[inside], Y.reshape(-1)[inside]
    acc = torch.zeros(len(inside), depth, dtype=torch.float64, device=sino.device)
    for a, (c, s) in enumerate(zip(*_cos_sin(angles_deg))):
        row = torch.zeros(depth, length, dtype=torch.float64, device=sino.device)
        row[:, pad:pad + bins] = sino[:, a].double()
        q = torch.fft.irfft(torch.fft.rfft(row) * H, n=length)[:, :sq].t().contiguous()
        u = X * float(c) - Y * float(s) + sq // 2
        i0 = torch.floor(u)
        frac = u - i0
        i0 = i0.long()
        ok = ((i0 >= 0) & (i0 + 1 < sq)).double()
        i0 = i0.clamp(0, sq - 2)
        acc.addcmul_(q[i0], (ok * (1.0 - frac))[:, None])
        acc.addcmul_(q[i0 + 1], (ok * frac)[:, None])
    out = torch.zeros(depth, n * n, dtype=torch.float64, device=sino.device)
    out[:, inside] = (acc * (math.pi / (2.0 * angles))).t()
    return out.reshape(depth, n, n)


def exact(case, seed):
    op = case["op"]
    if op in ("sinogram", "forward"):
        ang = _angles(case["angles"], 0, uniform=op == "sinogram")
        h, w, depth = (case["h"], case["w"], 1) if op == "sinogram" else (case["n"], case["n"], case["depth"])
        sino, lo, hi = _exact_forward(_volume(case["data"], depth, h, w, seed), ang, case["bins"])
        if op == "sinogram":
            return sino[0], np.arange(case["angles"]) * (180.0 / case["angles"]), float(lo), float(hi)
        span = hi - lo
        one = torch.ones_like(span)
        return sino, torch.stack([lo, hi, torch.where(span < 1e-6, one, span), torch.where(span <= 0, one, span)], 1)
    if op in ("volume", "host"):
        vol = _volume(case["data"], case["depth"], case["n"], case["n"], seed)
        ang = _angles(case["angles"], seed)
        sino, lo, hi = _exact_forward(vol, ang, case["bins"])
        span = torch.where(hi - lo <= 0, torch.ones_like(lo), hi - lo)
        return _exact_fbp(sino, ang, case["n"], case["filter"]) * span[:, None, None] + lo[:, None, None]
    if op in ("slice", "fbp"):
        ang = _angles(case["angles"], seed)
        sino = _sinograms(case.get("depth", 1), ang, case["bins"], case["n"], seed)
        out = _exact_fbp(sino, ang, case["n"], case["filter"])
        return out[0] if op == "slice" else out
    if op == "stack":
        ang = _angles(case["angles"], seed)
        sino = _sinograms(case["depth"], ang, case["bins"], int(case["bins"] / 1.5), seed)
        lo, hi = sino.amin((1, 2)).double(), sino.amax((1, 2)).double()
        span = torch.where(hi - lo <= 0, torch.ones_like(lo), hi - lo)
        return _exact_fbp(sino, ang, case["bins"], case["filter"]) * span[:, None, None] + lo[:, None, None]
    out = []
    for k, j in enumerate(_mix(case)):
        ang = _angles(j["angles"], seed)
        out.append(_exact_fbp(_sinograms(j["depth"], ang, j["bins"], j["n"], seed + 101 * k), ang, j["n"], j["filter"]))
    return out
