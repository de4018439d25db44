"""Every read of the forward projector's prepared rows stays inside the planes (CPU).

k_forward (csrc/forward_proj.cu) prepares 32 rows at a time, blocks starting at
multiples of 32: a lane evaluates its row's crossing of the strip's lower edge in
double, q = p dq + q0, and the walk reads the 32 columns from rint(q) on (to the left
where kq < 0), with no clamp, in whole groups of 8 rows of which at least one is
needed: in the strip's row range, its columns meeting the non-zero box. The planes
have a zero border of 64 columns on both sides and 16 zero rows below. The bins 0 and
nd - 1 are read again by edge_bin, over row ranges of their own, clamped to the image.

This replays the set-up (row ranges, clamped in double before they become integers,
and the disc test, with its single-precision roots) and the walk on the host, over
random images, detectors and boxes, with angles at and a float step beside the axes
and the diagonals, and checks each row and column that can be read. The non-zero
bands only leave reads out, so the box alone is used.
"""
import math

import numpy as np
import pytest

GUARD, ROWS, LANES, KREACH = 64, 16, 32, 2.0
F = np.float32


def _prange(qa, qb, dq, idq, cl, ch, rl, rh):
    lo, hi = rl, rh
    if dq != 0.0:
        p = [(cl - KREACH - qa) * idq, (ch + KREACH - qa) * idq, (cl - KREACH - qb) * idq, (ch + KREACH - qb) * idq]
        lo = int(min(max(math.floor(min(p)) - 1.0, rl), rh + 1.0))
        hi = int(max(min(math.ceil(max(p)) + 1.0, rh), rl - 1.0))
    elif max(qa, qb) < cl - KREACH or min(qa, qb) > ch + KREACH:
        hi = -1
    return lo, hi


def _sincospi(t):
    """Exact at multiples of a half, as the device function."""
    t = math.fmod(t, 2.0)
    if (2.0 * t).is_integer():
        return [(0.0, 1.0), (1.0, 0.0), (0.0, -1.0), (-1.0, 0.0)][int(2.0 * t) % 4]
    return math.sin(math.pi * t), math.cos(math.pi * t)


def _check(w, h, nd, deg, box, r4):
    s, c = _sincospi(float(F(deg)) / 180.0)
    rows = abs(c) >= abs(s)
    kq, kp = (c, s) if rows else (s, c)
    K = max(1, int(math.floor(31.5 * max(abs(kq), 0.7071))) - 1)
    np_, nq = (h, w) if rows else (w, h)
    cq, cp, dcf = 0.5 * (nq - 1), 0.5 * (np_ - 1), float(nd // 2)
    rl, rh, cl, ch = (box[2], box[3], box[0], box[1]) if rows else box
    inv = 1.0 / kq
    dq = -kp * inv
    idq = 1.0 / dq if dq != 0.0 else 0.0
    reach = 0
    for b_lo in range(-1, nd - 1, K):
        q0 = cq + (b_lo - dcf + cp * kp) * inv
        p_lo, p_hi = _prange(q0, q0 + (K + 1) * inv, dq, idq, cl, ch, rl, rh)
        rad = 0.5 * float(np.sqrt(F(r4))) + 1.5
        u0, u1 = b_lo - dcf, b_lo - dcf + K + 1
        a0, a1 = max(min(u0, u1), -rad), min(max(u0, u1), rad)
        if a0 > a1:
            p_hi = -1
        else:
            m = 0.0 if a0 <= 0.0 <= a1 else min(abs(a0), abs(a1))
            vm = float(np.sqrt(F(max(0.0, rad * rad - m * m))))
            p_lo = max(p_lo, int(math.floor(cp + min(a0 * kp, a1 * kp) - vm * abs(kq))) - 2)
            p_hi = min(p_hi, int(math.ceil(cp + max(a0 * kp, a1 * kp) + vm * abs(kq))) + 2)
        if p_hi >= p_lo:
            p = np.arange(p_lo & ~(LANES - 1), (p_hi | (LANES - 1)) + 1)
            col = np.rint(p * dq + q0)
            first = col - (LANES - 1 if kq < 0.0 else 0)
            need = (p >= p_lo) & (p <= p_hi) & (first + LANES - 1 >= cl) & (first <= ch)
            read = need.reshape(-1, 8).any(1).repeat(8)
            if read.any():
                assert p[read].min() >= 0 and p[read].max() <= np_ - 1 + ROWS, (w, h, nd, deg, box)
                lo, hi = first[read].min(), first[read].max() + LANES - 1
                assert lo >= -50 and hi <= nq - 1 + 50, (w, h, nd, deg, box, lo, hi)
                # the row records hold unsigned pixel offsets from the block's first row
                assert ((p[read] % LANES) * (nq + 2 * GUARD) + col[read] + GUARD >= 0).all()
                reach = max(reach, -lo, hi - (nq - 1))
        for side, (ea, eb) in ((b_lo < 0, (-1, 2)), (b_lo + min(K, nd - 1 - b_lo) == nd - 1, (nd - 3, nd + 1))):
            if not side:
                continue
            e0, e1 = _prange(q0 + (ea - b_lo) * inv, q0 + (eb - b_lo) * inv, dq, idq, cl, ch, rl, rh)
            assert e1 < e0 or (e0 >= 0 and e1 <= np_ - 1), (w, h, nd, deg, box, e0, e1)
            if e1 < e0:
                continue
            # a row's candidate columns: at most three, which edge_bin of a single slice takes unrolled
            lo, hi = (0.0, 1.0) if ea == -1 else (nd - 2.0, float(nd))
            da, db = (lo - 1.0 / 64 - b_lo) * inv, (hi + 1.0 / 64 - b_lo) * inv
            q = np.arange(e0, e1 + 1) * dq + q0
            count = np.floor(q + max(da, db)) - np.ceil(q + min(da, db)) + 1
            assert count.max() <= 3, (w, h, nd, deg, count.max())
    return reach


@pytest.mark.parametrize("seed", range(6))
def test_reads_stay_in_the_planes(seed):
    rng = np.random.default_rng(seed)
    step = [np.nextafter(F(a), F(b)) for a in (45, 90, 135, 180) for b in (0, 360)]
    worst = 0
    for _ in range(40):
        w = int(np.exp(rng.uniform(0.0, np.log(1500.0))))
        h = int(np.exp(rng.uniform(0.0, np.log(1500.0)))) if rng.random() < 0.3 else w
        nd = int(rng.integers(2, max(4, 3 * max(w, h))))
        if rng.random() < 0.3:  # bounds off: the whole image and a disc through its corners
            box, r4 = (0, w - 1, 0, h - 1), (w - 1) ** 2 + (h - 1) ** 2
        else:
            x0, x1 = sorted(int(v) for v in rng.integers(0, w, 2))
            y0, y1 = sorted(int(v) for v in rng.integers(0, h, 2))
            box = (x0, x1, y0, y1)
            r4 = max((2 * x - w + 1) ** 2 + (2 * y - h + 1) ** 2 for x in (x0, x1) for y in (y0, y1))
        for deg in [*rng.uniform(0.0, 360.0, 8), 0.0, 45.0, 90.0, 135.0, 180.0, 1e-30, 1e-5, *step]:
            worst = max(worst, _check(w, h, nd, deg, box, r4))
    assert 0 < worst <= 50
