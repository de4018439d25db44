"""The slab schedule of the host-buffer pipelines (CPU).

plan_slabs (csrc/host_math.cpp) over random stacks: whole groups of 8 slices in
order, nothing left out; slabs whose buffers would take more than 4 GiB hold no more
than an eighth or a sixteenth of the stack; and where an FBP is bound by copies that
take alike both ways, a slab is a few megabytes.
"""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "qtctreconstruction_b200", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"

MAIN = r"""
#include <cmath>
#include <cstdio>
#include "ctb_internal.h"
int main() {
    int depth, n, sms, lead;
    ctb::SlabWork w;
    while (std::scanf("%d %d %d %zu %zu %zu %d", &depth, &n, &sms, &w.in, &w.out, &w.scratch, &lead) == 7) {
        w.copies_lead = lead;
        for (const int2& s : ctb::plan_slabs(depth, n, sms, w)) std::printf("%d,%d ", s.x, s.y);
        std::printf("\n");
    }
}
"""


def _least(depth):
    sixteenth = 8 * -(-depth // 128)
    return 2 * sixteenth if sixteenth >= 32 else sixteenth


def test_schedule(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "main.cpp", tmp_path / "slabs"
    src.write_text(MAIN)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
                        "-I" + CUDA_INCLUDE, str(src), os.path.join(CSRC, "host_math.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = random.Random(7)
    cases = [(256, 64, 148, 4 * 64 * 64, 4 * 64 * 64, 2800 << 20, 0),   # 65536 angles of 3393 bins
             (50, 384, 148, 4 * 180 * 545, 4 * 384 * 384, 5 << 20, 1), (256, 256, 148, 4 * 256 ** 2, 4 * 256 ** 2, 3 << 20, 0)]
    for _ in range(3000):
        n, lead = rng.choice([2, 33, 64, 128, 200, 256, 387, 512, 1024]), rng.randint(0, 1)
        out = 4 * n * n
        size_in = int(out * 10 ** rng.uniform(-1.5, 1.5)) // 4 * 4 if lead else out
        cases.append((int(10 ** rng.uniform(0, 3.3)), n, rng.choice([1, 132, 148]), max(4, size_in), out,
                      int((size_in + out) * 10 ** rng.uniform(0.3, 4)), lead))
    r = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases), capture_output=True, text=True,
                       timeout=120)
    lines = r.stdout.splitlines()
    assert len(lines) == len(cases)
    for (depth, n, sms, size_in, out, scratch, lead), line in zip(cases, lines):
        slabs = [tuple(map(int, s.split(","))) for s in line.split()]
        z = 0
        for k, (first, count) in enumerate(slabs):
            assert first == z and count > 0 and (depth <= 16 or k + 1 == len(slabs) or count % 8 == 0), (depth, slabs)
            z += count
        assert z == depth
        if depth <= 16:
            continue
        most = max(c for _, c in slabs)
        # a piece is at most half a slab larger than the middle slab it is one of
        assert most * scratch <= max(1.5 * 4 * 2 ** 30, (_least(depth) + 7) * scratch), (depth, n, scratch, slabs)
        larger = max(size_in, out)
        if lead and 2 * size_in >= out and 5 * size_in <= 8 * out and 8 * larger >= 1000000:
            assert most <= max(8, 4400000 // larger) + 7, (depth, n, size_in, out, slabs)
