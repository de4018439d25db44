"""The forward projector's plan walks every angle along the axis its slope allows (CPU).

The kernel takes cos and sin from sincospi, which is exact for any angle; the plan
(forward_plan, csrc/host_math.cpp) chooses the walked axis and the strip width on the
host. Whatever the angle, also after very many turns, the coefficient along the walked
axis has to be the larger one: the reads' bounds rest on it.
"""
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "qtctreconstruction_b200", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"

MAIN = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "ctb_internal.h"
int main() {
    std::vector<float> angles;
    float a;
    while (std::scanf("%f", &a) == 1) angles.push_back(a);
    const ctb::FwdPlan p = ctb::forward_plan(angles.data(), static_cast<int>(angles.size()), 64, 64, 91);
    for (size_t g = 0; g < p.groups.size(); g += 4)
        for (int k = 0; k < p.groups[g + 1]; ++k)
            std::printf("%d %d %d\n", p.order[p.groups[g] + k], p.groups[g + 2], p.groups[g + 3]);
}
"""


def test_axis_of_every_angle(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "main.cpp", tmp_path / "plan"
    src.write_text(MAIN)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
                        "-I" + CUDA_INCLUDE, str(src), os.path.join(CSRC, "host_math.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = np.random.default_rng(0)
    angles = np.concatenate([rng.uniform(-720.0, 720.0, 500), [0.0, 45.0, 90.0, 135.0, 180.0, 1e-30],
                             rng.choice([-1.0, 1.0], 500) * 10.0 ** rng.uniform(3.0, 38.0, 500)]).astype(np.float32)
    r = subprocess.run([str(exe)], input="\n".join(f"{a:.9g}" for a in angles), capture_output=True, text=True)
    seen = set()
    for line in r.stdout.splitlines():
        a, axis, K = map(int, line.split())
        seen.add(a)
        t = math.fmod(float(angles[a]) / 180.0, 2.0)
        c, s = abs(math.cos(math.pi * t)), abs(math.sin(math.pi * t))
        walked = c if axis == 0 else s
        assert walked >= max(c, s) - 1e-12, (angles[a], axis)
        assert K + 1 <= 31.5 * max(walked, 0.7071) + 1e-9, (angles[a], K)
    assert seen == set(range(len(angles)))
