"""slab_step (device_math.cuh): the step the column counts of boxes divide by is no further than its least size from the real one,
whatever the sign; the bound of those counts takes that as given."""
import os
import subprocess

import pytest

from sdfibm_gb300 import build

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <limits>
#include "sdfibm_cuda.h"
#include "device_math.cuh"
int main() {
    int bad = 0;
    for (float least : {1e-30f, 1e-9f, 0.37f, 1e5f})
        for (int i = -4000; i <= 4000; ++i) {
            const float d = least * (float)i / 1000.f, s = sdfibm_dev::slab_step(d, least);
            bad += !(std::fabs((double)s - (double)d) <= (double)least && std::fabs(s) >= least && s * (1.f / least) * d >= 0.f);
            bad += std::fabs(d) >= least && s != d;
        }
    bad += sdfibm_dev::slab_step(0.f, 1e-9f) != 1e-9f;
    std::printf("%d\n", bad);
}
"""


def test_slab_step(tmp_path):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "slab.cu", tmp_path / "slab"
    src.write_text(SOURCE)
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I", build.CSRC, "-I", os.path.join(build.HERE, "..", "include"), str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.strip() == "0"
