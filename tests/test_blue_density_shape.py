"""Blue noise's density sums: the launch shape and, on a GPU, the ranks where a
block has several warps.

Each pixel's sum is one chain of additions, so blocks that wait for room on
an SM repeat its whole length: for every table size the blocks are on the SMs
at once."""
import os
import subprocess

import numpy as np
import pytest

from sfsim_gb300 import noise

SOURCE = r"""
#include <cstdio>
#include "blue_density.h"
int main() {
  for (int m = 2; m <= 256; m++) std::printf("%d %zu %d\n", m, sfsim::blue_density_smem(m), sfsim::blue_density_warps(m, 152));
}
"""


def test_one_wave(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src, exe = tmp_path / "shape.cpp", tmp_path / "shape"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(root, "sfsim_gb300", "csrc"), "-o", str(exe), str(src)], check=True)
    rows = [tuple(map(int, r.split())) for r in subprocess.run([str(exe)], capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == 255
    for m, smem, warps in rows:
        assert smem <= 220 * 1024 and 1 <= warps <= 16
        blocks = -(-m * m // (32 * warps))
        resident = 152 * min(32, 227 * 1024 // (smem + 1024), 64 // warps)
        assert blocks <= resident, (m, blocks, resident)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [150, 200])
def test_ranks_exactly(m):
    from oracle import oracle as O
    pixels = np.random.default_rng(m).permutation(m * m)[:m * m // 10]
    np.testing.assert_array_equal(noise.blue_noise(m, sigma=1.5, seed_pixels=pixels), O.blue(m, pixels, 1.5))
