"""Ray scatter where the threads of its blocks change: rows of up to 320, 512
and 1024 heading columns (sun elevations times headings + 2), on both sides of
each, and more, in passes; against the FP64 oracle with the bounds of
test_gpu_ray_scatter.py.  And rows of more than 320 columns keep what those
below have (corners kept in registers, planes built once): rows of as many
cells with a fifth more columns take 1.24 times as long, 2.2 times without."""
import pytest
import torch

from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C
from tests.test_gpu_ray_scatter import test_ray_scatter_shapes as check

pytestmark = pytest.mark.gpu

# 325, 512, 513, 1024 and 1028 columns
CASES = [((2, 3, 65, 3), 9), ((2, 3, 128, 2), 33), ((2, 3, 57, 7), 20), ((2, 3, 256, 2), 10), ((2, 2, 257, 2), 18)]


@pytest.mark.parametrize("shape,steps", CASES, ids=[f"{'x'.join(map(str, s))}-S{n}" for s, n in CASES])
@pytest.mark.parametrize("precision", [C.FP64, C.FP32], ids=["fp64", "fp32"])
def test_columns(shape, steps, precision):
    check(shape, steps, precision)


def test_time_follows_the_columns():
    def ray_scatter_ms(n2, n3):
        cfg = C.make_config(height=100000.0, transmittance_shape=(4, 8), surface_radiance_shape=(4, 8),
                            ray_scatter_shape=(16, 100, n2, n3), ray_steps=100, sphere_steps=6, iterations=2)
        out = A.build_device(cfg)
        read = A.stage_timings(True)
        try:
            times = []
            for _ in range(7):
                A.build_device(cfg, out)
                torch.cuda.synchronize()
                times.append(read()["ray_scatter"])
        finally:
            A.stage_timings(False)
        return sorted(times)[3]

    assert ray_scatter_ms(64, 4) < 1.7 * ray_scatter_ms(32, 8)
