"""An atmosphere of a batch has the bits of its own build, whatever the batch's
size: batches on both sides of the sizes at which a batch fills the GPU by
itself (ray scatter's groups of samples, point scatter's slices of
directions, the parts of a first-order row)."""
import numpy as np
import pytest

from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu

SHAPES = [(8, 16, 8, 4), (4, 11, 6, 3), (6, 30, 16, 8)]


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("precision", [C.FP32, C.FP64], ids=["fp32", "fp64"])
def test_batch_sizes(shape, precision):
    cfgs = C.parameter_sweep(30, precision=precision, ray_scatter_shape=shape, transmittance_shape=(16, 16),
                             surface_radiance_shape=(4, 8), ray_steps=24, sphere_steps=10, iterations=2)
    singles = [A.build(c) for c in cfgs]
    for size in (2, 5, 12, 30):
        batch = A.build_batch(cfgs[:size])
        for n in range(size):
            for key, value in singles[n].items():
                assert np.array_equal(batch[key][n], value), (size, n, key)


def test_unlike_atmospheres():
    """Atmospheres whose own builds take 8 or 16 segments of fitted sun rays, or
    integrate every sun ray, keep that in a batch, in whatever order."""
    def mk(height, mie_scale, base):
        return C.make_config(radius=base.radius, height=height, mie=C.component((2e-5,) * 3, mie_scale, 0.9, 0.76),
                             rayleigh=base.rayleigh, transmittance_shape=(4, 8), surface_radiance_shape=(3, 5),
                             ray_scatter_shape=(8, 101, 32, 8), ray_steps=100, sphere_steps=6, iterations=1)
    sweep = C.parameter_sweep(7)
    kinds = [(100000.0, 1200.0), (60000.0, 20.0), (60000.0, 200.0), (60000.0, 20.0), (35000.0, 1200.0),
             (60000.0, 250.0), (100000.0, 900.0)]
    cfgs = [mk(h, m, b) for (h, m), b in zip(kinds, sweep)]
    batch = A.build_batch(cfgs)
    for n, cfg in enumerate(cfgs):
        for key, value in A.build(cfg).items():
            assert np.array_equal(batch[key][n], value), (n, key)
