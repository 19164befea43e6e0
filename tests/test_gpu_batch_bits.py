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
