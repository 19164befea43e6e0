"""Ray scatter against the FP64 oracle where its launch shapes change: column
strides of the planes (sun elevations 2 to 33), no and few inner headings,
more columns than a block has threads (passes), odd and even ray steps on
both sides of a batch of 128 samples and of a buffer of 8 planes.

The oracle integrates the GPU's own point-scatter table.  FP64 within 2e-6.
FP32 within 1e-4 of the value and, at nodes darker than their neighbours along
the sun-elevation axis, within what the coordinate's rounding lets in: the
coordinate e <= n2 - 1 carries a few roundings, so its fraction is off by at
most 8 * 2^-24 (n2 - 1) and the result by that times the ray scatter of J's
largest value over sun elevations and headings."""
import numpy as np
import pytest

from oracle import oracle as O
from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu

# (height, elevation, sun elevation, sun heading), ray steps
CASES = [((2, 3, 2, 2), 4), ((3, 5, 3, 3), 7), ((2, 4, 4, 8), 8), ((3, 4, 16, 5), 9), ((2, 5, 19, 6), 16),
         ((2, 3, 31, 7), 17), ((3, 6, 32, 8), 127), ((2, 3, 32, 9), 30), ((2, 2, 33, 8), 24), ((4, 9, 8, 4), 128),
         ((2, 5, 5, 5), 129), ((2, 3, 7, 3), 258)]


@pytest.mark.parametrize("shape,steps", CASES, ids=[f"{'x'.join(map(str, s))}-S{n}" for s, n in CASES])
@pytest.mark.parametrize("precision", [C.FP64, C.FP32], ids=["fp64", "fp32"])
def test_ray_scatter_shapes(shape, steps, precision):
    mk = lambda p: C.make_config(height=100000.0, transmittance_shape=(3, 4), surface_radiance_shape=(3, 5),
                                 ray_scatter_shape=shape, ray_steps=steps, sphere_steps=6, iterations=1, precision=p)
    gpu = A.build(mk(precision), intermediates=True)
    J, got = gpu["point_scatter"][0].astype(np.float64), gpu["ray_scatter_delta"][0].astype(np.float64)
    bright = np.broadcast_to(J.max(axis=(2, 3), keepdims=True), J.shape).copy()
    want, most = np.empty_like(got), np.empty_like(got)
    for node in np.ndindex(*shape):
        want[node] = O.ray_scatter_node(mk(C.FP64), J, *node)
        if node[2:] == (0, 0):
            most[node[:2]] = O.ray_scatter_node(mk(C.FP64), bright, *node)
    assert np.isfinite(got).all()
    if precision == C.FP64:
        bound = 2e-6 * np.maximum(np.abs(want), 1e-6 * np.abs(want).max())
    else:
        bound = 1e-4 * np.maximum(np.abs(want), 1e-6 * np.abs(want).max()) + 8 * 2.0 ** -24 * (shape[2] - 1) * most
    assert (np.abs(got - want) <= bound).all(), float((np.abs(got - want) / bound).max())


# fewer columns than a block holds in few rows: the ray's samples are shared by
# groups of threads (4, 4, 2 and, with too many rows, 1), over parts that are
# uneven, shorter than a group's planes, empty, and of several batches
SPLIT = [((2, 5, 3, 3), 4), ((2, 5, 3, 3), 6), ((3, 7, 8, 4), 64), ((3, 7, 8, 4), 301), ((2, 9, 16, 8), 131),
         ((20, 150, 4, 4), 9)]


@pytest.mark.parametrize("shape,steps", SPLIT, ids=[f"{'x'.join(map(str, s))}-S{n}" for s, n in SPLIT])
@pytest.mark.parametrize("precision", [C.FP64, C.FP32], ids=["fp64", "fp32"])
def test_samples_shared_by_groups(shape, steps, precision):
    test_ray_scatter_shapes(shape, steps, precision)
