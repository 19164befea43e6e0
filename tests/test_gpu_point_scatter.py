"""Point scatter against the FP64 oracle where its launch shapes change: the
groupings of headings (pairs per thread, several groups, no inner heading),
the edges of a block of elevations, the fewest rings, and a surface-radiance
row that fills shared memory.  FP32 within 1e-4, FP64 within 2e-6 (the bounds
of the whole build's parity tests)."""
import numpy as np
import pytest

from oracle import oracle as O
from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu
TOL = {C.FP32: 1e-4, C.FP64: 2e-6}

# (height, elevation, sun elevation, sun heading), sphere steps, surface-radiance shape
CASES = [((2, 5, 3, 2), 6, (3, 5)), ((2, 5, 3, 3), 6, (3, 5)), ((3, 127, 3, 4), 5, (3, 5)),
         ((2, 128, 4, 5), 7, (2, 9)), ((2, 129, 3, 6), 6, (3, 5)), ((2, 43, 3, 8), 9, (2, 64)),
         ((2, 65, 3, 9), 2, (3, 5)), ((2, 33, 4, 16), 3, (3, 5)), ((2, 4, 3, 8), 4, (2, 8400))]


@pytest.mark.parametrize("shape,sphere,eshape", CASES,
                         ids=[f"{'x'.join(map(str, s))}-sphere{p}-E{'x'.join(map(str, e))}" for s, p, e in CASES])
@pytest.mark.parametrize("precision", [C.FP64, C.FP32], ids=["fp64", "fp32"])
def test_point_scatter_shapes(shape, sphere, eshape, precision):
    if precision == C.FP64 and eshape[1] > 4000:
        pytest.skip("the FP64 table of that size exceeds shared memory")
    mk = lambda p: C.make_config(height=100000.0, transmittance_shape=(3, 4), surface_radiance_shape=eshape,
                                 ray_scatter_shape=shape, ray_steps=8, sphere_steps=sphere, iterations=2, precision=p)
    ref = O.build(mk(C.FP64), intermediates=True)
    gpu = A.build(mk(precision), intermediates=True)
    # the first iteration against the oracle's build, the second against the
    # oracle's point scatter of the GPU's own tables of the first (the FP32 ray
    # scatter between them carries its own error at the darkest nodes)
    second = np.empty_like(ref["point_scatter"][1])
    dS, dE = (gpu[k][0].astype(np.float64) for k in ("ray_scatter_delta", "surface_delta"))
    for node in np.ndindex(*shape):
        second[node] = O.point_scatter_node(mk(C.FP64), dS, dE, *node)
    for g, r in ((gpu["point_scatter"][0], ref["point_scatter"][0]), (gpu["point_scatter"][1], second)):
        err = np.abs(g - r) / np.maximum(np.abs(r), 1e-6 * np.abs(r).max())
        assert np.isfinite(g).all() and err.max() <= TOL[precision], float(err.max())


# (n0, n1, n2, n3), sphere steps, atmospheres: directions shared by 8, 4 (with
# lanes left over) and 2 threads an item, by as many as fill a warp in a large
# batch, and more threads than a ring has directions
SHARED = [((2, 16, 3, 4), 9, 1), ((2, 11, 3, 6), 12, 1), ((2, 30, 3, 9), 7, 1), ((3, 63, 2, 5), 8, 1),
          ((8, 5, 16, 8), 8, 15), ((2, 3, 2, 3), 2, 1)]


@pytest.mark.parametrize("shape,sphere,batch", SHARED,
                         ids=[f"{'x'.join(map(str, s))}-sphere{p}-B{b}" for s, p, b in SHARED])
@pytest.mark.parametrize("precision", [C.FP64, C.FP32], ids=["fp64", "fp32"])
def test_shared_directions(shape, sphere, batch, precision):
    cfg = C.make_config(height=100000.0, transmittance_shape=(3, 4), surface_radiance_shape=(3, 5),
                        ray_scatter_shape=shape, ray_steps=8, sphere_steps=sphere, iterations=1, precision=precision)
    if batch > 1:
        # every atmosphere of the batch as the build of one
        one, many = A.build(cfg), A.build_batch([cfg] * batch)
        for key, value in one.items():
            err = np.abs(many[key] - value[None]) / np.maximum(np.abs(value), 1e-6 * np.abs(value).max())
            assert err.max() <= TOL[precision], (key, float(err.max()))
        return
    gpu = A.build(cfg, intermediates=True)
    t64 = lambda k: np.asarray(gpu[k], dtype=np.float64)
    ref = np.empty_like(t64("point_scatter")[0])
    for node in np.ndindex(*shape):
        ref[node] = O.point_scatter_node(cfg, t64("rayleigh_first"), t64("surface_base"), *node,
                                         mie_first=t64("mie_first"))
    err = np.abs(t64("point_scatter")[0] - ref) / np.maximum(np.abs(ref), 1e-6 * np.abs(ref).max())
    assert err.max() <= TOL[precision], float(err.max())
