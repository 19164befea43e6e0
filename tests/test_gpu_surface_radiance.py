"""Surface radiance against the FP64 oracle where its ring sums change shape
(one ring, odd ring sizes, the fewest headings, more texels than a block has
threads, node coordinates on and off the table), and the allocation-free
build where it keeps only some lights' weights at a time.  FP32 within 1e-4,
FP64 within 2e-6 (the bounds of the whole build's parity tests)."""
import ctypes
import re

import numpy as np
import pytest

from oracle import oracle as O
from sfsim_gb300 import _lib
from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu
TOL = {C.FP32: 1e-4, C.FP64: 2e-6}
STATIC_BYTES = 64 << 20

# (height, elevation, sun elevation, sun heading), ray steps, surface-radiance shape
CASES = [((2, 5, 3, 2), 4, (2, 3)), ((3, 6, 2, 3), 5, (3, 4)), ((2, 7, 4, 4), 11, (2, 9)), ((4, 5, 3, 7), 37, (3, 3)),
         ((2, 8, 3, 16), 36, (3, 5)), ((3, 5, 5, 8), 64, (5, 5)), ((2, 4, 3, 33), 21, (2, 2))]


@pytest.mark.parametrize("shape,steps,eshape", CASES,
                         ids=[f"{'x'.join(map(str, s))}-steps{n}-E{'x'.join(map(str, e))}" for s, n, e in CASES])
@pytest.mark.parametrize("precision", [C.FP64, C.FP32], ids=["fp64", "fp32"])
def test_surface_radiance_shapes(shape, steps, eshape, precision):
    cfg = C.make_config(height=100000.0, transmittance_shape=(3, 4), surface_radiance_shape=eshape,
                        ray_scatter_shape=shape, ray_steps=steps, sphere_steps=4, iterations=2, precision=precision)
    gpu = A.build(cfg, intermediates=True)
    # each iteration against the oracle's surface radiance of the GPU's own tables before it
    t64 = lambda k: np.asarray(gpu[k], dtype=np.float64)
    sources = [(t64("rayleigh_first"), t64("mie_first")), (t64("ray_scatter_delta")[0], None)]
    for it, (dS, mie) in enumerate(sources):
        g = np.asarray(gpu["surface_delta"][it])
        r = np.empty_like(g, dtype=np.float64)
        for i, k in np.ndindex(*eshape):
            r[i, k] = O.surface_radiance_node(cfg, dS, i, k, mie_first=mie)
        err = np.abs(g - r) / np.maximum(np.abs(r), 1e-6 * np.abs(r).max())
        assert np.isfinite(g).all() and err.max() <= TOL[precision], float(err.max())


def test_static_build_with_weights_in_parts():
    """The allocation-free build of the largest transmittance table that it
    accepts beside many lights: their weights do not all fit its array, and
    the tables are those of the ordinary build."""
    import torch

    L = _lib.load()
    lights, rows = 4000, 1024

    def config(columns):
        return C.make_config(height=100000.0, transmittance_shape=(rows, columns), surface_radiance_shape=(2, lights),
                             ray_scatter_shape=(2, 5, 3, 8), ray_steps=64, sphere_steps=4, iterations=2)

    def static(columns):
        cfg = config(columns)
        out = [torch.empty(tuple(s), dtype=torch.float32, device="cuda") for s in A.table_shapes(cfg)]
        rc = L.sfsim_atmo_build_static(ctypes.byref(cfg), *[t.data_ptr() for t in out],
                                       torch.cuda.current_stream().cuda_stream)
        _lib.check(rc, "sfsim_atmo_build_static")
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in out]

    with pytest.raises(_lib.AtmoError) as refused:
        static(2048)
    needs = int(re.search(r"needs (\d+) bytes", str(refused.value)).group(1))
    columns = 2048 - -(-(needs - STATIC_BYTES) // (32 * rows))  # 32 bytes of scratch a transmittance node
    got = static(columns)
    launches = A.last_launch_count()
    want = A.build(config(columns))
    assert launches > A.last_launch_count()
    for g, k in zip(got, ("transmittance", "surface_radiance", "ray_scatter", "mie_strength")):
        assert np.array_equal(g, want[k]), k


# the scratch that the allocation-free build counts for a configuration is part
# of its contract: it decides what is refused
@pytest.mark.parametrize("precision,shape,sphere,tshape,eshape,needs",
                         [(C.FP32, (12, 400, 20, 8), 4, (99, 99), (16, 64), 147622144),
                          (C.FP64, (20, 180, 31, 7), 2, (9, 11), (5, 13), 273119744)], ids=["fp32", "fp64"])
def test_static_build_counts_the_same_scratch(precision, shape, sphere, tshape, eshape, needs):
    cfg = C.make_config(height=100000.0, transmittance_shape=tshape, surface_radiance_shape=eshape,
                        ray_scatter_shape=shape, ray_steps=100, sphere_steps=sphere, precision=precision)
    import torch
    out = [torch.empty(tuple(t), dtype=torch.float32, device="cuda") for t in A.table_shapes(cfg)]
    rc = _lib.load().sfsim_atmo_build_static(ctypes.byref(cfg), *[t.data_ptr() for t in out], None)
    with pytest.raises(_lib.AtmoError, match=f"needs {needs} bytes"):
        _lib.check(rc, "sfsim_atmo_build_static")
