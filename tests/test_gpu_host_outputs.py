"""Host outputs inside one larger buffer, at odd word offsets: the build makes
the outputs' pages present before it copies into them and touches nothing
else."""
import ctypes

import numpy as np
import pytest

from sfsim_gb300 import _lib
from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu


def test_outputs_inside_a_larger_buffer():
    cfg = C.make_config(height=100000.0, transmittance_shape=(300, 301), surface_radiance_shape=(5, 7),
                        ray_scatter_shape=(8, 64, 16, 12), ray_steps=8, sphere_steps=4, iterations=1)
    want = A.build(cfg)
    keys = ("transmittance", "surface_radiance", "ray_scatter", "mie_strength")
    assert sum(want[k].nbytes > 1 << 20 for k in keys) == 3  # the sizes that are populated
    buf = np.full(sum(want[k].size + 101 for k in keys) + 101, -7.0, np.float32)
    at, ptrs = 101, []
    for k in keys:
        ptrs.append((at, want[k].size))
        at += want[k].size + 101
    fp = ctypes.POINTER(ctypes.c_float)
    args = [ctypes.cast(buf.ctypes.data + 4 * o, fp) for o, _ in ptrs]
    _lib.check(_lib.load().sfsim_atmo_build(ctypes.byref(cfg), *args), "build")
    for (o, n), k in zip(ptrs, keys):
        assert np.array_equal(buf[o:o + n], want[k].ravel()), k
        buf[o:o + n] = -7.0
    assert (buf == -7.0).all()
