"""The FP32 first order with fitted sun rays against the FP64 build, which
integrates every sun ray: passes over more cells than a block has threads, few
cells with the samples split over warps, odd step counts, segment counts that
follow the scale heights, batches of unlike atmospheres.  Within 1e-4 per
node (the bound of the FP32 parity tests) and 5e-6 in the 2-norm: the fits are
within 3e-6 of an optical depth, 8e-7 of a transmittance."""
import ctypes

import numpy as np
import pytest

from sfsim_gb300 import _lib
from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu


def config(shape, steps, precision, height=100000.0, mie_scale=1200.0, radius=6378000.0, rayleigh_scale=8000.0):
    return C.make_config(radius=radius, height=height, mie=C.component((2e-5,) * 3, mie_scale, 0.9, 0.76),
                         rayleigh=C.component((5.8e-6, 13.5e-6, 33.1e-6), rayleigh_scale),
                         transmittance_shape=(3, 4), surface_radiance_shape=(3, 5), ray_scatter_shape=shape,
                         ray_steps=steps, sphere_steps=4, iterations=0, precision=precision)


def check(got, want):
    for key in ("ray_scatter", "mie_strength"):
        g, w = got[key].astype(np.float64), want[key].astype(np.float64)
        err = np.abs(g - w) / np.maximum(np.abs(w), 1e-6 * np.abs(w).max())
        assert np.isfinite(g).all() and err.max() < 1e-4, (key, float(err.max()))
        assert np.linalg.norm(g - w) < 5e-6 * np.linalg.norm(w), key


# n0 n1 n2 n3 * steps / 3 above the size where fits are taken (18 * 8192 rays per segment)
CASES = [((4, 40, 32, 9), 90, {}), ((4, 101, 19, 6), 129, {}), ((6, 200, 8, 4), 100, {}),
         ((3, 100, 31, 7), 64, dict(radius=3000e3, mie_scale=800.0, rayleigh_scale=6000.0)),
         ((4, 101, 32, 8), 100, dict(height=60000.0, mie_scale=200.0)),
         ((5, 101, 16, 8), 61, dict(height=35000.0))]


@pytest.mark.parametrize("shape,steps,physics", CASES, ids=["x".join(map(str, s)) + f"-S{n}" for s, n, _ in CASES])
def test_fitted_first_order(shape, steps, physics):
    check(A.build(config(shape, steps, C.FP32, **physics)), A.build(config(shape, steps, C.FP64, **physics)))


def test_batch_of_unlike_atmospheres():
    """One batch shares its segments: those of the atmosphere that needs most."""
    physics = [dict(), dict(height=60000.0, mie_scale=200.0), dict(radius=3000e3, mie_scale=2000.0)]
    shape, steps = (4, 101, 32, 8), 100
    got = A.build_batch([config(shape, steps, C.FP32, **p) for p in physics])
    for n, p in enumerate(physics):
        check({k: v[n] for k, v in got.items()}, A.build(config(shape, steps, C.FP64, **p)))


def test_static_build_takes_the_same_fits():
    import torch
    cfg = config((6, 200, 8, 4), 100, C.FP32)
    want = A.build(cfg)
    out = [torch.empty(s, device="cuda") for s in A.table_shapes(cfg)]
    _lib.check(_lib.load().sfsim_atmo_build_static(ctypes.byref(cfg), *[t.data_ptr() for t in out],
                                                   torch.cuda.current_stream().cuda_stream), "static")
    for t, key in zip(out, ("transmittance", "surface_radiance", "ray_scatter", "mie_strength")):
        assert np.array_equal(t.cpu().numpy(), want[key]), key
