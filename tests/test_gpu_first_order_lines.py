"""Which FP32 builds take fitted sun rays in the first order.

Below 1.9e7 ray-scatter cells times ray steps every sun ray is integrated: a
node's first order then depends on its own coordinates alone, so the nodes
that a small and a larger table share are equal bit for bit.  Above it the
fits are taken (one launch more), within 1e-4 per node and 5e-6 in the 2-norm
of the FP64 build, over cells in several passes, few cells with their samples
split over warps, odd step counts, segment counts that follow the scale
heights, and steps that do not resolve the density peak."""
import ctypes

import numpy as np
import pytest

from sfsim_gb300 import _lib
from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C
from tests.test_gpu_first_order_fit import check, config

pytestmark = pytest.mark.gpu


def launches(cfg):
    A.build(cfg)
    return A.last_launch_count()


@pytest.mark.parametrize("steps,physics", [(36, {}), (70, dict(height=60000.0, mie_scale=2000.0))],
                         ids=["earth-S36", "60km-S70"])
def test_integrated_below(steps, physics):
    small, large = [A.build(config((5, 80, 32, n3), steps, C.FP32, **physics), intermediates=True) for n3 in (3, 9)]
    for key in ("rayleigh_first", "mie_first"):
        assert np.array_equal(large[key][..., ::4, :], small[key]), key


CASES = [((8, 101, 32, 9), 90, {}), ((14, 101, 19, 6), 129, {}), ((25, 250, 8, 4), 100, {}),
         ((14, 100, 31, 7), 64, dict(radius=3000e3, mie_scale=800.0, rayleigh_scale=6000.0)),
         ((8, 101, 32, 8), 100, dict(height=60000.0, mie_scale=200.0)),
         ((16, 160, 16, 8), 61, dict(height=35000.0)),
         # steps that do not resolve the density peak (3 sqrt(H / h) = 67 and 52)
         ((15, 255, 32, 8), 64, dict(mie_scale=200.0)), ((21, 255, 32, 8), 45, dict(height=60000.0, mie_scale=200.0))]


@pytest.mark.parametrize("shape,steps,physics", CASES, ids=["x".join(map(str, s)) + f"-S{n}" for s, n, _ in CASES])
def test_fitted_above(shape, steps, physics):
    got = A.build(config(shape, steps, C.FP32, **physics))
    assert A.last_launch_count() == launches(config((2, 3, 4, 4), steps, C.FP32, **physics)) + 1
    check(got, A.build(config(shape, steps, C.FP64, **physics)))


def test_static_build_takes_the_same_fits():
    import torch

    def static(cfg):
        out = [torch.empty(s, device="cuda") for s in A.table_shapes(cfg)]
        _lib.check(_lib.load().sfsim_atmo_build_static(ctypes.byref(cfg), *[t.data_ptr() for t in out],
                                                       torch.cuda.current_stream().cuda_stream), "static")
        return out, A.last_launch_count()
    cfg = config((6, 200, 8, 4), 510, C.FP32)
    out, count = static(cfg)
    assert count == static(config((2, 3, 4, 4), 510, C.FP32))[1] + 1
    want = A.build(cfg)
    for t, key in zip(out, ("transmittance", "surface_radiance", "ray_scatter", "mie_strength")):
        assert np.array_equal(t.cpu().numpy(), want[key]), key
