"""The fitted first order's sums are compensated: with thousands of ray steps
the FP32 Mie strength is as good as its last roundings.

The atmosphere is transparent (every transmittance rounds to 1), so that a
node's Mie strength is the sum of its lit samples' densities times two
constants.  The total, and each of the two products, is rounded once, by at
most 2^-24 relative: a spread of sqrt(3) 2^-24 / sqrt(3) at most.  The
samples' own roundings average out over the steps that matter (hundreds of
them, below 1e-8), so the spread over the nodes stays within 1.25 times
that.  What all nodes have in common is taken out."""
import numpy as np
import pytest

from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,steps", [((4, 12, 16, 8), 4096), ((4, 13, 19, 11), 2047)],
                         ids=["4x12x16x8-S4096", "4x13x19x11-S2047"])
def test_sums_to_the_last_rounding(shape, steps):
    def first(precision):
        cfg = C.make_config(height=35000.0, mie=C.component((1e-12,) * 3, 6000.0, 0.9, 0.76),
                            rayleigh=C.component((1e-12,) * 3, 8000.0), transmittance_shape=(2, 2),
                            surface_radiance_shape=(2, 2), ray_scatter_shape=shape, ray_steps=steps, sphere_steps=2,
                            iterations=0, precision=precision)
        return A.build(cfg, intermediates=True)["mie_first"].astype(np.float64)
    got, want = first(C.FP32), first(C.FP64)
    bright = want > 1e-2 * want.max()
    err = got[bright] / want[bright] - 1.0
    assert bright.sum() > 1000
    assert err.std() <= 1.25 * 2.0 ** -24, float(err.std())
    assert np.abs(err).max() < 2e-6
