"""Point scatter's sums are compensated: with a thousand and more directions
the FP32 result is as good as its last rounding.

A Rayleigh atmosphere without ground light, so that a term is a quadrature
weight, the flat phase and one lookup.  Relative to the result the last
rounding spreads by at most 2^-24 / sqrt(3) (uniform in half a unit, at the
least mantissa); the terms' own roundings average out over the directions and
runs (1e-8 with 1000 of them), so the spread stays within 1.25 times that.
What all nodes have in common (the rounding of the constants) is taken out.
The reference is the oracle's point scatter of the GPU's own first-order
tables."""
import numpy as np
import pytest

from oracle import oracle as O
from sfsim_gb300 import atmosphere_lut as A
from sfsim_gb300 import config as C

pytestmark = pytest.mark.gpu

CASES = [((3, 40, 4, 2), 48), ((2, 65, 3, 3), 60), ((2, 129, 4, 2), 56), ((2, 70, 3, 4), 50)]


@pytest.mark.parametrize("shape,sphere", CASES, ids=["x".join(map(str, s)) + f"-sphere{p}" for s, p in CASES])
def test_sums_to_the_last_rounding(shape, sphere):
    cfg = C.make_config(height=100000.0, brightness=(0.0,) * 3, mie=C.component((0.0,) * 3, 1200.0, 0.9, 0.76),
                        transmittance_shape=(3, 4), surface_radiance_shape=(3, 5), ray_scatter_shape=shape,
                        ray_steps=16, sphere_steps=sphere, iterations=1)
    gpu = A.build(cfg, intermediates=True)
    t64 = lambda k: np.asarray(gpu[k], dtype=np.float64)
    got = t64("point_scatter")[0]
    want = np.empty_like(got)
    for node in np.ndindex(*shape):
        want[node] = O.point_scatter_node(cfg, t64("rayleigh_first"), t64("surface_base"), *node,
                                          mie_first=t64("mie_first"))
    bright = want > 1e-2 * want.max()
    err = got[bright] / want[bright] - 1.0
    assert bright.sum() > 500
    assert err.std() <= 1.25 * 2.0 ** -24 / np.sqrt(3.0), float(err.std())
    assert np.abs(err).max() < 1e-6
