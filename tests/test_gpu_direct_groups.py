"""Direct queries against the FP64 oracle where the launch changes shape: fewer
queries than a group, a last group and a last warp that are not full, fewer
samples than a warp's lanes, and sun rays by the build's fits and integrated.
The bound of the existing direct-query test (1e-4 of the value, with its
floor)."""
import numpy as np
import pytest

from oracle import oracle as O
from sfsim_gb300 import config as C
from sfsim_gb300.query import Context
from tests.test_gpu_query import random_queries, rel_err

pytestmark = pytest.mark.gpu

# (height, elevation, sun elevation, sun heading), ray steps: the last two builds have fits
CASES = [((3, 9, 4, 4), 5, 3), ((3, 9, 4, 4), 31, 77), ((3, 9, 4, 4), 33, 64), ((4, 101, 32, 8), 100, 77),
         ((4, 200, 31, 7), 61, 130)]


@pytest.mark.parametrize("shape,steps,n", CASES, ids=[f"{'x'.join(map(str, s))}-S{t}-n{n}" for s, t, n in CASES])
def test_direct_query_groups(shape, steps, n):
    import torch
    cfg = C.make_config(height=100000.0, transmittance_shape=(4, 8), surface_radiance_shape=(3, 5),
                        ray_scatter_shape=shape, ray_steps=steps, sphere_steps=4, iterations=1)
    x, v, l = random_queries(cfg, n, steps)
    with Context(cfg) as ctx:
        got = ctx.direct(*[torch.tensor(a, dtype=torch.float64, device="cuda") for a in (x, v, l)]).cpu().numpy()
        jsum = ctx.point_scatter_sum().cpu().numpy()[..., :3].astype(np.float64)
    ref = np.array([O.rendered_inscatter(cfg, x[i], v[i], l[i], jsum) for i in range(n)])
    assert np.isfinite(got).all() and rel_err(got, ref).max() <= 1e-4, float(rel_err(got, ref).max())
