"""Loss and gradients of a training batch against the NumPy reference where the
launches change shape: the smallest batch, an odd number of row blocks, more
tiles than SMs with a partial last wave, and more rows than the head's blocks
take in one pass.  Bounds of the existing gradient test (2e-2 of each tensor's
norm, 1e-3 of the loss)."""
import numpy as np
import pytest

from sfsim_gb300 import config as C
from sfsim_gb300 import query
from tests.mlp_reference import SHAPES, loss_and_grads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    cfg = C.make_config(height=35000.0, transmittance_shape=(8, 16), surface_radiance_shape=(4, 8),
                        ray_scatter_shape=(4, 9, 4, 4), ray_steps=8, sphere_steps=4, iterations=1)
    with query.Context(cfg) as c:
        yield c


@pytest.mark.parametrize("n", [1024, 3072, 20480, 40960])
def test_gradients_by_batch_size(ctx, n):
    rng = np.random.default_rng(n)
    coords = rng.uniform(0, 1, (n, 10)).astype(np.float32)
    targets = rng.normal(0, 0.5, (n, 3)).astype(np.float32)
    loss, grads = ctx.surrogate_gradients(coords, targets)
    rloss, rgrads = loss_and_grads(ctx.surrogate_parameters(), coords, targets)
    assert abs(loss - rloss) <= 1e-3 * abs(rloss)
    o = 0
    for rows, cols in SHAPES:
        for size in (rows * cols, rows):
            g, rg = grads[o:o + size], rgrads[o:o + size]
            o += size
            assert np.linalg.norm(g - rg) <= 2e-2 * max(np.linalg.norm(rg), 1e-30), (rows, cols, size)
    assert o == grads.size
