"""Table lookups and attenuation where the 16-byte reads of neighbouring texels
meet every alignment and the tables' edges: the narrowest tables, odd widths,
and tables whose size is no multiple of 16 bytes.  The same comparisons and
bounds as on the production tables."""
import pytest

from sfsim_gb300 import config as C
from sfsim_gb300.query import Context
from tests.test_gpu_query import _check_attenuation, _check_table_queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tshape,shape", [((2, 2), (2, 2, 2, 2)), ((3, 5), (3, 3, 3, 3)), ((5, 7), (2, 5, 3, 7)),
                                          ((4, 9), (5, 6, 5, 3)), ((7, 3), (3, 7, 2, 5))],
                         ids=lambda s: "x".join(map(str, s)))
def test_lookups_on_odd_tables(tshape, shape):
    cfg = C.make_config(height=100000.0, transmittance_shape=tshape, surface_radiance_shape=(3, 4),
                        ray_scatter_shape=shape, ray_steps=8, sphere_steps=4, iterations=1)
    ctx = Context(cfg)
    try:
        _check_table_queries(cfg, ctx, 5)
        _check_attenuation(cfg, ctx, 6)
    finally:
        ctx.close()
