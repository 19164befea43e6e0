"""Blue-noise ranks against the FP64 oracle, exactly, where the tiled steps
change shape: tables smaller than a tile, ragged tiles, the most pixels that fit
and the first that do not, and widths of the weights around the line between
the tiles and the kernels that update every pixel."""
import numpy as np
import pytest

from oracle import oracle as O
from sfsim_gb300 import noise

pytestmark = pytest.mark.gpu

CASES = [(2, 1.5, 2), (3, 0.4, 1), (5, 1.5, 12), (8, 30.0, 6), (9, 1.0, 40), (33, 2.0, 1), (45, 1.5, 202),
         (48, 2.8, 1152), (48, 3.2, 200), (63, 0.6, 500), (64, 1.5, 2048), (66, 2.8, 400), (66, 2.9, 400),
         (100, 1.5, 1000), (133, 1.5, 1700), (137, 1.5, 1800)]


@pytest.mark.parametrize("m,sigma,n", CASES, ids=[f"{m}-sigma{s}-n{n}" for m, s, n in CASES])
def test_ranks_exactly(m, sigma, n):
    pixels = np.random.default_rng(m).permutation(m * m)[:n]
    np.testing.assert_array_equal(noise.blue_noise(m, sigma=sigma, seed_pixels=pixels), O.blue(m, pixels, sigma))


def test_regular_pattern():
    """Equal densities throughout: the order of equal keys decides."""
    m = 32
    pixels = np.array([y * m + x for y in range(0, m, 4) for x in range(0, m, 4)])
    np.testing.assert_array_equal(noise.blue_noise(m, sigma=1.5, seed_pixels=pixels), O.blue(m, pixels, 1.5))
