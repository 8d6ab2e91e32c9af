"""Fixed-point positions read back as floats: the product u * L / 2^32 computed
in double and rounded to float, word for word, for the smallest u as well as
across the range, at values next to a float rounding boundary, and for box
lengths from tiny to large."""
import numpy as np
import pytest

from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxsize", [1.0, 50000.0, 133337.3, 99999.17, 1e-3, 3.3e-22, 1.7e9])
def test_words(boxsize):
    L = float(np.float32(boxsize))
    rng = np.random.default_rng(3)
    u = np.concatenate([np.arange(6000), 2 ** rng.integers(0, 32, 6000) + rng.integers(-2, 3, 6000),
                        rng.integers(0, 2 ** 24, 30000), rng.integers(0, 2 ** 32, 60000),
                        2 ** 32 - 1 - np.arange(2000)])
    # words whose product is nearest to the middle of two floats
    some = rng.integers(2 ** 25, 2 ** 32, 400000)
    exact = some.astype(np.float64) * (L / 2.0 ** 32)
    f = exact.astype(np.float32)
    gap = np.abs(np.abs(exact - f.astype(np.float64)) / np.spacing(f).astype(np.float64) - 0.5)
    u = np.concatenate([u, some[np.argsort(gap)[:20000]]])
    u = (u[:len(u) // 3 * 3] & 0xFFFFFFFF).astype(np.uint32).reshape(-1, 3)
    box = Box(BoxConfig(n=len(u), pm_grid=32, cell_grid=8, boxsize=L, mass=1.0, G=ics.G_INTERNAL,
                        softening=0.01 * L, mode=MODE_FIXED))
    box.set_state_fixed(u)
    got = box.get_state()[0]
    box.close()
    assert np.array_equal(got, (u.astype(np.float64) * (L / 2.0 ** 32)).astype(np.float32))
