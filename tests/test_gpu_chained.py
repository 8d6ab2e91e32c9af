"""Steps whose kernels are launched chained (each may start while the one
before it ends) against the same steps with timing events between the phases,
which keeps the launches apart: the same bits after many steps, on meshes with
register and mixed-radix transforms, below and at the size where the PM's
launches are no longer chained, with sorts of one launch and of several."""
import numpy as np
import pytest

from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN

pytestmark = pytest.mark.gpu

L = 50000.0


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("n,M", [(500, 32), (5000, 36), (32768, 64), (65536, 128), (65537, 100), (90000, 256)])
def test_same_bits(n, M, mode):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, L, size=(n, 3)).astype(np.float32)
    vel = rng.normal(0, 50.0, size=(n, 3)).astype(np.float32)
    cfg = BoxConfig(n=n, pm_grid=M, cell_grid=max(8, M // 4), boxsize=L, mass=1.0, G=ics.G_INTERNAL,
                    softening=0.3 * L / M, mode=mode)
    states = []
    for timing in (False, True, False):
        box = Box(cfg)
        box.enable_timing(timing)
        box.set_state(pos, vel)
        for _ in range(20):
            box.step(0.5, 0.5)
        states.append(box.get_state())
        box.close()
    for other in states[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(states[0], other))
