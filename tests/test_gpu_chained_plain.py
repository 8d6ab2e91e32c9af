"""Steps whose kernels are launched chained against the same box in an ensemble
of one, whose transforms, cell order and drift are launched plainly: the same
bits after many steps, for register and mixed-radix transforms, one-launch and
three-kernel sorts, below the mesh where the chaining stops."""
import numpy as np
import pytest

from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN
from cuco_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu

L = 50000.0


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("n,M", [(700, 32), (5000, 36), (32768, 64), (65537, 100), (40000, 128), (30000, 216)])
def test_same_bits(n, M, mode):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, L, size=(n, 3)).astype(np.float32)
    vel = rng.normal(0, 50.0, size=(n, 3)).astype(np.float32)
    cfg = BoxConfig(n=n, pm_grid=M, cell_grid=max(16, M // 4), boxsize=L, mass=1.0, G=ics.G_INTERNAL,
                    softening=0.3 * L / M, mode=mode)
    box, ens = Box(cfg), Ensemble([cfg])
    box.set_state(pos, vel)
    ens.set_state(0, pos, vel)
    for _ in range(12):
        box.step(0.5, 0.5)
        ens.step(0.5, 0.5)
    ens.sync()
    assert all(np.array_equal(a, b) for a, b in zip(box.get_state(), ens.get_state(0)))
    box.close()
    ens.close()
