"""The PM on meshes that between them take every radix of the mixed-radix
transform (2 to 16, one to three stages) and every register transform, with an
odd half mesh among them: accelerations against the CPU oracle's PM, rms
relative over all particles, 1e-4 as in the other parity tests."""
import numpy as np
import pytest

import oracle
from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.ensemble import Ensemble
from conftest import rms_rel

pytestmark = pytest.mark.gpu

L = 50000.0
MESHES = [8, 10, 12, 16, 18, 20, 24, 30, 32, 36, 50, 54, 60, 64, 90, 96, 108, 120, 128, 150, 162, 180]


def case(M):
    rng = np.random.default_rng(M)
    pos = rng.uniform(0, L, size=(700, 3)).astype(np.float32)
    soft = 0.3 * L / M
    return pos, BoxConfig(n=700, pm_grid=M, cell_grid=max(8, M // 4), boxsize=L, mass=1.0, G=ics.G_INTERNAL,
                          softening=soft), oracle.reference_params(L, 1.0, ics.G_INTERNAL, M, soft)


@pytest.mark.parametrize("M", MESHES)
def test_one_box(port, M):
    pos, cfg, params = case(M)
    box = Box(cfg)
    box.set_state(pos)
    for _ in range(2):  # the second pass finds the deposit grid as the first left it
        box.forces(pm=True, pp=False)
    acc = box.get_state()[3]
    box.close()
    assert rms_rel(acc, port.pm(pos, params, M, 4)) < 1e-4


def test_ensemble_of_all():
    """Each box as it is alone, bit for bit."""
    cases = [case(M) for M in MESHES if M >= 32]
    ens = Ensemble([c for _, c, _ in cases])
    for b, (pos, _, _) in enumerate(cases):
        ens.set_state(b, pos)
    ens.forces()
    for b, (pos, cfg, _) in enumerate(cases):
        box = Box(cfg)
        box.set_state(pos)
        box.forces(pm=True, pp=False)
        alone = box.get_state()[3]
        box.close()
        assert np.array_equal(ens.get_state(b)[3], alone)
    ens.close()
