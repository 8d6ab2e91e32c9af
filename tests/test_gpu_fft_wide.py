"""The PM on meshes whose transforms take radices 18 and 24, first and last:
accelerations against the CPU oracle's PM, rms relative over all
particles, 1e-4 as in the other parity tests; in an ensemble beside a mesh with
small radices and a power of two, each box as it is alone, bit for bit; and 48,
whose last stage is the smallest radix, 3."""
import numpy as np
import pytest

import oracle
from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.ensemble import Ensemble
from conftest import rms_rel

pytestmark = pytest.mark.gpu

L = 50000.0


def case(M):
    rng = np.random.default_rng(M)
    pos = rng.uniform(0, L, size=(500, 3)).astype(np.float32)
    soft = 0.3 * L / M
    return pos, BoxConfig(n=500, pm_grid=M, cell_grid=max(8, M // 4), boxsize=L, mass=1.0, G=ics.G_INTERNAL,
                          softening=soft), oracle.reference_params(L, 1.0, ics.G_INTERNAL, M, soft)


def forces(pos, cfg):
    box = Box(cfg)
    box.set_state(pos)
    for _ in range(2):
        box.forces(pm=True, pp=False)
    acc = box.get_state()[3]
    box.close()
    return acc


@pytest.mark.parametrize("M", [48, 216, 288])
def test_one_box(port, M):
    pos, cfg, params = case(M)
    assert rms_rel(forces(pos, cfg), port.pm(pos, params, M, 4)) < 1e-4


def test_ensemble():
    cases = [case(M) for M in (162, 216, 50, 64)]
    ens = Ensemble([c for _, c, _ in cases])
    for b, (pos, _, _) in enumerate(cases):
        ens.set_state(b, pos)
    ens.forces()
    for b, (pos, cfg, _) in enumerate(cases):
        assert np.array_equal(ens.get_state(b)[3], forces(pos, cfg))
    ens.close()
