"""Boxes whose particles share a warp of the batched launches: equal boxes,
where a lane's particle and another box's have the same mesh cell, and boxes of
different meshes; each box's PM accelerations as it is alone, bit for bit."""
import numpy as np
import pytest

from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN
from cuco_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu

L = 1000.0


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("boxes", [[(16, 32)] * 4, [(5, 24), (5, 24), (70, 24)], [(40, 32), (40, 36), (33, 24), (1, 24)]])
def test_boxes_in_one_warp(boxes, mode):
    rng = np.random.default_rng(7)
    pos = rng.uniform(0, L, size=(70, 3)).astype(np.float32)
    cfgs = [BoxConfig(n=n, pm_grid=M, cell_grid=8, boxsize=L, mass=1.0, G=ics.G_INTERNAL, softening=0.3 * L / M,
                      mode=mode) for n, M in boxes]
    ens = Ensemble(cfgs)
    for b, c in enumerate(cfgs):
        ens.set_state(b, pos[:c.n])
    ens.forces()
    for b, c in enumerate(cfgs):
        box = Box(c)
        box.set_state(pos[:c.n])
        box.forces(pm=True, pp=False)
        assert np.array_equal(ens.get_state(b)[3], box.get_state()[3])
        box.close()
    ens.close()
