"""The PM of a scattered state (read in cell order, after the sort) against the
same particles in an order that does not scatter them (read as they come,
beside the sort): every particle's accelerations bit for bit, in both forms,
on both sides of the sizes where the schedule changes, alone and with the
short range, and after a step.  The small case is checked against the oracle
elsewhere; here the two routes check each other."""
import numpy as np
import pytest

from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN

pytestmark = pytest.mark.gpu

L = 100000.0


def run(cfg, pos, vel, order, pm_only):
    box = Box(cfg)
    box.set_state(pos[order], vel[order])
    if pm_only:
        box.forces(pm=True, pp=False)
    else:
        box.step(3e-5, 1e-3)
    p, v, app, apm = box.get_state()
    box.close()
    back = np.empty_like(order)
    back[order] = np.arange(len(order))
    return [a[back] for a in ((apm,) if pm_only else (p, v, app, apm))]


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("side,M,pm_only", [(79, 160, True), (80, 160, True), (80, 160, False), (80, 150, True),
                                            (104, 200, False)])
def test_order_does_not_change_the_forces(side, M, pm_only, mode):
    rng = np.random.default_rng(side)
    n = side ** 3
    pos = rng.uniform(0, L, size=(n, 3)).astype(np.float32)
    pos[pos >= np.float32(L)] = 0
    vel = rng.normal(0, 1e5, size=(n, 3)).astype(np.float32)
    cfg = BoxConfig(n=n, pm_grid=M, boxsize=L, mass=1.0, G=ics.G_INTERNAL, softening=0.07 * L / side, mode=mode)
    cell = np.minimum((pos / L * (M // 4)).astype(np.int64), M // 4 - 1)
    local = np.argsort((cell[:, 0] * M + cell[:, 1]) * M + cell[:, 2], kind="stable")
    for a, b in zip(run(cfg, pos, vel, np.arange(n), pm_only), run(cfg, pos, vel, local, pm_only)):
        # the order within a cell differs, and with it the short range's
        # summation order; the PM's accelerations do not depend on it
        if pm_only:
            assert np.array_equal(a, b)
        else:
            assert np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(b)
