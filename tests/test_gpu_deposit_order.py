"""The deposit's sums do not depend on how the particles fall into warps: a
particle's PM acceleration is the same bits in any input order, at counts whose
last warp is partial, with many particles in one mesh cell, others on the faces
where corners wrap, or no two of a warp in the same cell; and it agrees with
the CPU oracle's PM (rms relative over all particles, 1e-4 as in the other
parity tests)."""
import numpy as np
import pytest

import oracle
from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN
from conftest import rms_rel

pytestmark = pytest.mark.gpu

L, M = 1000.0, 32


def positions(n, kind):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, L, size=(n, 3))
    if kind == "clumped":  # two thirds in one mesh cell
        pos[: 2 * n // 3] = (np.array([5, 31, 0]) + rng.uniform(0.1, 0.9, size=(2 * n // 3, 3))) * (L / M)
    if kind == "faces":
        pos[:, n % 3] = np.where(np.arange(n) % 2, 0.0, L * (1 - 1e-4 / M))
    return pos.astype(np.float32)


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("kind", ["uniform", "clumped", "faces"])
@pytest.mark.parametrize("n", [3, 31, 32, 33, 63, 65, 1000])
def test_any_order(port, n, kind, mode):
    pos = positions(n, kind)
    cfg = BoxConfig(n=n, pm_grid=M, cell_grid=8, boxsize=L, mass=1.0, G=ics.G_INTERNAL, softening=0.3 * L / M,
                    mode=mode)

    def acc(order):
        box = Box(cfg)
        box.set_state(pos[order])
        box.forces(pm=True, pp=False)
        out = np.empty((n, 3), dtype=np.float32)
        out[order] = box.get_state()[3]
        box.close()
        return out

    first = acc(np.arange(n))
    assert np.array_equal(acc(np.arange(n)[::-1]), first)
    assert np.array_equal(acc(np.random.default_rng(1).permutation(n)), first)
    want = port.pm(pos, oracle.reference_params(L, 1.0, ics.G_INTERNAL, M, 0.3 * L / M), M, 4)
    assert rms_rel(first, want) < 1e-4
