"""Ensembles whose particle total passes the sizes at which a single box's short
range takes larger units (155,648 and 311,296), with every box below them: each
box's short-range forces are still those it has alone, bit for bit, and so are
a served job's trajectories while a mix grows and shrinks across such a total."""
import numpy as np
import pytest

from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN
from cuco_gb300.ensemble import Ensemble
from cuco_gb300.serve import Job, Server
from helpers import clustered

pytestmark = pytest.mark.gpu

L = 1000.0


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("boxes", [3, 6])  # 156,000 and 312,000 particles
def test_forces_of_small_boxes_in_a_large_total(boxes, mode):
    n = 52000
    rng = np.random.default_rng(boxes)
    pos = [rng.uniform(0, L, size=(n, 3)).astype(np.float32) for _ in range(boxes - 1)] + [clustered(n, L, 5)]
    cfg = BoxConfig(n=n, pm_grid=64, cell_grid=16, boxsize=L, mass=1.0, G=ics.G_INTERNAL, softening=0.5, mode=mode)
    ens = Ensemble([cfg] * boxes)
    for b in range(boxes):
        ens.set_state(b, pos[b])
    ens.forces()
    box = Box(cfg)
    for b in (0, boxes - 1):
        box.set_state(pos[b])
        box.forces(pm=False, pp=True)
        assert np.array_equal(ens.get_state(b)[2], box.get_state()[2]), f"box {b}"
    box.close()
    ens.close()


def test_served_jobs_across_a_total():
    def jobs():
        out = []
        for k, (side, steps, arrival) in enumerate([(40, 4, 0), (36, 3, 1), (45, 3, 1)]):  # 64,000 then 201,781
            ic = ics.zeldovich(side, 80.0, 49.0, 30 + k)
            cfg = BoxConfig(n=ic.n, pm_grid=2 * side, boxsize=ic.boxsize, mass=ic.mass, G=ics.G_INTERNAL,
                            softening=0.07 * ic.boxsize / side, mode=MODE_FIXED)
            out.append(Job(k, cfg, ic.pos, ic.canonical_velocity(), ic.a, steps, arrival=float(arrival)))
        return out

    def served(some):
        srv = Server(1 << 40, clock=None)
        srv.clock = lambda: float(srv.ticks)
        return {j.job_id: j for j in srv.run(some)}, srv.peak_active

    mix, peak = served(jobs())
    assert peak == 3
    for job in jobs():
        alone = served([job])[0][job.job_id]
        assert np.array_equal(mix[job.job_id].result_pos, alone.result_pos)
        assert np.array_equal(mix[job.job_id].result_vel, alone.result_vel)
