"""cuco_ensemble_footprint, which decides what a server admits, against what an
ensemble holds on the stand-in CUDA runtime: for given and tuned, even and odd
cell grids, small and ragged boxes, one and several; and, where no candidate of
the tuner has a finer cell grid than the box, against the most that it holds at
any time while it is created, the tuner's scratch included."""
import pytest

from fake_host import run

MEASURE = """
from cuco_gb300.serve import footprint
cfgs = [config(n, M, G, mode={mode}) for n, M, G in {boxes}]
for c, (_, _, G) in zip(cfgs, {boxes}):
    c.cell_grid = G or None
bound = footprint(cfgs)
before = fake.fake_live()
fake.fake_reset()
ens = Ensemble(cfgs)
held, peak = fake.fake_live() - before, fake.fake_peak() - before
"""


@pytest.mark.parametrize("mode", ["MODE_PLAIN", "MODE_FIXED"])
@pytest.mark.parametrize("boxes", [[(64 ** 3, 128, 64)], [(81 ** 3, 162, 41)], [(125 ** 3, 250, 63)], [(5000, 36, 17)],
                                   [(700, 24, 16)] * 5, [(32768, 64, 0)], [(4096, 32, 0), (5000, 100, 50), (80 ** 3, 160, 40)],
                                   [(1, 64, 33)], [(300, 24, 0)]])
def test_held(tmp_path, boxes, mode):
    run(tmp_path, MEASURE.format(mode=mode, boxes=boxes) + "assert held <= bound, (held, bound)")


@pytest.mark.parametrize("mode", ["MODE_PLAIN", "MODE_FIXED"])
@pytest.mark.parametrize("boxes", [[(64 ** 3, 128, 64)], [(81 ** 3, 162, 81)], [(5000, 36, 18)], [(700, 24, 16)] * 5,
                                   [(32768, 64, 0)], [(4096, 32, 0), (5000, 100, 50), (80 ** 3, 160, 0)], [(300, 24, 0)],
                                   [(200, 20, 20)] * 9 + [(20 ** 3, 200, 100)]])
def test_peak(tmp_path, boxes, mode):
    run(tmp_path, MEASURE.format(mode=mode, boxes=boxes) + "assert peak <= bound, (peak, bound)")


def test_peak_of_a_growing_ensemble(tmp_path):
    run(tmp_path, """
from cuco_gb300.serve import footprint
small, big = config(20 ** 3, 40, 20), config(64 ** 3, 128, 64)
before = fake.fake_live()
ens = Ensemble([small])
ens.set_state(0, np.zeros((20 ** 3, 3), np.float32))
fake.fake_reset()
ens.reshape([small, big], [0, -1])
peak = fake.fake_peak() - before
# (an array that grows to new sizes lives beside the state it carries over)
bound = footprint([small, big]) + footprint([small])
assert peak <= bound, (peak, bound)
""")
