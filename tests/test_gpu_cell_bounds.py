"""Bounds given to cudaForceEvaluateShortrange that leave particles out: cells
marked empty (0xffffffff, or an end not above the start) whose particles are
still in the sorted array, single cells and whole columns of them, at both ends
and in between.  The particles of
the other cells get the forces of a box that holds only them (against the CPU
oracle, rms relative 1e-4), the others are neither sources nor targets: their
accelerations are left as they were."""
import numpy as np
import pytest
import torch

from conftest import rms_rel
from test_gpu_cell_grids import L, Gravlist

pytestmark = pytest.mark.gpu

G = 32


@pytest.mark.parametrize("mark", [0xFFFFFFFF, 5])
@pytest.mark.parametrize("masked", ["column", "cells", "first", "last", "none"])
def test_masked_cells(port, masked, mark):
    rng = np.random.default_rng(11)
    n = 20000
    pos = rng.uniform(0, L, size=(n, 3)).astype(np.float32)
    g = Gravlist(pos, G, G, 0.02 * L / G)
    cells = torch.arange(g.ncell, device="cuda:0")
    keep = {"column": (cells // G) % 7 != 3, "cells": cells % 5 != 2, "first": cells >= 9 * G + 5,
            "last": cells < g.ncell - 6 * G - 11, "none": cells >= 0}[masked]
    g.start[~keep] = np.uint32(mark).astype(np.int32).item()
    if mark == 5:
        g.end[~keep] = 5
    covered = keep[g.keys.long()].cpu().numpy()  # in sorted order
    at = g.perm.cpu().numpy()[covered]
    g.acc[:] = 7.0
    got = g.forces()
    assert rms_rel(got[at], port.pp(np.ascontiguousarray(pos[at]), g.params, G, 8)) < 1e-4
    left = np.ones(n, dtype=bool)
    left[at] = False
    assert (got[left] == 7.0).all()


@pytest.mark.parametrize("shift", [1, 2])
def test_bounds_at_any_word(port, shift):
    """Bounds that do not lie on 16 bytes, contiguous and with cells left out."""
    rng = np.random.default_rng(shift)
    pos = rng.uniform(0, L, size=(9000, 3)).astype(np.float32)
    for G, left_out in ((21, False), (21, True), (110, False), (110, True)):
        g = Gravlist(pos, G, G, 0.02 * L / G)
        if left_out:
            g.start[::3] = -1
        want = g.forces()
        held = [torch.empty(g.ncell + shift, dtype=torch.int32, device="cuda:0") for _ in range(2)]
        for h, a in zip(held, (g.start, g.end)):
            h[shift:] = a
        g.start, g.end = held[0][shift:], held[1][shift:]
        g.acc[:] = 0
        assert np.array_equal(g.forces(), want)
