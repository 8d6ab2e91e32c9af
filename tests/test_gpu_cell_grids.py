"""The reference-named short range (cudaForceEvaluateShortrange) on cell grids
beyond 1024 an axis and on grids of many more cells than particles: forces
against the CPU oracle, rms relative 1e-4 as in the other parity tests, and a
cost that grows with the cells, not with their square."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from cuco_gb300 import _native, ics
from cuco_gb300._native import SoftParam
from conftest import rms_rel
from test_gpu_capi import simparam

pytestmark = pytest.mark.gpu

L = 1000.0


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


class Gravlist:
    """The reference's device calls on torch buffers."""

    def __init__(self, pos, G, pm_grid, soft):
        self.lib = lib = _native.load()
        lib.cudaInit()
        self.n, self.G, self.ncell = len(pos), G, G ** 3
        lib.cuco_dropin_configure(64, G)
        self.params = oracle.reference_params(L, 1.0, ics.G_INTERNAL, pm_grid, soft)
        lib.setSimParam(ctypes.byref(simparam(L, G, 1.0, self.params.asmth, self.params.rcut)))
        lib.setSoftParam(ctypes.byref(SoftParam(self.params.softening, 1.0 / self.params.softening,
                                                (1.0 / self.params.softening) ** 3)))
        n, dev = self.n, "cuda:0"
        self.pos = torch.zeros((n, 4), device=dev)
        self.pos[:, :3] = torch.from_numpy(pos)
        word = dict(dtype=torch.int32, device=dev)
        self.keys, self.perm = torch.zeros(n, **word), torch.zeros(n, **word)
        self.start, self.end = torch.zeros(self.ncell, **word), torch.zeros(self.ncell, **word)
        self.spos, self.acc = torch.zeros((n, 4), device=dev), torch.zeros((n, 4), device=dev)
        tmp = [torch.zeros(32 * ((n + 1023) // 1024), **word) for _ in range(3)]
        tk, tv = torch.zeros(n, **word), torch.zeros(n, **word)
        torch.cuda.synchronize()
        lib.calcHash(ptr(self.keys), ptr(self.perm), ptr(self.pos), n)
        lib.radixSort(ptr(self.keys), ptr(self.perm), ptr(tk), ptr(tv), *map(ptr, tmp), 0, n,
                      max(18, int(self.ncell - 1).bit_length()), False)
        lib.reorderDataAndFindCellStart(ptr(self.start), ptr(self.end), ptr(self.spos), ptr(self.keys),
                                        ptr(self.perm), ptr(self.pos), n, self.ncell)
        torch.cuda.synchronize()

    def forces(self):
        self.lib.cudaForceEvaluateShortrange(ptr(self.acc), ptr(self.spos), ptr(self.perm), ptr(self.start),
                                             ptr(self.end), self.n, self.ncell)
        torch.cuda.synchronize()
        return self.acc[:, :3].cpu().numpy()


def clumps(n, G, seed):
    """Particles in clumps a few cells wide: around the corner of the box, where
    cell coordinates are largest and the periodic images meet, and elsewhere."""
    rng = np.random.default_rng(seed)
    centres = np.vstack([[[0, 0, 0], [L, L, L / 2], [L / 2, 0.997 * L, 0.999 * L]], rng.uniform(0, L, (5, 3))])
    pos = centres[rng.integers(0, len(centres), n)] + rng.normal(0, 3 * L / G, (n, 3))
    pos = np.mod(pos, L).astype(np.float32)
    pos[pos >= np.float32(L)] = 0
    return pos


@pytest.mark.parametrize("G", [20, 150, 300, 1024, 1025, 1032])
def test_forces(port, G):
    pos = clumps(4000, G, G)
    g = Gravlist(pos, G, G, 0.1 * L / G)
    got = g.forces()
    assert rms_rel(got, port.pp(pos, g.params, 32, 8)) < 1e-4
    del g
    torch.cuda.empty_cache()


def test_cost_grows_with_the_cells():
    """768^3 cells, 1000 particles.  A call reads both bounds twice, writes the
    offsets and reads them at the segments' ends: at most 24 bytes a cell.  A
    copy of both bounds moves 16.  A work that is quadratic in the cells' blocks
    of 1024 (390 GB of block results here) takes tens of such copies."""
    g = Gravlist(clumps(1000, 768, 1), 768, 768, 0.1 * L / 768)
    copies = [torch.empty_like(g.start), torch.empty_like(g.end)]

    def best(f):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            f()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    def copy():
        copies[0].copy_(g.start)
        copies[1].copy_(g.end)

    force, moved = best(g.forces), best(copy)
    print(f"force {force:.3f} ms, copy {moved:.3f} ms")
    assert force < 6 * moved
