"""The short range's units, groups and source lists at the sizes where they
change shape: groups of 1 to 32 targets, segments just below and above a
unit and the dense limit, lists that are evaluated more than once, stencils
that wrap at every face, and the reference's start/end cell bounds (converted
to offsets) against the engine's own.

Forces against the CPU oracle, rms relative over all particles: 1e-4 for the
plain form and 1e-3 for fixed point, the bars of the other parity tests."""
import ctypes

import numpy as np
import pytest

import oracle
from cuco_gb300 import Box, BoxConfig, _native, ics
from cuco_gb300._native import SoftParam
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN
from conftest import rms_rel
from test_gpu_capi import dev_alloc, from_dev, simparam, to_dev

pytestmark = pytest.mark.gpu

L, M, SOFT = 64000.0, 64, 20.0


def particles(crowd, seed, corner=False, background=600):
    """`crowd` particles within one small cell (at the box corner: every
    stencil wraps) over a uniform background."""
    rng = np.random.default_rng(seed)
    at = 0.0 if corner else 0.53 * L
    pos = np.concatenate([rng.uniform(0, L, size=(background, 3)), at + rng.uniform(0, 0.015, size=(crowd, 3)) * L])
    pos = np.mod(pos, L).astype(np.float32)
    pos[pos >= np.float32(L)] = 0
    return pos


def check(port, pos, G, mode):
    params = oracle.reference_params(L, 1.0, ics.G_INTERNAL, M, SOFT)
    ref = port.pp(pos, params, M, 8)
    box = Box(BoxConfig(n=len(pos), pm_grid=M, cell_grid=G, boxsize=L, mass=1.0, G=ics.G_INTERNAL, softening=SOFT,
                        mode=mode))
    box.set_state(pos)
    box.count_pairs(True)
    box.forces(pm=False, pp=True)
    acc = box.get_state()[2]
    pairs = box.pair_count()
    box.close()
    assert rms_rel(acc, ref) < (1e-4 if mode == MODE_PLAIN else 1e-3)
    # fixed point rounds the positions: a pair at the cut may change sides
    assert abs(pairs - port.pair_count(pos, params, M, 8)) <= (0 if mode == MODE_PLAIN else 8)


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("crowd", [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 127, 129, 191, 193, 257, 1500])
def test_group_and_list_sizes(port, crowd, mode):
    check(port, particles(crowd, crowd), 16, mode)


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("G", [16, 20, 27, 32, 50, 64, 90])
def test_cell_grids_with_every_stencil_wrap(port, G, mode):
    check(port, particles(300, G, corner=True, background=3000), G, mode)


@pytest.mark.parametrize("n_background", [320000])
def test_large_units(port, n_background):
    """Enough particles that a unit is two groups of up to 16 targets and a
    dense slice one group of 32."""
    pos = particles(900, 5, background=n_background)
    params = oracle.reference_params(L, 1.0, ics.G_INTERNAL, M, SOFT)
    tg = np.concatenate([np.arange(0, n_background, 997), np.arange(n_background, len(pos))])
    ref = port.pp_targets(pos, tg, params, M, 8)
    box = Box(BoxConfig(n=len(pos), pm_grid=M, cell_grid=32, boxsize=L, mass=1.0, G=ics.G_INTERNAL, softening=SOFT))
    box.set_state(pos)
    box.forces(pm=False, pp=True)
    acc = box.get_state()[2]
    box.close()
    assert rms_rel(acc[tg], ref) < 1e-4


@pytest.mark.parametrize("crowd", [1, 40, 1500])
@pytest.mark.parametrize("G", [16, 33, 64])
def test_start_end_bounds_agree_with_the_engine(port, G, crowd):
    """cudaForceEvaluateShortrange on the reference's cell bounds, with whatever
    an empty cell's cellEnd holds."""
    lib = _native.load()
    lib.cudaInit()
    pos = particles(crowd, 11 * crowd)
    n, ncell = len(pos), G ** 3
    p = oracle.reference_params(L, 1.0, ics.G_INTERNAL, M, SOFT)
    lib.cuco_dropin_configure(M, G)
    lib.setSimParam(ctypes.byref(simparam(L, G, 1.0, p.asmth, p.rcut)))
    lib.setSoftParam(ctypes.byref(SoftParam(SOFT, 1.0 / SOFT, (1.0 / SOFT) ** 3)))
    keys = port.keys(pos, np.float32(np.float32(G) / np.float32(L)), G)
    order = np.argsort(keys, kind="stable").astype(np.uint32)
    start, end = port.cell_bounds(keys[order], ncell)
    end[start == 0xFFFFFFFF] = 0xDEADBEEF  # not read
    spos = np.zeros((n, 4), dtype=np.float32)
    spos[:, :3] = pos[order]
    d_spos, d_idx, d_start, d_end, d_acc = (to_dev(lib, spos), to_dev(lib, order), to_dev(lib, start),
                                            to_dev(lib, end), dev_alloc(lib, 16 * n))
    lib.cudaForceEvaluateShortrange(d_acc, d_spos, d_idx, d_start, d_end, n, ncell)
    acc = from_dev(lib, d_acc, (n, 4), np.float32)
    for d in (d_spos, d_idx, d_start, d_end, d_acc):
        lib.freeArray(d)
    assert rms_rel(acc[:, :3], port.pp(pos, p, M, 8)) < 1e-4
    assert np.all(acc[:, 3] == 0)
