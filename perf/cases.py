"""Performance cases of the force path: what a program that uses this framework
has it do, through its public entry points, over the range of sizes, states,
forms and options in use.

A case's kind says which entry points it goes through:

  steps     Box: the program hands over positions and velocities (device
            arrays), takes `steps` drift-force-kick steps and reads positions,
            velocities and both accelerations back into device arrays.  All
            kicks but the last are zero (the same work): a force evaluated at
            positions that depend on an earlier force would amplify rounding
            into other bins of the nearest-bin split table.
  forces    Box: positions in, one force evaluation (PM, short range or both), accelerations out
  batch     Ensemble: many uneven boxes in pinned host memory, set, stepped together, read back
  gravlist  the device calls of the reference's gravlist.cpp (calcHash, radixSort,
            reorderDataAndFindCellStart, cudaForceEvaluateShortrange) on device arrays
  sort      radixSort / radixSortKeysOnly alone
  dropin    compute_accelerations on the reference's globals, P[] in host memory

States: "early" is a Zel'dovich box at z = 49, "late" a clustered box near
z = 0 (a smoothed Zel'dovich field with 30 % of the mass in isothermal
haloes, cells holding up to about 10^3 particles), "uniform" random positions.
"""
import ctypes
import math

import numpy as np
import torch

from cuco_gb300 import Box, BoxConfig, _native, ics
from cuco_gb300._native import All, Header, SimParam, SoftParam, check
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN
from cuco_gb300.ensemble import Ensemble

NTAB = 1000
SOFT_FRAC = 0.025
A_OF = {"early": 0.02, "late": 0.98, "uniform": 0.5}
DLNA = math.log(50.0) / 200  # 200 log-a steps from z = 49 to 0
# in-range pairs per particle over the uniform value
CLUMPING = {"early": 0.9, "late": 3.9, "uniform": 1.0, "blobs": 8.0}
# particle grids per side whose mesh (twice the side) has no prime factor above 5
SIDES = (16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 120,
         125, 128, 135, 144, 150, 160, 162, 180, 192)


def listed():
    return [
        # the small configuration: one opening call and ten steps of 32^3, launch-bound
        {"name": "steps-32-plain", "kind": "steps", "side": 32, "mesh": 64, "box": 100.0, "form": "plain", "state": "early", "steps": 10},
        # the mid configuration at its start and at its clustered end
        {"name": "steps-128-plain-early", "kind": "steps", "side": 128, "mesh": 256, "box": 256.0, "form": "plain", "state": "early", "steps": 3},
        {"name": "steps-128-plain-late", "kind": "steps", "side": 128, "mesh": 256, "box": 256.0, "form": "plain", "state": "late", "steps": 3},
        # the precision form on a grid that is no power of two
        {"name": "steps-100-fixed-late", "kind": "steps", "side": 100, "mesh": 200, "box": 210.0, "form": "fixed", "state": "late", "steps": 3},
        # the precision form, large, and the largest configuration
        {"name": "steps-256-fixed-early", "kind": "steps", "side": 256, "mesh": 512, "box": 500.0, "form": "fixed", "state": "early", "steps": 1},
        {"name": "steps-512-fixed-early", "kind": "steps", "side": 512, "mesh": 1024, "box": 1000.0, "form": "fixed", "state": "early", "steps": 1},
        # the long range alone, and the short range alone on a ragged count with dense blobs
        {"name": "forces-pm-192", "kind": "forces", "count": 192 ** 3, "mesh": 384, "box": 300.0, "form": "plain", "state": "uniform", "pm": True, "pp": False},
        {"name": "forces-pp-ragged", "kind": "forces", "count": 200003, "mesh": 128, "box": 100.0, "form": "plain", "state": "blobs", "pm": False, "pp": True},
        # the batched form: uneven boxes, each at its own stage
        {"name": "batch-16-fixed", "kind": "batch", "boxes": 16, "lo": 16, "hi": 80, "form": "fixed", "steps": 4, "salt": 3},
        # the reference's own GPU pipeline on its own cell grid (64^3 cells)
        {"name": "gravlist-64", "kind": "gravlist", "count": 32 ** 3, "grid": 64, "box": 100.0, "state": "early"},
        # the sort by itself
        {"name": "sort-4m", "kind": "sort", "count": 4000037, "bits": 24, "values": True},
        # the reference's host program on a host P[]
        {"name": "dropin-64", "kind": "dropin", "side": 64},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["steps", "steps", "steps", "forces", "forces", "batch", "gravlist", "sort", "dropin"])
    if kind == "steps":
        side = min(SIDES, key=lambda s, x=log_int(24, 192): abs(s - x))
        return {"kind": kind, "side": side, "mesh": 2 * side, "box": round(rng.uniform(50.0, 500.0), 1),
                "form": rng.choice(["plain", "fixed"]), "state": rng.choice(["early", "late"]),
                "steps": rng.randint(4, 10) if side < 64 else rng.randint(1, 3)}
    if kind == "forces":
        pm, pp = rng.choice([(True, True), (True, False), (False, True)])
        mesh = 2 * min(SIDES[3:], key=lambda s, x=log_int(24, 160): abs(s - x))
        count = max(1000, int((mesh / 2) ** 3 * rng.uniform(0.3, 1.2)))
        return {"kind": kind, "count": count, "mesh": mesh, "box": round(rng.uniform(50.0, 500.0), 1),
                "form": rng.choice(["plain", "fixed"]), "state": rng.choice(["uniform", "blobs"] if mesh <= 200 else ["uniform"]),
                "pm": pm, "pp": pp}
    if kind == "batch":
        return {"kind": kind, "boxes": rng.randint(3, 16), "lo": rng.choice([16, 24]), "hi": rng.choice([48, 64, 72]),
                "form": rng.choice(["plain", "fixed"]), "steps": rng.randint(2, 5), "salt": rng.randint(0, 1000)}
    if kind == "gravlist":
        return {"kind": kind, "count": log_int(5000, 60000), "grid": rng.choice([32, 64]), "box": round(rng.uniform(50.0, 200.0), 1),
                "state": "uniform"}
    if kind == "sort":
        return {"kind": kind, "count": log_int(3000, 6000000), "bits": rng.randint(12, 30), "values": rng.random() < 0.7}
    return {"kind": kind, "side": rng.choice([32, 40, 48, 56, 72, 80, 96]) + rng.choice([0, 1, 3])}


# ------------------------------------------------------------------ inputs

_cosmo = {}


def _cosmology(a):
    """(cosmology, power amplitude, D(a), f(a)), computed once per process."""
    if a not in _cosmo:
        c = ics.Cosmology()
        _cosmo[a] = (c, c.power_amplitude(), *c.growth(a))
    return _cosmo[a]


def _step_factors(a):
    """Drift and kick integrals over one log-a step ending or starting at a (Simpson)."""
    x = np.linspace(0.0, DLNA, 65)
    w = np.ones(65)
    w[1:-1:2], w[2:-1:2] = 4.0, 2.0
    w *= DLNA / 64 / 3
    s = a * np.exp(x)
    h = ics.HUBBLE_INTERNAL * np.sqrt(0.3 / s ** 3 + 0.7)
    return float((w / (h * s * s)).sum()), float((w / (h * s)).sum())


def _zeldovich(side, box_mpc, a, seed, smooth_mpc=0.0):
    """Displacement field (side^3, 3) in kpc/h at scale factor a, float64, on the GPU."""
    cosmo, amp, d, _ = _cosmology(a)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed * 7919 + 11)
    dtype = torch.float64 if side <= 256 else torch.float32
    wk = torch.fft.rfftn(torch.randn((side, side, side), generator=g, device=dev, dtype=dtype))
    kf = 2 * math.pi / box_mpc
    idx = torch.fft.fftfreq(side, d=1.0 / side, device=dev, dtype=dtype)
    idz = torch.fft.rfftfreq(side, d=1.0 / side, device=dev, dtype=dtype)
    nyq = side // 2
    axes = [(idx * kf)[:, None, None], (idx * kf)[None, :, None], (idz * kf)[None, None, :]]
    k2 = axes[0] ** 2 + axes[1] ** 2 + axes[2] ** 2
    k = torch.sqrt(k2).clamp_min(1e-20)
    q = k / (cosmo.omega0 * cosmo.hubble_param)
    t = torch.log1p(2.34 * q) / (2.34 * q) * (1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3 + (6.71 * q) ** 4) ** -0.25
    pk = amp * k ** cosmo.ns * t * t * torch.exp(-k2 * smooth_mpc ** 2)
    wk = wk * torch.sqrt(pk / (box_mpc / side) ** 3) / k2.clamp_min(1e-30)
    del k, q, t, pk
    dead = (k2 == 0) | (idx.abs() == nyq)[:, None, None] | (idx.abs() == nyq)[None, :, None] | (idz == nyq)[None, None, :]
    wk[dead] = 0
    del dead, k2
    out = torch.empty((side ** 3, 3), device=dev, dtype=torch.float32 if dtype == torch.float32 else torch.float64)
    for j in range(3):
        out[:, j] = torch.fft.irfftn(1j * axes[j] * wk, s=(side,) * 3).reshape(-1) * (1000.0 * d)
    return out


def _wrapped(pos, length):
    p = torch.remainder(pos, length).to(torch.float32)
    p[p >= np.float32(length)] = 0.0
    return p.contiguous()


def _lattice(side, length):
    x = (torch.arange(side, device="cuda", dtype=torch.float64) + 0.5) * (length / side)
    return torch.stack(torch.meshgrid(x, x, x, indexing="ij"), dim=-1).reshape(-1, 3)


def _haloes(side, length, pos, seed):
    """30 % of the particles moved into isothermal haloes (20 to 2000 members each, mean overdensity 200)."""
    rng = np.random.default_rng(seed + 101)
    n, spacing = side ** 3, length / side
    members = np.minimum(20.0 * rng.random(n // 40 + 1) ** (-1.0 / 0.9), min(2000.0, n / 20)).astype(np.int64)
    members = members[: max(1, int(np.searchsorted(np.cumsum(members), 0.3 * n)))]
    centre = rng.integers(0, n, members.size)
    edge = np.ceil(np.cbrt(members)).astype(np.int64)
    which = np.repeat(np.arange(members.size), members)
    at = np.arange(which.size) - np.repeat(np.cumsum(members) - members, members)
    e = edge[which]
    # a halo's members come from the block of lattice sites around its centre's
    site = [(centre[which] // side ** 2 + at // (e * e) - e // 2) % side, (centre[which] // side % side + at // e % e - e // 2) % side,
            (centre[which] % side + at % e - e // 2) % side]
    target = (site[0] * side + site[1]) * side + site[2]
    target, first = np.unique(target, return_index=True)
    which = which[first]
    way = rng.standard_normal((which.size, 3))
    way /= np.linalg.norm(way, axis=1, keepdims=True)
    radius = np.cbrt(3.0 * members[which] / (4 * math.pi * 200.0)) * spacing * np.maximum(rng.random(which.size), 0.01)
    own = torch.from_numpy(centre[which]).cuda()
    moved = pos[own].double() + torch.from_numpy(way * radius[:, None]).cuda()
    pos = pos.clone()
    pos[torch.from_numpy(target).cuda()] = moved.to(pos.dtype)
    return pos


def _particles(state, side, box_mpc, seed):
    """Positions and canonical velocities (side^3, 3), float32, on the GPU."""
    length, a = box_mpc * 1000.0, A_OF[state]
    cosmo, _, _, f = _cosmology(a)
    psi = _zeldovich(side, box_mpc, a, seed, 0.0 if state == "early" else 2.0)
    pos = _lattice(side, length).to(psi.dtype) if side <= 256 else None
    if pos is None:  # the lattice row by row: no second array of the largest size
        x = (torch.arange(side, device="cuda", dtype=torch.float64) + 0.5) * (length / side)
        pos = torch.empty_like(psi)
        view = pos.view(side, side, side, 3)
        view[..., 0], view[..., 1], view[..., 2] = x[:, None, None].float(), x[None, :, None].float(), x[None, None, :].float()
    pos = pos + psi
    vel = (psi * (a * a * ics.HUBBLE_INTERNAL * float(cosmo.E(a)) * f)).to(torch.float32)
    if state == "late":
        pos = _haloes(side, length, pos, seed)
    return _wrapped(pos, length), vel.contiguous()


def _scattered(state, count, box_mpc, seed):
    """Random positions; "blobs": 60 % of them in tight Gaussian blobs."""
    length = box_mpc * 1000.0
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 104729 + 7)
    pos = torch.rand((count, 3), generator=g, device="cuda", dtype=torch.float64) * length
    if state == "blobs":
        blobs = max(3, count // 1500)
        nb = int(0.6 * count)
        centre = torch.rand((blobs, 3), generator=g, device="cuda", dtype=torch.float64) * length
        which = torch.randint(0, blobs, (nb,), generator=g, device="cuda")
        spread = 0.5 * length / count ** (1.0 / 3)
        pos[:nb] = centre[which] + spread * torch.randn((nb, 3), generator=g, device="cuda", dtype=torch.float64)
    return _wrapped(pos, length)


def _config(case, count=None, side=None, mesh=None, box=None):
    side = side or case.get("side")
    count = count if count is not None else case.get("count", (side or 0) ** 3)
    length = (box or case["box"]) * 1000.0
    return BoxConfig(n=count, pm_grid=mesh or case["mesh"], boxsize=length, mass=ics.particle_mass(count, length, 0.3), G=ics.G_INTERNAL,
                     softening=float(np.float32(2.8 * np.float32(SOFT_FRAC * length / count ** (1.0 / 3)))),
                     mode=MODE_FIXED if case.get("form") == "fixed" else MODE_PLAIN)


def _batch_boxes(case):
    """(side, box length, state) of each box: sides log-uniform, boxes at their own stages."""
    rng = np.random.default_rng(case["salt"])
    out = []
    for i in range(case["boxes"]):
        x = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        out.append((min(SIDES, key=lambda s, x=x: abs(s - x)), round(float(rng.uniform(50.0, 400.0)), 1), ("early", "late")[i % 2]))
    return out


# --------------------------------------------------------------- the cases

def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_steps(case, seed):
    pos, vel = _particles(case["state"], case["side"], case["box"], seed)
    return {"run": _run_steps, "box": Box(_config(case)), "pos": pos, "vel": vel, "steps": case["steps"],
            "factors": _step_factors(A_OF[case["state"]]), "out": [torch.empty_like(pos) for _ in range(4)]}


def _read(box, out):
    check(box.lib.cuco_box_get_state(box.h, *[ctypes.c_void_p(o.data_ptr() if o is not None else None) for o in out], 1),
          "cuco_box_get_state")


def _run_steps(s):
    box, (drift, kick) = s["box"], s["factors"]
    box.set_state_device(s["pos"].data_ptr(), s["vel"].data_ptr())
    for _ in range(s["steps"] - 1):
        box.step(drift, 0.0)
    box.step(drift, kick)
    _read(box, s["out"])
    return dict(zip(("pos", "vel", "acc_pp", "acc_pm"), s["out"]))


def _prepare_forces(case, seed):
    pos = _scattered(case["state"], case["count"], case["box"], seed)
    return {"run": _run_forces, "box": Box(_config(case)), "pos": pos, "pm": case["pm"], "pp": case["pp"],
            "out": [None, None, torch.empty_like(pos) if case["pp"] else None, torch.empty_like(pos) if case["pm"] else None]}


def _run_forces(s):
    s["box"].set_state_device(s["pos"].data_ptr(), None)
    s["box"].forces(pm=s["pm"], pp=s["pp"])
    _read(s["box"], s["out"])
    return {k: o for k, o in zip(("acc_pp", "acc_pm"), s["out"][2:]) if o is not None}


def _prepare_batch(case, seed):
    boxes = _batch_boxes(case)
    configs, ins, outs, drift, kick = [], [], [], [], []
    for i, (side, length, stage) in enumerate(boxes):
        c = _config(case, side=side, mesh=2 * side, box=length)
        c.cell_grid = max(c.pm_grid // 4, 8)  # a tuned grid may differ from run to run, and with it the rounding
        configs.append(c)
        ins.append([t.cpu().pin_memory().numpy() for t in _particles(stage, side, length, 64 * seed + i)])
        outs.append([torch.empty((side ** 3, 3), dtype=torch.float32, pin_memory=True) for _ in range(4)])
        d, k = _step_factors(A_OF[stage])
        drift.append(d)
        kick.append(k)
    s = {"run": _run_batch, "ens": Ensemble(configs), "in": ins, "out": outs, "drift": np.array(drift), "kick": np.array(kick),
         "none": np.zeros(len(boxes)), "steps": case["steps"]}
    _run_batch(s)  # the first step lays out the graph that the others replay
    return s


def _run_batch(s):
    ens = s["ens"]
    for b, (pos, vel) in enumerate(s["in"]):
        ens.set_state(b, pos, vel)
    for _ in range(s["steps"] - 1):
        ens.step(s["drift"], s["none"])
    ens.step(s["drift"], s["kick"])
    for b, out in enumerate(s["out"]):
        check(ens.lib.cuco_ensemble_get_state(ens.h, b, *[ctypes.c_void_p(o.data_ptr()) for o in out]), "cuco_ensemble_get_state")
    return s["out"]


def _split(length, mesh):
    asmth = np.float32(1.25 * float(np.float32(length)) / mesh)
    return float(asmth), float(np.float32(4.5 * float(asmth)))


def _table():
    u = 3.0 / NTAB * (np.arange(NTAB) + 0.5)
    return torch.erfc(torch.from_numpy(u)).numpy() + 2 * u / math.sqrt(math.pi) * np.exp(-u * u)


def _gravlist_particles(case, seed):
    if case["state"] == "early":
        return _particles("early", round(case["count"] ** (1.0 / 3)), case["box"], seed)[0]
    return _scattered(case["state"], case["count"], case["box"], seed)


def _prepare_gravlist(case, seed):
    lib = _native.load()
    n, grid, length = case["count"], case["grid"], case["box"] * 1000.0
    c = _config(case, mesh=grid)
    asmth, rcut = _split(length, grid)
    sp = SimParam()
    sp.shortrange_table[:] = _table().astype(np.float32).tolist()
    sp.boxsize, sp.boxhalf, sp.to_grid_fac = length, length / 2, float(np.float32(grid) / np.float32(length))
    sp.rcut, sp.rcut2, sp.asmth, sp.asmthfac = rcut, float(np.float32(rcut * rcut)), asmth, float(np.float32(0.5 / asmth * (NTAB / 3.0)))
    sp.mass, sp.G = c.mass, c.G
    lib.cuco_dropin_configure(grid, grid)
    lib.setSimParam(ctypes.byref(sp))
    h = c.softening
    lib.setSoftParam(ctypes.byref(SoftParam(h, 1.0 / h, 1.0 / h ** 3)))
    pos4 = torch.zeros((n, 4), device="cuda")
    pos4[:, :3] = _gravlist_particles(case, seed)

    def i32(count):
        return torch.zeros(count, device="cuda", dtype=torch.int32)

    words = 32 * ((n + 1023) // 1024)
    bufs = {"hash": i32(n), "index": i32(n), "tk": i32(n), "tv": i32(n), "c": i32(words), "cs": i32(words), "bo": i32(words),
            "start": i32(grid ** 3), "end": i32(grid ** 3), "spos": torch.zeros_like(pos4), "acc": torch.zeros_like(pos4)}
    return {"run": _run_gravlist, "lib": lib, "n": n, "cells": grid ** 3, "bits": (grid ** 3 - 1).bit_length(), "pos": pos4, "bufs": bufs}


def _run_gravlist(s):
    lib, n, b = s["lib"], s["n"], s["bufs"]
    p = {k: ctypes.c_void_p(v.data_ptr()) for k, v in b.items()}
    pos = ctypes.c_void_p(s["pos"].data_ptr())
    lib.calcHash(p["hash"], p["index"], pos, n)
    lib.radixSort(p["hash"], p["index"], p["tk"], p["tv"], p["c"], p["cs"], p["bo"], 0, n, s["bits"], False)
    lib.reorderDataAndFindCellStart(p["start"], p["end"], p["spos"], p["hash"], p["index"], pos, n, s["cells"])
    lib.cudaForceEvaluateShortrange(p["acc"], p["spos"], p["index"], p["start"], p["end"], n, s["cells"])
    return {k: b[k] for k in ("hash", "index", "start", "end", "spos", "acc")}


def _sort_keys(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 31 + 5)
    return torch.randint(0, 1 << case["bits"], (case["count"],), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def _prepare_sort(case, seed):
    n = case["count"]
    keys = _sort_keys(case, seed)
    s = {"run": _run_sort, "lib": _native.load(), "n": n, "bits": case["bits"], "values": case["values"], "in": keys, "keys": torch.empty_like(keys),
         "tk": torch.empty_like(keys), "c": torch.zeros(3 * 32 * ((n + 1023) // 1024), device="cuda", dtype=torch.int32)}
    if case["values"]:
        s.update(first=torch.arange(n, device="cuda", dtype=torch.int32), vals=torch.empty_like(keys), tv=torch.empty_like(keys))
    return s


def _run_sort(s):
    n, words = s["n"], s["c"].numel() // 3
    s["keys"].copy_(s["in"])  # the sort is in place
    c = [ctypes.c_void_p(s["c"].data_ptr() + 4 * words * k) for k in range(3)]
    k, tk = ctypes.c_void_p(s["keys"].data_ptr()), ctypes.c_void_p(s["tk"].data_ptr())
    if not s["values"]:
        s["lib"].radixSortKeysOnly(k, tk, *c, 0, n, s["bits"], False)
        return {"keys": s["keys"]}
    s["vals"].copy_(s["first"])
    s["lib"].radixSort(k, ctypes.c_void_p(s["vals"].data_ptr()), tk, ctypes.c_void_p(s["tv"].data_ptr()), *c, 0, n, s["bits"], False)
    return {"keys": s["keys"], "vals": s["vals"]}


def _dropin_case(case):
    """The mesh (a power of two, as the reference fixes it) and box of a side: the
    library keeps one engine per particle count."""
    return {"mesh": 1 << (2 * case["side"] - 1).bit_length(), "box": 2.0 * case["side"]}


def _prepare_dropin(case, seed):
    lib = _native.load()
    c = _dropin_case(case)
    side, length = case["side"], c["box"] * 1000.0
    n = side ** 3
    pos, vel = _particles("late", side, c["box"], seed)
    raw = np.empty(n * 60 + 64, dtype=np.uint8)
    raw = raw[-raw.ctypes.data % 64:][: n * 60]
    rec = raw.view(np.float32).reshape(n, 15)
    rec[:] = 0
    rec[:, 0:3], rec[:, 4:7] = pos.cpu().numpy(), vel.cpu().numpy()
    rec[:, 3] = ics.particle_mass(n, length, 0.3)
    s = {"run": _run_dropin, "lib": lib, "rec": rec, "n": n, "length": length, "mass": float(rec[0, 3]), "mesh": c["mesh"], "a": A_OF["late"]}
    _point_at(s)
    lib.cuco_dropin_configure(c["mesh"], 0)
    lib.set_softenings()
    lib.long_range_init()
    lib.linklist_init()
    return s


def _point_at(s):
    """The host program's globals at this state's particles."""
    lib, n = s["lib"], s["n"]
    ctypes.c_void_p.in_dll(lib, "P").value = s["rec"].ctypes.data
    ctypes.c_uint.in_dll(lib, "NumPart").value = n
    hdr, al = Header.in_dll(lib, "header"), All.in_dll(lib, "All")
    hdr.NumPart, hdr.Mass, hdr.Time, hdr.BoxSize = n, s["mass"], s["a"], s["length"]
    al.NumPart, al.BoxSize, al.Mass, al.G, al.Hubble = n, s["length"], s["mass"], ics.G_INTERNAL, ics.HUBBLE_INTERNAL
    al.Omega0, al.OmegaLambda, al.HubbleParam = 0.3, 0.7, 0.7
    al.Time, al.TimeBegin, al.TimeMax = s["a"], 0.02, 1.0
    al.Ti_Current = al.PM_Ti_begstep = al.PM_Ti_endstep = 0
    al.SofteningHalo, al.SofteningHaloMaxPhys = SOFT_FRAC * s["length"] / n ** (1.0 / 3), 1e30


def _run_dropin(s):
    _point_at(s)
    s["lib"].compute_accelerations()
    rec = s["rec"]
    return {"pos": rec[:, 0:3], "acc_pp": rec[:, 7:10], "acc_pm": rec[:, 10:13]}


# ------------------------------------------------------------------- work

def _force_work(n, mesh, clumping, pm=True, pp=True):
    """Flops of one force: 20 per in-range pair, the FFT pair, deposit and interpolation."""
    f = 0.0
    if pp:
        f += 20.0 * n * (clumping * n * 4 / 3 * math.pi * (5.625 / mesh) ** 3)
    if pm:
        f += 2 * 2.5 * mesh ** 3 * 3 * math.log2(mesh) + 6.0 * mesh ** 3 / 2 + 130.0 * n
    return f


def work(case):
    kind = case["kind"]
    if kind == "steps":
        # per step: positions and velocities in and out, both accelerations out
        n = case["side"] ** 3
        return {"bytes": 72.0 * n * case["steps"], "flops": case["steps"] * _force_work(n, case["mesh"], CLUMPING[case["state"]])}
    if kind == "forces":
        n = case["count"]
        return {"bytes": n * (12.0 + 12 * case["pm"] + 12 * case["pp"]),
                "flops": _force_work(n, case["mesh"], CLUMPING[case["state"]], case["pm"], case["pp"])}
    if kind == "batch":
        boxes = _batch_boxes(case)
        return {"bytes": 72.0 * case["steps"] * sum(s ** 3 for s, _, _ in boxes),
                "flops": case["steps"] * sum(_force_work(s ** 3, 2 * s, CLUMPING[t]) for s, _, t in boxes)}
    if kind == "gravlist":
        n = case["count"]
        return {"bytes": n * (16.0 + 8 + 16 + 16) + 8.0 * case["grid"] ** 3, "flops": _force_work(n, case["grid"], 1.0, pm=False)}
    if kind == "sort":
        return {"bytes": case["count"] * (16.0 if case["values"] else 8.0), "flops": 0.0}
    n = case["side"] ** 3
    return {"bytes": 120.0 * n, "flops": _force_work(n, _dropin_case(case)["mesh"], CLUMPING["late"])}


# ------------------------------------------------------------ in 64 bits

MOST_PAIRS = 4e10  # candidate pairs that a minute of torch is not spent on


def _pair_forces(pos, length, mesh, mass, h):
    """Short-range accelerations: every pair within the cut, 1/r^2 (the spline inside
    h) times the split function at the centre of the pair's table bin; None where the
    box is too small for a cell list or there are too many pairs."""
    length = float(np.float32(length))
    asmth, rcut = _split(length, mesh)
    tab = torch.from_numpy(_table()).cuda()
    scale = 0.5 / asmth * (NTAB / 3.0)
    n, cells = pos.shape[0], int(length / (rcut * (1 + 1e-6)))
    if cells < 3:
        return None
    cell = (pos * (cells / length)).long().clamp_(0, cells - 1)
    key = (cell[:, 0] * cells + cell[:, 1]) * cells + cell[:, 2]
    order = torch.argsort(key)
    p, cell = pos[order].contiguous(), cell[order]
    count = torch.bincount(key, minlength=cells ** 3)
    start = torch.cumsum(count, 0) - count
    cube = count.view(cells, cells, cells)
    near = sum(torch.roll(cube, (a, b, c), (0, 1, 2)) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1))
    if float((cube * near).sum()) > MOST_PAIRS:
        return None
    acc = torch.zeros_like(p)
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for c in (-1, 0, 1):
                other = [(cell[:, j] + d) % cells for j, d in enumerate((a, b, c))]
                other = (other[0] * cells + other[1]) * cells + other[2]
                size, total = count[other], torch.cumsum(count[other], 0)
                lo = 0
                while lo < n:
                    done = int(total[lo - 1]) if lo else 0
                    hi = max(lo + 1, int(torch.searchsorted(total, done + 30_000_000)))
                    s = size[lo:hi]
                    t = torch.repeat_interleave(torch.arange(lo, hi, device=p.device), s)
                    first = torch.repeat_interleave(start[other[lo:hi]] - (total[lo:hi] - s - done), s)
                    d = p[first + torch.arange(t.numel(), device=p.device)] - p[t]
                    d -= length * torch.round(d / length)
                    r2 = (d * d).sum(1)
                    keep = ((r2 <= rcut * rcut) & (r2 > 0)).nonzero().squeeze(1)
                    d, r, t = d[keep], r2[keep].sqrt(), t[keep]
                    f = r ** -3
                    u = r / h
                    inner = torch.where(u < 0.5, 10.66667 + u * u * (32.0 * u - 38.4),
                                        21.33333 - 48.0 * u + 38.4 * u * u - 10.66667 * u ** 3 - 0.06667 / u ** 3) / h ** 3
                    f = torch.where(u < 1.0, inner, f) * tab[(r * scale).long().clamp_(max=NTAB - 1)]
                    acc.index_add_(0, t, d * f[:, None])
                    lo = hi
    out = torch.empty_like(acc)
    out[order] = acc * (float(np.float32(mass)) * ics.G_INTERNAL)
    return out


def _mesh_forces(pos, length, mesh, mass):
    """Long-range accelerations: CIC mass, the filtered and deconvolved potential, four-point differences, CIC back."""
    m, length = mesh, float(np.float32(length))
    asmth, _ = _split(length, m)
    t = pos * (m / length)
    cell = t.floor().clamp_(max=m - 1)
    frac, cell = t - cell, cell.long()
    corners = []
    for a in (0, 1):
        for b in (0, 1):
            for c in (0, 1):
                w = torch.ones_like(t[:, 0])
                for j, o in enumerate((a, b, c)):
                    w = w * (frac[:, j] if o else 1 - frac[:, j])
                at = [(cell[:, j] + o) % m for j, o in enumerate((a, b, c))]
                corners.append(((at[0] * m + at[1]) * m + at[2], w))
    rho = torch.zeros(m ** 3, device=pos.device, dtype=torch.float64)
    for at, w in corners:
        rho.index_add_(0, at, w)
    rho = torch.fft.rfftn(rho.view(m, m, m) * float(np.float32(mass)))
    k = torch.fft.fftfreq(m, d=1.0 / m, device=pos.device, dtype=torch.float64)
    kz = torch.fft.rfftfreq(m, d=1.0 / m, device=pos.device, dtype=torch.float64)

    def filt(x):
        return torch.exp(-x * x * (2 * math.pi * asmth / length) ** 2) / torch.sinc(x / m) ** 4

    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    rho *= -filt(k)[:, None, None] * filt(k)[None, :, None] * filt(kz)[None, None, :] / k2.clamp_min(1e-30)
    rho[0, 0, 0] = 0
    phi = torch.fft.irfftn(rho, s=(m, m, m)) * float(m) ** 3
    del rho, k2
    scale = ics.G_INTERNAL / (math.pi * length) * (m / (2.0 * length))
    out = torch.zeros_like(pos)
    for j in range(3):
        g = (scale * (4.0 / 3 * (torch.roll(phi, 1, j) - torch.roll(phi, -1, j)) - 1.0 / 6 * (torch.roll(phi, 2, j) - torch.roll(phi, -2, j)))).view(-1)
        for at, w in corners:
            out[:, j] += g[at] * w
    return out


def _after(pos, vel, length, drift, steps, fixed):
    """Positions after `steps` drifts, as the state holds them: float32, or
    multiples of length / 2^32; and the positions that a caller reads."""
    if fixed:
        unit = 2.0 ** 32 / float(np.float32(length))
        x = torch.round(pos.double() * unit).long() & 0xFFFFFFFF
        move = torch.round(vel * np.float32(drift * 2.0 ** 32 / float(np.float32(length)))).long()
        x = (x + steps * move) & 0xFFFFFFFF
        x = x.double() / unit
        return x, x.to(torch.float32).double()
    length = torch.tensor(np.float32(length), device=pos.device)
    step = float(np.float32(drift))
    for _ in range(steps):
        pos = (vel.double() * step + pos.double()).to(torch.float32)
        for _ in range(4):
            pos = torch.where(pos < 0, pos + length, pos)
        for _ in range(4):
            pos = torch.where(pos >= length, pos - length, pos)
    return pos.double(), pos.double()


def _exact_box(pos, vel, c, steps, factors):
    drift, kick = factors
    x, seen = _after(pos, vel, c.boxsize, drift, steps, c.mode == MODE_FIXED)
    app = _pair_forces(x, c.boxsize, c.pm_grid, c.mass, c.softening)
    apm = _mesh_forces(x, c.boxsize, c.pm_grid, c.mass)
    new = None if app is None else vel.double() + (app + apm) * kick
    return {"pos": seen, "vel": new, "acc_pp": app, "acc_pm": apm}


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        if case["mesh"] > 512:
            return None
        pos, vel = _particles(case["state"], case["side"], case["box"], seed)
        return _exact_box(pos, vel, _config(case), case["steps"], _step_factors(A_OF[case["state"]]))
    if kind == "forces":
        c = _config(case)
        none = torch.zeros((case["count"], 3), device="cuda")
        x = _after(_scattered(case["state"], case["count"], case["box"], seed), none, c.boxsize, 0.0, 0, c.mode == MODE_FIXED)[0]
        out = {}
        if case["pp"]:
            out["acc_pp"] = _pair_forces(x, c.boxsize, c.pm_grid, c.mass, c.softening)
        if case["pm"]:
            out["acc_pm"] = _mesh_forces(x, c.boxsize, c.pm_grid, c.mass)
        return out
    if kind == "batch":
        out = []
        for i, (side, length, stage) in enumerate(_batch_boxes(case)):
            c = _config(case, side=side, mesh=2 * side, box=length)
            got = _exact_box(*_particles(stage, side, length, 64 * seed + i), c, case["steps"], _step_factors(A_OF[stage]))
            out.append([got["pos"], got["vel"], got["acc_pp"], got["acc_pm"]])
        return out
    if kind == "gravlist":
        length, grid = case["box"] * 1000.0, case["grid"]
        c = _config(case, mesh=grid)
        acc = _pair_forces(_gravlist_particles(case, seed).double(), length, grid, c.mass, c.softening)
        return {"hash": None, "index": None, "start": None, "end": None, "spos": None,
                "acc": None if acc is None else torch.cat([acc, torch.zeros_like(acc[:, :1])], 1)}
    if kind == "sort":
        keys = _sort_keys(case, seed)
        keys, order = torch.sort(keys, stable=True)
        return {"keys": keys, "vals": order.to(torch.int32)} if case["values"] else {"keys": keys}
    c = _dropin_case(case)
    length = c["box"] * 1000.0
    n = case["side"] ** 3
    pos = _particles("late", case["side"], c["box"], seed)[0].double()
    h = float(np.float32(2.8 * float(np.float32(SOFT_FRAC * length / n ** (1.0 / 3)))))
    mass = ics.particle_mass(n, length, 0.3)
    return {"pos": pos, "acc_pp": _pair_forces(pos, length, c["mesh"], mass, h), "acc_pm": _mesh_forces(pos, length, c["mesh"], mass)}
