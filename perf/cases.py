"""The work a user of this framework has it do, as measured cases.

Kinds of case, each through the public Python entry points:

* ``tunnel``: an airfoil tunnel stepped by ``LBMSolver.step_n`` -- plain, with
  the wall model, with a 2:1 .. 4:1 refinement patch, with a finer level
  nested in it; FP32 or FP16 populations.
* ``box``: an all-fluid periodic lattice (Taylor-Green vortex) stepped with
  the A/B or the AA layout.
* ``polar``: an angle-of-attack polar stepped by ``BatchSolver.step_n``.
* ``aoa``: a change of the angle of attack: flag fields built on the device,
  ``set_flags`` (and ``set_refined_flags``), which restart the flow.
* ``edit``: vanes moved on a running tunnel (``apply_edited_flags``).
* ``train``: the wall model's learned seed trained from scratch
  (``wallnet.train_wallnet``).
* ``labels``: u_tau solves of a sample set (``wallnet.utau_solve``).

A ``tunnel`` or ``box`` pass takes ``steps`` steps from wherever the last pass
left the flow and returns the population array of every level (and the wall
model's slip velocities); the viscosities are high enough for the flows to
stay stable however long they run. ``exact`` replays the first pass in 64
bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from foil_cfd_gb300 import geometry, wallnet
from foil_cfd_gb300.batch import BatchSolver, polar_tunnels
from foil_cfd_gb300.solver import Box, LBMSolver, fine_anchor, layout_anchor, naca4, scaling_direct

U_LAT = 0.08
TAU = 0.56          # with u 0.08 and Cs 0.1 every tunnel below is stable
LES_CS = 0.1
LAMBDA = 3.0 / 16.0
AOA = 6.0
SHELL = 2           # interface cells around a refined level
BAND = 2            # coarse cells of a patch that the restriction leaves alone
POP_BYTES = {"fp32": 4, "fp16": 2}
METHODS = {"reference": wallnet.REFERENCE, "newton64": wallnet.NEWTON64}


# ---- the cases --------------------------------------------------------------------


def _tunnel_case(nx, ny, nz, chord, steps, storage="fp32", factor=0, finer=False, wall=False, force=False):
    return {"kind": "tunnel", "nx": nx, "ny": ny, "nz": nz, "chord": chord, "storage": storage, "factor": factor,
            "finer": finer, "wall": wall, "force": force, "steps": steps}


def listed():
    return [
        # One step and the force of a small section with the wall model: a control or optimisation loop.
        dict(_tunnel_case(160, 64, 8, 64, 1, wall=True, force=True), name="section_160x64x8_step"),
        # The smallest validation flow, a lattice that stays in L2: launches and latency.
        {"name": "taylor_green_64", "kind": "box", "nx": 64, "ny": 64, "nz": 64, "storage": "fp32", "layout": "ab",
         "steps": 100},
        # The plain tunnel the headline rate is quoted on.
        dict(_tunnel_case(768, 320, 96, 256, 10), name="tunnel_768x320x96"),
        # A periodic box of odd extents in the in-place layout with half-precision storage, read back every 40 steps.
        {"name": "box_aa_fp16_333x170x149", "kind": "box", "nx": 333, "ny": 170, "nz": 149, "storage": "fp16",
         "layout": "aa", "steps": 40},
        # The full airfoil tunnel with its patch and wall model, both storages: the production run.
        dict(_tunnel_case(640, 192, 192, 256, 10, factor=2, wall=True), name="airfoil_640_fp32"),
        dict(_tunnel_case(640, 192, 192, 256, 10, storage="fp16", factor=2, wall=True), name="airfoil_640_fp16"),
        # A small three-level tunnel, as the interactive and harvesting runs use them.
        dict(_tunnel_case(320, 96, 32, 128, 5, factor=2, finer=True, wall=True), name="nested_320x96x32"),
        # The 24-tunnel polar with half-precision storage: one chunk of 100 steps and its force sample.
        {"name": "polar_24_fp16", "kind": "polar", "count": 24, "span": 16, "storage": "fp16", "steps": 100},
        # A new angle of attack on the full tunnel and its patch.
        {"name": "aoa_change_640", "kind": "aoa", "nx": 640, "ny": 192, "nz": 192, "chord": 256, "storage": "fp32",
         "factor": 2},
        # Vortex generators moved on a running mid-size tunnel.
        {"name": "edit_320x96x96", "kind": "edit", "nx": 320, "ny": 96, "nz": 96, "chord": 128, "storage": "fp32"},
        # Training of the learned wall seed at its usual batch size, and the labels of its sample set.
        {"name": "train_131072", "kind": "train", "samples": 131072, "batch": 2048, "epochs": 4},
        {"name": "labels_3m", "kind": "labels", "samples": 3000000, "method": "newton64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tunnel", "tunnel", "patch", "patch", "box", "polar", "aoa", "edit", "train", "labels"])
    storage = rng.choice(["fp32", "fp16"])
    if kind == "train":
        batch = 64 * _log_int(rng, 4, 64)
        return {"kind": "train", "samples": _log_int(rng, 8192, 131072), "batch": batch, "epochs": rng.randint(1, 4)}
    if kind == "labels":
        return {"kind": "labels", "samples": _log_int(rng, 1000, 3000000),
                "method": rng.choice(["reference", "newton64"])}
    if kind == "polar":
        return {"kind": "polar", "count": rng.randint(2, 24 if storage == "fp16" else 12), "span": rng.randint(5, 16), "storage": storage,
                "steps": 100}
    if kind == "box":
        nx, ny, nz = (_log_int(rng, 24, 300) for _ in range(3))
        return {"kind": "box", "nx": nx, "ny": ny, "nz": nz, "storage": storage,
                "layout": rng.choice(["ab", "aa"]), "steps": max(2, min(100, int(3e8 / (nx * ny * nz))))}
    nx = _log_int(rng, 150, 640)
    ny, nz = int(nx * rng.uniform(0.3, 0.45)), _log_int(rng, 6, 96)
    chord = int(nx * rng.uniform(0.3, 0.4))
    if kind == "aoa":
        return {"kind": "aoa", "nx": nx, "ny": ny, "nz": nz, "chord": chord, "storage": storage,
                "factor": rng.choice([0, 2])}
    if kind == "edit":
        return {"kind": "edit", "nx": nx, "ny": ny, "nz": nz, "chord": chord, "storage": storage}
    if kind == "tunnel":
        steps = max(1, min(20, int(1e8 / (nx * ny * nz))))
        return _tunnel_case(nx, ny, nz, chord, steps, storage, wall=rng.random() < 0.5)
    factor = rng.choice([2, 2, 2, 3])
    finer = factor == 2 and rng.random() < 0.3
    if factor == 3 or finer:
        nz = min(nz, 24)
    return _tunnel_case(nx, ny, nz, chord, rng.randint(1, 8), storage, factor, finer, wall=rng.random() < 0.7)


# ---- inputs -------------------------------------------------------------------------


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _levels(case, aoa):
    """Flag fields of every level, built on the device: [(dims, flags, box in the parent, factor), ...]."""
    dims, chord = _dims(case), case["chord"]
    flags = geometry.clean_foil_flags(dims, "0012", aoa, chord)
    levels = [(dims, flags, None, 1)]
    anchor, scale = layout_anchor(dims), 1
    for factor in [case.get("factor")] * bool(case.get("factor")) + [2] * bool(case.get("finer")):
        m = int(round(0.1 * chord)) if scale == 1 else 6
        # The box of the patch follows the nominal angle, so that every angle of a run fits in it.
        base = geometry.clean_foil_flags(dims, "0012", AOA, chord) if scale == 1 else flags
        box = geometry.derive_patch_box(levels[-1][0], base, m, m, m, m, 3 if scale == 1 else SHELL + 2)
        anchor, scale = fine_anchor(anchor, box, factor), scale * factor
        fd = (factor * (box.x1 - box.x0), factor * (box.y1 - box.y0), factor * levels[-1][0][2])
        placed = geometry.foil(naca4("0012", 200), aoa, scale * chord, *anchor)
        flags = geometry.build_flags(fd, "fluid", placed, True, SHELL, count_closed=False)[0]
        levels.append((fd, flags, box, factor))
    return levels


def _fields(dims, seed, periodic=False):
    """(rho, u, v, w) of a developed-looking start: the stream (or a
    Taylor-Green vortex) with a few seeded waves on it."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    ax = [(2 * math.pi / n) * torch.arange(n, device="cuda", dtype=torch.float32) for n in (nz, ny, nx)]
    z, y, x = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    out = []
    for k in range(4):
        f = torch.zeros((nz, ny, nx), device="cuda")
        for _ in range(3):
            kx, ky, kz = (int(v) for v in rng.integers(1, 5, 3))
            p = rng.uniform(0, 2 * math.pi, 3)
            amp = float(rng.uniform(0.002, 0.004))
            f += amp * torch.sin(kx * x + p[0]) * torch.sin(ky * y + p[1]) * torch.cos(kz * z + p[2])
        out.append(f)
    out[0] += 1.0
    if periodic:
        out[1] += 0.05 * torch.sin(x) * torch.cos(y) * torch.cos(z)
        out[2] -= 0.05 * torch.cos(x) * torch.sin(y) * torch.cos(z)
    else:
        out[1] += U_LAT
    return [f.reshape(-1) for f in out]


class _Device:
    """A device array of a solver, for torch.as_tensor; a tensor over it keeps the solver alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": typestr, "version": 2}


class _Flow:
    """A solver and tensors over the buffers its steps leave their results in."""

    def __init__(self, sol, storage, levels, wall=False):
        self.sol, self.storage, self.levels, self.wall = sol, storage, levels, wall
        self.seen = {}

    def _tensor(self, ptr, shape, typestr):
        t = self.seen.get(ptr)
        if t is None:
            t = self.seen[ptr] = torch.as_tensor(_Device(self.sol, ptr, shape, typestr), device="cuda")
        return t

    def populations(self):
        out = []
        for level in range(self.levels):
            v = self.sol.lattice_view(level)
            out.append(self._tensor(v.f, (19, v.cells), "<f4" if self.storage == "fp32" else "<f2"))
        return out

    def slip(self):
        out = []
        for level in range(self.levels) if self.wall else ():
            v = self.sol.lattice_view(level)
            out += [self._tensor(p, (v.cells,), "<f2") for p in (v.uwx, v.uwy, v.uwz) if p]
        return out


def _blank(flow):
    """Cells that no step writes (inside solids) hold zeros in both buffers of a refined level."""
    for t in flow.populations()[1:]:
        t.zero_()
    flow.sol.mirror_buffers()


def _solver(case, levels):
    sol = LBMSolver()
    dims, flags = levels[0][:2]
    sol.init(dims, scaling_direct(TAU, U_LAT, case["chord"]), flags, storage=case["storage"], les_cs=LES_CS)
    if case.get("wall") or case["kind"] == "edit":
        sol.set_wall_model_enabled(True)
    sol.set_startup_ramp_enabled(False)
    sol.reset()
    if len(levels) > 1:
        sol.init_refinement(levels[1][2], levels[1][3], levels[1][1])
    if len(levels) > 2:
        sol.init_finer_refinement(levels[2][2], levels[2][3], levels[2][1])
    return sol


def _warm_start(sol, fields):
    sol.restore_from_macroscopic(*[f.cpu().numpy() for f in fields])


def _vaned(case, levels, at):
    """The tunnel's flags with a row of vanes standing on the upper side, `at` cells downstream of the anchor."""
    nx, ny, nz = _dims(case)
    f = levels[0][1].clone().reshape(nz, ny, nx)
    x0, y0 = int(0.3 * nx) + at, ny // 2 + max(4, int(0.08 * case["chord"]))
    vane = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda")
    for z in range(0, nz, 12):
        vane[z : z + 2, y0 : y0 + 6, x0 : x0 + 10] = True
    f[vane & (f == 0)] = 1
    return f.reshape(-1)


def _edits(case, levels, seed):
    at = int(np.random.default_rng(seed).integers(0, case["chord"] // 4))
    return _vaned(case, levels, at), _vaned(case, levels, at + 5)


def _polar(case, seed):
    turn = float(np.random.default_rng(seed).uniform(-0.5, 0.5))
    return polar_tunnels(case["count"], span=case["span"], aoas=[-4.0 + 2.5 * k + turn for k in range(9)],
                         reynolds=400.0, device=True)


def _samples(case, seed):
    return [torch.from_numpy(a).cuda() for a in wallnet.synthetic_samples(case["samples"], seed)]


def _new_angle(seed):
    return AOA - 3.0 * float(np.random.default_rng(seed).uniform(0.2, 1.0))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        ut, ys, nu = _samples(case, seed)
        return case, (ut, ys, nu, wallnet.utau_solve(wallnet.NEWTON64, ut, ys, nu, stats=False)[0])
    if kind == "labels":
        return case, _samples(case, seed)
    if kind == "polar":
        batch = BatchSolver()
        batch.init(_polar(case, seed), storage=case["storage"], les_cs=LES_CS, force_every=case["steps"])
        return case, batch
    if kind == "box":
        dims = _dims(case)
        sol = LBMSolver()
        sol.init(dims, scaling_direct(0.53, 0.05, 64), np.zeros(int(np.prod(dims)), np.uint8),
                 storage=case["storage"], les_cs=LES_CS, layout=case["layout"])
        sol.set_startup_ramp_enabled(False)
        sol.reset()
        _warm_start(sol, _fields(dims, seed, periodic=True))
        return case, _Flow(sol, case["storage"], 1)
    levels = _levels(case, AOA)
    if kind == "edit":
        first, second = _edits(case, levels, seed)
        clean = levels[0][1]
        levels[0] = (levels[0][0], first, None, 1)
        sol = _solver(case, levels)
        sol.set_surface_reference(clean)
        _warm_start(sol, _fields(_dims(case), seed))
        return case, [_Flow(sol, case["storage"], 1), second, first]
    sol = _solver(case, levels)
    flow = _Flow(sol, case["storage"], len(levels), case.get("wall", False))
    _blank(flow)
    if kind == "aoa":
        return case, [flow, levels[1][2] if len(levels) > 1 else None, _new_angle(seed)]
    _warm_start(sol, _fields(_dims(case), seed))
    return case, flow


def _done(rc):
    if rc:
        raise RuntimeError(f"a step failed ({rc})")


def run(state):
    case, s = state
    kind = case["kind"]
    if kind == "train":
        net, loss = wallnet.train_wallnet(*s, epochs=case["epochs"], batch=case["batch"])
        master, working, norm = net.params()
        return {"loss": loss, "master": master, "bf16": working, "norm": norm}
    if kind == "labels":
        return wallnet.utau_solve(METHODS[case["method"]], *s, stats=False)[0]
    if kind == "polar":
        _done(s.step_n(case["steps"]))
        return {"force": s.force_history(1), "latched": s.latched()}
    if kind == "aoa":
        flow, box, aoa = s
        dims, chord = _dims(case), case["chord"]
        flags = [geometry.clean_foil_flags(dims, "0012", aoa, chord)]
        _done(flow.sol.set_flags(flags[0]))
        if box is not None:
            flags.append(geometry.fine_patch_flags(dims, box, case["factor"], "0012", aoa, chord, shell=SHELL)[1])
            _done(flow.sol.set_refined_flags(flags[1]))
        return {"flags": flags, "f": flow.populations()}
    if kind == "edit":
        flow, new, old = s
        s[1], s[2] = old, new      # the next pass moves the vanes back
        edited = flow.sol.apply_edited_flags(new)
        return {"edited": edited, "wall_cells": flow.sol.wall_count(0), "f": flow.populations()}
    _done(s.sol.step_n(case["steps"]))
    out = {"f": s.populations(), "slip": s.slip()}
    if case.get("force"):
        out["force"] = s.sol.force_raw()
    return out


# ---- what a pass cannot do without ----------------------------------------------------


def _patch_cells(case):
    """About the cells of the patch (and of the finer box in it)."""
    m, c = case["factor"], case["chord"]
    if not m:
        return []
    fine = (m * 1.2 * c) * (m * 0.35 * c) * (m * case["nz"])
    finer = (2 * (m * c + 12)) * (2 * (0.15 * m * c + 12)) * (2 * m * case["nz"])
    return [fine] + ([finer] if case.get("finer") else [])


def work(case):
    kind = case["kind"]
    if kind == "train":
        # 16 bytes a sample; about 2.3 kFLOP forward and twice that backward.
        n = case["samples"] * case["epochs"]
        return {"bytes": 16 * n, "flops": 6900 * n}
    if kind == "labels":
        return {"bytes": 16 * case["samples"], "flops": 4 * 60 * case["samples"]}
    pop = 19 * POP_BYTES[case["storage"]]
    if kind == "polar":
        cells = case["count"] * 2.5 * 1.5 * 144 * 144 * case["span"] * case["steps"]
        return {"bytes": 2 * pop * cells, "flops": 250 * cells}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "aoa":      # flags out, both population buffers written
        cells = n + sum(_patch_cells(case))
        return {"bytes": (1 + 2 * pop) * cells, "flops": 100 * cells}
    if kind == "edit":     # flags in; the cells of the vanes are few
        return {"bytes": n, "flops": 20 * n}
    cells = n
    m = case.get("factor", 0)
    for fine in _patch_cells(case) if kind == "tunnel" else []:
        cells += m * fine
        m *= 2
    return {"bytes": 2 * pop * cells * case["steps"], "flops": 250 * cells * case["steps"]}


# ---- the same in 64 bits ---------------------------------------------------------------

C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
     (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1)]
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [C.index((-a, -b, -c)) for a, b, c in C]
MIRROR_Y = [C.index((a, -b, c)) for a, b, c in C]


def _dot(c, u):
    t = 0.0
    for k in range(3):
        if c[k]:
            t = t + c[k] * u[k]
    return t


def _feq(q, rho, u, usq):
    cu = 3.0 * _dot(C[q], u)
    return W[q] * rho * (1.0 + cu + 0.5 * cu * cu - usq)


def _usq(u):
    return 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])


def _moments(f):
    rho = sum(f[1:], f[0])
    j = [sum(C[q][k] * f[q] for q in range(19) if C[q][k]) for k in range(3)]
    return rho, j


def _limited(f):
    rho, j = _moments(f)
    rho = rho.clamp_min(0.05)
    u = [a / rho for a in j]
    speed = (u[0] ** 2 + u[1] ** 2 + u[2] ** 2).sqrt()
    cut = torch.where(speed > 0.3, 0.3 / speed, torch.ones_like(speed))
    return rho, [a * cut for a in u]


def _pull(a, c):
    return torch.roll(a, (c[2], c[1], c[0]), (0, 1, 2))


STRESS = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]


def _stress(fneq):
    """Second moments of a list of 19 fields."""
    return [sum(C[q][a] * C[q][b] * fneq[q] for q in range(19) if C[q][a] * C[q][b]) for a, b in STRESS]


def _regular(fneq):
    p = _stress(fneq)
    trace = (p[0] + p[1] + p[2]) / 3.0
    for q in range(19):
        t = -trace
        for (a, b), v in zip(STRESS, p):
            if C[q][a] * C[q][b]:
                t = t + (1.0 if a == b else 2.0) * C[q][a] * C[q][b] * v
        fneq[q] = 4.5 * W[q] * t
    return fneq


class _Level64:
    """One level's A/B pair in 64 bits, [19, nz, ny, nx] each."""

    def __init__(self, dims, flags, box=None, factor=1):
        self.dims, self.box, self.m = dims, box, factor
        self.flags = flags.reshape(dims[2], dims[1], dims[0])
        self.f = None

    def start(self, init):
        self.f = [init, init.clone()]

    def collide(self, tau, u_in):
        src, dst, flags = self.f[0], self.f[1], self.flags
        f = []
        for q in range(19):
            v = _pull(src[q], C[q])
            nf = _pull(flags, C[q])
            v = torch.where(nf == 1, src[OPP[q]], v)
            slip = (nf == 4) | (nf == 5)
            f.append(torch.where(slip, _pull(src[MIRROR_Y[q]], (C[q][0], 0, C[q][2])), v))
        rho, u = _limited(f)
        usq = _usq(u)
        fneq = [f[q] - _feq(q, rho, u, usq) for q in range(19)]
        p = _stress(fneq)
        qbar = (p[0] ** 2 + p[1] ** 2 + p[2] ** 2 + 2.0 * (p[3] ** 2 + p[4] ** 2 + p[5] ** 2)).sqrt()
        pre = 18.0 * math.sqrt(2.0) * LES_CS * LES_CS
        tau_eff = 0.5 * (tau + (tau * tau + pre * qbar / rho).sqrt())
        om_p = 1.0 / tau_eff
        om_m = 1.0 / (0.5 + LAMBDA / (tau_eff - 0.5))
        fluid = flags == 0
        for q in range(19):
            a, b = fneq[q], fneq[OPP[q]]
            new = f[q] - 0.5 * om_p * (a + b) - 0.5 * om_m * (a - b)
            dst[q] = torch.where(fluid, new, dst[q])
        del f, fneq
        for x, flag in ((0, 2), (self.dims[0] - 1, 3), (self.dims[0] - 1, 9)):
            at = flags[:, :, x] == flag
            if not bool(at.any()):
                continue
            if flag == 2:
                for q in range(19):
                    dst[q][:, :, x][at] = W[q] * (1 + 3 * C[q][0] * u_in + 4.5 * (C[q][0] * u_in) ** 2 - 1.5 * u_in ** 2)
                continue
            up = [src[q][:, :, x - 1] for q in range(19)]
            r, j = _moments(up)
            v = [t / r for t in j]
            for q in range(19):
                e = up[q] if flag == 3 else _feq(q, torch.ones_like(r), v, _usq(v))
                dst[q][:, :, x] = torch.where(at, e, dst[q][:, :, x])

    def swap(self):
        self.f.reverse()

    def inner_shell(self):
        """Interface cells that a collide of this level reads."""
        wet = (self.flags == 0) | (self.flags == 3) | (self.flags == 9)
        near = torch.zeros_like(wet)
        for q in range(1, 19):
            near |= _pull(wet, C[q])
        return torch.nonzero(((self.flags == 8) & near).reshape(-1)).reshape(-1)

    def fill(self, parent, dst, targets, weight, scale):
        """Coarse-to-fine fill of `targets` (flat cells) of the buffer dst."""
        for part in torch.split(targets, 4_000_000):
            self._fill(parent, dst, part, weight, scale)

    def _fill(self, parent, dst, t, weight, scale):
        nx, ny, _ = self.dims
        pnx, pny, pnz = parent.dims
        g = [(t % nx + 0.5) / self.m - 0.5 + self.box.x0, ((t // nx) % ny + 0.5) / self.m - 0.5 + self.box.y0,
             (t // (nx * ny) + 0.5) / self.m - 0.5]
        g = [a.double() for a in g]
        lo = [a.floor() for a in g]
        fr = [a - b for a, b in zip(g, lo)]
        lo = [a.long() for a in lo]
        corners, weights = [], []
        for c in range(8):
            d = (c & 1, (c >> 1) & 1, (c >> 2) & 1)
            cell = (lo[0] + d[0]) % pnx + pnx * ((lo[1] + d[1]) % pny + pny * ((lo[2] + d[2]) % pnz))
            w = 1.0
            for k in range(3):
                w = w * (fr[k] if d[k] else 1.0 - fr[k])
            weights.append(torch.where(parent.flags.reshape(-1)[cell] == 1, torch.zeros_like(w), w))
            corners.append(cell)
        total = sum(weights)
        keep = total >= 1e-6
        weights = [w / torch.where(keep, total, torch.ones_like(total)) for w in weights]
        f = []
        for q in range(19):
            s = [sum(w * p[q].reshape(-1)[c] for w, c in zip(weights, corners)) for p in
                 (parent.f if weight else parent.f[:1])]
            f.append(s[0] + weight * (s[1] - s[0]) if weight else s[0])
        rho, u = _limited(f)
        usq = _usq(u)
        fneq = _regular([f[q] - _feq(q, rho, u, usq) for q in range(19)])
        for q in range(19):
            dst[q].view(-1)[t[keep]] = (_feq(q, rho, u, usq) + scale * fneq[q])[keep]

    def restrict_into(self, parent, dst, scale):
        """Fine-to-coarse restriction of this level's current state."""
        m, b = self.m, self.box
        x0, y0, x1, y1 = b.x0 + BAND, b.y0 + BAND, b.x1 - BAND, b.y1 - BAND
        w, h, nz = x1 - x0, y1 - y0, parent.dims[2]

        def kids(a):
            a = a[:, m * BAND : m * (BAND + h), m * BAND : m * (BAND + w)]
            return a.reshape(nz, m, h, m, w, m).sum((1, 3, 5))

        wet = self.flags != 1
        count = kids(wet.double())
        valid = count > 0
        f = [kids(torch.where(wet, self.f[0][q], 0.0)) / count.clamp_min(1.0) for q in range(19)]
        f = [torch.where(valid, a, torch.full_like(a, W[q])) for q, a in enumerate(f)]
        rho, u = _limited(f)
        usq = _usq(u)
        pad = torch.nn.functional.pad
        ok = pad(valid.double(), (1, 1, 1, 1))

        def near(a):
            """Sum of a (padded in x and y, periodic in z) over the stencil."""
            return sum(torch.roll(a, -C[q][2], 0)[:, 1 + C[q][1] : 1 + C[q][1] + h, 1 + C[q][0] : 1 + C[q][0] + w]
                       for q in range(19))

        n = near(ok).clamp_min(1.0)
        fneq = _regular([near(pad(torch.where(valid, f[q] - _feq(q, rho, u, usq), 0.0), (1, 1, 1, 1))) / n
                         for q in range(19)])
        ex = torch.arange(w, device="cuda")
        ey = torch.arange(h, device="cuda")
        edge = torch.minimum(torch.minimum(ex, w - 1 - ex)[None, :], torch.minimum(ey, h - 1 - ey)[:, None])
        blend = ((edge + 1).double() / 4.0).clamp_max(1.0)[None]
        at = valid & (parent.flags[:, y0:y1, x0:x1] == 0)
        for q in range(19):
            old = dst[q][:, y0:y1, x0:x1]
            new = old + blend * (_feq(q, rho, u, usq) + scale * fneq[q] - old)
            dst[q][:, y0:y1, x0:x1] = torch.where(at, new, old)


def _equilibrium64(dims, flags, fields):
    shape = (dims[2], dims[1], dims[0])
    solid = flags.reshape(shape) == 1
    rho, *u = (torch.where(solid, 1.0 if k == 0 else 0.0, a.double().reshape(shape)) for k, a in enumerate(fields))
    usq = _usq(u)
    return torch.stack([_feq(q, rho, u, usq) for q in range(19)])


def _speck64(f, flags, u_lat):
    """The seeded spanwise perturbation of a cold start, added to the fluid cells of f."""
    nz, ny, nx = f.shape[1:]

    def phase(salt):
        h = ((0x5EED + salt) * 2654435761) & 0xFFFFFFFF
        h ^= h >> 16
        return 6.2831853 * (h & 0xFFFFFF) / 16777216.0

    tz = 6.2831853 * (torch.arange(nz, device="cuda").double() + 0.5) / nz
    tx = 6.2831853 * (torch.arange(nx, device="cuda").double() + 0.5) / nx
    wz = 1e-3 * u_lat * (0.6 * torch.sin(3 * tz + phase(1)) + 0.4 * torch.sin(7 * tz + phase(2)))[:, None, None]
    wz = wz * (1 + 0.3 * torch.sin(2 * tx + phase(3)))[None, None, :]
    fluid = flags.reshape(nz, ny, nx) == 0
    for q in range(1, 19):
        if C[q][2]:
            f[q] += torch.where(fluid, 3.0 * W[q] * C[q][2] * wz, torch.zeros_like(wz))
    return f


def _uniform64(dims, flags, u_lat):
    n = dims[0] * dims[1] * dims[2]
    one = torch.ones(n, device="cuda")
    return _speck64(_equilibrium64(dims, flags, [one, u_lat * one, 0 * one, 0 * one]), flags, u_lat)


def _stored(case, f):
    """A level's populations as the solver's storage holds them: f, or f - w_q with half-precision storage."""
    if case["storage"] == "fp16":
        f = f - torch.tensor(W, device="cuda", dtype=torch.float64)[:, None, None, None]
    return f.reshape(19, -1)


def _empty64(case, dims):
    """A buffer of stored zeros."""
    f = torch.zeros((19, dims[2], dims[1], dims[0]), device="cuda", dtype=torch.float64)
    if case["storage"] == "fp16":
        f += torch.tensor(W, device="cuda", dtype=torch.float64)[:, None, None, None]
    return f


def _fine_tau(tau, m):
    return m * (tau - 0.5) + 0.5


def _seed64(level, parent, tau_parent):
    every = torch.nonzero(level.flags.reshape(-1) != 1).reshape(-1)
    scale = _fine_tau(tau_parent, level.m) / (level.m * tau_parent)
    level.fill(parent, level.f[0], every, 0.0, scale)
    level.f[1].copy_(torch.where((level.flags != 1)[None], level.f[0], level.f[1]))


def _sub_steps(levels, shells, tau):
    """m sub-steps of levels[1] between the two time levels of levels[0], then its restriction into the newer one."""
    parent, fine = levels[0], levels[1]
    m, tf = fine.m, _fine_tau(tau, fine.m)
    for k in range(m):
        fine.fill(parent, fine.f[0], shells[0], k / m, tf / (m * tau))
        fine.collide(tf, U_LAT)
        if len(levels) > 2:
            _sub_steps(levels[1:], shells[1:], tf)
        fine.swap()
    fine.restrict_into(parent, parent.f[1], m * tau / tf)


def _force64(level):
    f, flags = level.f[0], level.flags
    out = [0.0, 0.0, 0.0]
    for q in range(1, 19):
        at = (flags == 0) & (_pull(flags, C[OPP[q]]) == 1)
        t = 2.0 * f[q][at].sum()
        out = [o + C[q][k] * t for k, o in enumerate(out)]
    return torch.stack([torch.as_tensor(o, device="cuda", dtype=torch.float64) for o in out])


def _exact_train(case, seed):
    """Adam on the 3-32-32-1 tanh network in 64 bits, its weights rounded to BF16 before each step."""
    ut, ys, nu, tau = (a.double() for a in prepare(case, seed)[1])
    h, n, mask = 32, case["samples"], (1 << 64) - 1

    class Rng:
        s = 0

        def u64(self):
            self.s = (self.s + 0x9E3779B97F4A7C15) & mask
            z = self.s
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            return z ^ (z >> 31)

        def uniform(self, lim):
            return float(np.float32((2.0 * ((self.u64() >> 11) / 9007199254740992.0) - 1.0) * np.float32(lim)))

    rng = Rng()
    limits = [math.sqrt(6.0 / (3 + h)), math.sqrt(6.0 / (h + h)), math.sqrt(6.0 / (h + 1))]
    w1, w2, w3 = ([rng.uniform(lim) for _ in range(k)] for lim, k in zip(limits, (3 * h, h * h, h)))
    master = torch.tensor(w1 + [0.0] * h + w2 + [0.0] * h + w3 + [0.0], device="cuda", dtype=torch.float64)
    cuts = [3 * h, h, h * h, h, h, 1]
    cols = [ut.log(), ys.log(), nu.log(), tau.log() - ut.log()]
    mean, std = ([float(np.float32(float(g))) for g in v] for v in
                 ([c.mean() for c in cols], [c.std(unbiased=False) for c in cols]))
    x = torch.stack([(c - a) / b for c, a, b in zip(cols[:3], mean, std)], 1)
    target = (cols[3] - mean[3]) / std[3]
    rng = Rng()
    per = -(-n // case["batch"])
    total = per * case["epochs"]
    up = max(1, int(0.3 * total))
    lr_max = float(np.float32(3e-3))
    lr0 = lr_max / 25.0
    end = lr0 / 1e4
    m, v, t, loss = torch.zeros_like(master), torch.zeros_like(master), 0, []
    b1, b2 = float(np.float32(0.9)), float(np.float32(0.999))
    for _ in range(case["epochs"]):
        while True:
            a = 1 + rng.u64() % (n - 1)
            if math.gcd(a, n) == 1:
                break
        c = rng.u64() % n
        order = (a * torch.arange(n, device="cuda") + c) % n
        for at in torch.split(order, case["batch"]):
            w1, c1, w2, c2, w3, c3 = master.float().bfloat16().double().split(cuts)
            w1, w2 = w1.view(h, 3), w2.view(h, h)
            h1 = torch.tanh(x[at] @ w1.T + c1)
            h2 = torch.tanh(h1 @ w2.T + c2)
            err = h2 @ w3 + c3 - target[at]
            dy = 2.0 * err / len(at)
            dz2 = dy[:, None] * w3 * (1 - h2 * h2)
            dz1 = (dz2 @ w2) * (1 - h1 * h1)
            g = torch.cat([(dz1.T @ x[at]).reshape(-1), dz1.sum(0), (dz2.T @ h1).reshape(-1), dz2.sum(0), dy @ h2,
                           dy.sum()[None]])
            lr = (lr0 + (lr_max - lr0) * 0.5 * (1 - math.cos(math.pi * t / up)) if t < up else
                  end + (lr_max - end) * 0.5 * (1 + math.cos(math.pi * (t - up) / max(1, total - up))))
            t += 1
            m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
            master = master - lr * (m / (1 - b1 ** t)) / ((v / (1 - b2 ** t)).sqrt() + 1e-8)
        loss.append((err * err).mean())
    # The normalisation is two roundings of its own and comes back as numbers.
    return {"loss": torch.stack(loss), "master": master, "bf16": master.float().bfloat16().double(),
            "norm": {"in_mean": mean[:3], "in_std": std[:3], "out_mean": mean[3], "out_std": std[3]}}


def _exact_labels(case, seed):
    """Reichardt's law solved for u_tau by bisection in log u_tau."""
    ut, ys, nu = (a.double() for a in _samples(case, seed))
    lo, hi = (ut * 1e-4).log(), (ut * 2.0).log()
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        yp = mid.exp() * ys / nu
        up = torch.log1p(0.41 * yp) / 0.41 + 7.8 * (1 - (-yp / 11).exp() - (yp / 11) * (-yp / 3).exp())
        over = mid.exp() * up > ut
        lo, hi = torch.where(over, lo, mid), torch.where(over, mid, hi)
    return (0.5 * (lo + hi)).exp()


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "labels":
        # The reference's fixed iteration count is an approximation of its own.
        return _exact_labels(case, seed) if case["method"] == "newton64" else None
    if kind == "polar":
        force = []
        for t in _polar(case, seed):
            level = _Level64(t.dims, t.flags)
            level.start(_uniform64(t.dims, t.flags, t.u_lat))
            for _ in range(case["steps"]):
                level.collide(t.tau, t.u_lat)
                level.swap()
            force.append(_force64(level))
        return {"force": torch.stack(force)[None], "latched": None}
    if kind == "box":
        dims = _dims(case)
        level = _Level64(dims, torch.zeros(int(np.prod(dims)), dtype=torch.uint8, device="cuda"))
        level.start(_equilibrium64(dims, level.flags, _fields(dims, seed, periodic=True)))
        for _ in range(case["steps"]):
            level.collide(0.53, 0.05)
            level.swap()
        return {"f": [_stored(case, level.f[0])], "slip": []}
    levels = _levels(case, AOA)
    if kind == "edit":
        return _exact_edit(case, levels, seed)
    if kind == "aoa":
        new = _levels(case, _new_angle(seed))
        top = _Level64(*new[0])
        top.start(_uniform64(top.dims, top.flags, U_LAT))
        out = [top]
        if len(new) > 1:
            fine = _Level64(*levels[1])
            fine.start(_empty64(case, fine.dims))
            _seed64(fine, top, TAU)          # set_flags seeds by the old flags, set_refined_flags by the new
            fine.flags = new[1][1].reshape(fine.flags.shape)
            _seed64(fine, top, TAU)
            out.append(fine)
        return {"flags": None, "f": [_stored(case, lv.f[0]) for lv in out]}
    stack = [_Level64(*lv) for lv in levels]
    stack[0].start(_equilibrium64(stack[0].dims, stack[0].flags, _fields(_dims(case), seed)))
    tau = TAU
    for parent, lv in zip(stack, stack[1:]):
        lv.start(_empty64(case, lv.dims))
        _seed64(lv, parent, tau)
        tau = _fine_tau(tau, lv.m)
    shells = [lv.inner_shell() for lv in stack[1:]]
    for _ in range(case["steps"]):
        stack[0].collide(TAU, U_LAT)
        if len(stack) > 1:
            _sub_steps(stack, shells, TAU)
        stack[0].swap()
    # The slip velocities follow from wall lists that are not rebuilt here; the first pass steps without slip.
    out = {"f": [_stored(case, lv.f[0]) for lv in stack], "slip": None}
    if case.get("force"):
        out["force"] = _force64(stack[0])
    return out


def _exact_edit(case, levels, seed):
    dims = _dims(case)
    shape = (dims[2], dims[1], dims[0])
    first, second = (t.reshape(shape) for t in _edits(case, levels, seed))
    f = _equilibrium64(dims, first, _fields(dims, seed))
    gone, back = (first != 1) & (second == 1), (first == 1) & (second != 1)
    usable = (second == 0) & ~back
    rho, j = _moments([f[q] for q in range(19)])
    sums, n = [torch.zeros(shape, device="cuda", dtype=torch.float64) for _ in range(4)], 0.0
    for q in range(1, 19):
        at = _pull(usable, C[OPP[q]])        # vanes stand clear of the x and y faces
        n = n + at
        for k, v in enumerate((rho, j[0] / rho, j[1] / rho, j[2] / rho)):
            sums[k] += torch.where(at, _pull(v, C[OPP[q]]), 0.0)
    mean = [torch.where(n > 0, s / n.clamp_min(1), float(k == 0)) for k, s in enumerate(sums)]
    usq = _usq(mean[1:])
    for q in range(19):
        f[q] = torch.where(gone, 0.0, torch.where(back, _feq(q, mean[0], mean[1:], usq), f[q]))
    return {"edited": None, "wall_cells": None, "f": [_stored(case, f)]}
