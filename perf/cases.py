"""Workloads for timing and checking the framework through its public entry points.

A case is a dict of plain values.  `prepare` makes what a simulation program
has in hand before the call (inputs drawn from the seed, the objects it
keeps), `run` is one pass through the public API, `work` the bytes and
operations one pass cannot do without, `exact` the pass's results in 64 bits
by plain torch.

Kinds, and what each stands for in a PhysiCell-style main loop:

    substep    one diffusion sub-step through the main loop's own three calls
               (sweeps, Dirichlet reset, secretion): the smallest call
    period     one mechanics period of a single simulation: 10 sub-steps and
               a mechanics update, optionally with voxel refresh, motility
               between forces and integration, and net export
    diffuse    one diffusion step of a large 2-D domain, no cells
    mechanics  CellMechanics.update alone, on a dense cell population
    batch      many uneven simulations advanced together for some periods,
               then the state read back into pinned host buffers (with
               'upload', the host-owned fields are sent up first)
    serve      requests of mixed sizes submitted to the server, run to
               completion and fetched
    gradients  computeGradients with its read-back
    sort       the allocation-free pair sort on device buffers
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DT, DT_MECH, SUB_STEPS = 0.01, 0.1, 10
L2_BYTES = 126e6


def _package():
    if "pcg" not in sys.modules:
        pkg = os.path.join(ROOT, "physicell-mac-metal_b200")
        spec = importlib.util.spec_from_file_location("pcg", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["pcg"] = mod
        spec.loader.exec_module(mod)
    from pcg import workloads
    return sys.modules["pcg"], workloads


_ctx = None


def _context():
    """The program's one context on the GPU."""
    global _ctx
    if _ctx is None:
        _ctx = _package()[0].Context(0)
    return _ctx


# ---------------------------------------------------------------- the cases


def listed():
    return [
        # the 50 x 50 plain 2-D simulation, one sub-step as its main loop calls it
        {"name": "substep_2d", "kind": "substep", "nx": 50, "ny": 50, "nz": 1, "S": 1, "cells": 500},
        # the same simulation, one mechanics period
        {"name": "period_2d", "kind": "period", "nx": 50, "ny": 50, "nz": 1, "S": 1, "cells": 500,
         "refresh": False, "motile": False, "export": False},
        # an odd-sized 2-D tissue of three substrates with motile, exporting cells
        {"name": "period_2d_motile", "kind": "period", "nx": 181, "ny": 117, "nz": 1, "S": 3, "cells": 8191,
         "refresh": True, "motile": True, "export": True},
        # a centimetre-scale 2-D domain: lines past every shared-memory tile
        {"name": "diffuse_2d_long", "kind": "diffuse", "nx": 701, "ny": 530, "nz": 1, "S": 2},
        # the plain 3-D simulation, one mechanics period
        {"name": "period_3d", "kind": "period", "nx": 150, "ny": 150, "nz": 150, "S": 4, "cells": 200000,
         "refresh": False, "motile": False, "export": False},
        # a small odd-sized 3-D spheroid whose voxel indices follow its cells
        {"name": "period_3d_odd", "kind": "period", "nx": 61, "ny": 47, "nz": 53, "S": 2, "cells": 30011,
         "refresh": True, "motile": False, "export": False},
        # mechanics alone: a dense 3-D population
        {"name": "mechanics_3d", "kind": "mechanics", "nx": 75, "ny": 75, "nz": 75, "S": 1, "cells": 99991},
        # the batched 2-D configuration: 256 simulations, side 32..256, 1-3 substrates
        {"name": "batch_2d", "kind": "batch", "dims": 2, "instances": 256, "side_lo": 32, "side_hi": 256,
         "cells_lo": 100, "cells_hi": 20000, "periods": 10, "upload": False, "sizes": 1236},
        # the batched 3-D configuration (the benchmark's), with the host's phenotype fields sent up
        {"name": "batch_3d", "kind": "batch", "dims": 3, "instances": 64, "side_lo": 40, "side_hi": 120,
         "cells_lo": 1000, "cells_hi": 100000, "periods": 10, "upload": True, "sizes": 1237},
        # a parameter sweep of mixed 2-D / 3-D requests served to completion
        {"name": "serve_mixed", "kind": "serve", "requests": 6, "side2_hi": 256, "side3_hi": 100,
         "cells_hi": 20000, "steps_lo": 100, "steps_hi": 300, "sizes": 1238},
        # field gradients of a 3-D simulation, read back
        {"name": "gradients_3d", "kind": "gradients", "nx": 97, "ny": 64, "nz": 33, "S": 2},
        # cells sorted by mechanics voxel without device allocation
        {"name": "sort_200k", "kind": "sort", "n": 200003, "bits": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["substep", "period", "period", "diffuse", "mechanics", "batch", "batch", "serve", "gradients",
                       "sort"])
    if kind in ("substep", "period"):
        two_d = kind == "substep" or rng.random() < 0.5
        if two_d:
            nx, ny, nz, S = _log_int(rng, 20, 300), _log_int(rng, 20, 300), 1, rng.randint(1, 4)
            cells = _log_int(rng, 100, 20000)
        else:
            nx, ny, nz = (_log_int(rng, 20, 150) for _ in range(3))
            S = rng.randint(1, 4)
            cells = _log_int(rng, 1000, 200000)
        c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "S": S, "cells": cells}
        if kind == "period":
            c.update(refresh=rng.random() < 0.5, motile=rng.random() < 0.3, export=rng.random() < 0.3)
        return c
    if kind == "diffuse":
        return {"kind": kind, "nx": _log_int(rng, 260, 1100), "ny": _log_int(rng, 260, 1100), "nz": 1,
                "S": rng.randint(1, 3)}
    if kind == "mechanics":
        side = _log_int(rng, 30, 120)
        nz = side if rng.random() < 0.6 else 1
        cells = _log_int(rng, 500, 200000 if nz > 1 else 20000)
        return {"kind": kind, "nx": side, "ny": side, "nz": nz, "S": 1, "cells": cells}
    if kind == "batch":
        dims = rng.choice([2, 3])
        lo, hi = (32, 256) if dims == 2 else (40, 120)
        return {"kind": kind, "dims": dims, "instances": _log_int(rng, 4, 128 if dims == 2 else 32), "side_lo": lo,
                "side_hi": hi, "cells_lo": 100 if dims == 2 else 1000, "cells_hi": 20000 if dims == 2 else 60000,
                "periods": 10, "upload": rng.random() < 0.5, "sizes": rng.randint(1, 1 << 20)}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(2, 8), "side2_hi": 256, "side3_hi": 80, "cells_hi": 10000,
                "steps_lo": 60, "steps_hi": 300, "sizes": rng.randint(1, 1 << 20)}
    if kind == "gradients":
        return {"kind": kind, "nx": _log_int(rng, 20, 120), "ny": _log_int(rng, 20, 120), "nz": _log_int(rng, 1, 60),
                "S": rng.randint(1, 3)}
    return {"kind": kind, "n": _log_int(rng, 1000, 1 << 18), "bits": rng.randint(8, 32)}


# ---------------------------------------------------------------- inputs


def _sizes(case):
    """Sizes of the simulations of a batch or of a server's requests, by the case alone:
    (nx, ny, nz, substrates, cells, steps) each."""
    r = np.random.default_rng(case["sizes"])
    out = []
    if case["kind"] == "batch":
        for _ in range(case["instances"]):
            side = int(r.integers(case["side_lo"], case["side_hi"] + 1))
            S = int(r.integers(1, 4)) if case["dims"] == 2 else 2
            n = int(r.integers(case["cells_lo"], case["cells_hi"] + 1))
            out.append((side, side, 1 if case["dims"] == 2 else side, S, n, case["periods"] * SUB_STEPS))
        return out
    for k in range(case["requests"]):
        two_d = k % 10 < 7
        side = int(r.integers(64, case["side2_hi"] + 1)) if two_d else int(r.integers(40, case["side3_hi"] + 1))
        out.append((side, side, 1 if two_d else side, int(r.integers(1, 5)), int(r.integers(500, case["cells_hi"] + 1)),
                    int(r.integers(case["steps_lo"], case["steps_hi"] + 1))))
    return out


def _instance(nx, ny, nz, S, n, rng, refresh=False, export=False):
    """One simulation: an oxygen-like substrate and drug-like ones, a random field about the
    targets, cells over the domain (2-D) or in a central ball (3-D)."""
    pcg, wl = _package()
    two_d = nz == 1
    grid = pcg.make_grid(nx, ny, nz, S, dx=20.0, dt=DT, z_min=-10.0 if two_d else 0.0)
    subs = [(1e5, 0.1, True, 38.0)]
    for s in range(1, S):   # the third substrate has no Dirichlet boundary
        subs.append((float(np.exp(rng.uniform(np.log(1e3), np.log(1e5)))), float(rng.uniform(0, 1)), s != 2,
                     float(rng.uniform(1, 40))))
    targets = np.array([p[3] for p in subs], np.float32)
    nv = nx * ny * nz
    density = (targets[:, None] * (np.float32(0.5) + np.float32(0.5) * rng.random((S, nv), dtype=np.float32))).ravel()
    lo = np.zeros(3)
    size = np.array([nx, ny, nz]) * 20.0
    if two_d:
        pos = np.zeros((n, 3), np.float32)
        pos[:, :2] = rng.uniform(0, 1, (n, 2)) * size[:2]
    else:
        v = rng.normal(size=(n, 3))
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        pos = (lo + size / 2 + v * (0.4 * size) * (rng.random(n) ** (1 / 3))[:, None]).astype(np.float32)
    radius = np.clip(rng.normal(8.4, 0.5, n), 5.0, 12.0).astype(np.float32)
    upt = np.tile(np.r_[10.0, np.ones(S - 1)], n) * rng.uniform(0.5, 1.5, n * S)
    # the 3-D simulations of more than two substrates secrete as well
    sec = rng.uniform(0, 10, n * S) if (not two_d and S > 2) else np.zeros(n * S)
    ne = rng.uniform(0, 5, n * S) if export else None
    inst = wl.instance(grid, subs, pos, radius, 10.0, 0.4, 1.25, sec=sec, upt=upt, sat=np.tile(targets, n).astype(float),
                       ne=ne, two_d=two_d, flags=pcg.INST_REFRESH_VOXELS if refresh else 0)
    inst.density = density
    return inst


def _instances(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        refresh = kind == "batch" and case["dims"] == 3
        return [_instance(nx, ny, nz, S, n, np.random.default_rng([seed, i]), refresh)
                for i, (nx, ny, nz, S, n, _) in enumerate(_sizes(case))]
    return [_instance(case["nx"], case["ny"], case["nz"], case["S"], case.get("cells", 0),
                      np.random.default_rng([seed, 0]), case.get("refresh", False), case.get("export", False))]


def _motility_state(n, S, rng):
    return {"persistence_time": rng.uniform(5.0, 30.0, n), "elapsed": rng.uniform(0.0, 5.0, n),
            "bias": rng.uniform(0, 1, n), "vec": rng.normal(0, 0.2, 3 * n),
            "is_motile": (rng.random(n) < 0.8).astype(np.uint32), "restrict_2d": np.ones(n, np.uint32),
            "chemotaxis_index": rng.integers(0, S, n).astype(np.int32),
            "chemotaxis_direction": np.where(rng.random(n) < 0.5, 1, -1).astype(np.int32),
            "sensitivity": rng.uniform(-1, 1, n * S)}


class _DeviceArray:
    """A block of the library's device memory, for torch; keeps its owner alive."""

    def __init__(self, owner, ptr, shape, strides, kind="<f4"):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": kind, "data": (ptr, False), "version": 3,
                                         "strides": tuple(4 * s for s in strides)}


class _HostArray:
    """A library-pinned host buffer, for numpy; keeps its owner alive."""

    def __init__(self, pinned):
        self.owner = pinned
        self.__array_interface__ = {"shape": pinned.array.shape, "typestr": "<f4",
                                    "data": (pinned.array.ctypes.data, False), "version": 3}


def _pinned(pcg, n):
    return np.asarray(_HostArray(pcg.PinnedArray((n,))))


def _density_view(pcg, me):
    ptr, rp, sp = ctypes.POINTER(ctypes.c_float)(), ctypes.c_size_t(), ctypes.c_size_t()
    me.ctx.check(pcg.lib().pcg_me_device_density(me.h, ctypes.byref(ptr), ctypes.byref(rp), ctypes.byref(sp)))
    g = me.grid
    shape = (g.n_substrates, g.nz, g.ny, g.nx)
    return torch.as_tensor(_DeviceArray(me, ctypes.cast(ptr, ctypes.c_void_p).value, shape,
                                        (sp.value, rp.value * g.ny, rp.value, 1)), device="cuda")


def _cell_views(pcg, cells):
    ptr, mc = ctypes.POINTER(ctypes.c_float)(), ctypes.c_uint32()
    cells.ctx.check(pcg.lib().pcg_cells_device_soa(cells.h, ctypes.byref(ptr), ctypes.byref(mc)))
    base, m, n = ctypes.cast(ptr, ctypes.c_void_p).value, mc.value, cells.n

    def fields(first, count, kind="<f4"):
        return torch.as_tensor(_DeviceArray(cells, base + 4 * first * m, (count, n), (m, 1), kind), device="cuda")
    return {"position": fields(0, 3), "velocity": fields(3, 3), "previous_velocity": fields(6, 3),
            "pressure": fields(22, 1), "voxel": fields(26, 1, "<i4"), "mech_voxel": fields(27, 1, "<i4")}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g = torch.Generator("cuda").manual_seed(seed)
        n = case["n"]
        keys = torch.randint(0, 1 << case["bits"], (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
        vals = torch.arange(n, device="cuda", dtype=torch.int32)
        return {"kind": kind, "bits": case["bits"], "keys": keys, "vals": vals, "keys_out": torch.empty_like(keys),
                "vals_out": torch.empty_like(vals)}
    pcg, _ = _package()
    ctx = _context()
    insts = _instances(case, seed)
    if kind == "serve":
        return {"kind": kind, "server": pcg.Server(ctx), "instances": insts, "steps": [z[5] for z in _sizes(case)]}
    if kind == "batch":
        batch = pcg.Batch(ctx, insts)
        n = batch.totals()[2]
        st = {"kind": kind, "batch": batch, "steps": case["periods"] * SUB_STEPS, "n": n,
              "soa": _pinned(pcg, pcg.NUM_FIELDS * n), "density": _pinned(pcg, batch.layout(0)[3])}
        if case["upload"]:
            st["fields"] = _pinned(pcg, pcg.NUM_FIELDS * n)
            off, host = 0, st["fields"].reshape(pcg.NUM_FIELDS, n)
            for inst in insts:
                host[:, off:off + inst.n_cells] = inst.soa.reshape(pcg.NUM_FIELDS, -1)[:, :inst.n_cells]
                off += inst.n_cells
        return st
    inst = insts[0]
    me = pcg.Microenvironment(ctx, inst.grid, inst.substrates)
    me.setDensityAll(inst.density)
    st = {"kind": kind, "me": me, "out": {"density": _density_view(pcg, me)}}
    if inst.n_cells:
        cells = pcg.Cells(ctx, inst.n_cells, inst.grid.n_substrates)
        cells.upload(inst.soa, inst.n_cells, inst.soa_max)
        cells.set_secretion(*inst.rates)
        if case.get("refresh"):
            cells.set_voxel_refresh(me)
        st["cells"] = cells
    if kind in ("period", "mechanics"):
        g = inst.grid
        st["mech"] = pcg.CellMechanics(ctx, inst.mech, (g.x_min, g.y_min, g.z_min), inst.n_cells)
        if kind == "mechanics":
            st["out"] = {}
        st["out"].update(_cell_views(pcg, cells))
    if case.get("motile"):
        rng = np.random.default_rng([seed, 1])
        mot = pcg.Motility(ctx, inst.n_cells, case["S"])
        mot.upload(_motility_state(inst.n_cells, case["S"], rng))
        cells.upload_fields(pcg.F_MOT_SPEED, 1, _speed_block(pcg, inst, rng), inst.soa_max)
        cells.upload_fields(pcg.F_IS_ALIVE, 1, _alive_block(pcg, inst), inst.soa_max)
        st.update(motility=mot, step=0, seed=seed)
    return st


def _speed_block(pcg, inst, rng):
    b = inst.soa.copy()
    b[pcg.F_MOT_SPEED * inst.soa_max:pcg.F_MOT_SPEED * inst.soa_max + inst.n_cells] = rng.uniform(0.2, 1.0, inst.n_cells)
    return b


def _alive_block(pcg, inst):
    b = inst.soa.copy()
    a = pcg.F_IS_ALIVE * inst.soa_max
    b[a:a + inst.n_cells] = np.ones(inst.n_cells, np.uint32).view(np.float32)
    return b


# ---------------------------------------------------------------- one pass


def run(st):
    kind = st["kind"]
    if kind == "substep":
        st["me"].simulateDiffusionDecay(1)
        st["me"].applyDirichletBC()
        st["me"].applySecretion(st["cells"], DT)
        return st["out"]
    if kind == "period":
        st["me"].step(st["cells"], SUB_STEPS)
        if "motility" in st:
            st["mech"].computeForces(st["cells"])
            st["motility"].update(st["cells"], st["me"], DT_MECH, st["seed"], st["step"], 1)
            st["mech"].integratePositions(st["cells"], DT_MECH)
            st["step"] += 1
        else:
            st["mech"].update(st["cells"], DT_MECH)
        return st["out"]
    if kind == "diffuse":
        st["me"].simulateDiffusionDecay(1)
        return st["out"]
    if kind == "mechanics":
        st["mech"].update(st["cells"], DT_MECH)
        return st["out"]
    if kind == "batch":
        b, soa = st["batch"], st["soa"]
        if "fields" in st:
            b.upload_cell_fields(st["fields"])
        b.step(st["steps"])
        b.download_cell_fields(soa)
        b.download_all_density(st["density"])
        f = soa.reshape(-1, st["n"])
        return {"density": st["density"], "position": f[0:3], "velocity": f[3:6], "previous_velocity": f[6:9],
                "pressure": f[22:23], "voxel": f[26:27].view(np.int32), "mech_voxel": f[27:28].view(np.int32)}
    if kind == "serve":
        srv = st["server"]
        ids = [srv.submit(inst, k) for inst, k in zip(st["instances"], st["steps"])]
        while True:
            running, queued, _ = srv.tick()
            if running == 0 and queued == 0:
                break
        out = []
        for i in ids:
            dens, soa = srv.fetch(i)
            f = soa.reshape(28, -1)
            out.append({"density": dens, "floats": f[:23], "words": f[23:].view(np.int32)})
        return out
    if kind == "gradients":
        return list(st["me"].computeGradients())
    ctx = _context()
    ptr = [ctypes.c_void_p(st[k].data_ptr()) for k in ("keys", "vals", "keys_out", "vals_out")]
    ctx.check(_package()[0].lib().pcg_sort_pairs_static(ctx.h, *ptr, st["keys"].numel(), st["bits"]))
    return {"keys": st["keys_out"], "values": st["vals_out"]}


# ---------------------------------------------------------------- what a pass cannot do without


def _sim_work(nx, ny, nz, S, n, substeps, mech, resident):
    """Bytes and operations of one simulation: the density and the cells' secretion terms read
    (and the density written) once per pass where all of the pass's state fits on the chip, else
    once per sub-step; positions, strengths and the mechanics step's results once per step."""
    vs = nx * ny * nz * S
    times = 1 if resident else substeps
    b = times * (8 * vs + (8 * S + 4) * n)
    f = substeps * (5 * (2 if nz == 1 else 3) * vs + 4 * S * n)
    if mech:
        # 3 positions, 4 strengths, 6 velocity terms in; 10 fields and 2 indices out; ~10 neighbours
        b += (1 if resident else mech) * n * 4 * (13 + 12)
        f += mech * n * 10 * 30
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 16 * case["n"], "flops": 0}
    if kind in ("diffuse", "gradients"):
        vs = case["nx"] * case["ny"] * case["nz"] * case["S"]
        return {"bytes": 8 * vs, "flops": 10 * vs} if kind == "diffuse" else {"bytes": 16 * vs, "flops": 9 * vs}
    if kind == "mechanics":
        b, f = _sim_work(0, 0, 0, 1, case["cells"], 0, 1, True)
        return {"bytes": b, "flops": f}
    if kind in ("substep", "period"):
        sub, mech = (1, 0) if kind == "substep" else (SUB_STEPS, 1)
        b, f = _sim_work(case["nx"], case["ny"], case["nz"], case["S"], case["cells"], sub, mech, True)
        return {"bytes": b, "flops": f}
    sizes = _sizes(case)
    resident = sum(4 * x * y * z * s + n * (112 + 32 * s) for x, y, z, s, n, _ in sizes) < L2_BYTES
    tot = [_sim_work(x, y, z, s, n, k, k // SUB_STEPS, resident) for x, y, z, s, n, k in sizes]
    return {"bytes": sum(t[0] for t in tot), "flops": sum(t[1] for t in tot)}


# ---------------------------------------------------------------- the same in 64 bits

_F64 = torch.float64


class _Exact:
    """Sweeps, Dirichlet reset, secretion and mechanics of some simulations in 64 bits, on one
    flat array of all densities and one of all cells."""

    def __init__(self, insts):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=_F64, device=self.dev)   # noqa: E731
        self.insts = insts
        self.blocks, self.ops, dens, off = [], [], [], 0
        for inst in insts:
            g = inst.grid
            shape = (g.n_substrates, g.nz, g.ny, g.nx)
            self.blocks.append((off, shape))
            off += int(np.prod(shape))
            dens.append(t(inst.density))
            self.ops.append([self._axis(inst, a) for a in range(3 if g.nz > 1 else 2)])
        self.dens = torch.cat(dens)
        f = lambda k: t(np.concatenate([i.soa.reshape(28, -1)[k, :i.n_cells] for i in insts]))   # noqa: E731
        rep = lambda v: torch.repeat_interleave(t(v), self.count)                                 # noqa: E731
        self.count = torch.as_tensor([i.n_cells for i in insts], device=self.dev)
        self.n = int(self.count.sum())
        self.owner = torch.repeat_interleave(torch.arange(len(insts), device=self.dev), self.count)
        self.pos = torch.stack([f(0), f(1), f(2)])
        self.vel, self.prev = torch.stack([f(3), f(4), f(5)]), torch.stack([f(6), f(7), f(8)])
        self.radius, self.rep, self.adh, self.relmax = f(9), f(13), f(14), f(15)
        self.pressure = f(22)
        self.volume = f(11)
        vox = np.concatenate([i.soa.reshape(28, -1)[26, :i.n_cells].view(np.uint32) for i in insts]).astype(np.int64)
        self.voxel = torch.as_tensor(vox, device=self.dev)
        self.refresh = rep([float(i.flags & 1) for i in insts]) > 0
        g = [i.grid for i in insts]
        self.dims = torch.stack([rep([x.nx for x in g]), rep([x.ny for x in g]), rep([x.nz for x in g])]).long()
        self.h = torch.stack([rep([x.dx for x in g]), rep([x.dy for x in g]), rep([x.dz for x in g])])
        self.lo = torch.stack([rep([x.x_min for x in g]), rep([x.y_min for x in g]), rep([x.z_min for x in g])])
        m = [i.mech for i in insts]
        self.mdims = torch.stack([rep([x.mech_grid_nx for x in m]), rep([x.mech_grid_ny for x in m]),
                                  rep([x.mech_grid_nz for x in m])]).long()
        vs = m[0].mechanics_voxel_size
        self.hi = (self.lo.float() + self.mdims.float() * np.float32(vs)).to(_F64)
        mv = [x.mech_grid_nx * x.mech_grid_ny * x.mech_grid_nz for x in m]
        self.mtotal = int(sum(mv))
        self.mbase = torch.repeat_interleave(torch.as_tensor(np.r_[0, np.cumsum(mv)[:-1]].astype(np.int64),
                                                             device=self.dev), self.count)
        self.vs, self.maxd = float(vs), float(m[0].max_interaction_distance)
        # per cell and substrate (padded to the widest instance): terms of the secretion update
        self.S = max(x.n_substrates for x in g)
        self.terms, self.nv, self.base = [], rep([x.nx * x.ny * x.nz for x in g]).long(), \
            torch.repeat_interleave(torch.as_tensor([b[0] for b in self.blocks], device=self.dev), self.count)
        self.has = []
        for s in range(self.S):
            cols = []
            for q in range(4):
                cols.append(t(np.concatenate([i.rates[q].reshape(-1, i.grid.n_substrates)[:, s] if s < i.grid.n_substrates
                                              else np.zeros(i.n_cells) for i in insts])))
            self.terms.append(cols)
            self.has.append(rep([float(s < x.n_substrates) for x in g]) > 0)
        self._order()

    def _axis(self, inst, a):
        """The sweep along axis a as out = A in + b, per substrate."""
        g = inst.grid
        n, h = (g.nx, g.ny, g.nz)[a], float((g.dx, g.dy, g.dz)[a])
        A, b = [], []
        for s in range(g.n_substrates):
            p = inst.substrates[s]
            c = float(p.diffusion_coefficient) * float(g.dt) / (h * h)
            hd = float(p.decay_rate) * float(g.dt) / (3 if g.nz > 1 else 2)
            T, dirichlet = float(p.target_value), bool(p.dirichlet_enabled)
            full, add = np.eye(n), np.zeros(n)
            if n >= 3:
                m = n - 2
                M = np.diag(np.full(m, 1 + 2 * c + hd)) - c * (np.eye(m, k=1) + np.eye(m, k=-1))
                fold = np.zeros(m)
                if m > 1:
                    M[0, 0] = M[-1, -1] = 1 + c + hd
                if dirichlet:
                    fold[0] += c * T
                    fold[-1] += c * T
                inv = np.linalg.inv(M)
                full[1:-1, :] = 0
                full[1:-1, 1:-1] = inv
                add[1:-1] = inv @ fold
            if dirichlet:
                full[0] = full[-1] = 0
                add[0] = add[-1] = T
            A.append(full)
            b.append(add)
        t = lambda v: torch.as_tensor(np.stack(v), dtype=_F64, device=self.dev)   # noqa: E731
        return t(A), t(b)

    def diffuse(self, reset):
        for inst, (off, shape), ops in zip(self.insts, self.blocks, self.ops):
            S, nz, ny, nx = shape
            view = self.dens[off:off + S * nz * ny * nx].view(shape)
            d = torch.matmul(view.reshape(S, nz * ny, nx), ops[0][0].transpose(1, 2)) + ops[0][1][:, None, :]
            d = torch.matmul(ops[1][0][:, None], d.view(shape)) + ops[1][1][:, None, :, None]
            if nz > 1:
                d = (torch.matmul(ops[2][0], d.reshape(S, nz, ny * nx)) + ops[2][1][:, :, None]).view(shape)
            view.copy_(d)
            if reset:
                self._faces(inst, view)

    def _faces(self, inst, view):
        for s in range(view.shape[0]):
            p = inst.substrates[s]
            if not p.dirichlet_enabled:
                continue
            v, T = view[s], float(p.target_value)
            v[:, 0], v[:, -1], v[:, :, 0], v[:, :, -1] = T, T, T, T
            if view.shape[1] > 1:
                v[0], v[-1] = T, T

    def _order(self):
        """Cells by (voxel, index) and each cell's place among its voxel's cells."""
        key = self.base + self.voxel
        order = torch.argsort(key, stable=True)
        k = key[order]
        first = torch.ones_like(k, dtype=torch.bool)
        first[1:] = k[1:] != k[:-1]
        at = torch.arange(self.n, device=self.dev)
        rank = at - torch.cummax(torch.where(first, at, torch.zeros_like(at)), 0).values
        by_rank = torch.argsort(rank, stable=True)
        counts = torch.bincount(rank) if self.n else torch.zeros(0, dtype=torch.long)
        self.waves = torch.split(order[by_rank], counts.tolist())

    def secrete(self, dt):
        if self.n == 0:
            return
        V = self.h[0] * self.h[1] * self.h[2]
        ic = dt * self.volume / V
        for s in range(self.S):
            sec, upt, sat, ne = self.terms[s]
            c0, c1, c2 = dt * ne / V, ic * sec * sat, 1 + ic * (sec + upt)
            for w in self.waves:
                w = w[self.has[s][w]]
                at = self.base[w] + s * self.nv[w] + self.voxel[w]
                self.dens[at] = ((self.dens[at] + c0[w] + c1[w]) / c2[w]).clamp_min(0)

    def forces(self):
        b = [((self.pos[a] - self.lo[a]) / self.vs).long() for a in range(3)]
        b = [torch.minimum(b[a].clamp_min(0), self.mdims[a] - 1) for a in range(3)]
        mx, my, mz = self.mdims
        self.mech_voxel = (b[2] * my + b[1]) * mx + b[0]
        bins = self.mbase + self.mech_voxel
        order = torch.argsort(bins, stable=True)
        start = torch.zeros(self.mtotal + 1, dtype=torch.long, device=self.dev)
        start[1:] = torch.cumsum(torch.bincount(bins, minlength=self.mtotal), 0)
        force, press = torch.zeros_like(self.vel), torch.zeros_like(self.pressure)
        for dk in (-1, 0, 1):
            for dj in (-1, 0, 1):
                k, j = b[2] + dk, b[1] + dj
                ok = (k >= 0) & (k < mz) & (j >= 0) & (j < my)
                row = self.mbase + (k.clamp_min(0) * my + j.clamp_min(0)) * mx
                row = torch.where(ok, row, torch.zeros_like(row))
                q0 = start[row + (b[0] - 1).clamp_min(0)]
                q1 = start[row + torch.minimum(b[0] + 1, mx - 1) + 1]
                cnt = torch.where(ok, q1 - q0, torch.zeros_like(q0))
                ends = torch.cumsum(cnt, 0)
                total, i0 = int(ends[-1]), 0
                while i0 < self.n and total:   # blocks of cells with at most ~2e7 candidates
                    done = int(ends[i0 - 1]) if i0 else 0
                    i1 = max(i0 + 1, int(torch.searchsorted(ends, torch.tensor(done + 20_000_000, device=self.dev))))
                    i1 = min(i1, self.n)
                    c = cnt[i0:i1]
                    i = torch.repeat_interleave(torch.arange(i0, i1, device=self.dev), c)
                    if i.numel():
                        local = torch.arange(i.numel(), device=self.dev) - (ends[i] - cnt[i] - done)
                        self._pairs(i, order[q0[i] + local], force, press)
                    i0 = i1
        self.vel, self.pressure = force, press

    def _pairs(self, i, j, force, press):
        d = self.pos[:, i] - self.pos[:, j]
        d2 = (d * d).sum(0)
        near = (d2 < self.maxd ** 2) & (d2 >= 1e-12)
        i, j, d, dist = i[near], j[near], d[:, near], d2[near].sqrt()
        u = dist / (self.radius[i] + self.radius[j])
        ov, t = (1 - u).clamp_min(0), (1 - u / self.relmax[i]).clamp_min(0)
        F = ov ** 2 * (self.rep[i] * self.rep[j]).sqrt() - t ** 2 * (self.adh[i] * self.adh[j]).sqrt()
        press.index_add_(0, i, ov ** 2 / 0.027288820670331)
        for a in range(3):
            force[a].index_add_(0, i, F * d[a] / dist)

    def integrate(self, dt):
        self.pos = torch.maximum(torch.minimum(self.pos + dt * (1.5 * self.vel - 0.5 * self.prev), self.hi), self.lo)
        self.prev = self.vel
        if bool(self.refresh.any()):
            v = [torch.minimum(((self.pos[a] - self.lo[a]) / self.h[a]).long().clamp_min(0), self.dims[a] - 1)
                 for a in range(3)]
            new = (v[2] * self.dims[1] + v[1]) * self.dims[0] + v[0]
            self.voxel = torch.where(self.refresh, new, self.voxel)
            self._order()

    def cells(self):
        return {"position": self.pos, "velocity": self.vel, "previous_velocity": self.prev,
                "pressure": self.pressure[None], "voxel": None, "mech_voxel": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sort", "serve"):   # whole numbers; many sub-steps of whole simulations
        return None
    dt, dt_mech = float(np.float32(DT)), float(np.float32(DT_MECH))
    e = _Exact(_instances(case, seed))
    if kind == "substep":
        e.diffuse(True)
        e.secrete(DT)
        return {"density": e.dens.view(e.blocks[0][1])}
    if kind == "diffuse":
        e.diffuse(False)
        return {"density": e.dens.view(e.blocks[0][1])}
    if kind == "gradients":
        d, out = e.dens.view(e.blocks[0][1]), []
        for ax in (3, 2, 1):
            n, g = d.shape[ax], torch.zeros_like(d)
            if n > 1:
                s = lambda a, b: d.narrow(ax, a, b)   # noqa: B023,E731
                g.narrow(ax, 0, 1).copy_((s(1, 1) - s(0, 1)) / 20)
                g.narrow(ax, n - 1, 1).copy_((s(n - 1, 1) - s(n - 2, 1)) / 20)
                if n > 2:
                    g.narrow(ax, 1, n - 2).copy_((s(2, n - 2) - s(0, n - 2)) / 40)
            out.append(g.reshape(-1))
        return out
    if kind == "mechanics":
        e.forces()
        e.integrate(dt_mech)
        return e.cells()
    if kind == "period":
        for _ in range(SUB_STEPS):
            e.diffuse(True)
            e.secrete(dt)
        if case["motile"]:   # the random walk's draws are the library's own
            return {"density": e.dens.view(e.blocks[0][1]), **{k: None for k in e.cells()}}
        e.forces()
        e.integrate(dt_mech)
        return {"density": e.dens.view(e.blocks[0][1]), **e.cells()}
    for _ in range(case["periods"]):
        for _ in range(SUB_STEPS):
            e.diffuse(True)
            e.secrete(dt)
        e.forces()
        e.integrate(dt_mech)
    arena = []   # the device layout: rows padded to 4 values, substrates to 32, the padding zero
    for off, (S, nz, ny, nx) in e.blocks:
        px = (nx + 3) // 4 * 4
        pitch = (nz * ny * px + 31) // 32 * 32
        block = torch.zeros(S, pitch, dtype=_F64, device=e.dev)
        block[:, :nz * ny * px].view(S, nz * ny, px)[:, :, :nx] = e.dens[off:off + S * nz * ny * nx].view(S, nz * ny, nx)
        arena.append(block.reshape(-1))
    return {"density": torch.cat(arena), **e.cells()}
