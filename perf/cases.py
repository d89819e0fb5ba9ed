"""The work that users of this framework have it do, as cases that can be timed and checked.

Each case is a dict of plain values; ``kind`` says which part of the public API one pass goes through:

* ``md``       a run of velocity-Verlet LJ steps by the MD driver (Verlet list with skin, or a cell list
               every step; FP64, FP32 or the precision form), then a snapshot of the state in id order
* ``sph``      a dam break from a given state: the state in, a driver on it, weakly compressible SPH steps, the
               same snapshot out
* ``serve``    a batch of independent LJ systems of uneven size through the serving loop, host to host
* ``forces``   a program with its own integrator: new positions, map, ghost_get, list update, LJ forces
               (full Verlet list, half list with ghost_put, or cell list)
* ``functor``  the cell-list functor pattern: map, ghost_get, updateCellListGPU with reorder, a neighbour
               functor over the sorted cells, restoreOrder
* ``compact``  particles injected and removed: new particles in, get_indexes_by_type, a reduction,
               remove_marked, the kept particles out

Inputs are made on the GPU from the seed; ``exact`` restates each path in 64-bit torch.
"""
import math

import numpy as np
import torch

from openfpm_pdata_b200 import pd

R_CUT, SKIN, DT = 2.5, 0.3, 0.005
DEV = "cuda"


def listed():
    return [
        # the main workload: 160^3 LJ particles in FP64, list rebuilt by displacement
        {"name": "md_f64_4m", "kind": "md", "n": 4096000, "layout": "lattice", "precision": "f64", "cells": False,
         "steps": 10},
        # a medium system, an odd cube (63^3)
        {"name": "md_f64_250k", "kind": "md", "n": 250047, "layout": "lattice", "precision": "f64", "cells": False,
         "steps": 10},
        # a small system with the cell list rebuilt every step: latency between the phases of a step
        {"name": "md_cells_4k", "kind": "md", "n": 4096, "layout": "lattice", "precision": "f64", "cells": True,
         "steps": 20},
        # the precision form on clusters: uneven cells, frequent rebuilds, a ragged count
        {"name": "md_mixed_clusters_1m", "kind": "md", "n": 1000003, "layout": "clusters", "precision": "mixed",
         "cells": False, "steps": 10},
        # dam break at dp = 1/128 in FP64 (0.75M particles, mostly empty tank)
        {"name": "sph_f64_128", "kind": "sph", "k": 128, "dtype": "f64", "steps": 15},
        # dam break at dp = 1/180 in FP32 (1.9M particles)
        {"name": "sph_f32_180", "kind": "sph", "k": 180, "dtype": "f32", "steps": 15},
        # the serving loop: 24 systems of 512 to 262144 particles at once, 50 steps each
        {"name": "serve_24", "kind": "serve", "systems": 24, "largest": 262144, "mix": 6, "steps": 50},
        # forces for a program's own integrator, full Verlet list rebuilt
        {"name": "forces_verlet_f64_1m", "kind": "forces", "n": 1000000, "dtype": "f64", "list": "verlet"},
        # the same through the half list, reactions folded back by ghost_put
        {"name": "forces_half_f64_200k", "kind": "forces", "n": 200001, "dtype": "f64", "list": "half"},
        # neighbour functor over a reordered cell list, FP32, about 6 particles a cell
        {"name": "functor_f32_700k", "kind": "functor", "n": 700001, "dtype": "f32", "occ": 6.0},
        # the same calls on a few thousand particles: launches and synchronisations
        {"name": "functor_f64_4k", "kind": "functor", "n": 4099, "dtype": "f64", "occ": 6.0},
        # injection and removal: 10 % of 4,096,000 FP64 particles go
        {"name": "compact_f64_4m", "kind": "compact", "n": 4096000, "dtype": "f64", "frac": 0.1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "sph", "serve", "forces", "functor", "compact"])
    if kind == "md":
        cells = rng.random() < 0.3
        if cells:  # lists rebuilt every step: small systems
            return {"kind": "md", "n": _log_int(rng, 512, 100000), "layout": "lattice",
                    "precision": rng.choice(["f64", "f32"]), "cells": True, "steps": rng.randint(5, 20)}
        return {"kind": "md", "n": _log_int(rng, 2000, 2500000), "layout": rng.choice(["lattice", "clusters"]),
                "precision": rng.choice(["f64", "f64", "f32", "mixed"]), "cells": False, "steps": rng.randint(5, 12)}
    if kind == "sph":
        return {"kind": "sph", "k": _log_int(rng, 24, 160), "dtype": rng.choice(["f64", "f32"]),
                "steps": rng.randint(8, 20)}
    if kind == "serve":
        return {"kind": "serve", "systems": rng.randint(4, 24), "largest": _log_int(rng, 4096, 200000),
                "mix": rng.randint(0, 10 ** 6), "steps": rng.randint(10, 50)}
    dtype = rng.choice(["f64", "f32"])
    if kind == "forces":
        return {"kind": "forces", "n": _log_int(rng, 1000, 1500000), "dtype": dtype,
                "list": rng.choice(["verlet", "half", "cells"])}
    if kind == "functor":
        return {"kind": "functor", "n": _log_int(rng, 1000, 1500000), "dtype": dtype,
                "occ": round(rng.uniform(2.0, 12.0), 2)}
    return {"kind": "compact", "n": _log_int(rng, 1000, 4000000), "dtype": dtype,
            "frac": round(math.exp(rng.uniform(math.log(0.005), math.log(0.6))), 4)}


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _sites(side, spacing):
    k = (torch.arange(side, device=DEV, dtype=torch.float64) + 0.5) * spacing
    z, y, x = torch.meshgrid(k, k, k, indexing="ij")
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)


def _lattice(n, spacing, g):
    """n particles on a simple cubic lattice with vacancies, jitter +-0.05 of a spacing; (x, box side)."""
    side = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    pos = _sites(side, spacing)
    if pos.shape[0] > n:
        keep = torch.randperm(pos.shape[0], device=DEV, generator=g)[:n]
        pos = pos[torch.sort(keep).values]
    pos = pos + (torch.rand(pos.shape, device=DEV, dtype=torch.float64, generator=g) - 0.5) * (0.1 * spacing)
    return pos, side * spacing


def _clusters(n, g):
    """n of the 4 n lattice sites (spacing 1.1), drawn by the density of Gaussian clusters: dense cores of
    lattice density, thin outskirts, empty space; (x, box side)."""
    side = int(math.ceil((4.0 * n) ** (1.0 / 3.0)))
    pos = _sites(side, 1.1)
    L = side * 1.1
    nc = max(3, min(64, n // 16000))
    sigma = 0.30 * L / nc ** (1.0 / 3.0)
    centres = torch.rand((nc, 3), device=DEV, dtype=torch.float64, generator=g) * L
    w = torch.full((pos.shape[0],), 1e-30, device=DEV, dtype=torch.float64)
    for c in centres:
        d = pos - c
        d -= L * torch.round(d / L)
        w += torch.exp(-(d * d).sum(1) / (2 * sigma * sigma))
    u = torch.rand(w.shape, device=DEV, dtype=torch.float64, generator=g).clamp_(1e-12, 1 - 1e-12)
    key = torch.log(w) - torch.log(-torch.log(u))  # weighted draw without replacement
    keep = torch.sort(torch.topk(key, n).indices).values
    pos = pos[keep]
    return pos + (torch.rand(pos.shape, device=DEV, dtype=torch.float64, generator=g) - 0.5) * 0.1, L


def _velocities(n, g):
    v = torch.randn((n, 3), device=DEV, dtype=torch.float64, generator=g)
    return v - v.mean(0, keepdim=True)


def _md_inputs(case, seed):
    g = _gen(seed)
    if case["layout"] == "clusters":
        x, L = _clusters(case["n"], g)
    else:
        x, L = _lattice(case["n"], 1.0 if case["cells"] else 1.1, g)
    v = _velocities(case["n"], g)
    if case["precision"] == "f32":
        x = x.float()
        v = v.float()
    elif case["precision"] == "mixed":
        v = v.float()
    return x, v, L


def _sph_inputs(case, seed):
    """Dam break in a unit tank with three layers of wall particles: the fluid block of the usual geometry
    with hydrostatic density, slightly disordered, already in motion."""
    g = _gen(seed)
    k, wl = case["k"], 3
    dp = 1.0 / k
    f64 = dict(device=DEV, dtype=torch.float64)
    nf = [int(round(s * k)) for s in (0.4, 1.0, 0.6)]
    i, j, m = [(torch.arange(c, **f64) + 0.5) * dp for c in nf]
    z, y, x = torch.meshgrid(m, j, i, indexing="ij")
    flu = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    w = (torch.arange(-wl, k + wl, **f64) + 0.5) * dp
    wz = (torch.arange(-wl, k, **f64) + 0.5) * dp
    z, y, x = torch.meshgrid(wz, w, w, indexing="ij")
    wal = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    inside = (wal[:, 0] > 0) & (wal[:, 0] < 1) & (wal[:, 1] > 0) & (wal[:, 1] < 1) & (wal[:, 2] > 0)
    wal = wal[~inside]
    a, b = flu.shape[0], wal.shape[0]
    flu = flu + (torch.rand(flu.shape, generator=g, **f64) - 0.5) * (0.1 * dp)
    pos = torch.cat([flu, wal])
    typ = torch.cat([torch.zeros(a, device=DEV, dtype=torch.int32), torch.ones(b, device=DEV, dtype=torch.int32)])
    depth = (0.6 - pos[:, 2]).clamp(min=0)
    rho = 1000.0 * (1.0 + 7.0 * 9.81 * depth / 400.0) ** (1.0 / 7.0)
    vel = torch.zeros(pos.shape, **f64)
    vel[:a, 0] = 0.5 * torch.sin(3.0 * flu[:, 2])
    vel[:a, 1] = 0.2 * torch.cos(5.0 * flu[:, 0])
    vel[:a] += 0.02 * torch.randn((a, 3), generator=g, **f64)
    lo = [-(wl + 1) * dp] * 3
    hi = [1.0 + (wl + 1) * dp] * 3
    if case["dtype"] == "f32":
        pos, vel, rho = pos.float(), vel.float(), rho.float()
    return pos, vel, rho, typ, 1000.0 * dp ** 3, lo, hi


def _sph_dt(case):
    return 1e-4 * 128.0 / case["k"]  # the same fraction of the sound speed's limit at every resolution


def _serve_sizes(case):
    r = np.random.default_rng(case["mix"])
    return np.rint(np.exp(r.uniform(math.log(512), math.log(case["largest"]), case["systems"]))).astype(int).tolist()


def _serve_inputs(case, seed):
    g = _gen(seed)
    out = []
    for n in _serve_sizes(case):
        side = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
        x, L = _lattice(n, (n / 0.8) ** (1.0 / 3.0) / side, g)
        out.append((x.cpu().numpy(), _velocities(n, g).cpu().numpy(), L))
    return out


def _forces_inputs(case, seed):
    g = _gen(seed)
    x, L = _lattice(case["n"], 1.1, g)
    # as an integrator leaves them: a little outside the box on every side
    x = x + 0.2 * torch.randn((1, 3), device=DEV, dtype=torch.float64, generator=g)
    return (x.float() if case["dtype"] == "f32" else x), L


def _functor_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    x = torch.rand((n, 3), device=DEV, dtype=torch.float64, generator=g).to(dt)
    x = torch.where(x >= 1, torch.zeros_like(x), x)
    q = (torch.rand(n, device=DEV, dtype=torch.float64, generator=g) + 0.5).to(dt)
    return x, q, float((case["occ"] / n) ** (1.0 / 3.0))


def _compact_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    x = torch.rand((n, 3), device=DEV, dtype=torch.float64, generator=g).to(dt) * 100
    v = torch.randn((n, 3), device=DEV, dtype=torch.float64, generator=g).to(dt)
    mark = torch.zeros(n, device=DEV, dtype=torch.int32)
    mark[torch.randperm(n, device=DEV, generator=g)[: max(1, int(case["frac"] * n))]] = 1
    return x, v, mark


# ---------------------------------------------------------------- what a program keeps

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    f = np.float32 if case.get("dtype", case.get("precision")) == "f32" else np.float64
    t = pd.PD_F32 if f == np.float32 else pd.PD_F64
    if kind == "md":
        x, v, L = _md_inputs(case, seed)
        vt = pd.PD_F32 if case["precision"] == "mixed" else t
        skin = 0.0 if case["cells"] else SKIN
        vd = pd.VectorDist(case["n"], np.zeros(3), np.full(3, L), np.ones(3, np.int32), R_CUT + skin, dtype=f,
                           props=[(vt, 3), (vt, 3), (pd.PD_I64, 1)])
        vd.hostToDevicePos(x)
        vd.hostToDeviceProp(0, v)
        vd.hostToDeviceProp(2, torch.arange(case["n"], device=DEV))
        s["vd"], s["vel"], s["id"] = vd, 0, 2
        s["run"] = pd.MD(vd, 0, 1, dt=DT, skin=skin, r_cut=R_CUT, use_cell_list=case["cells"],
                         precision=pd.PREC_MIXED if case["precision"] == "mixed" else pd.PREC_FP64)
    elif kind == "sph":
        x, v, rho, typ, m, lo, hi = _sph_inputs(case, seed)
        n, dp = x.shape[0], 1.0 / case["k"]
        vd = pd.VectorDist(n, lo, hi, np.zeros(3, np.int32), 0.0, dtype=f,
                           props=[(t, 3), (t, 3), (t, 1), (t, 1), (pd.PD_I32, 1), (pd.PD_I64, 1)])
        s["vd"], s["vel"], s["id"] = vd, 0, 5
        s["start"] = {0: v, 2: rho, 4: typ, 5: torch.arange(n, device=DEV)}
        s["x"], s["dp"], s["m"] = x, dp, m
    elif kind == "serve":
        s["systems"] = _serve_inputs(case, seed)
        s["server"] = pd.Server(6 << 30, max_slots=64, dt=DT, skin=SKIN, autotune=False)
    elif kind == "forces":
        x, L = _forces_inputs(case, seed)
        vd = pd.VectorDist(case["n"], np.zeros(3), np.full(3, L), np.ones(3, np.int32), R_CUT, dtype=f,
                           props=[(t, 3)])
        vd.hostToDevicePos(x)
        vd.map()
        vd.ghost_get([])
        if case["list"] == "cells":
            s["cl"] = vd.getCellListGPU(R_CUT)
        else:
            s["vl"] = vd.getVerletSym(R_CUT) if case["list"] == "half" else vd.getVerlet(R_CUT)
        s["vd"], s["x"] = vd, x
    elif kind == "functor":
        x, q, r = _functor_inputs(case, seed)
        vd = pd.VectorDist(case["n"], np.zeros(3), np.ones(3), np.ones(3, np.int32), r, dtype=f,
                           props=[(t, 1), (t, 3)])
        s["cl"] = vd.getCellListGPU(r, opt=pd.CL_NON_SYMMETRIC | pd.CL_GPU_REORDER)
        s["vd"], s["x"], s["q"] = vd, x, q
    else:
        s["x"], s["v"], s["mark"] = _compact_inputs(case, seed)
        s["vd"] = pd.VectorDist(case["n"], np.zeros(3), np.full(3, 100.0), np.ones(3, np.int32), 1.0, dtype=f,
                                props=[(t, 3), (pd.PD_I32, 1)])
    return s


def _snapshot(s, *props):
    """Positions, velocities and further properties in id order, as a program keeps them between runs."""
    vd = s["vd"]
    ids = vd.deviceToHostProp(s["id"], with_ghost=False, device=True)
    out = []
    for a in [vd.deviceToHostPos(with_ghost=False, device=True)] + [
            vd.deviceToHostProp(p, with_ghost=False, device=True) for p in (s["vel"],) + props]:
        b = torch.empty_like(a)
        b[ids] = a
        out.append(b)
    return out


def run(s):
    kind, case, vd = s["kind"], s["case"], s.get("vd")
    if kind == "md":
        E = s["run"].run(case["steps"])
        x, v = _snapshot(s)
        return {"E": E[:, :3], "x": x, "v": v}
    if kind == "sph":
        vd.hostToDevicePos(s["x"])
        for p, a in s["start"].items():
            vd.hostToDeviceProp(p, a)
        dp = s["dp"]
        sph = pd.SPH(vd, 0, 1, 2, 3, 4, 1.3 * dp, s["m"], 20.0, 1000.0, 0.1, -9.81, _sph_dt(case), skin=0.3 * dp)
        E = sph.run(case["steps"])
        x, v, rho = _snapshot(s, 2)
        return {"E": E[:, :2], "x": x, "v": v, "rho": rho}
    if kind == "serve":
        srv = s["server"]
        tickets = [srv.submit(x, v, L, case["steps"]) for x, v, L in s["systems"]]
        srv.run_until_done(tickets)
        got = [srv.result(t) for t in tickets]
        for t in tickets:
            srv.release(t)
        srv.completed()
        return {"x": [r[0] for r in got], "E": [r[1][:, :3] for r in got]}
    if kind == "forces":
        vd.hostToDevicePos(s["x"])
        vd.map()
        vd.ghost_get([])
        if case["list"] == "cells":
            vd.updateCellListGPU(s["cl"])
            e = vd.lj_forces(0, cl=s["cl"], r_cut=R_CUT)
        else:
            vd.updateVerlet(s["vl"])
            e = vd.lj_forces(0, vl=s["vl"], r_cut=R_CUT)
            if case["list"] == "half":
                vd.ghost_put([0])
        return {"e": np.array(e), "f": vd.deviceToHostProp(0, with_ghost=False, device=True)}
    if kind == "functor":
        vd.hostToDevicePos(s["x"])
        vd.hostToDeviceProp(0, s["q"])
        vd.map()
        vd.ghost_get([0])
        vd.updateCellListGPU(s["cl"], [0])
        vd.test_force(s["cl"], 0, 1, sorted=True)
        vd.restoreOrder(s["cl"], [1])
        return vd.deviceToHostProp(1, with_ghost=False, device=True)
    vd.resize(case["n"])
    vd.hostToDevicePos(s["x"])
    vd.hostToDeviceProp(0, s["v"])
    vd.hostToDeviceProp(1, s["mark"])
    gone = vd.get_indexes_by_type(1, 1, device=True)
    vmax = vd.reduce_local(0, comp=0, op=pd.RED_MAX)
    vd.remove_marked(1)
    return {"gone": gone, "vmax": vmax, "x": vd.deviceToHostPos(device=True),
            "v": vd.deviceToHostProp(0, device=True)}


# ---------------------------------------------------------------- what a pass cannot do without

def _near(density, r):
    return density * 4.0 / 3.0 * math.pi * r ** 3


def work(case):
    kind = case["kind"]
    w = 4 if case.get("dtype", case.get("precision")) == "f32" else 8
    if kind == "md":
        wv = 4 if case["precision"] == "mixed" else w
        pairs = 0.5 * _near((1.0 if case["cells"] else 1.1) ** -3, R_CUT)
        n, st = case["n"], case["steps"]
        # a step reads and writes every position and velocity; each pair once, 35 operations
        return {"bytes": st * n * 2.0 * 3 * (w + wv), "flops": st * n * (pairs * 35 + 18)}
    if kind == "sph":
        k = case["k"]
        n = round(0.4 * k) * round(0.6 * k) * k + (k + 6) ** 2 * (k + 3) - k ** 3
        pairs = 0.5 * _near(1.0, 2.6) * 0.8
        # x, v and rho read and written each step, the type read; each pair once, 60 operations
        return {"bytes": case["steps"] * n * (2.0 * 7 * w + 4), "flops": case["steps"] * n * (pairs * 60 + 30)}
    if kind == "serve":
        n = float(sum(_serve_sizes(case)))
        pairs = 0.5 * _near(0.8, R_CUT)
        return {"bytes": n * (48 + 24 + case["steps"] * 2.0 * 36), "flops": case["steps"] * n * (pairs * 35 + 18)}
    n = case["n"]
    if kind == "forces":
        return {"bytes": n * 6.0 * w, "flops": n * 0.5 * _near(1.1 ** -3, R_CUT) * 35}
    if kind == "functor":
        return {"bytes": n * 7.0 * w, "flops": n * case["occ"] * 27 * 0.5 * 20}
    kept = n * (1 - case["frac"])
    return {"bytes": n * (6.0 * w + 4) + kept * 6 * w + 4 * (n - kept), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "md":
        return {"f64": {"rel": 1e-11, "max": 1e-8}, "f32": {"rel": 2e-4, "max": 5e-2},
                "mixed": {"rel": 4e-5, "max": 1e-2}}[case["precision"]]
    if kind == "sph":
        return {"rel": 1e-11, "max": 1e-8} if case["dtype"] == "f64" else {"rel": 1e-4, "max": 5e-2}
    if kind == "serve":
        return {"rel": 2e-5, "max": 5e-3}
    if kind == "forces":
        return {"rel": 1e-11, "max": 1e-8} if case["dtype"] == "f64" else {"rel": 1e-4, "max": 2e-2}
    if kind == "functor":
        return {"rel": 1e-13, "max": 1e-10} if case["dtype"] == "f64" else {"rel": 1e-5, "max": 1e-3}
    return "exact"


# ---------------------------------------------------------------- the same in 64 bits, in plain torch

def _pairs(x, r, L):
    """Every pair i < j nearer than r, as two index tensors; L: side of the periodic box, or None. Blocks of
    particles against the padded 27 cells around them."""
    lo = torch.zeros(3, **{"device": DEV, "dtype": torch.float64}) if L else x.amin(0)
    span = [L] * 3 if L else (x.amax(0) - lo + 1e-12).tolist()
    nc = [max(1, int(c / r)) for c in span]
    n = x.shape[0]
    if L and min(nc) < 3:  # too few cells around: all pairs
        out = []
        for a in range(0, n, 2048):
            d = x[a:a + 2048, None] - x[None]
            d -= L * torch.round(d / L)
            hit = ((d * d).sum(2) < r * r).nonzero()
            i, j = hit[:, 0] + a, hit[:, 1]
            out.append(torch.stack([i, j])[:, i < j])
        return torch.cat(out, 1)
    side = torch.tensor([c / m for c, m in zip(span, nc)], device=DEV, dtype=torch.float64)
    u = torch.minimum(((x - lo) / side).floor().long().clamp_(min=0), torch.tensor(nc, device=DEV) - 1)
    cell = u[:, 0] + nc[0] * (u[:, 1] + nc[1] * u[:, 2])
    cell, order = torch.sort(cell, stable=True)
    u, xs = u[order], x[order]
    start = torch.searchsorted(cell, torch.arange(nc[0] * nc[1] * nc[2] + 1, device=DEV))
    cap = int((start[1:] - start[:-1]).max())
    lane = torch.arange(cap, device=DEV)
    step = max(1, 24000000 // cap)
    out = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) < (0, 0, 0):
                    continue  # half of the cells: each pair once
                for a in range(0, n, step):
                    w = u[a:a + step] + torch.tensor([dx, dy, dz], device=DEV)
                    ok = torch.ones(w.shape[0], device=DEV, dtype=torch.bool)
                    for d in range(3):
                        if L:
                            w[:, d] %= nc[d]
                        else:
                            ok &= (w[:, d] >= 0) & (w[:, d] < nc[d])
                            w[:, d].clamp_(0, nc[d] - 1)
                    c = w[:, 0] + nc[0] * (w[:, 1] + nc[1] * w[:, 2])
                    j = start[c][:, None] + lane
                    live = (j < start[c + 1][:, None]) & ok[:, None]
                    if (dx, dy, dz) == (0, 0, 0):
                        live &= j > torch.arange(a, a + w.shape[0], device=DEV)[:, None]
                    hit = live.nonzero()
                    i, j = hit[:, 0] + a, j[live]
                    d = xs[i] - xs[j]
                    if L:
                        d -= L * torch.round(d / L)
                    near = (d * d).sum(1) < r * r
                    out.append(torch.stack([order[i[near]], order[j[near]]]))
    return torch.cat(out, 1)


class _List:
    """Pairs within r, found again when a particle has moved more than half the margin."""

    def __init__(self, r, margin, L):
        self.r, self.L = r, L
        self.margin = max(0.0, min(margin, L / 3.0 - r - 1e-9)) if L and L > 3 * r else (0.0 if L else margin)
        self.at = None

    def get(self, x):
        if self.at is None or float(((x - self.at) ** 2).sum(1).max()) ** 0.5 * 2 >= self.margin:
            self.at, self.ij = x.clone(), _pairs(x % self.L if self.L else x, self.r + self.margin, self.L)
        return self.ij


def _blocks(ij, size=1 << 25):
    for a in range(0, ij.shape[1], size):
        yield ij[0, a:a + size], ij[1, a:a + size]


def _lj(x, ij, L):
    f = torch.zeros_like(x)
    pe = vir = 0.0
    for i, j in _blocks(ij):
        d = x[i] - x[j]
        d -= L * torch.round(d / L)
        r2 = (d * d).sum(1)
        keep = r2 < R_CUT * R_CUT
        i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
        s6 = 1.0 / (r2 * r2 * r2)
        pe = pe + (4.0 * s6 * (s6 - 1.0)).sum()
        fr = 24.0 * s6 * (2.0 * s6 - 1.0)
        vir = vir + fr.sum()
        fd = d * (fr / r2)[:, None]
        f.index_add_(0, i, fd)
        f.index_add_(0, j, fd, alpha=-1)
    return f, pe, vir


def _exact_lj_run(x, v, L, steps):
    """(E, x wrapped into the box, v) after velocity-Verlet steps."""
    near = _List(R_CUT, 0.35, L)
    x = x.clone()
    v = v.clone()
    f, _, _ = _lj(x, near.get(x), L)
    E = []
    for _ in range(steps):
        v += 0.5 * DT * f
        x += DT * v
        f, pe, vir = _lj(x, near.get(x), L)
        v += 0.5 * DT * f
        E.append([float(0.5 * (v * v).sum()), float(pe), float(vir)])
    return np.array(E), x, v


def _exact_sph(case, seed):
    x, v, rho, typ, m, _, _ = _sph_inputs(case, seed)
    x, v, rho = x.double(), v.double(), rho.double()
    dp = 1.0 / case["k"]
    h, c0, rho0, alpha, gz, dt = 1.3 * dp, 20.0, 1000.0, 0.1, -9.81, _sph_dt(case)
    B, fluid = c0 * c0 * rho0 / 7.0, typ == 0
    near = _List(2 * h, 0.3 * dp, None)

    def rates():
        p2 = B * ((rho / rho0) ** 7 - 1.0) / (rho * rho)
        acc, dr = torch.zeros_like(x), torch.zeros_like(rho)
        for i, j in _blocks(near.get(x), 1 << 24):
            d = x[i] - x[j]
            r2 = (d * d).sum(1)
            keep = r2 < 4 * h * h
            i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
            r = r2.sqrt()
            q = r / h
            dw = torch.where(q < 1, -3 * q + 2.25 * q * q, -0.75 * (2 - q) ** 2) / (math.pi * h ** 4) / r
            vr = ((v[i] - v[j]) * d).sum(1)
            visc = torch.where(vr < 0, -alpha * c0 * h * vr / (r2 + 0.01 * h * h) / (0.5 * (rho[i] + rho[j])),
                               torch.zeros_like(vr))
            a = d * (-m * (p2[i] + p2[j] + visc) * dw)[:, None]
            acc.index_add_(0, i, a)
            acc.index_add_(0, j, a, alpha=-1)
            g = m * vr * dw
            dr.index_add_(0, i, g)
            dr.index_add_(0, j, g)
        acc[:, 2] += gz
        acc[~fluid] = 0
        return acc, dr

    a, dr = rates()
    E = []
    for _ in range(case["steps"]):
        v += 0.5 * dt * a
        x += dt * v
        rho += 0.5 * dt * dr
        a, dr = rates()
        v += 0.5 * dt * a
        rho += 0.5 * dt * dr
        E.append([0.5 * m * float((v[fluid] ** 2).sum()), float(rho.sum())])
    return {"E": np.array(E), "x": x, "v": v, "rho": rho}


def _exact_functor(case, seed):
    """The sum of q unit vectors over the 27 cells of the library's documented grid (box enlarged by the
    ghost times 1.013, cells of side r, one layer of padding), in 64 bits on the same cells."""
    x, q, r = _functor_inputs(case, seed)
    T = np.float32 if case["dtype"] == "f32" else np.float64
    enl = T(np.float32(1.013))
    lo, hi = -T(r) * enl, T(1) + T(r) * enl
    div = int((hi - lo) / T(r)) + 1
    sp = ((lo + T(div) * T(r)) - lo) / T(div)
    xs, qs = [x], [q]
    for l in range(27):  # periodic images within the ghost, in the vector's precision
        c = (l % 3 - 1, l // 3 % 3 - 1, l // 9 - 1)
        if c == (0, 0, 0):
            continue
        sel = torch.ones(x.shape[0], device=DEV, dtype=torch.bool)
        for d in range(3):
            if c[d] == 1:
                sel &= x[:, d] < float(T(0) + T(r))
            elif c[d] == -1:
                sel &= x[:, d] >= float(T(1) + -T(r))
        im = x[sel].clone()
        for d in range(3):
            im[:, d] -= -float(c[d])
        xs.append(im)
        qs.append(q[sel])
    p, w = torch.cat(xs), torch.cat(qs)
    gs = div + 2
    u = ((p - torch.tensor(lo, device=DEV, dtype=p.dtype)) / torch.tensor(sp, device=DEV, dtype=p.dtype)).floor()
    u = (u.long() + 1).clamp_(0, gs - 1)
    cell, order = torch.sort(u[:, 0] + gs * (u[:, 1] + gs * u[:, 2]), stable=True)
    start = torch.searchsorted(cell, torch.arange(gs ** 3 + 1, device=DEV))
    cap = int((start[1:] - start[:-1]).max())
    ps, ws, lane = p.double()[order], w.double()[order], torch.arange(cap, device=DEV)
    n = x.shape[0]
    out = torch.zeros((n, 3), device=DEV, dtype=torch.float64)
    step = max(1, 8000000 // cap)
    for a in range(0, n, step):
        xi, ui = x[a:a + step].double(), u[a:min(a + step, n)]
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    c = ui + torch.tensor([dx, dy, dz], device=DEV)
                    ok = ((c >= 0) & (c < gs)).all(1)
                    c = c.clamp(0, gs - 1)
                    c = c[:, 0] + gs * (c[:, 1] + gs * c[:, 2])
                    j = start[c][:, None] + lane
                    live = (j < start[c + 1][:, None]) & ok[:, None]
                    j = torch.where(live, j, torch.zeros_like(j))
                    d = ps[j] - xi[:, None]
                    nrm = (d * d).sum(2).sqrt()
                    live &= nrm > 1e-6
                    g = torch.where(live, ws[j] / nrm.clamp(min=1e-30), torch.zeros_like(nrm))
                    out[a:a + step] += (d * g[:, :, None]).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "md":
        x, v, L = _md_inputs(case, seed)
        E, x, v = _exact_lj_run(x.double(), v.double(), L, case["steps"])
        return {"E": E, "x": None, "v": v}  # positions are wrapped when the list is rebuilt, which is the driver's choice
    if kind == "sph":
        return _exact_sph(case, seed)
    if kind == "serve":
        got = [_exact_lj_run(torch.from_numpy(x).to(DEV), torch.from_numpy(v).to(DEV), L, case["steps"])
               for x, v, L in _serve_inputs(case, seed)]
        return {"x": [None] * len(got), "E": [g[0] for g in got]}
    if kind == "forces":
        x, L = _forces_inputs(case, seed)
        x = x.double()
        f, pe, vir = _lj(x, _pairs(x % L, R_CUT, L), L)
        return {"e": np.array([float(pe), float(vir)]), "f": f}
    if kind == "functor":
        return _exact_functor(case, seed)
    x, v, mark = _compact_inputs(case, seed)
    keep = mark == 0
    return {"gone": None, "vmax": float(v[:, 0].max()), "x": x[keep], "v": v[keep]}
