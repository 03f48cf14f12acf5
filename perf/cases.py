"""The work that a landscape model on the GPU is asked for: whole steps of a
run and the stages that programs call by themselves, over the sizes of this
repository's own configurations (2,500 to 2.6 million vertices, planar and
spherical meshes, ensembles, deposition, the adjoint).

A case is a plain dict:

* ``kind``: the entry point (``flow``, ``fill``, ``direction``, ``spl``,
  ``hillslope``, ``step``, ``adjoint``);
* ``mesh``: ``sphere`` (icosahedral, ``level`` refinements, 10 * 4^level + 2
  vertices numbered along a Morton curve), ``planar`` (jittered hexagonal
  lattice of about ``n`` vertices) or ``ensemble`` (``members`` planar
  landscapes of uneven size, largest about ``n`` vertices);
* ``R``: flow directions per vertex; further options by name.

Meshes depend on their size alone and are made once per process, as a
program makes them once per run; relief, rain, uplift and erodibility come
from the seed.
"""
import functools
import math

import numpy as np
import torch

from gospl_b200 import adjoint as A
from gospl_b200 import synthetic as S
from gospl_b200.ensemble import Ensemble
from gospl_b200.mesh import FVMesh
from gospl_b200.model import Model

DEV = "cuda"
SPACING = 750.0      # vertex spacing of the planar landscapes, m (20,000 vertices over about 100 km)


def listed():
    return [
        # the 20,000-vertex planar landscape: the smallest run in use, bound by launches and round trips
        {"name": "flow_planar_20k", "kind": "flow", "mesh": "planar", "n": 20000, "R": 3},
        # a whole step of it, 200 of which make its run
        {"name": "step_planar_20k", "kind": "step", "mesh": "planar", "n": 20000, "R": 3},
        # depressions of the inversion's landscape filled with sediment, as a program that inspects lakes asks
        {"name": "fill_sed_planar_160k", "kind": "fill", "mesh": "planar", "n": 160647, "R": 3, "sed": True},
        # flow directions alone at the default number of directions
        {"name": "direction_r8_sphere_655k", "kind": "direction", "mesh": "sphere", "level": 8, "R": 8},
        # flow accumulation of the 2.6M sphere: the largest part of the headline step
        {"name": "flow_sphere_2621k", "kind": "flow", "mesh": "sphere", "level": 9, "R": 3},
        # implicit diffusion of the same mesh, step after step
        {"name": "hillslope_sphere_2621k", "kind": "hillslope", "mesh": "sphere", "level": 9, "R": 3},
        # transport-limited erosion: many sweeps of one graph
        {"name": "spl_transport_sphere_164k", "kind": "spl", "mesh": "sphere", "level": 7, "R": 3, "G": 1.0},
        # the headline step: 2.6M-vertex sphere
        {"name": "step_sphere_2621k", "kind": "step", "mesh": "sphere", "level": 9, "R": 3},
        # a step with continental deposition and lake smoothing
        {"name": "step_sediment_sphere_655k", "kind": "step", "mesh": "sphere", "level": 8, "R": 3, "sed": True},
        # a step with marine deposition
        {"name": "step_marine_sphere_164k", "kind": "step", "mesh": "sphere", "level": 7, "R": 3, "sed": True,
         "marine": True},
        # an ensemble of uneven landscapes advanced together
        {"name": "step_ensemble_12", "kind": "step", "mesh": "ensemble", "n": 60000, "members": 12, "R": 3},
        # gradients of an elevation misfit on the inversion's mesh, by checkpointed replay
        {"name": "adjoint_planar_160k", "kind": "adjoint", "mesh": "planar", "n": 160647, "R": 3, "steps": 4,
         "every": 2},
    ]


def _log_size(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1


def draw(rng):
    kind = rng.choice(["flow", "flow", "fill", "direction", "spl", "hillslope", "step", "step", "step", "adjoint"])
    case = {"kind": kind}
    shape = rng.choice(["planar", "sphere"])
    if kind == "step" and rng.random() < 0.2:
        shape = "ensemble"
    if kind == "adjoint":
        shape = "planar"
    case["mesh"] = shape
    if shape == "sphere":
        case["level"] = rng.choice([5, 6, 7, 8])
    elif shape == "planar":
        case["n"] = _log_size(rng, 2500, 160000)
    else:
        case["members"] = rng.randint(3, 12)
        case["n"] = _log_size(rng, 8000, 60000)
    case["R"] = 3 if kind in ("adjoint", "step") else rng.choice([1, 2, 3, 4, 5, 8])
    case["dt"] = float(rng.randint(500, 9999))
    if kind == "fill":
        case["sed"] = rng.random() < 0.5
    elif kind == "direction":
        case["down"] = rng.random() < 0.5
    elif kind == "spl":
        case["G"] = rng.choice([0.0, 0.0, 0.5, 1.0])
        if case["G"] and shape == "sphere":
            case["level"] = min(case["level"], 7)
    elif kind == "step" and shape != "ensemble":
        case["sed"] = rng.random() < 0.4
        case["marine"] = case["sed"] and shape == "sphere" and case["level"] <= 7 and rng.random() < 0.5
        if not case["sed"]:
            case["precision"] = rng.choice([64, 64, 32])
    elif kind == "adjoint":
        case["n"] = _log_size(rng, 2500, 80000)
        case["steps"] = rng.randint(1, 4)
        case["every"] = rng.choice([1, 2])
    return case


# ----------------------------------------------------------------------------
# meshes
# ----------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sphere(level):
    coords, cells = S.icosphere(level)
    coords, cells = S.renumber(coords, cells, S.morton_order(coords))
    return coords, cells, FVMesh(coords, cells, "oooo", device=DEV)


@functools.lru_cache(maxsize=None)
def _planar(n, spacing):
    side = spacing * math.sqrt(n * math.sqrt(3.0) / 2.0)
    coords, cells, onb = S.planar_hex_mesh(n, side, 7 + n)
    return coords, cells, FVMesh(coords, cells, "ffff", device=DEV), onb, side


def _waves(coords, seed, kmax, count, beta):
    """Smooth random field on the sphere: `count` plane waves with wave numbers
    spread over the logarithm of 1.5..kmax and power per degree ~ k^-beta
    (a stand-in for the spherical-harmonic relief that is quick to make)."""
    rng = np.random.default_rng(seed)
    k = np.exp(rng.uniform(math.log(1.5), math.log(kmax), count))
    d = rng.standard_normal((count, 3))
    d *= (k / np.linalg.norm(d, axis=1))[:, None]
    amp = k ** ((1.0 - beta) / 2.0)
    phase = rng.uniform(0.0, 2.0 * math.pi, count)
    x = torch.as_tensor(coords / np.linalg.norm(coords, axis=1)[:, None], device=DEV)
    out = torch.zeros(len(coords), dtype=torch.float64, device=DEV)
    for q in range(count):
        arg = x[:, 0] * d[q, 0] + x[:, 1] * d[q, 1] + x[:, 2] * d[q, 2]
        out += amp[q] * torch.cos(arg + phase[q])
    return out.cpu().numpy()


def _inputs(case, seed):
    """(coords, cells, mesh, elevation, rain, uplift, params) of one landscape."""
    if case["mesh"] == "sphere":
        coords, cells, mesh = _sphere(case["level"])
        z = S.rescale(_waves(coords, seed, 256.0, 768, 2.0), -4000.0, 3000.0)
        g = _waves(coords, seed + 1, 32.0, 96, 2.0)
        rain = np.exp(0.5 * (g - g.mean()) / g.std())
        up = S.belt_uplift(coords, seed + 2)
        params = dict(dt=case.get("dt", 1.0e4), K=5.0e-7, Cda=0.05, Cdm=0.05, sealevel=0.0, bc="oooo")
    else:
        coords, cells, mesh, onb, side = _planar(case["n"], SPACING)
        z = S.rescale(S.fractal_field(coords[:, :2], side, seed), 0.0, 100.0)
        z[onb] = 0.0
        rain = np.ones(len(z))
        up = np.full(len(z), 1.0e-3)
        up[onb] = 0.0
        params = dict(dt=case.get("dt", 1.0e3), K=2.0e-6, Cda=0.1, Cdm=0.1, sealevel=-100.0, bc="ffff")
    params.update(tStart=0.0, tEnd=float("inf"), flowDir=case["R"], d=0.0, m=0.5, oFill=-6000.0, rain=rain, upsub=up)
    return coords, cells, mesh, z, params


def _ensemble(case, seed):
    members = []
    for q in range(case["members"]):
        # uneven sizes, the last the largest
        n = int(case["n"] * 6.0 ** ((q + 1.0) / case["members"] - 1.0)) | 1
        coords, cells, mesh, onb, side = _planar(n, 250.0)
        z = S.rescale(S.fractal_field(coords[:, :2], side, seed + 10 * q), 0.0, 100.0)
        z[onb] = 0.0
        g = S.fractal_field(coords[:, :2], side, seed + 10 * q + 1, beta=4.0)
        rain = np.exp(0.7 * (g - g.mean()) / g.std())
        K = float(np.exp(np.random.default_rng(seed + 10 * q + 2).uniform(math.log(1e-7), math.log(1e-5))))
        params = dict(dt=case.get("dt", 500.0), tStart=0.0, tEnd=1.0e30, flowDir=case["R"], K=K, d=0.0, m=0.5,
                      Cda=0.1, Cdm=0.1, sealevel=-100.0, oFill=-6000.0, bc="ffff")
        members.append((coords, cells, z, rain, np.zeros(len(z)), params))
    return Ensemble(members)


def prepare(case, seed):
    state = {"case": case, "turn": 1}
    if case["mesh"] == "ensemble":
        state["ens"] = _ensemble(case, seed)
        m = state["ens"].model
    else:
        coords, cells, mesh, z, params = _inputs(case, seed)
        if case.get("sed") and case["kind"] == "step":
            params.update(nodep=False, marineSolver="picard", seadepo=bool(case.get("marine")))
        if case.get("G"):
            params["G"] = case["G"]
        m = Model(coords=coords, cells=cells, elev=z, params=params, mesh=mesh, device=DEV,
                  precision=case.get("precision", 64))
    state["model"] = m
    if case["kind"] in ("step", "spl"):
        # two elevations that a program restarts from in turn: the relief, and the relief a step of uplift later
        h0 = m.hGlobal.clone()
        h1 = h0 + (m.upsub * m.dt if m.upsub is not None else 0.0)
        state["start"] = (h0, h1) if case["kind"] == "step" else (h0, h0)
    elif case["kind"] == "fill":
        # the depressions' tables, in buffers that hold any number of them
        f64 = dict(dtype=torch.float64, device=m.dev)
        state["tables"] = [torch.zeros((m.lpoints + 1, 3), **f64),
                           torch.zeros((m.lpoints + 1, 2), dtype=torch.int32, device=m.dev),
                           torch.zeros((m.lpoints + 1, 5), **f64), torch.zeros((m.lpoints + 1, 5), **f64)]
    elif case["kind"] == "adjoint":
        n = m.lpoints
        rng = np.random.default_rng(seed + 5)
        g = S.gp_field(m.mesh_coords[:, :2], float(m.mesh_coords[:, 0].max()), seed + 3, 20.0e3)
        state["K"] = torch.as_tensor(np.exp(S.rescale(g, -14.0, -11.0)), device=DEV)
        state["U"] = m.upsub.clone()
        state["rain"] = torch.as_tensor(rng.uniform(0.8, 1.2, n), device=DEV)
        state["h0"] = m.hGlobal.clone()
    return state


def _flow_outputs(m):
    return {"FAL": m.FAL, "fillFAL": m.fillFAL, "waterFilled": m.waterFilled, "lFill": m.lFill, "pitIDs": m.pitIDs,
            "flatDirs": m.flatDirs, "rcvID": m.rcv_i, "distRcv": m.dist_i, "wghtVal": m.wgt_i,
            "lsink": m.lsink_mask, "seaID": m.sea_mask}


def run(state):
    case, m = state["case"], state["model"]
    kind = case["kind"]
    if kind == "flow":
        m.flowAccumulation()
        return _flow_outputs(m)
    if kind == "fill":
        m.fillElevation(sed=bool(case["sed"]))
        for kept, table in zip(state["tables"], m.pit_tables()):
            kept[:m.npits + 1].copy_(table)
        return {"lFill": m.lFill, "pitIDs": m.pitIDs, "flatDirs": m.flatDirs, "tables": state["tables"]}
    if kind == "direction":
        m._buildFlowDirection(m.hGlobal, down=bool(case.get("down")))
        return {"rcvID": m.rcv_live, "distRcv": m.dist_live, "wghtVal": m.wgt_live, "lsink": m.lsink_mask,
                "seaID": m.sea_mask}
    if kind == "hillslope":
        m.getHillslope()
        return {"h": m.hGlobal, "cumED": m.cumED, "Eb": m.EbLocal}
    if kind == "adjoint":
        K, U, rain, h0 = (state[k] for k in ("K", "U", "rain", "h0"))
        ns, ev = case["steps"], case["every"]
        hT, ckpt = A.run(m, K, U, rain, h0, ns, ev)
        # misfit 0.5 |h_T - h_0|^2: its gradient is h_T - h_0
        gK, gU, gr, gh = A.backward(m, K, U, rain, ckpt, ns, ev, hT - h0)
        return {"h": hT, "gK": gK, "gU": gU, "grain": gr, "gh0": gh}
    # restart from one of the two elevations in hand, then the stage or the step
    state["turn"] ^= 1
    m.hGlobal.copy_(state["start"][state["turn"]])
    m.cumED.zero_()
    if kind == "spl":
        m.erodepSPL()
        return {"h": m.hGlobal, "cumED": m.cumED, "Eb": m.EbLocal}
    (state["ens"] if "ens" in state else m).step()
    out = {"h": m.hGlobal, "cumED": m.cumED, "Eb": m.EbLocal}
    out.update(_flow_outputs(m))
    if case.get("sed"):
        out["vSed"] = m.vSed
    return out


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def _vertices(case):
    """(vertices, neighbour entries per vertex)."""
    if case["mesh"] == "sphere":
        return 10 * 4 ** case["level"] + 2, 6
    if case["mesh"] == "planar":
        return case["n"], 6
    return sum(int(case["n"] * 6.0 ** ((q + 1.0) / case["members"] - 1.0)) | 1 for q in range(case["members"])), 6


def work(case):
    n, W = _vertices(case)
    R = case["R"]
    ids, edges, faces = 4 * W, 8 * W, 8 * W
    direction = 8 + ids + edges + 20 * R + 2                        # h, ids, edge lengths -> rcv, dist, wgt, masks
    fill = 8 + ids + 1 + 8 + 4 + 4                                  # h, ids, outlets -> lFill, pitIDs, flatDirs
    flow = direction + fill + 8 + 24                                # + rain -> FAL, fillFAL, waterFilled
    spl = 24 + 20 * R + 2 + 16 + 24                                 # h, FAL, rain, graph, masks, cumED -> h, cumED, Eb
    hill = ids + edges + faces + 8 + 24 + 24                        # mesh rows, area, h, cumED, Eb -> h, cumED, Eb
    force = 8 + 8 + 8 + 16
    kind = case["kind"]
    if kind == "step":
        b = flow + spl + hill + force
        if case.get("sed"):
            b += flow + fill + 24 + 8 + 24 + 16                     # second accumulation; xyz, vSed, h, cumED
        if case.get("marine"):
            b += ids + edges + faces + 24 + 8 + 40
    elif kind == "adjoint":
        b = case["steps"] * 2 * (flow + spl + hill + force) + 5 * 8
    else:
        b = {"flow": flow, "fill": fill, "direction": direction, "spl": spl, "hillslope": hill}[kind]
    return {"bytes": float(b) * n, "flops": 0.0}


# ----------------------------------------------------------------------------
# the same results in plain 64-bit arithmetic
# ----------------------------------------------------------------------------
def exact(case, seed):
    if case["mesh"] == "ensemble" or case["kind"] not in ("direction", "hillslope") or case.get("down"):
        return None
    _, _, mesh, z, p = _inputs(case, seed)
    h = z + p["upsub"] * p["dt"]     # the forcing of the model's set-up
    if case["kind"] == "direction":
        # receiver ids are whole numbers; the masks read the fill, a graph search
        dist, wgt = _exact_direction(mesh, h, p["sealevel"], case["R"])
        return {"rcvID": None, "distRcv": dist, "wghtVal": wgt, "lsink": None, "seaID": None}
    x = _exact_diffusion(mesh, h, p)
    dz = x - h
    return {"h": x, "cumED": dz, "Eb": dz / p["dt"]}


def _exact_direction(mesh, h, sea, R):
    n = mesh.n
    W = int(mesh.nnb.max())
    ngb, L = mesh.ngb[:, :W], mesh.elgt[:, :W]
    ok = (ngb >= 0) & (L > 0.0) & (np.arange(W)[None, :] < mesh.nnb[:, None])
    d = h[:, None] - h[np.maximum(ngb, 0)]
    with np.errstate(divide="ignore", invalid="ignore"):
        e = np.maximum(np.where(ok, d / L, 0.0).max(axis=1), 0.0)
        fexp = np.where(e > 0, 5.0 * np.minimum(e, 1.0) + 1.1, 1.0)
        val = np.where(ok & (d > 0.0), np.power(np.maximum(d, 0.0), fexp[:, None]) / L, 0.0)
    val[h <= sea] = 0.0
    slp = val * (1.0 - 1.0e-15 * np.maximum(ngb, 0))
    slp[val <= 0.0] = -1.0
    kk = (slp > 0).sum(axis=1)
    # more candidates than R: by slope, descending; else in slot order
    key = np.where(slp > 0, np.where((kk > R)[:, None], -slp, np.arange(W)[None, :]), np.inf)
    top = np.argsort(key, axis=1, kind="stable")
    slots = np.argsort(np.where(slp > 0, np.arange(W)[None, :], W), axis=1, kind="stable")
    dist = np.zeros((R, n))
    wgt = np.zeros((R, n))
    tot = np.zeros(n)
    rows = np.arange(n)
    for o in range(min(R, W)):
        has = kk > o
        tot += np.where(has, slp[rows, top[:, o]], 0.0)
    for o in range(min(R, W)):
        has = kk > o
        # receiver o of a full set carries the edge length of the (o+1)-th last candidate slot
        sl = np.where(kk > R, slots[rows, np.maximum(kk - 1 - o, 0)], slots[:, o])
        dist[o] = np.where(has, L[rows, sl], 0.0)
        wgt[o] = np.where(has, slp[rows, top[:, o]] / np.where(tot > 0, tot, 1.0), 0.0)
    flat = mesh.outlet if mesh.flat else np.zeros(0, np.int64)
    dist[:, flat] = 0.0
    wgt[:, flat] = 0.0
    return dist, wgt


def _exact_diffusion(mesh, h, p):
    """(I + L) x = h: the change c = x - h solves (I + L) c = -L h, by Jacobi-preconditioned
    CG in the area-weighted inner product, in which the operator is symmetric."""
    W = int(mesh.nnb.max())
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEV)
    ngb = mesh.ngb[:, :W]
    j = torch.as_tensor(np.maximum(ngb, 0).astype(np.int64), device=DEV)
    ok = T((ngb >= 0) & (np.arange(W)[None, :] < mesh.nnb[:, None]) & (mesh.vdist[:, :W] > 0))
    area = T(mesh.farea)
    ht = T(h)
    kd = torch.where(ht <= p["sealevel"], p["Cdm"], p["Cda"]).to(torch.float64) * p["dt"]
    L = T(np.where(mesh.elgt[:, :W] > 0, mesh.elgt[:, :W], 1.0))
    v = ok * 0.5 * (kd[:, None] + kd[j]) / area[:, None] * T(mesh.vdist[:, :W]) / L
    free = torch.ones_like(ht)
    if mesh.flat:
        free[torch.as_tensor(mesh.outlet, device=DEV)] = 0.0
    v = v * free[:, None]

    def lap(x):
        return (v * (x[:, None] - x[j])).sum(dim=1)

    # symmetric form: weights A; fixed rows carry no change
    diag = 1.0 + v.sum(dim=1)
    b = -lap(ht)
    c = b / diag
    r = (b - c - lap(c)) * free
    zz = r / diag
    q = zz.clone()
    rz = (area * r * zz).sum()
    for _ in range(400):
        if float((area * r * r).sum()) <= 1e-34 * float((area * b * b).sum()):
            break
        Aq = (q + lap(q)) * free
        alpha = rz / (area * q * Aq).sum()
        c = c + alpha * q
        r = r - alpha * Aq
        zz = r / diag
        rn = (area * r * zz).sum()
        q = zz + (rn / rz) * q
        rz = rn
    return (ht + c).cpu().numpy()
