"""The basin levels of the fill against the oracle's priority flood.

Surfaces that stretch the contraction of the basin graph: noise (a basin every
few cells), a staircase of basins whose levels hang on a chain from one end to
the other, terraces of a few heights (equal passes, which join many basins in
one round), open borders, and a mesh with edges that only one end lists, which
takes the relaxation (there against the basin graph of the cells' own lists:
the oracle's flood follows the other direction of such an edge).  The levels
are heights of the surface: lFill is equal bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _surface(kind, coords, rng):
    x, y = coords[:, 0] / coords[:, 0].max(), coords[:, 1] / coords[:, 1].max()
    if kind == "noise":
        return rng.uniform(0.0, 100.0, len(x))
    if kind == "chain":
        return 50.0 + 30.0 * np.sin(90.0 * x) + 40.0 * x + 400.0 * np.abs(y - 0.5)
    if kind == "terraces":
        return np.floor(rng.uniform(0.0, 4.0, len(x))) * 5.0
    return 100.0 * (x - 0.5) ** 2 + rng.uniform(0.0, 3.0, len(x))


def _fill_by_lists(h, ngb, outlet):
    """Basins by steepest descent, minimax levels relaxed over the listed edges."""
    n = len(h)
    ids = np.arange(n)
    seed = np.zeros(n, bool)
    seed[outlet] = True
    z = h - h.min()
    par = ids.copy()
    best = z.copy()
    for s in range(ngb.shape[1]):
        j = np.where(ngb[:, s] >= 0, ngb[:, s], ids)
        better = ~seed & ((z[j] < best) | ((z[j] == best) & (j < par)))
        par, best = np.where(better, j, par), np.where(better, z[j], best)
    while not np.array_equal(par, par[par]):
        par = par[par]
    c, s = np.nonzero((ngb >= 0) & ~seed[par][:, None])
    j = ngb[c, s]
    u, v, w = par[c], par[j], np.maximum(z[c], z[j])
    L = np.where(seed, -np.inf, np.inf)
    while True:
        new = L.copy()
        np.minimum.at(new, u, np.maximum(w, L[v]))
        if np.array_equal(new, L):
            return np.where(z > 0.0, np.maximum(L[par], z), z) + h.min()
        L = new


@pytest.mark.parametrize("kind,n,jitter,bc", [("noise", 40, 0.25, "ffff"), ("noise", 30000, 0.25, "ffff"),
                                              ("chain", 12000, 0.25, "offf"), ("terraces", 8000, 0.25, "ffff"),
                                              ("bowl", 3000, 0.25, "oooo"), ("noise", 20000, 0.9, "ffff"),
                                              ("noise", 160000, 0.25, "ffff")])
def test_basin_levels_equal_the_priority_flood(kind, n, jitter, bc):
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from oracle.model import OracleModel

    coords, cells, _ = S.planar_hex_mesh(n, 1000.0 * np.sqrt(n), 9, jitter=jitter)
    z = _surface(kind, coords, np.random.default_rng(4))
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=1, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0, sealevel=-500.0,
             bc=bc, rain=np.ones(len(coords)), upsub=None)
    if jitter > 0.5:
        om = OracleModel(coords, cells, z, p, init_flow=False)
        expect, pits = _fill_by_lists(om.h, om.FVmesh_ngbID, om.outletIDs), None
    else:
        om = OracleModel(coords, cells, z, p)
        expect, pits = om.lFill, om.pitIDs
    gm = Model(coords=coords, cells=cells, elev=z, params=p, mesh=FVMesh(coords, cells, bc, device="cuda:0"),
               device="cuda:0")
    for _ in range(2):
        gm.flowAccumulation()
        assert np.array_equal(gm.lFill.cpu().numpy(), expect)
        assert pits is None or np.array_equal(gm.pitIDs.cpu().numpy(), pits)
    gm.destroy()


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_an_input_that_is_not_finite_leaves_the_fill_as_it_was(bad):
    """The check is read with the fill's sizes, after its kernels have run."""
    import torch
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model

    coords, cells, z, rain, up, p = S.planar_config(n=3000, side=30.0e3, seed=3)
    m = Model(coords=coords, cells=cells, elev=z, params=dict(p, rain=rain, upsub=up), mesh=FVMesh(coords, cells, p["bc"]),
              device="cuda:0")
    m.flowAccumulation()
    keep = [x.clone() for x in (m.lFill, m.pitIDs, m.seaID, m.FAL)]
    h0 = m.hGlobal.clone()
    m.hGlobal[1234] = bad
    with pytest.raises(Exception, match="non-finite"):
        m.flowAccumulation()
    assert torch.equal(m.lFill, keep[0]) and torch.equal(m.pitIDs, keep[1]) and torch.equal(m.seaID, keep[2])
    m.hGlobal.copy_(h0)
    m.flowAccumulation()
    assert all(torch.equal(a, b) for a, b in zip((m.lFill, m.pitIDs, m.seaID, m.FAL), keep))
    m.destroy()
