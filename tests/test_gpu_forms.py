"""Tile sweeps against solves that share no code with them.

The drainage area on surfaces that cannot hold a pit (heights grow with the hop
distance from the sea or the border), on spheres, whose consecutive ids are the
tiles, and on lattices with records of 8 and 12 slots: equal bit for bit to the
oracle's sequential solve.  Whole steps with deposition and its lake cascades
against the same mesh with one edge listed twice, without length: that mesh
takes the ordered sweeps, the relaxed basin levels and the flat search over all
depressions, and every result is the same, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hops(ngb, start):
    from scipy.sparse import coo_matrix, csgraph
    n, w = ngb.shape
    i, c = np.repeat(np.arange(n), w), ngb.ravel()
    i, c = i[c >= 0], c[c >= 0]
    rows = np.concatenate([i, np.full(len(start), n)])
    cols = np.concatenate([c, start])
    g = coo_matrix((np.ones(len(rows)), (rows, cols)), shape=(n + 1, n + 1)).tocsr()
    return csgraph.shortest_path(g, unweighted=True, indices=n)[:n] - 1.0


@pytest.mark.parametrize("kind,n,R,slots", [("sphere", 5, 3, 6), ("sphere", 7, 6, 6), ("lattice", 30000, 3, 8),
                                            ("wide", 4000, 3, 12), ("wide", 4000, 8, 12)])
def test_flow_without_pits_equals_the_sequential_solve(kind, n, R, slots):
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from oracle import fortran as F
    rng = np.random.default_rng(7)
    if kind == "sphere":
        coords, cells = S.icosphere(n)
        coords, cells = S.renumber(coords, cells, S.morton_order(coords))
    else:
        coords, cells, _ = S.planar_hex_mesh(n, 1000.0 * np.sqrt(n), 5, jitter=0.6 if kind == "wide" else 0.25)
    fv = FVMesh(coords, cells, "ffff")
    assert slots - 3 < fv.nnb.max() <= slots
    start = np.where(coords[:, 2] < -0.6 * np.abs(coords[:, 2]).max())[0] if kind == "sphere" else fv.outlet
    d = _hops(fv.ngb, start)
    z = np.where(d > 0, 10.0 * d + rng.uniform(0.0, 6.0, fv.n), -50.0 if kind == "sphere" else 0.0)
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=R, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0,
             sealevel=0.0 if kind == "sphere" else -100.0, bc="ffff", rain=rng.uniform(0.5, 1.5, fv.n), upsub=None)
    m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0")
    assert int((m.pitIDs > -1).sum()) == 0
    b = np.where(m.seaID.cpu().numpy(), 0.0, m.bL.cpu().numpy())
    q, left = F.flow_solve(np.ascontiguousarray(m.rcvIDi.cpu().numpy()), np.ascontiguousarray(m.wghtVali.cpu().numpy()),
                           b)
    assert left == 0
    assert np.array_equal(m.FAL.cpu().numpy(), q)
    m.destroy()


@pytest.mark.parametrize("kind,n,R,marine", [("sphere", 7, 3, True), ("sphere", 6, 6, False), ("wide", 4000, 3, False)])
def test_a_step_on_tiles_equals_a_step_in_order(kind, n, R, marine):
    import torch
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    if kind == "sphere":
        coords, cells, z, rain, up, p = S.sphere_config(level=n, lmax=64)
    else:
        side = 1000.0 * np.sqrt(n)
        coords, cells, onb = S.planar_hex_mesh(n, side, 5, jitter=0.6)
        z = S.rescale(S.fractal_field(coords[:, :2], side, 6), 0.0, 100.0)
        z[onb] = 0.0
        rain, up = np.ones(len(z)), np.full(len(z), 1e-3)
        p = dict(dt=1000.0, tStart=0.0, tEnd=1e30, K=3e-6, d=0.0, m=0.5, Cda=0.1, Cdm=0.1, sealevel=-100.0,
                 oFill=-6000.0, bc="ffff")
    p = dict(p, rain=rain, upsub=up, flowDir=R, nodep=False, seadepo=marine, marineSolver="picard")
    plain = FVMesh(coords, cells, p["bc"])
    arrays = {k: getattr(plain, k).copy() for k in ("nnb", "ngb", "elgt", "vdist", "farea", "larea")}
    v = int(np.argmin(plain.nnb))
    k = plain.nnb[v]
    arrays["ngb"][v, k], arrays["elgt"][v, k], arrays["vdist"][v, k] = plain.ngb[v, 0], 0.0, 0.0
    arrays["nnb"][v] = k + 1
    twice = FVMesh.from_arrays(dict(arrays, outlet=plain.outlet, open_nodes=plain.open_nodes, flat=plain.flat,
                                    coords=coords, cells=cells))
    out = []
    for fv in (plain, twice):
        m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0")
        for _ in range(2):
            m.step()
        assert m.stats["flow"]["cascade_solves"] > 0
        assert kind != "sphere" or m.stats["sed"]["cascade_solves"] > 0   # (the lattice's lakes hold their sediment)
        out.append([getattr(m, q).clone() for q in ("FAL", "fillFAL", "waterFilled", "vSed", "lFill", "pitIDs",
                                                    "flatDirs", "hGlobal", "cumED")])
        m.destroy()
    assert all(torch.equal(a, b) for a, b in zip(*out))
