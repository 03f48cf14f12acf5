"""Flat distances on meshes with edges that only one of their ends lists.

A vertex keeps twelve of its neighbours; here some have twenty, and eight of
those list a vertex that does not list them.  The definition walks from a
reached cell along that cell's own list, so the direction of such an edge
matters.  Lakes of 22 cells and of about 200 lie around such vertices; the
flat directions have to be the definition's, also from the tiled search.
"""
import numpy as np
import pytest

import definitions as D


def fan_mesh(n, seed, centres, degree=20):
    """Jittered lattice in which each centre (in units of the side) is joined to
    `degree` vertices on a circle of 2.4 spacings."""
    from scipy.spatial import Delaunay
    from gospl_b200 import synthetic as S
    side = 537.0 * np.sqrt(n * np.sqrt(3) / 2)
    xy = S.planar_hex_mesh(n, side, seed)[0][:, :2]
    r = 2.4 * 537.0
    mids = np.asarray(centres) * side
    for c in mids:
        xy = xy[np.hypot(*(xy - c).T) > r + 0.5 * 537.0]
        t = 2.0 * np.pi * np.arange(degree) / degree
        xy = np.concatenate([xy, c[None], c + r * np.stack([np.cos(t), np.sin(t)], 1)])
    tri = Delaunay(xy).simplices.astype(np.int32)
    coords = np.concatenate([xy, np.zeros((len(xy), 1))], axis=1)
    a, b, c = (xy[tri[:, k]] for k in range(3))
    turn = (b - a)[:, 0] * (c - a)[:, 1] - (b - a)[:, 1] * (c - a)[:, 0] < 0
    tri[turn] = tri[turn][:, [0, 2, 1]]
    return coords, tri, mids


def lakes(seed):
    """(mesh, elevation, the centres' ids)"""
    from gospl_b200.mesh import FVMesh
    coords, cells, mids = fan_mesh(3000, seed, [(0.25, 0.3), (0.7, 0.65)])
    mesh = FVMesh(coords, cells, "ffff")
    z = 100.0 + 1.0e-3 * coords[:, 0] + 3.0e-4 * coords[:, 1]
    ids = []
    for c, r in zip(mids, (3.0, 8.0)):
        d = np.hypot(coords[:, 0] - c[0] - 0.8 * 537.0, coords[:, 1] - c[1]) / 537.0
        z = np.where(d < r, 50.0 + d / r, z)
        ids.append(int(np.argmin(np.hypot(coords[:, 0] - c[0], coords[:, 1] - c[1]))))
    z[mesh.outlet] = 0.0
    return mesh, z, ids


@pytest.mark.parametrize("seed", [3, 4])
def test_the_meshes_have_one_sided_edges(seed):
    mesh, _, ids = lakes(seed)
    i, c = D._edges(mesh.ngb)
    pairs = set(zip(i.tolist(), c.tolist()))
    one = [(a, b) for a, b in pairs if (b, a) not in pairs]
    assert len(one) == 16 and {b for _, b in one} == set(ids)


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [3, 4])
@pytest.mark.parametrize("sed", [False, True])
def test_flat_directions_follow_the_listed_edges(seed, sed):
    from gospl_b200 import _lib
    from gospl_b200.model import Model
    mesh, z, ids = lakes(seed)
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=3, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0, sealevel=-100.0,
             oFill=-6000.0, bc="ffff", rain=np.ones(mesh.n), upsub=None)
    m = Model(elev=z, params=p, mesh=mesh, coords=mesh.coords, cells=mesh.cells, device="cuda:0", init_flow=False)
    for window in (0, 3):
        _lib.check(_lib.load().gs_plan_tune(m._plan, 7, window))
        m.fillElevation(sed=sed)
        lf, pit, dirs = (getattr(m, k).cpu().numpy() for k in ("lFill", "pitIDs", "flatDirs"))
        counts = np.bincount(pit[pit > 0])
        assert 20 < counts[pit[ids[0]]] <= 32 and counts[pit[ids[1]]] > 100
        info = m.pit_tables()[1].cpu().numpy()
        spills = np.unique(info[(info[:, 1] == 0) & (info[:, 0] >= 0), 0])
        pd = D.flat_distance(spills, pit.astype(np.int64), lf, mesh.ngb)
        want = D.flat_dirs(pd, pit.astype(np.int64), lf, mesh.ngb, spills, -100.0)
        assert np.array_equal(dirs, want), window
    m.destroy()
