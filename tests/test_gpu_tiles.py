"""The tile dataflow sweeps against the oracle's sequential solves.

Sizes around the tile limits: one tile, a few tiles, a tile of one vertex more
than the smallest, consecutive-id tiles (a sphere along a Morton curve) and
grown ones (lattice rows, shuffled ids), records of 6, 8 and 12 slots, whole
records and the hot part only, and the meshes that take the ordered sweep: one
just above the largest tile, and one with vertices of more than twelve
neighbours, of which the mesh keeps twelve (an edge that only its donor lists
carries no flow, and erosion still follows it).  The surface is a tilted plane with a relief too weak
for a depression, so the drainage area is the one flow solve.  Both sides add
the donors in ascending id and the receivers in slot order, in the same IEEE
operations: the solutions are equal bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(kind, n, seed):
    from gospl_b200 import synthetic as S
    rng = np.random.default_rng(seed)
    if kind == "sphere":
        coords, cells = S.icosphere(n)
        return S.renumber(coords, cells, S.morton_order(coords))
    side = 1000.0 * np.sqrt(n)
    coords, cells, _ = S.planar_hex_mesh(n, side, seed, jitter=0.6 if kind == "wide" else 0.25)
    if kind == "shuffled":
        coords, cells = S.renumber(coords, cells, rng.permutation(len(coords)))
    return coords, cells


@pytest.mark.parametrize("kind,n,R", [("rows", 60, 3), ("rows", 430, 3), ("rows", 480, 1), ("shuffled", 3000, 3),
                                      ("wide", 4000, 3), ("wide", 2500, 8), ("sphere", 5, 3), ("sphere", 6, 8),
                                      ("rows", 160647, 3), ("shuffled", 260000, 3), ("rows", 480000, 3)])
def test_flow_and_spl_sweeps_equal_the_sequential_solves(kind, n, R):
    import torch
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from oracle import fortran as F

    coords, cells = _mesh(kind, n, 5)
    rng = np.random.default_rng(7)
    span = coords.max(axis=0) - coords.min(axis=0)
    z = 50.0 + 400.0 * (coords[:, 0] - coords[:, 0].min()) / span[0] + 37.0 * coords[:, 1] / span[1]
    if kind == "sphere":
        z = z - 120.0     # part of the sphere is sea
    fv = FVMesh(coords, cells, "ffff", device="cuda:0")
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=R, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0,
             sealevel=0.0 if kind == "sphere" else -100.0, bc="ffff", rain=rng.uniform(0.5, 1.5, fv.n), upsub=None)
    m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0")
    rcv = np.ascontiguousarray(m.rcvIDi.cpu().numpy())
    wgt = np.ascontiguousarray(m.wghtVali.cpu().numpy())
    sea = m.seaID.cpu().numpy()
    if int((m.pitIDs > -1).sum()) == 0:
        b = np.where(sea, 0.0, m.bL.cpu().numpy())
        listed = (fv.ngb[rcv] == np.arange(fv.n)[:, None, None]).any(axis=2)
        q, left = F.flow_solve(rcv, np.where(listed, wgt, 0.0), b)
        assert left == 0
        assert np.array_equal(m.FAL.cpu().numpy(), q)
    else:
        assert kind == "wide" or kind == "sphere"    # uneven meshes may hold a cell below its neighbours
    # stream power over the same graph, in the coefficients' own definition
    fal = m.FAL.cpu().numpy()
    h0 = m.hGlobal.cpu().numpy().copy()
    dist = m.distRcvi.cpu().numpy()
    kbr = np.where(sea, 0.0, 3e-6 * (1000.0 * np.sqrt(fal)))
    c = np.zeros_like(wgt)
    for k in range(R):
        dh = h0 - h0[rcv[:, k]]
        lim = np.where(dh != 0.0, dh / np.where(dh != 0.0, dh + 1.0e-2, 1.0), 0.0)
        data = np.where(dist[:, k] != 0.0, (kbr * lim) / np.where(dist[:, k] != 0.0, dist[:, k], 1.0), 0.0)
        c[:, k] = np.where(rcv[:, k] == np.arange(fv.n), 0.0, data * np.where(sea, 0.0, wgt[:, k]))
    s, left = F.spl_solve(rcv, np.ascontiguousarray(c), h0)
    assert left == 0
    m.erodepSPL()
    torch.cuda.synchronize()
    E = (s - h0) / 1000.0
    if fv.flat:
        E[fv.outlet] = 0.0
    E[m.lsink.cpu().numpy()] = 0.0
    assert np.array_equal(m.hGlobal.cpu().numpy(), h0 + E * 1000.0)
    m.destroy()


@pytest.mark.parametrize("level,R,sed", [(7, 3, True), (8, 3, True), (8, 1, False), (8, 6, False)])
def test_cascade_on_tiles_equals_the_ordered_sweeps(level, R, sed):
    """Above the size whose records fit shared memory the cascade's flow alone is
    solved on tiles; a model that records for the adjoint takes the ordered
    sweeps there.  Donors are added in ascending id on both: equal bit for bit
    (below that size both models run the same tiles)."""
    import torch
    from gospl_b200 import _lib
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    coords, cells, z, rain, up, p = S.sphere_config(level=level, lmax=128)
    p = dict(p, rain=rain, upsub=up, flowDir=R, nodep=not sed, nlPitVolume=float("inf"))
    fv = FVMesh(coords, cells, p["bc"], device="cuda:0")
    out = []
    for recorded in (False, True):
        m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0")
        if recorded:
            _lib.check(_lib.load().gs_plan_record(m._plan, 1))
        m.flowAccumulation()
        assert m.stats["flow"]["cascade_solves"] > 0
        if sed:
            m.erodepSPL()
            m.flowAccumulation()
            m.sedChange()
            assert m.stats["sed"]["cascade_solves"] > 0
        out.append([x.clone() for x in (m.FAL, m.fillFAL, m.waterFilled, m.hGlobal)])
        m.destroy()
    assert all(torch.equal(a, b) for a, b in zip(*out))
