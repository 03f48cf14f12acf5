"""Flow directions of the unfilled surface in one kernel, against the oracle:
receiver counts below, at and above the mesh's neighbour slots (ranked in
registers, ranked by the general form, every candidate kept), six, eight and
twelve slots, flat borders whose outlets drain to themselves, and sea.

Receivers, distances and masks are equal; weights to 1e-12, the bound of the
stage tests (pow differs by units in the last place, which is why the heights
are continuous: slopes equal to the last place would rank by it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,R", [("sphere", 1), ("sphere", 4), ("sphere", 5), ("sphere", 6), ("sphere", 8),
                                    ("rows", 3), ("rows", 7), ("rows", 12), ("wide", 2), ("wide", 6), ("wide", 12)])
def test_directions_match_the_oracle(kind, R):
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from oracle.model import OracleModel

    rng = np.random.default_rng(12)
    if kind == "sphere":
        coords, cells = S.icosphere(5)
        bc, sl = "oooo", 3.0
    else:
        coords, cells, _ = S.planar_hex_mesh(5000, 70.0e3, 4, jitter=0.7 if kind == "wide" else 0.25)
        bc, sl = "ffff", 2.0
    z = rng.uniform(0.0, 40.0, len(coords))
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=R, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0, sealevel=sl, bc=bc,
             rain=np.ones(len(coords)), upsub=None)
    fv = FVMesh(coords, cells, bc, device="cuda:0")
    mesh = dict(coords=coords, cells=cells, nb=fv.n, flat=fv.flat, nnb=fv.nnb, ngb=fv.ngb, elgt=fv.elgt,
                vdist=fv.vdist, farea=fv.farea, larea=fv.larea, maxarea=fv.maxarea, outlet=fv.outlet,
                open_nodes=fv.open_nodes, borders=fv.outlet)
    om = OracleModel(coords, cells, z, p, mesh=mesh)
    gm = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0")
    rcv = gm.rcvIDi.cpu().numpy()
    assert rcv.shape == om.rcvIDi.shape
    assert int((rcv != om.rcvIDi).sum()) == 0
    assert np.array_equal(gm.distRcvi.cpu().numpy(), om.distRcvi)
    assert np.abs(gm.wghtVali.cpu().numpy() - om.wghtVali).max() <= 1e-12
    sea = np.zeros(om.lpoints, bool)
    sea[om.seaID] = True
    assert np.array_equal(gm.seaID.cpu().numpy(), sea)
    gm.destroy()
