"""Receivers of meshes beyond two waves of the unrolled kernels, against their
definition: the loop over the slots for 8 and 12 slots and for four directions on
spheres, and the form that keeps every candidate.  Receivers and distances are
equal, weights to 1e-15, the masks follow.
"""
import numpy as np
import pytest

import definitions as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,Rs", [("lattice", 200000, (1, 3, 4, 8, 10)), ("wide", 160000, (2, 4, 12)),
                                       ("sphere", 8, (3, 4, 6))])
def test_large_meshes_match_the_definition(kind, n, Rs):
    import torch
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    rng = np.random.default_rng(5)
    if kind == "sphere":
        coords, cells = S.icosphere(n)
        coords, cells = S.renumber(coords, cells, S.morton_order(coords))
    else:
        coords, cells, _ = S.planar_hex_mesh(n, 700.0 * np.sqrt(n), 3, jitter=0.55 if kind == "wide" else 0.25)
    fv = FVMesh(coords, cells, "ffff", device="cuda:0")
    assert int(fv.nnb.max()) == dict(lattice=8, wide=12, sphere=6)[kind]
    z = rng.uniform(0.0, 40.0, fv.n)
    land = rng.permutation(fv.n) < fv.n // 2
    z[land] += 300.0 * np.abs(np.sin(1e-5 * coords[land, 0]))
    ngb, elgt = np.pad(fv.ngb, ((0, 0), (0, 1)), constant_values=-1), np.pad(fv.elgt, ((0, 0), (0, 1)))
    for R in Rs:
        p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=R, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0, sealevel=2.0,
                 bc="ffff", rain=np.ones(fv.n), upsub=None)
        m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0", init_flow=False)
        h = m.hGlobal.clone()
        m.fillElevation()
        m._buildFlowDirection(h, down=False)
        torch.cuda.synchronize()
        rcv, dist, wgt, ties, slp = D.mfd_receivers(z, ngb, elgt, 2.0, R)
        if fv.flat:
            rcv[fv.outlet], dist[fv.outlet], wgt[fv.outlet] = fv.outlet[:, None], 0.0, 0.0
        assert D.near_ties(slp, R) == 0 and not ties.any()
        got = [x.cpu().numpy() for x in (m.rcvID, m.distRcv, m.wghtVal)]
        assert np.array_equal(got[0], rcv), R
        assert np.array_equal(got[1], dist), R
        assert np.abs(got[2] - wgt).max() <= 1e-15, R
        sea = m.lFill.cpu().numpy() <= 2.0
        out = np.zeros(fv.n, bool)
        out[fv.outlet] = fv.flat
        assert np.array_equal(m.seaID.cpu().numpy(), sea)
        assert np.array_equal(m.lsink.cpu().numpy(), (got[2].sum(axis=1) == 0.0) & ~out & ~sea)
        m.destroy()
