"""Tile sweeps whose vertices mostly pass through the ready queue.

On a plane tilted across the rows of a lattice whole fronts become ready
together and every vertex has several successors, so that most are queued for
another thread, which has to see the values of all their predecessors.  Many
passes, each equal bit for bit to the oracle's sequential solve.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,tilt", [(2000, 3, (0.0, 1.0)), (90000, 3, (0.0, 1.0)), (90000, 6, (0.3, 1.0)),
                                      (300000, 3, (0.05, 1.0))])
def test_queued_vertices_see_all_their_predecessors(n, R, tilt):
    import torch
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from oracle import fortran as F
    side = 1000.0 * np.sqrt(n)
    coords, cells, _ = S.planar_hex_mesh(n, side, 5, jitter=0.02)
    z = 50.0 + 400.0 * (tilt[0] * coords[:, 0] + tilt[1] * coords[:, 1]) / side
    rng = np.random.default_rng(11)
    fv = FVMesh(coords, cells, "ffff", device="cuda:0")
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=R, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0, sealevel=-100.0,
             bc="ffff", rain=rng.uniform(0.5, 1.5, fv.n), upsub=None)
    m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0")
    assert int((m.pitIDs > -1).sum()) == 0
    rcv = np.ascontiguousarray(m.rcvIDi.cpu().numpy())
    wgt = np.ascontiguousarray(m.wghtVali.cpu().numpy())
    q, left = F.flow_solve(rcv, wgt, m.bL.cpu().numpy())
    assert left == 0
    want = torch.as_tensor(q, device=m.dev)
    for _ in range(40):
        m.FAL.zero_()
        m.flowAccumulation()
        assert torch.equal(m.FAL, want)
    m.destroy()
