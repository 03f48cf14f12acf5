"""The cooperative CG's thread groups and slot batches, against the operator of
the oracle.

Sizes: fewer rows than one thread group, a number of rows just above the rows
of all groups of a small launch, several rows to a thread, and rows with more
neighbours than one batch of slots holds; erosion coefficients that differ on
land and in the sea, flat and open borders.  The solver stops at a relative
residual of 1e-13 of its own recurrence; the true residual of the returned
surface adds the rounding of the matrix products, a few units in the last
place of (1 + 2 L) per row and iteration.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("n,jitter,bc", [(60, 0.25, "ffff"), (3000, 0.25, "offo"), (9000, 0.45, "ffff"),
                                         (152000, 0.25, "ffff"), (310000, 0.35, "ffff")])
def test_diffusion_leaves_the_stated_residual(n, jitter, bc):
    import torch
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from oracle.model import OracleModel

    coords, cells, _ = S.planar_hex_mesh(n, 1000.0 * np.sqrt(n), 11, jitter=jitter)
    rng = np.random.default_rng(3)
    z = rng.uniform(-200.0, 600.0, len(coords))
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=1, K=3e-6, d=0.0, m=0.5, Cda=300.0, Cdm=900.0, sealevel=0.0,
             bc=bc, rain=np.ones(len(coords)), upsub=None)
    fv = FVMesh(coords, cells, bc, device="cuda:0")
    m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0", init_flow=False)
    h0 = m.hGlobal.cpu().numpy().copy()
    om = OracleModel(coords, cells, z, p, init_flow=False)
    assert np.array_equal(om.h, h0)
    if jitter > 0.4:
        assert int((om.FVmesh_ngbID >= 0).sum(axis=1).max()) > 6
    A = om.diffusion_matrix(np.where(h0 <= 0.0, 900.0, 300.0) * 1000.0).tocsr()
    fixed = (np.asarray(abs(A).sum(axis=1)).ravel() == 1.0) & (A.diagonal() == 1.0)
    area = om.larea
    b = area * (h0 - A[:, fixed] @ h0[fixed])
    bnorm = np.linalg.norm(b[~fixed])
    for again in (False, True):      # the second solve starts from the first one's change: the solution
        m.hGlobal.copy_(torch.as_tensor(h0))
        m.getHillslope()
        x = m.hGlobal.cpu().numpy()
        its = m.stats["hillslope"]["cg_iters"]
        assert its > 0 or again
        assert np.array_equal(x[fixed], h0[fixed])
        r = area * (A @ x - h0)
        tol = 1e-13 + 8.0 * (its + 1) * EPS * (2.0 * A.diagonal().max() - 1.0)
        assert np.linalg.norm(r[~fixed]) <= tol * bnorm
    m.destroy()
