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


@pytest.mark.parametrize("n,nsub,npic", [(80, 1, 1), (700, 3, 1), (20000, 2, 3)])
def test_lagged_diffusivity_solves_match_the_oracle(n, nsub, npic):
    """seaChange's sub-steps and Picard iterations in one launch, over a part of
    one thread group, a few groups, and several rows to a thread.  The oracle
    solves the systems exactly, the GPU to a relative residual of 1e-13: the
    elevations agree to 1e-11 of their scale, as the marine stages do."""
    import torch
    from gospl_b200 import synthetic as S
    from oracle.model import OracleModel
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from test_gpu_parity import _np, _resync, _resync_flow

    coords, cells, _ = S.planar_hex_mesh(n, 700.0 * np.sqrt(n), 5)
    x = coords[:, 0] / coords[:, 0].max()
    z = 60.0 * (x - 0.75) + np.random.default_rng(2).uniform(0.0, 0.5, len(coords))
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=3, K=2e-6, d=0.0, m=0.5, Cda=0.1, Cdm=0.1, sealevel=0.0,
             bc="ffff", nodep=False, marineSolver="picard", picardSub=nsub, picardIts=npic, seadepo=True,
             rain=np.ones(len(coords)), upsub=None)
    om = OracleModel(coords, cells, z, p)
    gm = Model(coords=coords, cells=cells, elev=z, params=p, mesh=FVMesh(coords, cells, "ffff"), device="cuda:0")
    for m in (om, gm):
        m.flowAccumulation()
    _resync_flow(gm, om)
    for stage in ("erodepSPL", "flowAccumulation", "sedChange", "seaChange"):
        if stage == "seaChange":
            gm.vSed.copy_(torch.as_tensor(om.vSed))
            before = om.h.copy()
        for m in (om, gm):
            getattr(m, stage)()
        if stage != "seaChange":
            _resync(gm, om)
        if stage == "flowAccumulation":
            _resync_flow(gm, om)
    assert np.abs(om.h - before).max() > 0.0, "the stage must deposit"
    assert gm.stats["sea"]["marine_passes"] == om.marine_passes
    assert np.abs(_np(gm.hGlobal) - om.h).max() <= 1e-11 * np.abs(om.h).max()
    gm.destroy()
