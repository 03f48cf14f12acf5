"""Detachment-transport erosion (GMRES over ordered sweeps) against the oracle's
sparse solve, at sizes around one block of the orthogonalisation, a few blocks,
and several elements to a thread.

Both solve (I + B) x = a, the oracle by LU and the GPU to a relative residual of
1e-13; the stage tests of the same system allow 1e-11 of the elevation scale.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,G", [(60, 1.0), (900, 0.5), (1100, 1.0), (30000, 1.5), (170000, 1.0)])
def test_transport_matches_the_sparse_solve(n, G):
    import torch
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    from oracle.model import OracleModel
    from test_gpu_parity import _np, _resync_flow

    coords, cells, _ = S.planar_hex_mesh(n, 1000.0 * np.sqrt(n), 6)
    rng = np.random.default_rng(8)
    z = 50.0 + 300.0 * coords[:, 0] / coords[:, 0].max() + rng.uniform(0.0, 4.0, len(coords))
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=3, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0, G=G, sealevel=-100.0,
             bc="ffff", rain=np.ones(len(coords)), upsub=None)
    om = OracleModel(coords, cells, z, p)
    gm = Model(coords=coords, cells=cells, elev=z, params=p, mesh=FVMesh(coords, cells, "ffff"), device="cuda:0")
    assert om.fDepa > 0.0
    _resync_flow(gm, om)
    om.erodepSPL()
    for _ in range(2):
        gm.hGlobal.copy_(torch.as_tensor(z))
        gm.erodepSPL()
        assert np.abs(_np(gm.hGlobal) - om.h).max() <= 1e-11 * np.abs(om.h).max()
    assert np.abs(om.h - z).max() > 0.0
    gm.destroy()
