"""Meshes whose rows list a neighbour twice.

The second listing has no length and no face, so it carries nothing: every
stage gives what it gives on the mesh without it, bit for bit, and no sweep
waits for a donor that was counted twice.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("both", [False, True])
def test_a_second_listing_without_length_changes_nothing(both):
    import torch
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    n, side = 4000, 60.0e3
    coords, cells, onb = S.planar_hex_mesh(n, side, 17)
    z = S.rescale(S.fractal_field(coords[:, :2], side, 18), 0.0, 100.0)
    z[onb] = 0.0
    plain = FVMesh(coords, cells, "ffff")
    arrays = {k: getattr(plain, k).copy() for k in ("nnb", "ngb", "elgt", "vdist", "farea", "larea")}
    rng = np.random.default_rng(19)
    for a in rng.choice(plain.n, 300, replace=False):
        b = int(plain.ngb[a, rng.integers(plain.nnb[a])])
        for i, j in ((a, b), (b, a))[:2 if both else 1]:
            k = arrays["nnb"][i]
            if k < 12:
                arrays["ngb"][i, k], arrays["elgt"][i, k], arrays["vdist"][i, k] = j, 0.0, 0.0
                arrays["nnb"][i] = k + 1
    mesh = FVMesh.from_arrays(dict(arrays, outlet=plain.outlet, open_nodes=plain.open_nodes, flat=plain.flat,
                                   coords=coords, cells=cells))
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e30, flowDir=3, K=3e-6, d=0.0, m=0.5, Cda=0.1, Cdm=0.1, sealevel=-100.0,
             oFill=-6000.0, bc="ffff", rain=rng.uniform(0.5, 1.5, plain.n), upsub=None)
    out = []
    for fv in (plain, mesh):
        m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0")
        m.step()
        out.append([getattr(m, k).clone() for k in ("FAL", "lFill", "pitIDs", "flatDirs", "rcv_i", "wgt_i", "hGlobal")])
        m.destroy()
    assert int((out[0][2] > -1).sum()) > 0
    assert all(torch.equal(a, b) for a, b in zip(*out))
