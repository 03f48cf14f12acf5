"""Transport-limited erosion (G > 0) in the precision form, on a mesh that has
tiles and on one with vertices of too many neighbours, which has none.

From the same drainage area the coupled system is the same FP64 system in
either precision, and its sweeps add in the same order on tiles and in vertex
order: equal bit for bit.  A whole step agrees as tests/test_precision.py asks
of the detachment-limited one (1e-8 for a refinement to 1e-10).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kind):
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    if kind == "sphere":
        c, f, z, rain, up, p = S.sphere_config(level=5, seed=42, lmax=32)
    else:
        c, f, z, rain, up, p = S.planar_config(n=4000, side=50.0e3, seed=41)
    if kind == "wide":
        c, f, onb = S.planar_hex_mesh(2500, 50.0e3, 5, jitter=0.6)
        z = S.rescale(S.fractal_field(c[:, :2], 50.0e3, 6), 0.0, 100.0)
        z[onb] = 0.0
        rain, up = np.ones(len(z)), np.full(len(z), 1e-3)
    p = dict(p, rain=rain, upsub=up, tEnd=1e30)
    return c, f, z, p, FVMesh(c, f, p["bc"])


@pytest.mark.parametrize("kind,G", [("planar", 1.0), ("planar", 0.3), ("sphere", 1.0), ("wide", 1.0)])
def test_transport_limited_erosion_in_fp32(kind, G):
    import torch
    from gospl_b200.model import Model
    c, f, z, p, mesh = _case(kind)
    m64, m32 = (Model(coords=c, cells=f, elev=z, params=dict(p, G=G), mesh=mesh, device="cuda:0", precision=bits,
                      refine_tol=1e-10) for bits in (64, 32))
    m32.hGlobal.copy_(m64.hGlobal)
    h0 = m64.hGlobal.clone()
    for m in (m64, m32):
        m.flowAccumulation()
    fal = m64.FAL.clone()
    m64.FAL.copy_(m32.FAL)
    for m in (m64, m32):
        m.erodepSPL()
    assert not torch.equal(m32.hGlobal, h0)
    assert torch.equal(m32.hGlobal, m64.hGlobal)
    m64.FAL.copy_(fal)
    for m in (m64, m32):
        m.hGlobal.copy_(h0)
        m.step()
    assert torch.equal(m32.rcv_i, m64.rcv_i)
    for name in ("FAL", "hGlobal"):
        a, b = getattr(m32, name), getattr(m64, name)
        assert float((a - b).abs().max()) <= 1e-8 * max(float(b.abs().max()), 1.0), name
    m64.destroy()
    m32.destroy()
