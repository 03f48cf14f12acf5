"""A plan after a call that stopped on an error.

Every stage waits for its stream, so a capturing stream refuses it, after some
of its kernels were recorded and never ran.  The next calls on the plan give
what a new plan gives, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4000, 60000])
@pytest.mark.parametrize("stage", ["erodepSPL", "flowAccumulation"])
def test_a_call_refused_by_a_capture_leaves_nothing_behind(n, stage):
    import torch
    from gospl_b200 import _lib
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    side = 1000.0 * np.sqrt(n)
    coords, cells, onb = S.planar_hex_mesh(n, side, 23)
    fv = FVMesh(coords, cells, "ffff")
    zs = []
    for seed in (24, 25):
        z = S.rescale(S.fractal_field(coords[:, :2], side, seed), 0.0, 100.0)
        z[onb] = 0.0
        zs.append(z)
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e30, flowDir=3, K=3e-6, d=0.0, m=0.5, Cda=0.1, Cdm=0.1, sealevel=-100.0,
             oFill=-6000.0, bc="ffff", rain=np.ones(fv.n), upsub=None)
    make = lambda z: Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0", init_flow=False)

    def passes(m):
        m.flowAccumulation()
        m.erodepSPL()
        return [getattr(m, k).clone() for k in ("FAL", "waterFilled", "hGlobal")]

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        fresh = make(zs[1])
        want = passes(fresh)
        m = make(zs[0])
        h1 = fresh.hGlobal.clone()
        h1.copy_(torch.as_tensor(zs[1]))
        passes(m)
    torch.cuda.synchronize()
    with pytest.raises(Exception):
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream):
            with pytest.raises(_lib.GsError):
                getattr(m, stage)()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        try:
            m.flowAccumulation()     # may report the runtime's last error once more
        except _lib.GsError:
            pass
        m.hGlobal.copy_(h1)
        got = passes(m)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    m.destroy()
    fresh.destroy()
