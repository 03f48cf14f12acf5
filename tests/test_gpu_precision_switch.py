"""The precision set between two stages of one plan.

A flow accumulation leaves its graph as tile records (FP64) or as a vertex
order (FP32); erosion and deposition after a switch solve over the form that is
there.  The tile sweeps and the ordered FP64 sweeps add in the same order, so
every result equals, bit for bit, that of a plan that stayed in FP64 and was
given the same drainage area.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _models(count, **more):
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    c, f, z, rain, up, p = S.planar_config(n=3000, side=50.0e3, seed=43)
    p = dict(p, rain=rain, upsub=up, tEnd=1e30, nodep=False, **more)
    mesh = FVMesh(c, f, p["bc"])
    return [Model(coords=c, cells=f, elev=z, params=p, mesh=mesh, device="cuda:0", init_flow=False)
            for _ in range(count)]


def _precision(m, bits):
    from gospl_b200 import _lib
    _lib.check(_lib.load().gs_plan_set_precision(m._plan, bits, 1e-10))


# the precisions of an earlier accumulation (of another surface), of the last one, and after the switch
@pytest.mark.parametrize("earlier,last,after", [(None, 64, 32), (None, 32, 64), (64, 32, 64), (32, 64, 32)])
@pytest.mark.parametrize("stage", ["erodepSPL", "sedChange"])
def test_stages_after_a_switch(earlier, last, after, stage):
    import torch
    m, ref = _models(2)
    if earlier:
        _precision(m, earlier)
        h = m.hGlobal.clone()
        m.hGlobal.copy_(h.flip(0))
        m.flowAccumulation()
        m.hGlobal.copy_(h)
    _precision(m, last)
    m.flowAccumulation()
    ref.flowAccumulation()
    assert torch.equal(m.rcv_i, ref.rcv_i)
    ref.FAL.copy_(m.FAL)
    if stage == "sedChange":
        rate = torch.as_tensor(np.random.default_rng(3).uniform(-1e-3, 1e-4, m.lpoints), device=m.dev)
        m.EbLocal.copy_(rate)
        ref.EbLocal.copy_(rate)
    _precision(m, after)
    before = m.hGlobal.clone()
    for q in (m, ref):
        getattr(q, stage)()
    assert not torch.equal(m.hGlobal, before)
    names = ("hGlobal", "cumED", "EbLocal") + (("vSed",) if stage == "sedChange" else ())
    for name in names:
        assert torch.equal(getattr(m, name), getattr(ref, name)), name
    m.destroy()
    ref.destroy()
