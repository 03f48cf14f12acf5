"""A plan on a device without room for the records of the tile sweeps.

The plan's other arrays fit: it is created, takes the ordered sweeps and gives
the same results, bit for bit.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_plan_without_room_for_tile_records():
    import torch
    from gospl_b200 import _lib
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    n = 200000
    side = 1000.0 * np.sqrt(n)
    coords, cells, onb = S.planar_hex_mesh(n, side, 29)
    z = S.rescale(S.fractal_field(coords[:, :2], side, 30), 0.0, 100.0)
    z[onb] = 0.0
    fv = FVMesh(coords, cells, "ffff")
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e30, flowDir=3, K=3e-6, d=0.0, m=0.5, Cda=0.1, Cdm=0.1, sealevel=-100.0,
             oFill=-6000.0, bc="ffff", rain=np.ones(fv.n), upsub=None)
    make = lambda: Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0", init_flow=False)

    def passes(m):
        m.flowAccumulation()
        m.erodepSPL()
        return [getattr(m, k).clone() for k in ("FAL", "hGlobal")]

    MB = 1 << 20
    records = 3 * 96 * fv.n              # three graphs, 96 bytes a vertex at least
    spare = torch.empty(256 * MB, dtype=torch.uint8, device="cuda:0")
    free = lambda: torch.cuda.mem_get_info()[0]
    a = make()
    want = passes(a)
    del spare                            # stays with the allocator, for the second model's tensors
    torch.cuda.synchronize()
    f0 = free()
    b = make()                           # what a plan takes, all told
    taken = f0 - free()
    assert taken > records
    b.destroy()
    torch.cuda.synchronize()
    hog = torch.empty(free() - (taken - records // 2), dtype=torch.uint8, device="cuda:0")
    try:
        c = make()
    finally:
        del hog
        torch.cuda.empty_cache()
    L = _lib.load()
    _lib.check(L.gs_plan_profile(c._plan, 1))
    got = passes(c)
    names = ctypes.create_string_buffer(1 << 18)
    assert 0 < L.gs_plan_profile_report(c._plan, names, len(names)) < len(names)
    assert b"k_ordered" in names.value and b"k_tile_sweep" not in names.value
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    a.destroy()
    c.destroy()
