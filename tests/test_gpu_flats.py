"""Flat distances by depression against their definition.

Lakes of every size class of the search (one warp, one block, the larger block,
more than 65,536 cells) as circular bowls, and integer reliefs full of exact
ties, where lakes touch through several rim cells at one level: some distances
there run through a lower lake, which the search inside a depression cannot
give and the pass over the rims has to.  Exact, like every check of
tests/test_gpu_definitions.py.  A lake of more than a million cells takes the
search over all depressions and is compared with its tiled form.
"""
import numpy as np
import pytest

import definitions as D
from test_definitions import _planar_oracle, fill_level
from test_gpu_definitions import _model_like, check_gpu_fill

pytestmark = pytest.mark.gpu


def crossing_cells(om, h, sed):
    """Pit cells whose hop distance comes only through another depression."""
    ngb = om.FVmesh_ngbID
    outm = np.zeros(om.lpoints, dtype=bool)
    outm[om.outletIDs] = True
    level = fill_level(om, h)
    lf = D.filled_surface(h, level, ngb, outm, om.sealevel, sed=sed)
    pid = D.pit_ids(lf, ngb, level if sed else om.sealevel, om.outletIDs)
    om.h = h.copy()
    om.fillElevation(sed=sed)
    spills = np.unique(om.pitInfo[(om.pitInfo[:, 1] == 0) & (om.pitInfo[:, 0] >= 0), 0])
    pd = D.flat_distance(spills, pid, lf, ngb)
    is_spill = np.zeros(om.lpoints, dtype=bool)
    is_spill[spills] = True
    count = 0
    for v in np.where((pid > 0) & (pd > 1))[0]:
        c = ngb[v][ngb[v] >= 0]
        ok = (pd[c] == pd[v] - 1) & (lf[v] >= lf[c]) & ((pid[c] == pid[v]) | is_spill[c])
        count += 0 if ok.any() else 1
    return count


@pytest.mark.parametrize("seed,top", [(3, 4), (8, 6)])
def test_integer_relief_with_lakes_entered_from_lower_lakes(seed, top):
    om = _planar_oracle("ffff", n=4000, seed=11)
    xy = np.asarray(om.mesh["coords"])[:, :2]
    side = xy[:, 0].max()
    rng = np.random.default_rng(seed)
    # integer heights on blocks of cells: wide flats and lakes side by side
    cell = (np.floor(xy / side * 24.0).astype(int) @ np.array([1, 25]))
    z = rng.integers(1, top, 25 * 26).astype(np.float64)[cell] + rng.integers(0, 2, om.lpoints)
    z[om.outletIDs] = 0.0
    assert sum(crossing_cells(om, z, sed) for sed in (False, True)) > 0
    gm = _model_like(om)
    check_gpu_fill(gm, om, z, False, "integers")
    check_gpu_fill(gm, om, z, True, "integers sed")
    gm.destroy()


@pytest.mark.parametrize("n,radii", [(6000, (1.3, 2.9, 3.6, 11.0)), (16000, (25.3, 26.5)), (60000, (105.0,)),
                                     (90000, (150.0,))])
def test_bowls_of_every_size_class(n, radii):
    """Circular lakes of the given radii (in vertex spacings) on a slope; the
    last has more than 65,536 cells."""
    om = _planar_oracle("ffff", n=n, seed=13)
    xy = np.asarray(om.mesh["coords"])[:, :2]
    side = xy[:, 0].max()
    z = 100.0 + 1.0e-4 * xy[:, 0] + 3.0e-5 * xy[:, 1]
    x0 = 8.0 * 537.0
    for r in radii:
        r = r * 537.0
        x0 += r
        d = np.hypot(xy[:, 0] - (x0 if len(radii) > 1 else 0.5 * side), xy[:, 1] - 0.5 * side)
        z = np.where(d < r, 50.0 + d / r, z)
        x0 += r + 4.0 * 537.0
    z[om.outletIDs] = 0.0
    gm = _model_like(om)
    check_gpu_fill(gm, om, z, False, "bowls", large=n > 20000)
    assert int((gm.pitIDs > 0).sum()) > sum(r * r for r in radii)
    gm.destroy()


def test_a_lake_too_large_for_the_search_by_depressions():
    import torch
    from gospl_b200 import _lib
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    coords, cells = S.icosphere(9)
    fv = FVMesh(coords, cells, device="cuda:0")
    lat = coords[:, 2] / np.linalg.norm(coords, axis=1)
    # a lake around one pole with islands, a rim with one notch, and a sea around the other pole
    z = np.where(lat > 0.0, 300.0 * (1.0 - lat) + 40.0 * (np.sin(9.0 * np.arctan2(coords[:, 1], coords[:, 0])) > 0.97),
                 320.0 + 400.0 * lat)
    z[np.argmin(np.abs(lat) + (coords[:, 0] < 0))] -= 0.5
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e6, flowDir=3, K=3e-6, d=0.0, m=0.5, Cda=0.0, Cdm=0.0, sealevel=0.0,
             oFill=-6000.0, bc="oooo", rain=np.ones(fv.n), upsub=None)
    m = Model(coords=coords, cells=cells, elev=z, params=p, mesh=fv, device="cuda:0", init_flow=False)
    m.fillElevation()
    assert int(torch.bincount(m.pitIDs[m.pitIDs > 0].long()).max()) > 1 << 20
    one = m.flatDirs.clone()
    _lib.check(_lib.load().gs_plan_tune(m._plan, 7, 4096))
    m.fillElevation()
    assert torch.equal(one, m.flatDirs)
    assert int((one >= 0).sum()) > 1 << 20
    m.destroy()
