"""Plans of different sizes used by several threads at once, each on its own stream.

A launch asks for its own plan's shared memory; nothing that one plan sets may
change what the other's launches get.  Results equal those of one thread.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(n, seed):
    from gospl_b200 import synthetic as S
    from gospl_b200.mesh import FVMesh
    from gospl_b200.model import Model
    side = 1000.0 * np.sqrt(n)
    c, f, onb = S.planar_hex_mesh(n, side, seed)
    z = S.rescale(S.fractal_field(c[:, :2], side, seed + 1), 0.0, 100.0)
    z[onb] = 0.0
    p = dict(dt=1000.0, tStart=0.0, tEnd=1e30, flowDir=3, K=3e-6, d=0.0, m=0.5, Cda=0.1, Cdm=0.1, sealevel=-100.0,
             oFill=-6000.0, bc="ffff", rain=np.ones(len(z)), upsub=None)
    return Model(coords=c, cells=f, elev=z, params=p, mesh=FVMesh(c, f, "ffff"), device="cuda:0", init_flow=False)


def test_plans_of_two_sizes_in_four_threads():
    import torch
    sizes, rounds = (2500, 3200, 4000, 90000), 300
    models, streams, starts, wants = [], [], [], []
    for q, n in enumerate(sizes):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            m = _model(n, 31 + q)
            h0 = m.hGlobal.clone()
            m.flowAccumulation()
            m.erodepSPL()
            wants.append([getattr(m, k).clone() for k in ("FAL", "flatDirs", "hGlobal")])
        models.append(m)
        streams.append(s)
        starts.append(h0)
    torch.cuda.synchronize()
    stop, errors = threading.Event(), []

    def work(q):
        m = models[q]
        done = 0
        try:
            with torch.cuda.stream(streams[q]):
                # the small plans go on until the large one has had its rounds
                large = q == len(sizes) - 1
                while not (done == rounds if large else stop.is_set()):
                    m.hGlobal.copy_(starts[q])
                    if large:
                        m.flowAccumulation()
                    m.erodepSPL()
                    for k, w in zip(("FAL", "flatDirs", "hGlobal"), wants[q]):
                        if not torch.equal(getattr(m, k), w):
                            raise AssertionError("plan %d, pass %d: %s" % (q, done, k))
                    done += 1
        except Exception as e:      # noqa: BLE001 - reported by the test's own thread
            errors.append(repr(e))
        finally:
            stop.set()

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120.0)
    assert not any(t.is_alive() for t in threads)
    assert not errors, errors
    for m in models:
        m.destroy()
