"""Reads of small fields (through the handle's pinned staging up to 32768 cells,
straight into pinned memory and for larger fields into the caller's) return
the cells of the device view, and the status word that a run leaves on the host
serves the next run: after accepted, rejected and repaired runs."""
import numpy as np
import pytest

import nicr
from parity import smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 7), (61, 61), (128, 256), (182, 181), (11, 5, 7), (32, 32, 32), (33, 32, 32)])
def test_read_matches_device_view(require_gpu, shape):
    import torch
    kw = dict(nx=shape[0], ny=shape[1], grains=0, nucleation="off", bounds="legacy")
    if len(shape) == 3:
        kw["nz"] = shape[2]
    s = nicr.Solver(nicr.make_config(len(shape), **kw))
    o, cr, p, _ = smooth_fields(s.shape, 0, seed=3)
    s.set_fields(o, cr, p, None)
    s.run(3)
    for f in ("o", "cr", "p"):
        want = s.device_view(f).cpu().numpy().reshape(-1)
        pinned = torch.empty(s.n, dtype=torch.float64).pin_memory().numpy()
        assert np.array_equal(s.get(f).reshape(-1), want)
        assert np.array_equal(np.asarray(s.get(f, out=pinned)).reshape(-1), want)
    s.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_runs_after_a_rejected_one(require_gpu, dim):
    shape = (25, 15, 13)[:dim]
    kw = dict(nx=25, ny=15, grains=1, grain_diameter_grid=12., bounds="stop", nucleation="off", dt=1e-12)
    if dim == 3:
        kw["nz"] = 13
    a, b = (nicr.Solver(nicr.make_config(dim, **kw)) for _ in range(2))
    o, cr, p, eta = smooth_fields(shape, a.n_eta, seed=5)
    bad = cr.copy()
    bad[(20, 5, 4)[:dim]] = -0.1
    for s in (a, b):
        s.set_fields(o, cr, p, eta if eta else None)
        s.run(5)
    good = a.get("cr")
    a.set("cr", bad)
    rc, done = a.run(4, check=False)
    assert rc == nicr._abi.ERR_TRIAL_BOUNDS and done == 0
    a.set("cr", good)
    if dim == 2:
        a.set("o", b.get("o"))   # 2D keeps the enforced inlet layer of a rejected step
    for n in (1, 6):
        for s in (a, b):
            s.run(n)
        for f in ("o", "cr", "p"):
            assert np.array_equal(a.get(f), b.get(f)), (n, f)
    assert a.info().steps_done == b.info().steps_done == 12
