"""Each step's launch commits the step before it. A rejected step must stop
what is already enqueued behind it: later steps, and a Ksp scan due right after
it (its nuclei are not booked), in the 2D, two-kernel and one-pass forms, in a
single handle and in a batch."""
import numpy as np
import pytest

import nicr
from nicr import make_config
from oracle import Oracle
from parity import assert_bitexact, assert_budget, smooth_fields

pytestmark = pytest.mark.gpu

FORMS = {"2d": (2, (25, 140), dict(grains=1, grain_diameter_grid=12.)),
         "3d-split": (3, (9, 17, 40), dict(grains=1, grain_diameter_grid=9.)),
         "3d-split-eta": (3, (9, 17, 40), dict(grains=1, grain_evolution=1, grain_diameter_grid=16., step_form=2)),
         "3d-onepass": (3, (9, 32, 64), dict(grains=1, grain_evolution=1, grain_diameter_grid=20., step_form=1))}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("period", [2, 3])
@pytest.mark.parametrize("batch", [False, True])
def test_rejection_stops_what_is_enqueued(require_gpu, form, period, batch):
    dim, shape, extra = FORMS[form]
    kw = dict(nx=shape[0], ny=shape[1], bounds="stop", nucleation="ksp", dt=1e-12, radius_grid=2.5,
              nucleation_period=period * 1e-12, **extra)
    if dim == 3:
        kw["nz"] = shape[2]
    cfg = make_config(dim, **kw)
    orc = Oracle(cfg)
    b = nicr.Batch([cfg, cfg]) if batch else None
    sol = b.domains[1] if batch else nicr.Solver(cfg)
    o, cr, p, eta = smooth_fields(orc.shape, orc.neta, seed=6)
    cr[tuple(s - 2 for s in cr.shape)] = -0.1      # rejected by the first step
    orc.set_fields(o, cr, p, np.array(eta) if eta else None)
    sol.set_fields(o, cr, p, eta if eta else None)
    rc, done = orc.run(9)
    assert rc != 0
    if batch:
        dones, got = b.run(9, check=False)
        assert dones[1] == done
    else:
        got, n = sol.run(9, check=False)
        assert n == done
        assert sol.last_error == orc.error()
    assert got == rc
    for n in ("o", "cr", "p"):
        assert_bitexact(n, sol.get(n), orc.get(n))
    assert_budget(sol.budget(), orc.budget())
    assert sol.info().steps_done == done
    if batch:
        b.close()
    else:
        sol.close()
