"""A batch that is tuned between two runs: trial launches must leave nothing
that the next run reads (nicr_batch_tune measures on whatever the domains hold,
a state that the bounds reject included)."""
import numpy as np
import pytest

import nicr
from parity import assert_bitexact, assert_budget, smooth_fields

pytestmark = pytest.mark.gpu

KINDS = {"2d": (2, (21, 40), dict(grains=1, grain_diameter_grid=12.)),
         "3d-static": (3, (9, 17, 40), dict(grains=1, grain_diameter_grid=9.)),
         "3d-evolving": (3, (9, 17, 40), dict(grains=1, grain_evolution=1, grain_diameter_grid=16.))}


def batch(kind):
    dim, shape, extra = KINDS[kind]
    kw = dict(nx=shape[0], ny=shape[1], bounds="stop", nucleation="off", dt=1e-12, **extra)
    if dim == 3:
        kw["nz"] = shape[2]
    b = nicr.Batch([nicr.make_config(dim, **kw) for _ in range(2)])
    for i, d in enumerate(b.domains):
        o, cr, p, eta = smooth_fields(d.shape, d.n_eta, seed=i)
        d.set_fields(o, cr, p, eta if eta else None)
        d.reset_inventory()
    return b


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("steps", [2, 3])   # both buffer parities
def test_tune_on_a_rejected_state_leaves_no_error(require_gpu, kind, steps):
    a, b = batch(kind), batch(kind)
    for q in (a, b):
        q.run(steps)
        d = q.domains[1]
        good = d.get("cr")
        bad = good.copy()
        bad[tuple(s - 2 for s in bad.shape)] = -0.1     # the next step would be rejected
        d.set("cr", bad)
        if q is a:
            q.tune(1)
        d.set("cr", good)
        done, rc = q.run(5, check=False)
        assert (done, rc) == ([5, 5], 0), q.last_error
    for da, db in zip(a.domains, b.domains):
        for f in ("o", "cr", "p"):
            assert_bitexact(f, da.get(f), db.get(f))
        for g in range(da.n_eta):
            assert_bitexact("eta%d" % g, da.get("eta", g), db.get("eta", g))
        assert_budget(da.budget(), db.budget())
        assert da.info().steps_done == steps + 5
    a.close()
    b.close()


def test_tune_measures_after_a_rejection(require_gpu):
    """A rejected run leaves the domain stopped; tuning it and running the unrepaired state rejects it again."""
    b = batch("3d-static")
    d = b.domains[0]
    cr = d.get("cr")
    cr[3, 3, 3] = -0.1
    d.set("cr", cr)
    for _ in range(2):
        done, rc = b.run(4, check=False)
        assert rc != 0 and done == [0, 4]
        b.tune(1)
    assert np.array_equal(d.get("cr"), cr)
    b.close()
