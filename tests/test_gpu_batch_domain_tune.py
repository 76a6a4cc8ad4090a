"""A batch's domain tuned by its own handle between two runs of the batch: its
launches have another grid then, and its partial sums may have moved (a 64^3
grid has 1024 CTAs with the candidate chunk of one plane, above the room a
handle starts with), so the step pairs the batch captured before serve no more.
Fields equal an untuned batch's, bit for bit; budgets to 1e-13 (their per-CTA
sums group differently)."""
import pytest

import nicr
from parity import assert_bitexact, assert_budget, smooth_fields

pytestmark = pytest.mark.gpu


def batch():
    kw = dict(bounds="legacy", nucleation="off", dt=1e-12, bc="concentration")
    b = nicr.Batch([nicr.make_config(3, nx=64, ny=64, nz=64, grains=1, grain_diameter_grid=20., **kw),
                    nicr.make_config(3, nx=9, ny=17, nz=40, grains=1, grain_evolution=1, grain_diameter_grid=16., **kw),
                    nicr.make_config(3, nx=64, ny=64, nz=64, grains=0, **kw)])
    for i, d in enumerate(b.domains):
        o, cr, p, eta = smooth_fields(d.shape, d.n_eta, seed=i)
        d.set_fields(o, cr, p, eta if eta else None)
        d.reset_inventory()
    return b


def test_tuned_domain_of_a_batch(require_gpu):
    a, b = batch(), batch()
    for n in (4, 5, 6):           # pairs from both parities
        a.run(n)
        b.run(n)
        for i in (0, 1):
            a.domains[i].tune(1)
    a.run(8)
    b.run(8)
    for da, db in zip(a.domains, b.domains):
        assert da.info().steps_done == 23
        for f in ("o", "cr", "p"):
            assert_bitexact(f, da.get(f), db.get(f))
        for g in range(da.n_eta):
            assert_bitexact("eta%d" % g, da.get("eta", g), db.get("eta", g))
        assert_budget(da.budget(), db.budget())
    a.close()
    b.close()
