"""The reciprocal form's mobility in oxide at grain boundaries: the bulk oxide
value must not carry the rounding of the enhanced metal value. One step of an
all-oxide state with a boundary everywhere and an enhancement of 1e8 against
the drop-in form. Bound: two roundings of a value below one, and increments
that differ by the rounding of mu (about 2e-9 of 1e7) against its differences
(about 5e5 here), 4e-14, times five; the enhanced value's rounding would be
1e-6 of the increments."""
import numpy as np
import pytest

import nicr
from nicr import make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step_form", [1, 2])
def test_oxide_mobility_beside_enhanced_boundaries(require_gpu, step_form):
    shape = (9, 32, 64)
    rng = np.random.default_rng(5)
    o, cr = 0.4 + 0.02 * rng.random(shape), 0.2 + 0.02 * rng.random(shape)
    p = np.ones(shape)
    out = []
    for precision in (0, 1):
        cfg = make_config(3, nx=9, ny=32, nz=64, grains=1, grain_evolution=1, grain_diameter_grid=20., bounds="legacy",
                          nucleation="off", dt=2e-10, gb_factor_o=1e8, gb_factor_cr=1e8, step_form=step_form,
                          precision=precision)
        sol = nicr.Solver(cfg)
        eta = [np.full(shape, 0.5) for _ in range(sol.n_eta)]
        sol.set_fields(o, cr, p, eta)
        sol.step(1)
        out.append([sol.get(f) for f in ("o", "cr")])
    for start, a, b in zip((o, cr), *out):
        bound = 4.5e-16 + 2e-13 * np.abs(a[1:] - start[1:]).max()   # row 0 is the inlet's
        assert np.abs(a - start)[1:].max() > 0.
        assert np.abs(a - b).max() <= bound
