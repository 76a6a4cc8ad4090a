"""The reduction kernels behind log() and grain_log() at the sizes where they
can go wrong: rows shorter than a warp and just beyond one or several 32-column
segments, a single segment for the whole grid, more CTAs than segments, and
grain counts on both sides of the shared-memory counters' capacity (1024)."""
import numpy as np
import pytest

import nicr
from nicr import make_config
from oracle import Oracle
from parity import ld, smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,shape,diameter", [
    (2, (5, 3), 3.0), (2, (41, 33), 9.0), (2, (140, 97), 12.0),
    (3, (3, 3, 3), 2.5), (3, (7, 5, 31), 5.0), (3, (9, 6, 32), 6.0), (3, (6, 11, 33), 6.0), (3, (33, 18, 65), 14.0),
    (3, (26, 24, 22), 2.9),      # 1075 grains, above the capacity
    (3, (20, 16, 24), 2.45),     # 997 grains, below it
])
def test_statistics_equal_the_oracle(require_gpu, dim, shape, diameter):
    """Extrema and counts equal; the sums are double-double here and long double in the oracle, so they
    differ by at most n eps_ld relative to the sum of magnitudes (all terms of one sign): below 1e-14."""
    kw = dict(nx=shape[0], ny=shape[1], grains=1, grain_evolution=1, grain_diameter_grid=diameter, bounds="legacy",
              nucleation="off", max_eta_fields=2000, random_seed=7)
    if dim == 3:
        kw["nz"] = shape[2]
    cfg = make_config(dim, **kw)
    sol, orc = nicr.Solver(cfg), Oracle(cfg)
    if orc.neta <= 16:
        o, cr, p, eta = smooth_fields(orc.shape, orc.neta, seed=3)
        rng = np.random.default_rng(5)
        p = np.where(rng.random(orc.shape) < .2, rng.random(orc.shape), p)      # some cells count as oxide
        eta = [e * rng.random(orc.shape) for e in eta]                         # a dominant grain that changes cell by cell
        orc.set_fields(o, cr, p, np.array(eta))
        sol.set_fields(o, cr, p, eta)
    orc.refresh()
    d, e = sol.diagnostics(), orc.log_values()
    for k in ("sum_O", "sum_Cr", "sum_phi", "sum_h"):
        assert abs(ld(d[k]) - ld(e[k])) <= 1e-14 * (1e-300 + abs(ld(e[k]))), k
    for k in ("min_O", "max_O", "min_Cr", "max_Cr", "min_Ni", "min_phi", "max_phi"):
        assert d[k] == e[k], k
    a, b = sol.grain_stats(), orc.grain_values()
    for k in ("min_eta", "max_eta", "min_s2", "max_s2", "gb_max", "alive", "unassigned"):
        assert a[k] == b[k], k
    assert (a["cells"] == b["cells"]).all()
    for k in ("sum_s2", "mask", "energy"):
        assert abs(ld(a[k]) - ld(b[k])) <= 1e-14 * (1e-300 + abs(ld(b[k]))), k
    assert np.allclose(a["amount"].sum(axis=1), b["amount"].sum(axis=1), rtol=1e-14, atol=1e-300)
    sol.close()
