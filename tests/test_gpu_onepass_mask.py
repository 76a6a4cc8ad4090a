"""The mask fields behind the one-pass step (gb, eta_s2, and what is computed
from them) after steps that were replayed from a captured graph: the kernel
does not write them, so each read after a run rebuilds them from that run's
eta, also when an earlier read had rebuilt them."""
import numpy as np
import pytest

import nicr
from oracle import Oracle, make_config
from parity import compare_state, smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_mask_after_replayed_steps(require_gpu, precision):
    cfg = make_config(3, nx=19, ny=16, nz=32, grains=1, grain_evolution=1, grain_diameter_grid=16., bounds="legacy",
                      bc="mu", nucleation="off", dt=1e-9, step_form=1, precision=precision)
    o, cr, p, eta = smooth_fields((19, 16, 32), nicr.Solver(cfg).n_eta, seed=4)
    a, b = nicr.Solver(cfg), nicr.Solver(cfg)
    for s in (a, b):
        s.set_fields(o, cr, p, eta)
    for n in (2, 2, 4, 4, 16, 16):     # even runs: graph replays from the second of each length on
        a.step(n)
        for f in ("gb", "eta_s2"):
            a.get(f)                   # rebuilds the mask of this state
    for _ in range(44):
        b.step(1)
    for f in ("o", "cr", "p", "gb", "eta_s2", "mo", "mc", "muO", "muCr"):
        assert np.array_equal(a.get(f), b.get(f)), f
    ga, gb = a.grain_stats(), b.grain_stats()
    for k in ("min_s2", "max_s2", "gb_max", "mask", "sum_s2", "energy"):
        assert ga[k] == gb[k], k
    a.close()
    b.close()


def test_mask_of_a_run_equals_the_oracle(require_gpu):
    cfg = make_config(3, nx=19, ny=16, nz=32, grains=1, grain_evolution=1, grain_diameter_grid=16., bounds="legacy",
                      bc="mu", nucleation="off", dt=1e-9, step_form=1)
    sol, orc = nicr.Solver(cfg), Oracle(cfg)
    o, cr, p, eta = smooth_fields(orc.shape, orc.neta, seed=4)
    orc.set_fields(o, cr, p, np.array(eta))
    sol.set_fields(o, cr, p, eta)
    for n in (2, 2, 2):
        assert orc.step(n) == 0, orc.error()
        sol.run(n)
        compare_state(sol, orc)        # reads gb, eta_s2 and the mobilities
    sol.close()
