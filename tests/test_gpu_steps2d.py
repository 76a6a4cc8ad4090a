"""Many steps of a 2D domain in one cooperative launch: grids at the edges of its
tiles (rows of one to three column tiles, plane counts beside each tile size, the
smallest grid), grids for each tile size and one too large for it, runs longer
than one launch, rejections in the middle of a launch."""
import numpy as np
import pytest

import nicr
from nicr import make_config
from oracle import Oracle
from parity import assert_bitexact, assert_budget, compare_state, smooth_fields

pytestmark = pytest.mark.gpu

MODES = {"crystal": dict(grains=0), "static": dict(grains=1, grain_diameter_grid=9.),
         "evolving": dict(grains=1, grain_evolution=1, grain_diameter_grid=14.)}


def pair(shape, mode, **kw):
    base = dict(nx=shape[0], ny=shape[1], bounds="legacy", nucleation="off", dt=1e-12, **MODES[mode])
    base.update(kw)
    cfg = make_config(2, **base)
    sol, orc = nicr.Solver(cfg), Oracle(cfg)
    o, cr, p, eta = smooth_fields(orc.shape, orc.neta, seed=shape[0] + shape[1])
    orc.set_fields(o, cr, p, np.array(eta) if eta else None)
    sol.set_fields(o, cr, p, eta if eta else None)
    return sol, orc


@pytest.mark.parametrize("shape", [(3, 3), (4, 31), (5, 32), (7, 33), (8, 64), (9, 65), (200, 60), (300, 64), (151, 97),
                                   (600, 70)])
@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("bc", ["concentration", "mu"])
def test_grids(require_gpu, shape, mode, bc):
    if mode == "evolving" and shape[0] * shape[1] > 20000:
        pytest.skip("the oracle's evolving grains on the large grids: minutes")
    sol, orc = pair(shape, mode, bc=bc)
    for n in (1, 4, 2):
        assert orc.step(n) == 0, orc.error()
        sol.run(n)
    compare_state(sol, orc)
    sol.close()


def test_more_steps_than_a_launch(require_gpu):
    sol, orc = pair((12, 10), "static", bc="concentration")
    assert orc.step(4099) == 0
    sol.step(4099)
    compare_state(sol, orc)
    sol.close()


@pytest.mark.parametrize("mode", list(MODES))
def test_rejection_inside_a_launch(require_gpu, mode):
    """A step that is too long for the mesh leaves the bounds after 7, 1 and 3 accepted steps (by the oracle); the
    state is the last accepted one, as step by step."""
    sol, orc = pair((21, 40), mode, bc="mu", bounds="stop", dt=1e-6 if mode == "crystal" else 2e-7)
    rc = 0
    done = 0
    while rc == 0 and done < 400:
        rc = orc.step(1)
        done += rc == 0
    assert rc != 0 and done > 0, "the case must be rejected after its first step"
    got, n = sol.step(400, check=False)
    assert (got, n) == (rc, done)
    assert sol.last_error == orc.error()
    for name in ["o", "cr", "p"] + ["eta%d" % (g + 1) for g in range(orc.neta)]:
        assert_bitexact(name, sol.get(name), orc.get(name))
    assert_budget(sol.budget(), orc.budget())
    sol.close()


@pytest.mark.parametrize("mode", list(MODES))
def test_reciprocal_form(require_gpu, mode):
    a, orc = pair((61, 61), mode, bc="concentration")
    b, _ = pair((61, 61), mode, bc="concentration", precision=1)
    a.step(50)
    b.step(50)
    for name in ["o", "cr", "p"] + ["eta%d" % (g + 1) for g in range(orc.neta)]:
        x, y = a.get(name), b.get(name)
        assert np.max(np.abs(x - y)) <= 1e-10 * max(np.max(np.abs(x)), 1e-300), name
