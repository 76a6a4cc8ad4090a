"""The host's part of a long run() call is linear in its steps: one call takes
about as long as the same steps in calls of 10,000, with a Ksp schedule that
fires in none of them. (Looking ahead to the next scan before every group of
steps, 400,000 steps of the smallest 3D grid took 8.2 s in one call and 2.7 s
in forty.) The smallest 3D grid and a 2D grid too large for the many-step
launch take the stepwise path."""
import time

import pytest

import nicr
from parity import smooth_fields

pytestmark = pytest.mark.gpu


def test_one_long_call_costs_what_short_calls_do(require_gpu):
    cfg = nicr.make_config(3, nx=6, ny=5, nz=7, grains=0, bounds="legacy", bc="closed", nucleation="ksp",
                           nucleation_period=1e3, dt=1e-12)
    s = nicr.Solver(cfg)
    o, cr, p, _ = smooth_fields(s.shape, 0)
    s.set_fields(o, cr, p, None)
    s.run(2000)
    ratios = []
    for _ in range(3):        # the host may be disturbed: one undisturbed attempt decides
        t0 = time.perf_counter()
        s.run(400_000)
        t1 = time.perf_counter()
        for _ in range(40):
            s.run(10_000)
        ratios.append((t1 - t0) / (time.perf_counter() - t1))
        if ratios[-1] < 1.6:
            break
    assert ratios[-1] < 1.6, ratios
    s.close()


def test_schedule_of_a_stepwise_2d_call(require_gpu):
    """The same scans fire in one call and in calls of one step."""
    kw = dict(nx=400, ny=120, grains=0, bounds="legacy", bc="mu", nucleation="ksp", nucleation_period=7e-12, dt=1e-12,
              radius_grid=2.5)
    a, b = nicr.Solver(nicr.make_config(2, **kw)), nicr.Solver(nicr.make_config(2, **kw))
    o, cr, p, _ = smooth_fields(a.shape, 0)
    for s in (a, b):
        s.set_fields(60.0 * o, cr, p, None)
        s.reset_inventory()
    a.run(30)
    for _ in range(30):
        b.run(1)
    assert a.budget() == b.budget()
    for f in ("o", "cr", "p"):
        assert (a.get(f) == b.get(f)).all(), f
    a.close()
    b.close()
