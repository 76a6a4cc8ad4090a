"""Step graphs of 2D domains that the many-step launch does not take (more than
37,888 cells): replayed groups against plain launches (NICR_GRAPHS=0, in a child
process each), single crystal, static and evolving grains, across Ksp scans,
odd step counts, a read between replays and a rejected trial. The same state,
budgets, return codes and launch counts, bit for bit."""
import numpy as np
import pytest

from test_gpu_graphs import run_child

pytestmark = pytest.mark.gpu

KSP = dict(nucleation="ksp", nucleation_period=5e-12, radius_grid=2.5, dt=1e-12, bounds="legacy")
CASES = {
    "crystal": dict(chunks=[1, 7, 30], kw=dict(nx=211, ny=199, grains=0, nucleation="center", radius_grid=4.0,
                                               bc="concentration", ck="legacy", bounds="legacy")),
    "static-ksp": dict(chunks=[9, 13, 4], kw=dict(nx=300, ny=130, grains=1, grain_diameter_grid=25., bc="mu", **KSP)),
    "evolving-ksp": dict(chunks=[9, 13, 4], kw=dict(nx=220, ny=181, grains=1, grain_evolution=1, grain_diameter_grid=90.,
                                                    bc="mu", **KSP)),
    "evolving-rejection": dict(chunks=[6, 6], bad=[100, 90],
                               kw=dict(nx=200, ny=200, grains=1, grain_evolution=1, grain_diameter_grid=90., bounds="stop",
                                       nucleation="off", dt=1e-12)),
}


@pytest.mark.parametrize("mode", ["run", "step"])
@pytest.mark.parametrize("name", list(CASES))
def test_replayed_groups_match_plain_launches(require_gpu, tmp_path, name, mode):
    case = dict(CASES[name], dim=2, mode=mode)
    a, ja = run_child(case, tmp_path / "graphs", True)
    b, jb = run_child(case, tmp_path / "plain", False)
    for k in b.files:
        assert np.array_equal(a[k].view(np.int64), b[k].view(np.int64)), (name, k)
    assert ja["rcs"] == jb["rcs"] and ja["budget"] == jb["budget"] and ja["steps"] == jb["steps"]
    assert ja["launches"] == jb["launches"]
    if name == "evolving-rejection":
        assert ja["rcs"][0][0] != 0 and ja["rcs"][1][0] == 0
