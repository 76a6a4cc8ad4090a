"""Edges of the drop-in form's scaled exact division: quotients that overflow
times 2^128 or are not finite (noted through the trial value they reach), and
divisors outside the certified range (every chunk divided by IEEE division).
Results, status and message equal the oracle's in the 2D, the two-kernel 3D and
the one-pass 3D kernels, with the odd value on a tile corner and inside one."""
import numpy as np
import pytest

import nicr
from nicr import make_config
from oracle import Oracle
from parity import assert_bitexact, smooth_fields

pytestmark = pytest.mark.gpu

FORMS = {"2d": (2, (25, 140), dict(grains=0)), "3d-split": (3, (9, 17, 40), dict(grains=1, grain_diameter_grid=9.)),
         "3d-split-eta": (3, (9, 17, 40), dict(grains=1, grain_evolution=1, grain_diameter_grid=16., step_form=2)),
         "3d-onepass": (3, (9, 32, 64), dict(grains=1, grain_evolution=1, grain_diameter_grid=20., step_form=1))}


def pair(form, **kw):
    dim, shape, extra = FORMS[form]
    base = dict(nx=shape[0], ny=shape[1], bounds="legacy", nucleation="off", dt=1e-12, **extra)
    if dim == 3:
        base["nz"] = shape[2]
    base.update(kw)
    cfg = make_config(dim, **base)
    sol, orc = nicr.Solver(cfg), Oracle(cfg)
    if form == "3d-onepass":
        assert 1 <= orc.neta <= 8, orc.neta
    return sol, orc


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("field", ["o", "cr", "p", "eta"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e300, -1e272])
@pytest.mark.parametrize("at", [(0, 0, 0), (8, 16, 32), (4, 9, 13)])
def test_nonfinite_and_overflowing_quotients(require_gpu, form, field, value, at):
    sol, orc = pair(form)
    o, cr, p, eta = smooth_fields(orc.shape, orc.neta, seed=2)
    if field == "eta" and not eta:
        pytest.skip("no eta in this form")
    target = {"o": o, "cr": cr, "p": p, "eta": eta[0] if eta else None}[field]
    target[at if len(orc.shape) == 3 else (at[0], at[2])] = value
    orc.set_fields(o, cr, p, np.array(eta) if eta else None)
    sol.set_fields(o, cr, p, eta if eta else None)
    rc = orc.step()
    got, done = sol.step(1, check=False)
    assert got == rc and done == (1 if rc == 0 else 0)
    if rc:
        assert sol.last_error == orc.error()
    for n in ("o", "cr", "p"):
        a, b = sol.get(n), orc.get(n)
        assert np.array_equal(a, b, equal_nan=True), n
    sol.close()


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("kw", [dict(dx=1e-19, dt=1e-42), dict(eta_kappa=1e-160)])
def test_divisors_and_constants_out_of_range(require_gpu, form, kw):
    sol, orc = pair(form, **kw)
    o, cr, p, eta = smooth_fields(orc.shape, orc.neta, seed=4)
    orc.set_fields(o, cr, p, np.array(eta) if eta else None)
    sol.set_fields(o, cr, p, eta if eta else None)
    for _ in range(2):
        rc = orc.step()
        got, _ = sol.step(1, check=False)
        assert got == rc
        if rc:
            assert sol.last_error == orc.error()
            break
    # the fields only: the clipped amounts here are sums of huge cancelling terms
    for n in ["o", "cr", "p"] + ["eta%d" % (g + 1) for g in range(orc.neta)]:
        assert_bitexact(n, sol.get(n), orc.get(n))
    sol.close()
