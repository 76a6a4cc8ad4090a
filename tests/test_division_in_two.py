"""Two-operation division by a run constant: the library's decision
(nicr_division_in_two) against an exact rational restatement of the argument,
and both routes of the drop-in form against the oracle on the GPU."""
import ctypes
import math
import random
from fractions import Fraction as F

import numpy as np
import pytest

import nicr

# divisors whose two-operation quotient fails for some numerator
DX_FAILS, DT_FAILS = 9.466577983171802e-09, 4.3e-11


def rn(f):
    return f.numerator / f.denominator   # int / int is correctly rounded


def reciprocal(Y):
    zh = rn(F(1, Y))
    if F(zh) > F(1, Y):
        zh = math.nextafter(zh, 0)
    return zh, rn(F(1, Y) - F(zh))


def near_midpoints(Y, most):
    """Numerators X whose quotient X / Y lies k / (2^s Y) beside a rounding midpoint, 0 < |k| <= most."""
    t = (Y & -Y).bit_length() - 1
    for s in (53, 54):
        mod = 1 << (s - t)
        inv = pow(Y >> t, -1, mod)
        for k in range(-most, most + 1):
            if k == 0 or k % (1 << t) or (k // (1 << t)) % 2 == 0:
                continue
            for M in range((-(k // (1 << t)) * inv) % mod, 1 << 54, mod):
                X = (M * Y + k) >> s
                if M > 1 << 53 and 1 << 52 <= X < 1 << 53:
                    yield X


def two_operations(X, zh, zl):
    return rn(F(X) * F(zh) + F(rn(F(X) * F(zl))))


def decided(b):
    f = nicr.lib().nicr_division_in_two
    f.argtypes = [ctypes.c_double]
    return bool(f(b))


def divisors():
    r = random.Random(3)
    out = [1e-8, 1e-8 * 1e-8, 2e-10, 1e-12, 1e-9, 1e-18, 1.0, 0.5, 3.0, DX_FAILS, DT_FAILS, 1.9264783593120531]
    for i in range(150):
        out.append(float("%.2g" % (r.uniform(1, 10) * 10.0 ** r.randint(-16, 2))) if i % 2 else r.uniform(0.5, 2.0))
    return out


def test_decision_matches_exact_restatement():
    kept = 0
    for b in divisors():
        Y = int(math.frexp(b)[0] * 2 ** 53)
        zh, zl = reciprocal(Y)
        good = all(two_operations(X, zh, zl) == X / Y for X in near_midpoints(Y, 16))
        assert decided(b) == good, b
        if good:   # further from the midpoints nothing can fail: some of those numerators all the same
            kept += 1
            assert all(two_operations(X, zh, zl) == X / Y for X in near_midpoints(Y, 40))
    assert kept > 100
    assert not decided(DX_FAILS) and not decided(DT_FAILS)
    for b in (2.0 ** 61, -3.0, 0.0, 2.0 ** -61, math.inf, math.nan):   # outside the range: never
        assert not decided(b)


def test_a_failing_divisor_has_a_witness():
    for b in (DX_FAILS, DT_FAILS):
        Y = int(math.frexp(b)[0] * 2 ** 53)
        assert any(two_operations(X, *reciprocal(Y)) != X / Y for X in near_midpoints(Y, 16))


@pytest.mark.gpu
@pytest.mark.parametrize("spacing", [dict(), dict(dt=DT_FAILS / 64), dict(dx=DX_FAILS, dy=DX_FAILS)])
@pytest.mark.parametrize("dim,step_form,shape", [(2, 0, (37, 45)), (3, 0, (25, 15, 13)), (3, 2, (25, 15, 37)),
                                                 (3, 1, (9, 32, 64))])
def test_both_routes_match_oracle(require_gpu, spacing, dim, step_form, shape):
    from oracle import Oracle, make_config
    from parity import compare_state, smooth_fields
    if dim == 3 and "dx" in spacing:
        spacing = dict(spacing, dz=DX_FAILS)
    kw = dict(nx=shape[0], ny=shape[1], grains=1, grain_evolution=1, grain_diameter_grid=26., bc="concentration",
              ck="legacy", bounds="legacy", nucleation="off", dt=1e-12, step_form=step_form)
    if dim == 3:
        kw["nz"] = shape[2]
    cfg = make_config(dim, **{**kw, **spacing})
    sol, orc = nicr.Solver(cfg), Oracle(cfg)
    o, cr, p, eta = smooth_fields(orc.shape, orc.neta, seed=2)
    orc.set_fields(o, cr, p, np.array(eta) if eta else None)
    sol.set_fields(o, cr, p, eta if eta else None)
    for _ in range(5):
        assert orc.step() == 0, orc.error()
    sol.run(5)
    compare_state(sol, orc)


@pytest.mark.gpu
@pytest.mark.parametrize("b", [DX_FAILS, DT_FAILS, 1e-8 * 1e-8, 2e-10, 5e-10])
def test_device_division(require_gpu, b):
    L = nicr.lib()
    L.nicr_check_division.argtypes = [ctypes.c_double, ctypes.c_longlong, ctypes.c_ulonglong,
                                      ctypes.POINTER(ctypes.c_longlong)]
    L.nicr_check_division.restype = ctypes.c_longlong
    tested = ctypes.c_longlong(0)
    assert L.nicr_check_division(b, 1 << 25, 99, ctypes.byref(tested)) == 0
    assert tested.value > 1 << 24
