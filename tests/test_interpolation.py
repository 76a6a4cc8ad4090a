"""The reciprocal form's interpolation h(p) = p^3 (10 - 15 p + 6 p^2), compiled
here for the host from the library's header, against 80-bit arithmetic. Oxide
has p near 1, where the enhanced mobility of a grain boundary multiplies 1 - h,
so h must carry little more than its own rounding there.

With u = 2^-53: p^3 takes two roundings; 10 - 15 p + 6 p^2 = 1 + (p - 1)(6 p - 9)
takes, relative to its value on [0, 1], at most 1.1 u from 6 p - 9 (p below 1/6;
less above), 0.6 u from p - 1 (none from p = 1/2) and its own rounding; the
product one more. Together below 6 u. By Horner's rule 6 p - 15 alone rounds by
up to 8 u of the polynomial's value at p = 1."""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import PKG

SHIM = """
#include "nicr_physics.h"
extern "C" void h_of(const double* p, double* out, long long n) {
    for (long long i = 0; i < n; ++i) out[i] = nicr::h_fast(p[i]);
}
"""


@pytest.fixture(scope="module")
def h_of(tmp_path_factory):
    d = tmp_path_factory.mktemp("h")
    (d / "h.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-I" + str(PKG / "csrc"),
                    str(d / "h.cpp"), "-o", str(d / "h.so")], check=True)
    f = ctypes.CDLL(str(d / "h.so")).h_of

    def call(p):
        p = np.ascontiguousarray(p, dtype=np.float64)
        out = np.empty_like(p)
        ptr = ctypes.POINTER(ctypes.c_double)
        f(p.ctypes.data_as(ptr), out.ctypes.data_as(ptr), ctypes.c_longlong(p.size))
        return out
    return call


def test_relative_error_on_the_unit_interval(h_of):
    rng = np.random.default_rng(3)
    n = 200_000
    p = np.concatenate([rng.random(n), 1.0 - 10.0 ** rng.uniform(-12, -1, n), 10.0 ** rng.uniform(-12, -1, n),
                        1.0 - np.arange(64) * 2.0 ** -53, [0.0, 0.5, 1.0]])
    x = p.astype(np.longdouble)
    exact = x * x * x * (1 + (x - 1) * (6 * x - 9))
    err = np.abs(h_of(p).astype(np.longdouble) - exact)
    assert float((err / np.maximum(exact, np.longdouble(1e-300))).max()) <= 6 * 2.0 ** -53
    assert h_of(np.array([0.0, 1.0])).tolist() == [0.0, 1.0]
