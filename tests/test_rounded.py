"""The square root and quotient of the coarse factor (csrc/rounded.h), compiled for the host, against sqrt and / on
random operands over the range that takes them, for reciprocal roots that are up to two ulps off."""
import ctypes
import os
import subprocess

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-to_b200", "csrc")
SOURCE = """
#include "rounded.h"
extern "C" void roots(long n, const double *s, const double *y, double *d)
{
    for (long i = 0; i < n; ++i) d[i] = gputo::sqrt_by(s[i], y[i]);
}
extern "C" void quotients(long n, const double *s, const double *d, const double *y, double *q)
{
    for (long i = 0; i < n; ++i) q[i] = gputo::div_by(s[i], d[i], y[i]);
}
"""


def test_roots_and_quotients_are_those_of_sqrt_and_division(tmp_path):
    src, so = tmp_path / "r.cpp", tmp_path / "r.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}", str(src), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    ptr = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))   # noqa: E731
    rng = np.random.default_rng(3)
    n = 200000

    def values(e):
        return rng.uniform(1.0, 10.0, n) * 10.0 ** rng.uniform(-e, e - 1, n)

    for s, t in ((values(200), values(200)), (rng.uniform(0.5, 2.0, n), rng.uniform(-1.0, 1.0, n))):
        root = np.sqrt(s)
        for ulps in (-2, -1, 0, 1, 2):
            y = 1.0 / root
            y = y + ulps * np.spacing(y)
            d, q = np.empty(n), np.empty(n)
            lib.roots(ctypes.c_long(n), ptr(s), ptr(y), ptr(d))
            assert np.array_equal(d, root)
            normal = np.abs(t / root) > 1e-300
            lib.quotients(ctypes.c_long(n), ptr(t), ptr(root), ptr(y), ptr(q))
            assert np.array_equal(q[normal], (t / root)[normal])
