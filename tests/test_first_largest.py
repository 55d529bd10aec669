"""first_largest.h (the first maxr of a row of draws) on the host, against the
quotients themselves; crafted draws take it where the draws alone do not
decide."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "first_largest.h"
extern "C" int first(const unsigned long long* u, int n) {
  return pqdts::first_largest([=](int k) { return (uint64_t)u[k]; }, n);
}
extern "C" double value(unsigned long long u) { return pqdts::draw_value(u); }
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("first_largest")
    (d / "t.cpp").write_text(SOURCE)
    so = str(d / "t.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    "-I", os.path.join(ROOT, "pqdts_gb300", "csrc"), str(d / "t.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.value.restype = C.c_double
    lib.value.argtypes = [C.c_ulonglong]
    return lib


def _reference(u):
    x = np.array([int(v) * 2.0 ** -53 for v in u])
    s = 0.0
    for v in x:
        s = s + v
    with np.errstate(invalid="ignore"):
        q = x / s
    am = 0
    for n in range(1, len(q)):
        if q[n] > q[am]:
            am = n
    return am


def test_values(host):
    for u in [0, 1, 2, 3, 2**52 - 1, 2**52, 2**52 + 1, 2**53 - 1] + [3 << k for k in range(51)]:
        assert host.value(u) == u * 2.0 ** -53


def test_first_largest(host):
    rng = np.random.default_rng(1)
    rows = [[0], [7], [0, 0, 0], [0, 3], [3, 0], [5, 5, 5]]
    for top in (6, 2**20, 2**50, 2**53 - 1):
        for gap in range(7):  # an early maximum, and one or two just above it
            rows += [[1, top - gap, 2, top], [top - gap, top], [top - gap, 0, top - gap // 2, top, top]]
    for spread in (2, 8, 64, 2**53 - 2**52):
        for n in (2, 3, 5, 33, 200):
            rows += [list(2**53 - 1 - rng.integers(0, spread, n)) for _ in range(40)]
    decided = 0
    for row in rows:
        u = np.array(row, np.uint64)
        am = host.first(u.ctypes.data_as(C.c_void_p), len(u))
        assert am == _reference(u), row
        decided += am != int(np.argmax(u))
    assert decided > 0  # rows where two draws' quotients round to the same
