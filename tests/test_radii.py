"""The distinct radii of a pixel set (host code, compiled here): values, order and pixel map, and slots looked at
per pixel: the table is at most half full, so a spread hash needs 1.5 on average."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include "ytf_radii.h"
extern "C" long radii(int nx, const double* xs, int ny, const double* ys, double* ur, int* map, long* n) {
  std::vector<double> u;
  std::vector<int> m;
  const long probes = ytf::radii_map(nx, xs, ny, ys, u, m);
  std::memcpy(ur, u.data(), 8 * u.size());
  std::memcpy(map, m.data(), 4 * m.size());
  *n = (long)u.size();
  return probes;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("radii")
    (d / "r.cpp").write_text(SRC)
    so = d / "r.so"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "yellowthinfilms_b200", "csrc"), "-o", str(so), str(d / "r.cpp")])
    return ctypes.CDLL(str(so))


def _radii(lib, x, y):
    x, y = np.ascontiguousarray(x, np.float64), np.ascontiguousarray(y, np.float64)
    ur, m, n = np.zeros(len(x) * len(y)), np.zeros(len(x) * len(y), np.int32), ctypes.c_long()
    lib.radii.restype = ctypes.c_long
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    probes = lib.radii(len(x), p(x), len(y), p(y), p(ur), p(m), ctypes.byref(n))
    return ur[:n.value], m, probes


K = np.arange(65536.0)
SETS = {
    "whole": (K, [0.0]), "half": (0.5 * K, [0.0]), "hundreds": (100 * K, [0.0]), "2^-20": (2.0**-20 * K, [0.0]),
    "2^300": (2.0**300 * K[:4096], [0.0]), "powers of two": (2.0 ** np.arange(-500, 500), [0.0]),
    "whole grid": (K[:256], K[:256]), "symmetric": (K[:301] - 150, K[:201] - 100), "tenths": (0.1 * K, [0.0]),
    "offset": (K, [0.3]), "log": (np.geomspace(1e-3, 1e3, 65536), [0.0]), "one": ([0.0], [-0.0]),
}


@pytest.mark.parametrize("name", SETS)
def test_distinct_radii(lib, name):
    x, y = SETS[name]
    ur, m, probes = _radii(lib, x, y)
    r = np.hypot(np.asarray(x)[None, :], np.asarray(y)[:, None]).ravel()
    assert np.abs(ur[m] - r).max() <= 4e-16 * r.max()  # numpy's hypot may round otherwise
    assert len(np.unique(ur)) == len(ur)
    first = np.unique(m, return_index=True)[1]
    assert (np.diff(first) > 0).all()  # first-occurrence order
    assert probes <= 2 * len(m) + 8


def test_not_numbers(lib):
    """Each NaN is a radius of its own, found without a look at the others."""
    ur, m, probes = _radii(lib, np.full(20000, np.nan), [0.0, 1.0])
    assert len(ur) == 40000 and np.isnan(ur).all() and (m == np.arange(40000)).all() and probes <= 40000
    ur, m, _ = _radii(lib, [1.0, np.inf, np.nan, 1.0, -np.inf], [0.0])
    assert m.tolist() == [0, 1, 2, 0, 1] and ur[1] == np.inf and np.isnan(ur[2])
