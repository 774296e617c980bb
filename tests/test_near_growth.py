"""leaf_growth as the view computes it, in binary32, is never less than the
binary64 bound that it stands for, over sizes, thin and flat triangles."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from lucent_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def growth(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("growth") / "growth.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I" + inc,
                           "-I" + B.CSRC, os.path.join(HERE, "near_growth_host.cpp"), "-o", out])
    fn = C.CDLL(out).growth

    def call(tri, s):
        n = len(tri)
        g, r = np.zeros(n, np.float32), np.zeros(n, np.float32)
        fn(tri.ctypes.data_as(C.c_void_p), C.c_int(n), C.c_float(s), g.ctypes.data_as(C.c_void_p),
           r.ctypes.data_as(C.c_void_p))
        return g, r

    return call


def _bound(v, s):
    """Growth and its rise per unit of s, in binary64. A triangle in a coordinate plane needs next to none unless it is
    thin (|e1| |e2| above 65,536 of its area's double)."""
    e1, e2 = v[1] - v[0], v[2] - v[0]
    l1, l2 = math.sqrt(e1 @ e1), math.sqrt(e2 @ e2)
    area2 = math.sqrt(np.sum(np.cross(e1, e2) ** 2))
    k = 2.0 ** -28
    if not (np.any((v[0] == v[1]) & (v[0] == v[2])) and l1 * l2 <= 65536 * area2):
        w = 2.1e-3 * l1 * l2 / max(1 - 1.8e-3 * l1 * l2, 1e-6)
        if w >= 0.5:
            return math.inf, 0.0  # no bound at all: the box is as good as everywhere
        k += w / (1 - w)
    return k * (4 * s + 3 * max(l1, l2)), 4 * k


@pytest.mark.parametrize("size", [1e-12, 1e-6, 1e-3, 0.03, 1.0, 12.0, 16.0, 1e3, 1e6])
@pytest.mark.parametrize("thin", [1.0, 1e-3, 2e-5, 1.5e-5, 1e-6, 0.0])
@pytest.mark.parametrize("flat", [False, True])
def test_never_below_the_bound(growth, size, thin, flat):
    rng = np.random.Generator(np.random.PCG64(int(1e6 * thin) + flat))
    n = 2000
    a, e = rng.uniform(-1, 1, (n, 3)) * size, rng.normal(size=(n, 3)) * size
    off = np.cross(e, rng.normal(size=(n, 3)))
    if flat:
        e[:, 2] = 0
        off = np.cross(e, [0.0, 0.0, 1.0])
    off *= thin * np.linalg.norm(e, axis=1, keepdims=True) / np.maximum(np.linalg.norm(off, axis=1, keepdims=True), 1e-300)
    tri = np.stack([a, a + e, a + e * rng.uniform(0.3, 1.5, (n, 1)) + off], 1).astype(np.float32)
    s = 5 * size
    g, rise = growth(tri, s)
    s = float(np.float32(s))
    for k in range(n):
        want, up = _bound(tri[k].astype(np.float64), s)
        assert g[k] >= (want * (1 - 1e-6) if math.isfinite(want) else 1e29), (tri[k], g[k], want)
        assert not math.isfinite(want) or g[k] >= 1e29 or rise[k] >= up * (1 - 1e-6)
