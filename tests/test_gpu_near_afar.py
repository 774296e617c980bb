"""Rays from outside the range that the nearest-first view covers end in its
kernel where they meet none of the root's boxes, and are handed on otherwise:
aimed at, along and just past the tree's box and its corners, in and against
short t_max, ids, t, u, v equal the oracle's."""
import math

import numpy as np
import pytest

import oracle
from lucent_gb300 import DeviceBVH, mesh, workloads

pytestmark = pytest.mark.gpu

KNOT = mesh.torus_knot(tubular_segments=150, radial_segments=12).positions
ONE = np.array([[-0.5, -0.4, 0.1, 0.6, -0.3, 0.2, 0.0, 0.5, -0.3]], np.float32)


def _rays(pos, radius, n, seed):
    """A third each: chords, lines past the box, lines through points on its edges and corners (some a few ulps off)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    v = np.asarray(pos, np.float64).reshape(-1, 3)
    lo, hi = v.min(0), v.max(0)
    o = workloads.sphere_rays(rng, n)[:, :3].astype(np.float64)
    o *= radius * np.linalg.norm(hi - lo) / np.linalg.norm(o, axis=1, keepdims=True)
    to = rng.uniform(lo, hi, (n, 3))
    third = n // 3
    to[:third] += np.cross(o[:third], rng.normal(size=(third, 3))) / radius
    k = rng.integers(0, 8, (n, 3))  # per axis: one face, the other, or inside
    edge = np.where(k < 3, lo, np.where(k < 6, hi, to))
    to[third:2 * third] = edge[third:2 * third] * (1 + rng.integers(-2, 3, (third, 3)) * 2.0 ** -23)
    d = to - o
    d *= rng.choice([1.0, 0.1, 5.0], (n, 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("t_max", [math.inf, 1.0, 1e-3])
@pytest.mark.parametrize("radius", [0.3, 3.0, 70.0, 3e3, 1e6])
@pytest.mark.parametrize("pos", [KNOT, ONE], ids=["knot", "one"])
def test_afar(pos, radius, t_max):
    pos = np.asarray(pos, np.float32)
    rays = _rays(pos, radius, 9_999, int(radius * 10))
    t_max *= radius * 4 if t_max == 1.0 else 1.0  # about half of the hits
    ob = oracle.build_bvh(pos)
    dev = DeviceBVH(ob.nodes, ob.tri_indices, pos, ob.node_count)
    ids, t, u, v = oracle.intersect_bvh(ob, pos, rays, 0.0, t_max)
    got = dev.intersect(rays, 0.0, t_max)
    dev.close()
    assert np.array_equal(got[0], ids)
    hit = ids >= 0
    for a, b in zip(got[1:], (t, u, v)):
        assert np.array_equal(a[hit], b[hit].astype(np.float32))
    assert np.all(np.isinf(got[1][~hit]))
