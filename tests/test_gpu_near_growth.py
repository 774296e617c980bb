"""Nearest-first closest hit over triangles around the thinness at which the growth
of a leaf in a coordinate plane changes (edges' product 65,536 times the cross
product) and over tilted ones, from far below to far above it and at sizes whose
cross products binary32 can and cannot square: ids, t, u, v equal the oracle's
intersectBVH for rays that graze the triangles' edges."""
import numpy as np
import pytest

import oracle
from lucent_gb300 import DeviceBVH

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1e-7, 1e-3, 0.3])
@pytest.mark.parametrize("thin", [1e-6, 1.5e-5, 2e-5, 1e-3])
@pytest.mark.parametrize("flat", [False, True])
def test_thin_triangles(size, thin, flat):
    rng = np.random.Generator(np.random.PCG64(int(1 / thin) + int(1 / size)))
    n = 3000
    a = rng.uniform(-1, 1, (n, 3))
    e = rng.normal(size=(n, 3)) * size
    if flat:
        e[:, 2] = 0
    off = np.cross(e, rng.normal(size=(n, 3)) * (0, 0, 1) if flat else rng.normal(size=(n, 3)))
    off *= thin * np.linalg.norm(e, axis=1, keepdims=True) / np.linalg.norm(off, axis=1, keepdims=True)
    tri = np.stack([a, a + e, a + e * rng.uniform(0.3, 1.5, (n, 1)) + off], 1).astype(np.float32)
    w = rng.dirichlet((0.2, 0.2, 0.2), n)  # many near an edge or a corner
    target = (tri.astype(np.float64) * w[:, :, None]).sum(1) + rng.normal(size=(n, 3)) * size * thin * 0.3
    o = 3.0 * rng.normal(size=(n, 3))
    o /= np.maximum(1.0, np.linalg.norm(o, axis=1, keepdims=True) / 3.0)
    d = target - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    pos = tri.reshape(-1)
    ob = oracle.build_bvh(pos)
    dev = DeviceBVH(ob.nodes, ob.tri_indices, pos, ob.node_count)
    ids, t, u, v = oracle.intersect_bvh(ob, pos, rays)
    p, gt, gu, gv = dev.intersect(rays)
    assert np.array_equal(p, ids)
    hit = ids >= 0
    for x, y in ((gt, t), (gu, u), (gv, v)):
        assert np.array_equal(x[hit], y[hit].astype(np.float32))
    dev.close()
