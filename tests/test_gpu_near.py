"""Nearest-first closest hit (lucent_gb300/csrc/traverse_near.cuh) where it can
go wrong: ray counts around a warp and around one ray per warp, rays it hands
to the ordered kernels (far origins, long directions, tiny components), trees
it must not be used on (units where |det| >= 1e-12 bounds nothing, leaves that
do not hold their triangles, leaves of more than 255 triangles), one huge
triangle among small ones, and t_max exactly at hits. Ids, t, u, v equal the
oracle's intersectBVH."""
import math

import numpy as np
import pytest

import oracle
from lucent_gb300 import DeviceBVH, mesh, workloads
from refcases import LCG, random_soup

pytestmark = pytest.mark.gpu


def _check(pos, rays, t_min=1e-5, t_max=math.inf, ob=None, max_leaf=4):
    pos = np.asarray(pos, np.float32)
    ob = ob or oracle.build_bvh(pos, max_leaf)
    dev = DeviceBVH(ob.nodes, ob.tri_indices, pos, ob.node_count)
    ids, t, u, v = oracle.intersect_bvh(ob, pos, rays, t_min, t_max)
    p, gt, gu, gv = dev.intersect(rays, t_min, t_max)
    assert np.array_equal(p, ids)
    hit = ids >= 0
    for a, b in ((gt, t), (gu, u), (gv, v)):
        assert np.array_equal(a[hit], b[hit].astype(np.float32))
    assert np.all(np.isinf(gt[~hit]))
    dev.close()
    return ids, t


KNOT = mesh.torus_knot(tubular_segments=120, radial_segments=16).positions


@pytest.mark.parametrize("n", [1, 31, 33, 4097, 10_000, 40_001])
def test_ray_counts(n):
    ids, _ = _check(KNOT, workloads.sphere_rays(np.random.Generator(np.random.PCG64(n)), n))
    assert n < 1000 or 0.05 < (ids >= 0).mean() < 1


@pytest.mark.parametrize("scale", [1e-3, 30.0, 3000.0])
def test_units(scale):
    rays = workloads.sphere_rays(np.random.Generator(np.random.PCG64(1)), 5000)
    rays[:, :3] *= np.float32(scale)
    _check(KNOT * np.float32(scale), rays, 1e-5 * scale)


def test_rays_outside_the_proven_range():
    rays = workloads.sphere_rays(np.random.Generator(np.random.PCG64(2)), 6000)
    rays[:1000, :3] *= 20.0                 # far origins
    rays[1000:2000, 3:] *= 5.0              # |d| above 2
    rays[2000:3000, 3:] *= 0.01
    rays[3000:3500, 3] = 1e-12              # tiny components
    rays[3500:4000, 4] = 0.0
    _check(KNOT, rays)


def test_one_huge_triangle():
    pos = np.concatenate([KNOT.reshape(-1), np.array([-40, -0.3, -30, 45, 0.2, -35, 3, 0.4, 60], np.float32)])
    rays = workloads.sphere_rays(np.random.Generator(np.random.PCG64(4)), 8000)
    _check(pos, rays)
    _check(pos, workloads.adversarial_rays(pos, np.random.Generator(np.random.PCG64(5)), 500))


def test_leaves_that_do_not_hold_their_triangles():
    ob = oracle.build_bvh(KNOT)
    nodes = ob.nodes.reshape(-1, 8)
    leaf = nodes[:, 7] > 0
    mid = 0.5 * (nodes[leaf, 0:3] + nodes[leaf, 4:7])
    nodes[leaf, 0:3] = 0.5 * (nodes[leaf, 0:3] + mid)
    nodes[leaf, 4:7] = 0.5 * (nodes[leaf, 4:7] + mid)
    _check(KNOT, workloads.sphere_rays(np.random.Generator(np.random.PCG64(6)), 5000), ob=ob)


def test_leaves_of_many_triangles():
    soup = random_soup(1200, LCG(5))
    rays = workloads.sphere_rays(np.random.Generator(np.random.PCG64(7)), 3000)
    rays[:, :3] *= 4.0
    _check(soup, rays, max_leaf=300)
    _check(soup, rays, max_leaf=60)


def test_t_max_at_hits():
    rays = workloads.sphere_rays(np.random.Generator(np.random.PCG64(8)), 300)
    ids, t = _check(KNOT, rays)
    for k in np.nonzero(ids >= 0)[0][:6]:
        for t_max in (t[k], np.nextafter(t[k], 0), np.nextafter(t[k], 9)):
            _check(KNOT, rays, 1e-5, float(t_max))
