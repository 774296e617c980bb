"""Binary64 pick rays a warp each (k_pick, lucent_gb300/csrc/closest_hit.cu):
ray counts around the argument block and past the warp path, rays it hands to
one lane's walk (zero components, infinite ranges, equal distances), flat
geometry whose boxes begin at the hit, and trees whose leaves are not in slot
order (there for the binary32 path too). Ids, t, u, v equal the oracle's
intersectBVH in binary64."""
import math

import numpy as np
import pytest

import oracle
from lucent_gb300 import DeviceBVH, mesh, workloads
from refcases import LCG, random_soup

pytestmark = pytest.mark.gpu

KNOT = mesh.torus_knot(tubular_segments=120, radial_segments=16).positions
FLAT = mesh.merge_meshes([
    mesh.quad((-2, 0, 2), (2, 0, 2), (2, 0, -2), (-2, 0, -2)), mesh.quad((2, 0, 2), (2, 0, -2), (-2, 0, -2), (-2, 0, 2)),
    mesh.transform(mesh.box((-0.3, 0.0, -0.3), (0.3, 1.2, 0.3)), translate=(-0.4, 0.0, -0.35), rotate_y=0.4),
    mesh.quad((-1, 0.6, 1), (1, 0.6, 1), (1, 0.6, -1), (-1, 0.6, -1))]).positions


def _check(pos, rays, t_min=1e-5, t_max=math.inf, ob=None):
    pos = np.asarray(pos, np.float32)
    ob = ob or oracle.build_bvh(pos)
    dev = DeviceBVH(ob.nodes, ob.tri_indices, pos, ob.node_count)
    rays = np.asarray(rays, np.float64)
    ids, t, u, v = oracle.intersect_bvh(ob, pos, rays, t_min, t_max)
    p, gt, gu, gv = dev.intersect_f64(rays, t_min, t_max)
    assert np.array_equal(p, ids)
    hit = ids >= 0
    assert np.array_equal(gt[hit], t[hit]) and np.array_equal(gu[hit], u[hit]) and np.array_equal(gv[hit], v[hit])
    assert np.all(np.isinf(gt[~hit]))
    p32, t32, _, _ = dev.intersect(rays.astype(np.float32), t_min, t_max)
    i32, o32, _, _ = oracle.intersect_bvh(ob, pos, rays.astype(np.float32), t_min, t_max)
    assert np.array_equal(p32, i32) and np.array_equal(t32[i32 >= 0], o32[i32 >= 0].astype(np.float32))
    dev.close()
    return ids


@pytest.mark.parametrize("n", [1, 31, 32, 33, 700, 2736, 2737])
def test_ray_counts(n):
    _check(KNOT, workloads.sphere_rays(np.random.Generator(np.random.PCG64(n)), n))


@pytest.mark.parametrize("name", ["knot", "flat", "soup", "single"])
@pytest.mark.parametrize("t_min,t_max", [(1e-5, math.inf), (0.0, 1.5)])
def test_adversarial(name, t_min, t_max):
    pos = {"knot": KNOT, "flat": FLAT, "soup": random_soup(400, LCG(3)),
           "single": np.array([0, 0, 0, 1, 0, 0, 0, 1, 0], np.float32)}[name]
    rays = workloads.adversarial_rays(np.asarray(pos, np.float32), np.random.Generator(np.random.PCG64(1)), 150)
    _check(pos, rays, t_min, t_max)


def test_many_equal_triangles():
    soup = np.tile(np.array([0, 0, 0, 1, 0, 0, 0, 1, 0], np.float32), 300)
    rays = [[0.2, 0.2, -1, 0.0, 0.0, 1], [0.2, 0.3, -1, 0.01, 0.02, 1], [0.1, 0.1, 2, 0.001, 0.002, -1]]
    assert (_check(soup, rays) >= 0).all()


def test_leaves_out_of_slot_order():
    # the same tree with its leaves' triangles laid out in reverse, every triangle doubled
    pos = np.tile(np.asarray(random_soup(300, LCG(9)), np.float32).reshape(-1, 9), (2, 1)).reshape(-1)
    ob = oracle.build_bvh(pos, 2)
    nodes = ob.nodes.reshape(-1, 8)
    order, at = [], 0
    for n in sorted(np.nonzero(nodes[:, 7] > 0)[0], key=lambda n: -nodes[n, 3]):
        first, count = int(nodes[n, 3]), int(nodes[n, 7])
        order.extend(ob.tri_indices[first:first + count])
        nodes[n, 3] = at
        at += count
    ob.tri_indices[:] = order
    rays = workloads.sphere_rays(np.random.Generator(np.random.PCG64(2)), 2000)
    rays[:, :3] *= 4.0
    hits = _check(pos, rays, ob=ob)
    assert (hits >= 0).any()
