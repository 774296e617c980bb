"""The argument of the nearest-first traversal (lucent_gb300/csrc/traverse_near.cuh)
checked on the CPU, without a traversal: among all triangles the reference's
binary64 test accepts in leaves whose binary64 slab test passes, the least t
(the lowest slot among equals) is intersectBVH's hit whenever that triangle's
leaf begins at or before its t, or no other accepted t lies between the two.
The tests are the oracle's own (aabb_intersect, intersect_triangle); soups,
a closed mesh and coplanar, flat geometry with adversarial rays."""
import math

import numpy as np
import pytest

import oracle
from lucent_gb300 import mesh, workloads
from refcases import LCG, random_soup


def _leaf_of(nodes, node_count, n_tri):
    nd = np.asarray(nodes, np.float64).reshape(-1, 8)[:node_count]
    out = np.zeros(n_tri, np.int64)
    for n in range(node_count):
        if nd[n, 7] > 0:
            out[int(nd[n, 3]):int(nd[n, 3] + nd[n, 7])] = n
    return nd, out


def _flat():
    parts = [mesh.quad((-2, 0, 2), (2, 0, 2), (2, 0, -2), (-2, 0, -2)), mesh.quad((2, 0, 2), (2, 0, -2), (-2, 0, -2), (-2, 0, 2)),
             mesh.transform(mesh.box((-0.3, 0.0, -0.3), (0.3, 1.2, 0.3)), translate=(-0.4, 0.0, -0.35), rotate_y=0.4),
             mesh.quad((-1, 0.6, 1), (1, 0.6, 1), (1, 0.6, -1), (-1, 0.6, -1))]
    return mesh.merge_meshes(parts).positions


@pytest.mark.parametrize("name", ["soup", "knot", "flat", "single"])
def test_least_t_is_the_references_hit(name):
    pos = {"soup": lambda: random_soup(300, LCG(7)), "flat": _flat, "single": lambda: np.array([0, 0, 0, 1, 0, 0, 0, 1, 0], np.float32),
           "knot": lambda: mesh.torus_knot(tubular_segments=30, radial_segments=6).positions}[name]()
    pos = np.asarray(pos, np.float32)
    ob = oracle.build_bvh(pos)
    nd, leaf = _leaf_of(ob.nodes, ob.node_count, ob.tri_indices.size)
    rays = workloads.adversarial_rays(pos, np.random.Generator(np.random.PCG64(3)), 12)
    v = pos.reshape(-1, 3, 3).astype(np.float64)[ob.tri_indices]
    ids, _, _, _ = oracle.intersect_bvh(ob, pos, rays, 1e-6, math.inf)
    decided = 0
    for ray, want in zip(rays.astype(np.float64), ids):
        o, d = ray[:3], ray[3:]
        inv = np.array([1.0 / x if x != 0 else math.copysign(math.inf, x) for x in d])
        if not np.all(np.isfinite(inv)):
            continue  # the fast paths leave such rays to the binary64 kernel
        hits = []
        for s in range(leaf.size):
            e = oracle.aabb_intersect(nd[leaf[s], 0:3], nd[leaf[s], 4:7], o, inv, math.inf)
            if e == math.inf:
                continue
            h = oracle.intersect_triangle(o, d, v[s, 0], v[s, 1], v[s, 2], 1e-6, math.inf)
            if h is not None:
                hits.append((h[0], s, e))
        if not hits:
            assert want < 0
            decided += 1
            continue
        t, s, e = min(hits)
        if e <= t or not any(t <= x[0] <= e for x in hits if x[1] != s):
            assert ob.tri_indices[s] == want
            decided += 1
    assert decided > 0.5 * len(rays) or name == "single"


def _growth(v, diag):
    """leaf_growth (lucent_gb300/csrc/near_build.cu) in binary64."""
    e1, e2 = v[1] - v[0], v[2] - v[0]
    l1, l2, area2 = np.linalg.norm(e1), np.linalg.norm(e2), np.linalg.norm(np.cross(e1, e2))
    reach = 10 * diag + 3 * max(l1, l2)
    least = reach * 2.0 ** -28
    if np.any((v[0] == v[1]) & (v[0] == v[2])) and l1 * l2 <= 65536 * area2:
        return least
    k = 2.1e-3 * l1 * l2 / max(1 - 1.8e-3 * l1 * l2, 1e-6)
    return k * reach / (1 - k) + least if k < 0.5 else math.inf


@pytest.mark.parametrize("seed", range(3))
def test_accepted_points_lie_in_the_grown_box(seed):
    """Grazing and edge-on rays, where binary64's t, u, v are worst: the point
    the reference accepts is never outside its triangle's box by more than the
    growth the view allows for."""
    rng = np.random.Generator(np.random.PCG64(seed))
    worst = accepted = 0
    for _ in range(4000):
        v = rng.uniform(-1, 1, (3, 3)) if rng.random() < 0.5 else rng.uniform(-1, 1, 3) + rng.normal(0, 0.03, (3, 3))
        v = v.astype(np.float32).astype(np.float64)
        if rng.random() < 0.2:
            v[:, rng.integers(3)] = v[0, 0]
        diag = 2 * math.sqrt(3.0)
        g = _growth(v, diag)
        # a point of the triangle (a vertex, an edge point or inside) and a direction within 10^-k of its plane
        w = rng.dirichlet((0.3, 0.3, 0.3))
        p = w @ v
        d = (v[1] - v[0]) * rng.normal() + (v[2] - v[0]) * rng.normal()
        n = np.cross(v[1] - v[0], v[2] - v[0])
        d = d / np.linalg.norm(d) + n / max(np.linalg.norm(n), 1e-30) * 10.0 ** -rng.uniform(0, 12)
        d /= np.linalg.norm(d)
        o = (p - d * rng.uniform(0.01, 3)).astype(np.float32).astype(np.float64)
        d = d.astype(np.float32).astype(np.float64)
        h = oracle.intersect_triangle(o, d, v[0], v[1], v[2], 0.0, math.inf)
        if h is None:
            continue
        accepted += 1
        x = o + h[0] * d
        out = max(np.max(v.min(0) - x), np.max(x - v.max(0)), 0.0)
        assert out <= g, (v, o, d, out, g)
        worst = max(worst, out / g)
    assert accepted > 500 and worst < 1.0
