"""Which trees the default mode traverses nearest first, and that it answers
nearly all rays so: equal hits alone would not show it, as every ray may be
handed on to the ordered kernels and every tree left to them."""
import numpy as np
import pytest

import oracle
from lucent_gb300 import DeviceBVH, bvh, mesh, workloads
from refcases import LCG, random_soup

pytestmark = pytest.mark.gpu

KNOT = mesh.torus_knot(tubular_segments=120, radial_segments=16).positions


def _info(ob, pos, rays):
    dev = DeviceBVH(ob.nodes, ob.tri_indices, np.asarray(pos, np.float32), ob.node_count)
    assert dev.near_info() == (False, 0.0, 0)
    dev.intersect(rays)
    out = dev.near_info()
    dev.close()
    return out


def _rays(n, seed=1):
    return workloads.sphere_rays(np.random.Generator(np.random.PCG64(seed)), n)


@pytest.mark.parametrize("n", [1, 4099, 100_000])
def test_used_on_what_the_builder_makes(n):
    soup, chords = workloads.soup_and_rays(seed=0, n_tri=20_000, n_rays=n)
    for pos, rays in ((KNOT, _rays(n)), (soup, chords)):
        b = bvh.build_bvh(np.asarray(pos, np.float32).reshape(-1))
        b._device.intersect(rays)
        usable, reach, handed = b._device.near_info()
        diag = float(np.linalg.norm(np.subtract(b.bounds.max, b.bounds.min)))
        assert usable and reach >= 1.99 * diag * (1 - 1e-5)
        assert handed <= n // 100  # ties that the proof leaves open


def test_far_and_unsafe_rays_are_handed_on():
    ob = oracle.build_bvh(KNOT)
    rays = _rays(6000, 2)
    rays[:1000, :3] *= 1e6            # beyond any reach, towards the tree
    d = -rays[:1000, :3].astype(np.float64)
    rays[:1000, 3:] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[1000:1500, 4] = 0.0          # a zero component
    rays[1500:2000, 3:] *= 5.0        # |d| above 2
    usable, _, handed = _info(ob, KNOT, rays)
    assert usable and 500 <= handed <= 2000 + 60


def test_not_used_where_it_proves_nothing():
    pos = np.asarray(KNOT, np.float32)
    assert not _info(oracle.build_bvh(pos * np.float32(3000)), pos * np.float32(3000), _rays(1000) * 3000)[0]
    ob = oracle.build_bvh(pos)  # leaves that do not hold their triangles
    nodes = ob.nodes.reshape(-1, 8)
    leaf = nodes[:, 7] > 0
    half = 0.25 * (nodes[leaf, 4:7] - nodes[leaf, 0:3])
    nodes[leaf, 0:3] += half
    nodes[leaf, 4:7] -= half
    assert not _info(ob, pos, _rays(1000))[0]
    soup = np.asarray(random_soup(1200, LCG(5)), np.float32)
    assert not _info(oracle.build_bvh(soup, 300), soup, _rays(1000))[0]  # leaves of more than 255
    assert _info(oracle.build_bvh(soup, 60), soup, _rays(1000))[0]
