"""A caller's node array may hold leaves that the root never reaches. Such a
leaf must not stand in for the one that the reference visits: here the tree's
own leaf is flat and its binary64 box test rejects some rays that meet its
triangle at the border, which a stray, thicker leaf over the same triangle
would let through."""
import numpy as np
import pytest

import oracle
from lucent_gb300 import DeviceBVH

POS = np.array([[0, 0, 0.25, 1, 0, 0.25, 0, 1, 0.25],
                [2, 2, 2, 3, 2, 2.5, 2, 3, 2.5]], np.float32)


def _node(tris, first, count, grow=0.0):
    v = POS[tris].reshape(-1, 3)
    return [*(v.min(0) - grow), first, *(v.max(0) + grow), count]


def _tree(flat, strays=0):
    """Root, a leaf a triangle, and stray leaves over triangle 0 (thicker than its own when that is flat)."""
    nodes = [_node([0, 1], 1, 0, 0.5), _node([0], 0, 1, 0.0 if flat else 0.25), _node([1], 1, 1)]
    nodes = np.array(nodes + [_node([0], 0, 1, 0.25)] * min(1, strays), np.float32)
    nodes = np.concatenate([nodes, np.repeat(nodes[-1:], max(0, strays - 1), 0)])
    return oracle.BVH(nodes.reshape(-1), len(nodes), np.arange(2, dtype=np.uint32), None)


def _rays(n=20_000):
    """Exactly through points of the triangle's two sides that are its box's border: every number is a small multiple
    of a power of two, so only the box test's reciprocals round."""
    rng = np.random.Generator(np.random.PCG64(11))
    p = np.stack([np.zeros(n), rng.integers(100, 900, n) / 1024, np.full(n, 0.25)], 1)
    p[::2, :2] = p[::2, 1::-1]
    d = np.concatenate([rng.integers(-250, 250, (n, 2)) | 1, -(rng.integers(50, 250, (n, 1)) | 1)], 1) / 256
    return np.concatenate([p - 3 * d, d], 1).astype(np.float32)


def test_the_boxes_matter():
    rays = _rays()
    flat, thick = (oracle.intersect_bvh(_tree(f), POS, rays)[0] for f in (True, False))
    assert (thick == 0).sum() > (flat == 0).sum() + 100
    assert np.array_equal(oracle.intersect_bvh(_tree(True, 400), POS, rays)[0], flat)


@pytest.mark.gpu
@pytest.mark.parametrize("strays", [0, 1, 400, 600_000])  # of the last, most are read after the tree
def test_stray_leaves(strays):
    rays = _rays()
    ob = _tree(True, strays)
    dev = DeviceBVH(ob.nodes, ob.tri_indices, POS, ob.node_count)
    want = oracle.intersect_bvh(ob, POS, rays)[0]
    assert np.array_equal(dev.intersect(rays)[0], want)
    dev.close()
