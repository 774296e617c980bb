"""The builder where small builds change form: around their subtrees (256 and
512 triangles) and the sizes at which those and the cluster's share of the
levels end; node arrays and triIndices equal the oracle's buildBVH."""
import numpy as np
import pytest

import oracle
from lucent_gb300 import bvh as B
from lucent_gb300 import mesh, workloads

pytestmark = pytest.mark.gpu


def _same(pos, max_leaf=4, bins=12):
    pos = np.asarray(pos, np.float32).reshape(-1)
    ob = oracle.build_bvh(pos, max_leaf, bins)
    gb = B.build_bvh(pos, max_leaf, bins)
    assert gb.node_count == ob.node_count
    assert np.array_equal(gb.tri_indices, ob.tri_indices)
    assert np.array_equal(gb.nodes, ob.nodes)


@pytest.mark.parametrize("n", [255, 256, 257, 4095, 4096, 4097, 8193, 12287, 12288, 12289])
def test_small_sizes(n):
    _same(workloads.soup_and_rays(seed=n, n_tri=n, n_rays=1)[0])


@pytest.mark.parametrize("n,bins,leaf", [(4000, 32, 300), (4000, 2, 1), (12000, 32, 600), (12000, 3, 1)])
def test_small_options(n, bins, leaf):
    _same(workloads.soup_and_rays(seed=bins, n_tri=n, n_rays=1)[0], leaf, bins)


def test_small_uneven_splits():
    # every split leaves nearly all triangles on one side: many more levels than halving takes
    x = (2.0 ** -np.arange(0, 100, 0.0082)).astype(np.float32)
    t = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32) * 1e-3
    _same(t[None] * x[:, None, None] + np.stack([x, np.zeros_like(x), np.zeros_like(x)], 1)[:, None, :])


def test_small_knot():
    _same(mesh.torus_knot(tubular_segments=300, radial_segments=20).positions)
