"""The builder where its kernels meet: sizes around one subtree (1024
triangles) and one chunk, many equal centroids above and below a subtree, bins
at their least and most, centroids on bin boundaries, and scales whose
binary32 areas and extents leave its range; node arrays and triIndices equal
the oracle's buildBVH."""
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


@pytest.mark.parametrize("n", [2, 5, 31, 33, 511, 512, 513, 1023, 1024, 1025, 1026, 2047, 2049, 4097, 9999])
def test_sizes(n):
    _same(workloads.soup_and_rays(seed=n, n_tri=n, n_rays=1)[0])


@pytest.mark.parametrize("bins,leaf", [(2, 1), (3, 4), (12, 1), (31, 4), (32, 1), (12, 900), (12, 3000)])
def test_options(bins, leaf):
    _same(workloads.soup_and_rays(seed=bins, n_tri=5000, n_rays=1)[0], leaf, bins)


@pytest.mark.parametrize("scale", [1e-18, 1e-9, 3e-7, 1e6, 1e15, 3e18])
def test_scales(scale):
    pos = mesh.torus_knot(tubular_segments=90, radial_segments=12).positions
    _same(pos * np.float32(scale))


@pytest.mark.parametrize("cells", [6, 12, 24])
def test_centroids_on_bin_boundaries(cells):
    # a lattice of equal boxes: every centroid a multiple of the bin width, equal extents, equal costs
    g = np.stack(np.meshgrid(*[np.arange(cells + 1)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)
    t = np.array([[-0.25, -0.25, -0.25], [0.25, 0.25, -0.25], [0, 0, 0.25]], np.float32)
    _same(g[:, None, :] + t[None])


@pytest.mark.parametrize("n", [700, 1500, 5000])
def test_equal_centroids(n):
    one = np.tile(np.array([0, 0, 0, 1, 0, 0, 0, 1, 0], np.float32), n)
    _same(np.concatenate([one, workloads.soup_and_rays(seed=1, n_tri=600, n_rays=1)[0]]))


def test_long_chain_of_uneven_splits():
    # centroids in a geometric progression: every split leaves nearly all triangles on one side
    x = (2.0 ** -np.arange(0, 100, 0.03125)).astype(np.float32)
    t = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32) * 1e-3
    _same(t[None] * x[:, None, None] + np.stack([x, np.zeros_like(x), np.zeros_like(x)], 1)[:, None, :])
