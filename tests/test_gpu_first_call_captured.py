"""A tree whose first nearest-first call is in a stream capture, and is made
directly before the graph is replayed: both answer as the oracle does, over a
tree that is traversed nearest first and over one that is not."""
import numpy as np
import pytest

import oracle
from lucent_gb300 import bvh as B
from lucent_gb300 import workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shrink", [0.0, 0.5])
def test_first_call_captured(shrink):
    pos, rays = workloads.soup_and_rays(seed=4, n_tri=3000, n_rays=20_003)
    ob = oracle.build_bvh(pos)
    nodes = ob.nodes.reshape(-1, 8)
    leaf = nodes[:, 7] > 0
    half = 0.5 * shrink * (nodes[leaf, 4:7] - nodes[leaf, 0:3])
    nodes[leaf, 0:3] += half  # leaves that do not hold their triangles
    nodes[leaf, 4:7] -= half
    want = oracle.intersect_bvh(ob, pos, rays)
    dev = B.DeviceBVH(ob.nodes, ob.tri_indices, pos, ob.node_count)
    n = len(rays)
    r = torch.from_numpy(rays).cuda()

    def outs():
        return [torch.zeros(n, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(3)]

    def call(o, stream):
        dev.intersect_device(r.data_ptr(), n, *(x.data_ptr() for x in o), stream=stream.cuda_stream)

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graphed, direct = outs(), outs()
    dev.set_mode(False, True, False)
    with torch.cuda.stream(s):
        call(graphed, s)  # scratch is made outside the capture
    s.synchronize()
    dev.set_mode(False)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        call(graphed, s)
    call(direct, torch.cuda.current_stream())
    dev.check()
    for x in graphed:
        x.zero_()
    g.replay()
    torch.cuda.synchronize()
    hit = want[0] >= 0
    assert 0.01 < hit.mean() < 1
    for got in (direct, graphed):
        assert np.array_equal(got[0].cpu().numpy(), want[0])
        for x, y in zip(got[1:], want[1:]):
            assert np.array_equal(x.cpu().numpy()[hit], y[hit].astype(np.float32))
