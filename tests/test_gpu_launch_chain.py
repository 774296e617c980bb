"""intersect_device inside a caller's CUDA graph: its kernels start early behind
one another (programmatic launches), which a capture has to keep; a replay over
new rays answers them as a direct call does, bit for bit."""
import pytest

from lucent_gb300 import bvh as B
from lucent_gb300 import workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 4099, 200_003])
def test_captured_calls_replay(n):
    pos, rays = workloads.soup_and_rays(seed=3, n_tri=5000, n_rays=2 * n)
    b = B.build_bvh(pos)._device
    both = torch.from_numpy(rays).cuda().reshape(2, n, 6)
    r = both[0].clone()

    def outs():
        return [torch.zeros(n, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(3)]

    def call(o, stream):
        b.intersect_device(r.data_ptr(), n, *(x.data_ptr() for x in o), stream=stream.cuda_stream)

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    got = outs()
    with torch.cuda.stream(s):
        call(got, s)  # scratch and view are made outside the capture
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        call(got, s)
    for k in (1, 0):
        r.copy_(both[k])
        g.replay()
        torch.cuda.synchronize()
        want = outs()
        call(want, torch.cuda.current_stream())
        b.check()
        for x, y in zip(got, want):
            assert torch.equal(x, y)
