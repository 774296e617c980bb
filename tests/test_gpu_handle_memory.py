"""Handles closed while their queries are in flight, and built, queried and
closed by several threads: pooled memory that is handed on must not change an
answer."""
import threading

import numpy as np
import pytest

from lucent_gb300 import bvh as B
from lucent_gb300 import workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _soup(seed, tris, rays):
    pos, r = workloads.soup_and_rays(seed=seed, n_tri=tris, n_rays=rays)
    return torch.from_numpy(pos.reshape(-1, 9)).cuda(), torch.from_numpy(r).cuda()


def _query(dev, r, stream):
    prim = torch.full((len(r),), -7, dtype=torch.int32, device="cuda")
    t, u, v = (torch.empty(len(r), device="cuda") for _ in range(3))
    torch.cuda.current_stream().synchronize()
    dev.intersect_device(r.data_ptr(), len(r), *(x.data_ptr() for x in (prim, t, u, v)), stream=stream.cuda_stream)
    return prim, t, u, v  # all kept: the call is not over


def test_closed_in_flight():
    sets = [_soup(k, 20_000 + 3_001 * k, 200_000) for k in range(4)]
    want = []
    for pos, r in sets:
        dev = B.build_device(pos.data_ptr(), len(pos))
        want.append(_query(dev, r, torch.cuda.current_stream()))
        dev.check()
        dev.close()
    streams = [torch.cuda.Stream() for _ in range(6)]
    got = []
    for k in range(24):
        pos, r = sets[k % 4]
        dev = B.build_device(pos.data_ptr(), len(pos))
        for j in range(1 + k % 3):  # a handle has one scratch: its calls follow one another
            if j:
                streams[(k + j) % 6].wait_stream(streams[(k + j - 1) % 6])
            got.append((k % 4, _query(dev, r, streams[(k + j) % 6])))
        dev.close()  # its memory may go to the next build
    torch.cuda.synchronize()
    for k, (prim, t, _, _) in got:
        assert torch.equal(prim, want[k][0]) and torch.equal(t, want[k][1])


def test_replayed_after_the_scratch_grew():
    pos, r = _soup(7, 30_000, 300_000)
    dev = B.build_device(pos.data_ptr(), len(pos))
    few = r[:5_000].clone()
    want = _query(dev, few, torch.cuda.current_stream())
    dev.check()
    s = torch.cuda.Stream()
    o = [torch.zeros_like(x) for x in want]
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        dev.intersect_device(few.data_ptr(), len(few), *(x.data_ptr() for x in o), stream=s.cuda_stream)
    _query(dev, r, torch.cuda.current_stream())  # needs more scratch than the graph's call
    dev.check()
    other = B.build_device(pos.data_ptr(), len(pos))  # what was given back is taken again
    for x in o:
        x.fill_(-9)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(o[0], want[0]) and torch.equal(o[1], want[1])
    other.close()
    dev.close()
    B.trim()


def test_trim_returns_what_builds_leave():
    pos, r = _soup(9, 500_000, 1_000)
    kept = B.build_device(pos.data_ptr(), len(pos))
    want = _query(kept, r, torch.cuda.current_stream())[0]
    B.trim()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        B.build_device(pos.data_ptr(), len(pos)).close()
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    B.trim()
    after = torch.cuda.mem_get_info()[0]
    assert held < before - (64 << 20)  # 168 bytes a triangle of scratch and more of the tree
    assert after >= before - (8 << 20)
    assert torch.equal(_query(kept, r, torch.cuda.current_stream())[0], want)
    kept.check()
    B.build_device(pos.data_ptr(), len(pos)).close()


def test_threads():
    bad = []

    def work(seed):
        try:
            torch.cuda.set_device(0)
            s = torch.cuda.Stream()
            for k in range(6):
                n = 500 + 7_001 * ((seed + k) % 4)
                pos, rays = workloads.soup_and_rays(seed=seed, n_tri=n, n_rays=5_000)
                b = B.build_bvh(pos, stream=s.cuda_stream)
                prim = b._device.intersect(rays, stream=s.cuda_stream)[0]
                again = B.build_bvh(pos, stream=s.cuda_stream)
                if not (np.array_equal(b.nodes, again.nodes)
                        and np.array_equal(prim, again._device.intersect(rays, stream=s.cuda_stream)[0])):
                    bad.append(seed)
                b._device.close()
        except Exception as e:  # noqa: BLE001 (reported below)
            bad.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
