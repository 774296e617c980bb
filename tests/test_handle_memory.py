"""The pooled memory of BVH handles, on the fake runtime: it goes back to the
device that it came from, behind the work that may still use it, without a
wait on the host and without touching another thread's capture; what a graph
may still replay stays until the device can be waited for."""
import ctypes as C
import threading

import pytest

import fakecuda as F

L = None


@pytest.fixture(autouse=True)
def _fake():
    global L
    L = F.library()
    F.clear()
    yield
    F.fail(0, 0, 0)
    L.cudaSetDevice(0)


def _on_device(d):
    L.cudaSetDevice(d)
    b = F.create()
    L.cudaSetDevice(0)
    return b


def _order():
    """Each block given back, with the events its stream waited for before."""
    waited, out = {}, []
    for x in F.log():
        w = x.split()
        if w[0] == "wait":
            waited.setdefault(w[3], set()).add(w[1])
        elif x.startswith("give back"):
            out.append((w[2], set(waited.get(w[4], ()))))
    return out


def test_closed_while_another_device_is_current():
    b = _on_device(1)
    own = [x.split()[1] for x in F.calls("alloc", "device 1 pool")]
    assert len(own) == 2  # nodes and triangles
    F.clear()
    L.lucent_bvh_destroy(b.h)
    assert sorted(x.split()[2] for x in F.calls("give back")) == sorted(own)
    assert not F.calls("device 0")  # neither a pool, a stream nor a wait there
    assert L.cudaGetLastError() == 0


def test_grown_while_another_device_is_current():
    b = _on_device(1)
    L.lucent_bvh_set_mode(b.h, 0)  # no views: scratch alone
    F.clear()
    F.fail(1, 1 << 40)  # the first attempt: its own device's pool is trimmed for the second
    F.intersect(b, 1_000)
    assert F.calls("trim device 1") and F.calls("alloc", "device 1 pool") and not F.calls("device 0")
    L.lucent_bvh_destroy(b.h)
    assert L.fake_live(1) == 0


def test_closed_on_another_thread():
    b = _on_device(1)
    F.clear()
    t = threading.Thread(target=L.lucent_bvh_destroy, args=(b.h,))  # device 0 is current there
    t.start()
    t.join()
    assert len(F.calls("give back")) == 2 and not F.calls("device 0")


@pytest.mark.parametrize("streams", [1, 3, 4, 5, 9])
def test_given_back_behind_every_stream(streams):
    b = F.create()
    last = {}
    ss = [F.stream() for _ in range(streams)]
    for s in ss + ss[::2]:
        at = len(F.log())
        assert F.intersect(b, 10, s) == 0
        sid = "stream %d" % F.stream_id(s)
        event = [x for x in F.log()[at:] if x.startswith("event") and x.endswith(sid)]
        assert len(event) == 1 and F.log()[-1] == event[0]  # behind all of the call's work
        last[sid] = (event[0].split()[1], len(F.log()))
    L.lucent_bvh_destroy(b.h)
    text = F.log()
    first_back = next(k for k in reversed(range(len(text))) if not text[k].startswith("give back")) + 1
    for event, at in last.values():  # an event used again stands for another stream: waited for in between
        assert any(x.split()[1] == event for x in text[at:first_back] if x.startswith("wait"))
    assert not F.calls("sync device")


def test_grown_behind_its_last_call():
    b = F.create()
    s, t = F.stream(), F.stream()
    for n, q in ((10, s), (10, t)):
        assert F.intersect(b, n, q) == 0
    events = {x.split()[1] for x in F.calls("event")}
    assert F.intersect(b, 100_000, s) == 0  # more scratch
    (back,) = [x for x in _order() if x[1]]
    assert events <= back[1]
    L.lucent_bvh_destroy(b.h)


def test_another_capture_is_left_alone():
    b, s, other = F.create(), F.stream(), F.stream()
    assert F.intersect(b, 10, s) == 0
    F.begin_capture(other)  # somebody else's, on the same device
    assert F.intersect(b, 100_000, s) == 0
    L.lucent_bvh_destroy(b.h)
    F.end_capture(other)
    assert not F.calls("spoiled") and not F.calls("sync device")
    assert L.fake_live(1) == 0


def test_what_a_graph_holds_stays():
    b, s, other = F.create(), F.stream(), F.stream()
    assert F.intersect(b, 10, s) == 0
    F.begin_capture(s)
    assert F.intersect(b, 10, s) == 0
    F.end_capture(s)
    F.clear()
    assert F.intersect(b, 100_000, s) == 0  # the graph's scratch is not given back
    assert F.calls("alloc") and not F.calls("give back")
    F.begin_capture(other)
    L.lucent_bvh_destroy(b.h)  # replays may be in flight and the device cannot be waited for
    F.end_capture(other)
    kept = L.fake_live(1)
    assert kept >= 4
    F.clear()
    L.lucent_bvh_destroy(F.create().h)
    assert L.fake_live(1) == 0
    text = F.log()
    assert text.index("sync device 0") < [k for k, x in enumerate(text) if x.startswith("give back")][2]


def test_trimmed_without_a_renderer():
    b, s, other = F.create(), F.stream(), F.stream()
    assert F.intersect(b, 10, s) == 0
    F.begin_capture(s)
    assert F.intersect(b, 10, s) == 0
    F.end_capture(s)
    F.begin_capture(other)
    L.lucent_bvh_destroy(b.h)
    assert L.lucent_trim() != 0  # a capture is under way: nothing can be waited for
    F.end_capture(other)
    F.clear()
    assert L.lucent_trim() == 0
    assert L.fake_live(1) == 0 and F.log()[0] == "sync device 0" and F.log()[-1] == "trim device 0"


def test_allocation_after_the_pool_is_trimmed():
    F.fail(1, 1 << 40)
    b = F.create()
    text = F.log()
    refused = next(k for k, x in enumerate(text) if x.startswith("refuse"))
    assert text[refused + 1] == "trim device 0" and text[refused + 2].startswith("alloc")
    F.fail(1, 1 << 40, 100)
    h = C.c_void_p()
    pos = F.triangles(5)
    assert L.lucent_bvh_build_device(pos.ctypes.data, 5, None, C.byref(h), None) == 3  # out of memory
    F.fail(0, 0, 0)
    assert F.intersect(b, 10) == 0
    L.lucent_bvh_destroy(b.h)
    assert L.fake_live(1) == 0
