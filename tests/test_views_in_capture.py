"""A handle's views in a stream capture, on the fake runtime: what a capture
records has not run, so a view built in one would be read before it is there."""
import pytest

import fakecuda as F

USABLE, UNUSABLE = 1.0, 1e10  # beyond 1e9 across, a tree is not traversed nearest first


@pytest.mark.parametrize("size", [USABLE, UNUSABLE])
def test_first_call_captured(size):
    b, s = F.create(size=size), F.stream()
    L = F.library()
    L.lucent_bvh_set_mode(b.h, 0)
    assert F.intersect(b, 10, s) == 0  # scratch is there, views are not
    L.lucent_bvh_set_mode(b.h, 3)
    F.clear()
    F.begin_capture(s)
    assert F.intersect(b, 10, s) == 0
    F.end_capture(s)
    # the binary nodes, nothing of a view: neither built nor read
    assert F.calls("record", "k_closest_fast_t") and F.calls("record", "k_closest_exact_t")
    assert not F.calls("record", "_wide") and not F.calls("near")
    F.clear()
    assert F.intersect(b, 10, s) == 0  # before any replay: builds them itself
    view = "k_near_records" if size == USABLE else "k_build_wide"
    use = "k_closest_near" if size == USABLE else "k_closest_wide"
    assert len(F.calls("launch", view)) == len(F.calls("launch", use)) == 1
    F.clear()
    F.begin_capture(s)
    assert F.intersect(b, 10, s) == 0
    F.end_capture(s)
    assert F.calls("record", use) and not F.calls("record", view)
    F.library().lucent_bvh_destroy(b.h)


@pytest.mark.parametrize("size", [USABLE, UNUSABLE])
def test_another_stream_finds_them_complete(size):
    b, s, t = F.create(size=size), F.stream(), F.stream()
    F.clear()
    assert F.intersect(b, 10, s) == 0
    built = max(k for k, x in enumerate(F.log()) if "k_build_wide" in x or "k_near_records" in x)
    read = min(k for k, x in enumerate(F.log()) if "k_closest" in x)
    assert "sync stream %d" % F.stream_id(s) in F.log()[built:read]
    F.clear()
    assert F.intersect(b, 10, t) == 0
    assert not F.calls("k_build_wide") and not F.calls("k_near_records")
    F.library().lucent_bvh_destroy(b.h)
