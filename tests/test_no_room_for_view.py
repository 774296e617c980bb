"""The nearest-first view only saves time: where there is no memory for it, a
scene loads and a handle answers in the reference's order, as without it."""
import pytest

import fakecuda as F

N_TRIS = 300
N_NODES = 2 * N_TRIS - 1
RECORDS, SCRATCH = N_NODES * 128, N_NODES * 44 + 64


@pytest.fixture(autouse=True)
def _fake():
    F.clear()
    yield
    F.fail(0, 0, 0)


# An allocation is tried twice; the four-wide view is as large as the records.
@pytest.mark.parametrize("size", [RECORDS, SCRATCH])
def test_handle(size):
    b = F.create(N_TRIS)
    F.fail(size, size, 2)
    assert F.intersect(b, 10) == 0
    assert len(F.calls("refuse")) == 2 and F.calls("launch", "k_closest_wide") and not F.calls("launch", "near")
    F.clear()
    assert F.intersect(b, 10) == 0  # not tried again
    assert F.calls("k_closest_wide") and not F.calls("near") and not F.calls("alloc")
    F.library().lucent_bvh_destroy(b.h)


@pytest.mark.parametrize("size,after", [(RECORDS, 1), (SCRATCH, 0)])
def test_scene(size, after):
    L = F.library()
    r = F.renderer()
    assert F.load_scene(r, F.triangles(N_TRIS)) == 0
    F.clear()
    assert L.lucent_renderer_trace(r, 1, None) == 0
    assert F.calls("k_closest_near")
    L.lucent_renderer_destroy(r)
    r = F.renderer()
    F.clear()
    F.fail(size, size, 2, after)
    assert F.load_scene(r, F.triangles(N_TRIS)) == 0, L.lucent_last_error()
    assert len(F.calls("refuse")) == 2
    F.clear()
    assert L.lucent_renderer_trace(r, 1, None) == 0, L.lucent_last_error()
    assert F.calls("k_closest_wide") and F.calls("k_anyhit_wide") and not F.calls("near")
    L.lucent_renderer_destroy(r)
