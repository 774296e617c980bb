"""The backward pass keeps 9 bytes a path and bounce beside the paths
themselves. Where that does not fit for all samples at once it takes them in
smaller waves; it gives up only where one sample does not fit. It is sized by
its own samples, not by the largest wave the renderer ever traced. On the fake
runtime."""
import ctypes as C

import numpy as np
import pytest

import fakecuda as F
from lucent_gb300 import _native as N
from lucent_gb300 import _native_render as R

SIDE, BOUNCES, SAMPLES = 16, 64, 8


def _bytes(samples):
    paths = SIDE * SIDE * samples
    return paths * 16 + paths * (BOUNCES + 1) * 9 + (BOUNCES + 1) * 4


@pytest.fixture
def renderer():
    L = F.library()
    r = F.renderer(SIDE, SIDE)
    assert F.load_scene(r, F.triangles(20)) == 0
    s = R.SettingsDesc(BOUNCES, 10.0, 0)
    assert L.lucent_renderer_apply_settings(r, C.byref(s)) == 0
    F.clear()
    yield r
    F.fail(0, 0, 0)
    L.lucent_renderer_destroy(r)


def _backward(r):
    dl, dm = np.ones((SIDE, SIDE, 4), np.float32), np.zeros((1, 6), np.float32)
    return F.library().lucent_renderer_backward(r, SAMPLES, 1, N.ptr(dl, C.c_float), N.ptr(dm, C.c_float), None, None)


@pytest.mark.parametrize("fits,waves", [(8, 1), (4, 2), (3, 4), (1, 8)])
def test_waves_that_fit(renderer, fits, waves):
    # the path state is larger than some of this: made before the limit
    assert F.library().lucent_renderer_trace(renderer, SAMPLES, None) == 0
    F.clear()
    F.fail(_bytes(fits) + 1, 1 << 40, 100)
    assert _backward(renderer) == 0, F.library().lucent_last_error()
    assert len(F.calls("launch", "k_seed_lrem")) == waves


def test_one_sample_does_not_fit(renderer):
    assert F.library().lucent_renderer_trace(renderer, SAMPLES, None) == 0
    F.fail(_bytes(1), 1 << 40, 100)
    assert _backward(renderer) == 3
    F.fail(0, 0, 0)
    assert _backward(renderer) == 0


def test_sized_by_its_own_samples(renderer):
    assert F.library().lucent_renderer_trace(renderer, 100 * SAMPLES, None) == 0
    F.clear()
    assert _backward(renderer) == 0
    assert max(int(x.split()[2]) for x in F.calls("alloc")) <= _bytes(SAMPLES)
