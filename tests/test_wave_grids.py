"""shade_blocks sets how many threads a batch's shade, sort and shadow kernels
get, in blocks of 128 for shading whatever block size a wave's size selects,
and trace_blocks those of its closest-hit kernels, in blocks of 256; 0: all
resident blocks. On the fake runtime (152 SMs)."""
import ctypes as C

import pytest

import fakecuda as F
from lucent_gb300 import _native_render as R


def _grids(word):
    out = set()
    for x in F.calls("launch", word) + F.calls("record", word):
        w = x.split()
        out.add((int(w[w.index("grid") + 1]), int(w[w.index("block") + 1])))
    return out


@pytest.mark.parametrize("near", [True, False])
@pytest.mark.parametrize("shade_blocks", [0, 1, 152, 152 * 3, 152 * 8])
@pytest.mark.parametrize("trace_blocks", [0, 100, 10_000])
@pytest.mark.parametrize("side", [64, 1024])  # waves of 2^13 and 2^21 paths
def test_batch_grids(side, trace_blocks, shade_blocks, near):
    L = F.library()
    r = F.renderer(side, side)
    assert F.load_scene(r, F.triangles(20, 1.0 if near else 1e10)) == 0
    b = C.c_void_p()
    assert L.lucent_batch_create((C.c_void_p * 1)(r), 1, C.byref(b)) == 0
    o = R.BatchOptions(0, 1 << 21, 1, trace_blocks, shade_blocks, 1, 1, 1, 0, 1)
    assert L.lucent_batch_set_options(b, C.byref(o)) == 0
    F.clear()
    assert L.lucent_batch_trace(b, 2, None) == 0, L.lucent_last_error()
    ((grid, threads),) = _grids("k_shade_t")
    assert threads == (512 if side == 1024 else 256)
    assert grid == (max(1, shade_blocks * 128 // threads) if shade_blocks else 152 * 512 // threads)
    if near:
        ((grid, threads),) = _grids("k_anyhit_near")
        assert grid == min(4 * shade_blocks or 1 << 30, 152 * 4) and threads == 128
    else:
        ((grid, threads),) = _grids("k_anyhit_wide")
        assert threads == 256 and (not shade_blocks or grid == 2 * shade_blocks)
    if near:
        ((grid, threads),) = _grids("k_closest_near")
        assert grid == min(2 * trace_blocks or 1 << 30, 152 * 4) and threads == 128
    ((grid, threads),) = _grids("k_closest_wide")
    assert threads == 256 and (not trace_blocks or grid == trace_blocks)
    ((grid, threads),) = _grids("k_sort_keys")
    assert threads == 256 and (not shade_blocks or grid == shade_blocks)
    L.lucent_batch_destroy(b)
    L.lucent_renderer_destroy(r)
