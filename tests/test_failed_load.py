"""After a scene load that failed midway (here a tree too deep for the
reference's stack) a renderer has no scene: parts of the last one are already
overwritten, so tracing it is refused until a load succeeds."""
import numpy as np

import fakecuda as F


def _chain(pos):
    """A tree that splits one triangle off at a time."""
    nodes = []
    for k in range(len(pos)):
        for a, b in ((k - 1, k), (k, len(pos))) if k else ((0, len(pos)),):
            lo, hi = pos[a:b].min((0, 1)), pos[a:b].max((0, 1))
            leaf = b - a == 1
            nodes.append([*lo, a if leaf else len(nodes) + (2 if a < k else 1), *hi, 1 if leaf else 0])
    out = np.array(nodes, np.float32)
    inner = np.nonzero(out[:, 7] == 0)[0]
    out[inner, 3] = 2 * np.arange(len(inner)) + 1
    return out.reshape(-1)


def test_no_scene_after_a_failed_load():
    L = F.library()
    r = F.renderer()
    assert L.lucent_renderer_trace(r, 1, None) == 1  # no scene yet
    assert F.load_scene(r, F.triangles(200)) == 0, L.lucent_last_error()
    assert L.lucent_renderer_trace(r, 1, None) == 0, L.lucent_last_error()
    pos = F.triangles(100)
    assert F.load_scene(r, pos, _chain(pos)) == 5 and b"deeper" in L.lucent_last_error()
    F.clear()
    assert L.lucent_renderer_trace(r, 1, None) == 1
    assert not F.calls("launch") and not F.calls("replay")
    assert F.load_scene(r, pos) == 0
    assert L.lucent_renderer_trace(r, 1, None) == 0
    L.lucent_renderer_destroy(r)


def test_a_refused_description_changes_nothing():
    L = F.library()
    r = F.renderer()
    assert F.load_scene(r, F.triangles(20)) == 0
    bad = F.triangles(20)
    bad[3, 1, 2] = np.nan
    assert F.load_scene(r, bad, F.tree(F.triangles(20))) == 5
    assert F.load_scene(r, F.triangles(20), sphere_count=65) == 1
    assert L.lucent_renderer_trace(r, 1, None) == 0
    L.lucent_renderer_destroy(r)
