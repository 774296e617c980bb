"""The library on a CUDA runtime without a GPU (fake_cudart.cpp): its own
objects, linked against host memory and a log of what it asked CUDA to do."""
import ctypes as C
import functools
import os
import subprocess
import tempfile
import types

import numpy as np

from lucent_gb300 import _native as N
from lucent_gb300 import _native_render as R
from lucent_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@functools.lru_cache(maxsize=None)
def library():
    B.build()
    objs = [os.path.join(B.BUILD, s[:-3] + ".o") for s in B.sources()]
    out = os.path.join(tempfile.mkdtemp(prefix="lucent_fake_"), "liblucent_fake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    # -Bsymbolic: the fake answers this library only, whatever runtime the process has loaded
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + inc,
                           os.path.join(HERE, "fake_cudart.cpp"), *objs, "-o", out])
    L = C.CDLL(out)
    N._declare(L)
    L.fake_log.restype = C.c_char_p
    L.fake_fail.argtypes = [C.c_size_t, C.c_size_t, C.c_int, C.c_int]
    L.fake_fail.restype = L.fake_clear.restype = None
    L.fake_live.restype = C.c_size_t
    L.fake_id.argtypes = [C.c_void_p]
    L.fake_id.restype = C.c_ulonglong
    L.cudaStreamCreateWithFlags.argtypes = [C.POINTER(C.c_void_p), C.c_uint]
    L.cudaStreamBeginCapture.argtypes = [C.c_void_p, C.c_int]
    L.cudaStreamEndCapture.argtypes = [C.c_void_p, C.POINTER(C.c_void_p)]
    return L


def log():
    return library().fake_log().decode().splitlines()


def clear():
    library().fake_clear()


def calls(*words):
    """The log's lines that hold all of the words."""
    return [x for x in log() if all(w in x for w in words)]


def fail(low, high, times=1, after=0):
    """Refuses `times` allocations of low to high bytes, once `after` of them were made; fail(0, 0, 0): none."""
    library().fake_fail(low, high, times, after)


def stream():
    s = C.c_void_p()
    assert library().cudaStreamCreateWithFlags(C.byref(s), 1) == 0
    return s


def stream_id(s):
    return int(library().fake_id(s))


def begin_capture(s):
    assert library().cudaStreamBeginCapture(s, 1) == 0


def end_capture(s):
    assert library().cudaStreamEndCapture(s, C.byref(C.c_void_p())) == 0


def triangles(n, size=1.0):
    """n triangles in a row along x."""
    p = np.zeros((n, 3, 3), np.float32)
    p[:, 1, 1] = p[:, 2, 2] = 0.5
    p[:, :, 0] = np.arange(n, dtype=np.float32)[:, None]
    return p * np.float32(size)


def tree(pos):
    """Reference-layout nodes over the triangles in order, halved down to single ones."""
    lo, hi = pos.min(1), pos.max(1)
    nodes = []

    def fill(at, a, b):
        box = [*lo[a:b].min(0)], [*hi[a:b].max(0)]
        if b - a == 1:
            nodes[at] = [*box[0], a, *box[1], 1]
            return
        kids = len(nodes)
        nodes[at] = [*box[0], kids, *box[1], 0]
        nodes.extend([None, None])
        m = (a + b) // 2
        fill(kids, a, m)
        fill(kids + 1, m, b)

    nodes.append(None)
    fill(0, 0, len(pos))
    return np.array(nodes, np.float32).reshape(-1)


def create(n=5, size=1.0):
    """A handle over n triangles, and the memory that its calls are given."""
    L = library()
    pos = triangles(n, size)
    nodes, idx = tree(pos), np.arange(n, dtype=np.uint32)
    h = C.c_void_p()
    st = L.lucent_bvh_create(N.ptr(nodes, C.c_float), nodes.size // 8, N.ptr(idx, C.c_uint32), n,
                             N.ptr(pos, C.c_float), C.byref(h))
    assert st == 0, L.lucent_last_error()
    return types.SimpleNamespace(h=h, n=n)


def intersect(b, n, s=None):
    L = library()
    mem = [np.zeros(max(1, n) * w, np.float32) for w in (6, 1, 1, 1, 1)]
    return L.lucent_bvh_intersect_device(b.h, mem[0].ctypes.data, n, 0.0, float("inf"), *(m.ctypes.data for m in mem[1:]),
                                         s)


def renderer(w=8, h=8):
    L = library()
    r = C.c_void_p()
    assert L.lucent_renderer_create(w, h, C.byref(r)) == 0, L.lucent_last_error()
    env = np.ones((4, 8, 3), np.float32)
    light = R.LightingDesc(env_width=8, env_height=4, env_rgb=N.ptr(env, C.c_float), env_rotation_cos=1.0,
                           env_intensity=1.0)
    assert L.lucent_renderer_upload_lighting(r, C.byref(light)) == 0, L.lucent_last_error()
    return r


def load_scene(r, pos, nodes=None, **more):
    """Loads triangles with their tree (halved in order unless given) and a grey material; the call's status."""
    L = library()
    n = len(pos)
    nodes = tree(pos) if nodes is None else nodes
    idx, mat, grey = np.arange(n, dtype=np.uint32), np.zeros(n, np.int32), np.zeros(40, np.float32)
    grey[:3], grey[16:20] = 0.5, -1
    d = R.SceneDesc(tri_count=n, positions=N.ptr(pos, C.c_float), normals=N.ptr(pos, C.c_float),
                    tri_material=N.ptr(mat, C.c_int32), bvh_nodes=N.ptr(nodes, C.c_float),
                    bvh_node_count=nodes.size // 8, bvh_tri_indices=N.ptr(idx, C.c_uint32),
                    materials=N.ptr(grey, C.c_float), material_count=1, ground_material=-1, **more)
    return L.lucent_renderer_load_scene(r, C.byref(d))
