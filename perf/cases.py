"""The work that programs using this framework have it do, as cases to be timed.

Every case goes through the public entry points (lucent_gb300.bvh, renderer, adjoint): ray queries against a BVH,
BVH builds, path-traced frames with their denoise and display passes, inverse-rendering steps and multi-scene batches.
Sizes come from this repository's tests, workloads and benchmark; `draw` spreads over the same ranges.
"""
import math

import numpy as np
import torch

from lucent_gb300 import adjoint as AD
from lucent_gb300 import bvh as B
from lucent_gb300 import mesh as M
from lucent_gb300 import scene as S
from lucent_gb300 import workloads as W
from lucent_gb300.renderer import Batch, Renderer


def listed():
    return [
        # An editor's click: one binary64 pick ray against a loaded mesh; all latency.
        {"name": "pick", "kind": "pick", "mesh": "knot", "tris": 81_920},
        # A few thousand visibility queries from a device program (line of sight, placement), an odd count.
        {"name": "rays_4k", "kind": "rays", "mesh": "knot", "tris": 20_480, "rays": 4_099, "aim": "sphere",
         "host": False},
        # The benchmark's intersection workload: 10^6 incoherent rays into a soup of 65,536 triangles.
        {"name": "rays_1m_soup", "kind": "rays", "mesh": "soup", "tris": 65_536, "rays": 1_000_000, "aim": "sphere",
         "host": False},
        # A 720p image of primary rays answered for a host program: copies in and out are part of the call.
        {"name": "rays_720p_host", "kind": "rays", "mesh": "knot", "tris": 300_000, "rays": 921_600, "aim": "camera",
         "host": True},
        # buildBVH of a small edited object, a size that is no multiple of anything.
        {"name": "build_2k", "kind": "build", "mesh": "soup", "tris": 2_503},
        # buildBVH of an imported model from host positions (the tests' 300,000-triangle knot).
        {"name": "build_300k", "kind": "build", "mesh": "knot", "tris": 300_000},
        # An animated mesh of 2,000,000 triangles on the device: rebuilt, then queried, each step.
        {"name": "rebuild_2m", "kind": "rebuild", "mesh": "knot", "tris": 2_000_000, "rays": 262_144},
        # The viewer: one sample a frame of a textured model with cut-out alpha while the camera moves
        # (temporal reprojection, denoise, display), a canvas with odd sides.
        {"name": "preview_textured", "kind": "frame", "scene": "textured", "width": 641, "height": 359, "spp": 1,
         "depth": 6, "view": True},
        # The benchmark's frame: the box scene at 512 x 512, 16 samples, depth 8, colour read back.
        {"name": "frame_box", "kind": "frame", "scene": "box", "width": 512, "height": 512, "spp": 16, "depth": 8,
         "view": False},
        # The largest frame: a 2,000,000-triangle knot of layered, glass and blended materials under an HDRI with a
        # thin lens at 1080p, depth 12, with denoise and display.
        {"name": "frame_knot_hd", "kind": "frame", "scene": "knot", "tris": 2_000_000, "width": 1920, "height": 1080,
         "spp": 4, "depth": 12, "view": True},
        # One view of an inverse-rendering iteration: parameters set, forward image, gradients of materials and
        # environment.
        {"name": "inverse_step", "kind": "inverse", "width": 512, "height": 512, "spp": 8, "depth": 8},
        # Progressive updates of several small scenes as one wavefront.
        {"name": "batch_progressive", "kind": "batch", "scenes": 6, "tris": 20_000, "width": 256, "height": 256,
         "spp": 2, "depth": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "build", "rebuild", "frame", "frame", "frame", "inverse", "batch", "pick"])
    if kind == "pick":
        return {"kind": "pick", "mesh": rng.choice(["knot", "soup"]), "tris": _log(rng, 1_000, 300_000)}
    if kind == "rays":
        mesh = rng.choice(["knot", "soup"])
        return {"kind": "rays", "mesh": mesh, "tris": _log(rng, 1_000, 300_000), "rays": _log(rng, 1_000, 1_000_000),
                "aim": rng.choice(["sphere", "camera"]), "host": rng.random() < 0.3}
    if kind == "build":
        return {"kind": "build", "mesh": rng.choice(["knot", "soup"]), "tris": _log(rng, 1_000, 500_000)}
    if kind == "rebuild":
        return {"kind": "rebuild", "mesh": "knot", "tris": _log(rng, 10_000, 2_000_000),
                "rays": _log(rng, 1_000, 262_144)}
    if kind == "frame":
        scene = rng.choice(["box", "knot", "sky", "textured"])
        c = {"kind": "frame", "scene": scene, "width": _log(rng, 64, 1024), "height": _log(rng, 64, 1024),
             "spp": _log(rng, 1, 8), "depth": rng.randint(2, 12), "view": rng.random() < 0.5}
        if scene == "knot":
            c["tris"] = _log(rng, 10_000, 1_000_000)
        return c
    if kind == "inverse":
        return {"kind": "inverse", "width": _log(rng, 64, 512), "height": _log(rng, 64, 512), "spp": _log(rng, 1, 8),
                "depth": rng.randint(3, 8)}
    return {"kind": "batch", "scenes": rng.randint(2, 8), "tris": _log(rng, 10_000, 100_000),
            "width": _log(rng, 64, 256), "height": _log(rng, 64, 256), "spp": _log(rng, 1, 4),
            "depth": rng.randint(3, 8)}


# --------------------------------------------------------------------------- inputs
def _rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _knot(seed, tris, normals=False):
    """About `tris` triangles of a (2, 3) torus knot with three octaves of smooth displacement (the proportions of the
    large-mesh workload), made on the GPU: float32 positions [n, 9] (and vertex normals [n, 9])."""
    radial = max(3, int(round(math.sqrt(tris / 50.0))))
    tubular = max(3, int(round(tris / (2.0 * radial))))
    ph = torch.tensor(_rng(seed).uniform(0, 2 * math.pi, 12), dtype=torch.float64, device="cuda")
    i = torch.arange(tubular, dtype=torch.float64, device="cuda")[:, None] / tubular * (4 * math.pi)
    j = torch.arange(radial, dtype=torch.float64, device="cuda")[None, :] / radial * (2 * math.pi)

    def curve(a):
        q = 1.5 * a
        r = 0.5 * (2 + torch.cos(q))
        return torch.stack([r * torch.cos(a), r * torch.sin(a), 0.5 * torch.sin(q)], -1)

    p0, p1 = curve(i), curve(i + 0.01)
    t = p1 - p0
    b = torch.linalg.cross(t, p1 + p0)
    n = torch.linalg.cross(b, t)
    b, n = b / b.norm(dim=-1, keepdim=True), n / n.norm(dim=-1, keepdim=True)
    disp = 0.0
    for o in range(3):
        f = 4 * 2 ** o
        disp = disp + 0.05 / 2 ** o * torch.sin(f * i + ph[o]) * torch.sin(f * j + ph[3 + o])
    r = 0.32 + disp
    v = p0 + (-r * torch.cos(j))[..., None] * n + (r * torch.sin(j))[..., None] * b  # [tubular, radial, 3]
    w = v.roll(-1, 0)
    quads = (v, w, v.roll(-1, 1), w.roll(-1, 1))
    pos = torch.stack([quads[0], quads[1], quads[2], quads[1], quads[3], quads[2]], 2).reshape(-1, 9)
    pos = pos.to(torch.float32).contiguous()
    if not normals:
        return pos
    m = torch.linalg.cross(v.roll(-1, 0) - v.roll(1, 0), v.roll(-1, 1) - v.roll(1, 1))
    m = m / m.norm(dim=-1, keepdim=True)
    x = m.roll(-1, 0)
    nq = (m, x, m.roll(-1, 1), x.roll(-1, 1))
    nrm = torch.stack([nq[0], nq[1], nq[2], nq[1], nq[3], nq[2]], 2).reshape(-1, 9)
    return pos, nrm.to(torch.float32).contiguous()


def _positions(case, seed):
    """float32 [n, 9] on the GPU."""
    if case["mesh"] == "knot":
        return _knot(seed, case["tris"])
    rng = _rng(seed)
    n = case["tris"]
    p = rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.normal(0.0, 0.01, (n, 3, 3))
    return torch.from_numpy(p.reshape(n, 9).astype(np.float32)).cuda()


def _chords(rng, n):
    """float32 [n, 6]: from a sphere of radius 3 towards points of the cube [-1, 1]^3, unit directions."""
    g = rng.normal(size=(n, 3))
    o = (3.0 * g / np.linalg.norm(g, axis=1, keepdims=True)).astype(np.float32)
    d = rng.uniform(-1.0, 1.0, (n, 3)) - o
    return np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)


def _pick_ray(pos, seed):
    """A binary64 ray aimed at the middle of one of the triangles, 6 values."""
    o = _chords(_rng(seed + 1), 1)[0, :3].astype(np.float64)
    k = int(_rng(seed + 2).integers(0, pos.size // 9))
    d = pos.reshape(-1, 3, 3)[k].astype(np.float64).mean(0) - o
    return np.concatenate([o, d / np.linalg.norm(d)])


def _rays(case, seed):
    """float32 [n, 6] on the GPU: chords through a sphere around the mesh, or a camera's pixels row by row."""
    n = case["rays"]
    if case.get("aim", "sphere") == "sphere":
        return torch.from_numpy(_chords(_rng(seed + 7919), n)).cuda()
    w = max(1, int(round(math.sqrt(n * 16.0 / 9.0))))
    h = -(-n // w)
    a, e = _rng(seed + 7919).uniform(-0.6, 0.6, 2)
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    x = ((k % w + 0.5) / w * 2 - 1) * 0.75
    y = (torch.floor(k / w) + 0.5) / h * 2 - 1
    y = y * 0.75 * h / w
    eye = torch.tensor([4.2 * math.sin(a) * math.cos(e), 4.2 * math.sin(e), 4.2 * math.cos(a) * math.cos(e)],
                       dtype=torch.float64, device="cuda")
    f = -eye / eye.norm()
    r = torch.linalg.cross(f, torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device="cuda"))
    r = r / r.norm()
    u = torch.linalg.cross(r, f)
    d = f[None] + x[:, None] * r[None] + y[:, None] * u[None]
    d = d / d.norm(dim=1, keepdim=True)
    return torch.cat([eye[None].expand(n, 3), d], 1).to(torch.float32).contiguous()


def _materials(rng, n, glass=0, blend=0):
    out = []
    for k in range(n):
        if k < glass:
            out.append(S.material(albedo=(1.0, 1.0, 1.0), transmission=1.0, ior=float(rng.uniform(1.3, 1.8)),
                                  roughness=float(rng.uniform(0.0, 0.3)), attenuation_distance=1.0,
                                  attenuation_color=tuple(float(x) for x in np.exp(-rng.uniform(0, 2, 3)))))
            continue
        extra = {"alpha": 0.5, "alpha_mode": "blend"} if k >= n - blend else {}
        out.append(S.material(albedo=tuple(float(x) for x in rng.uniform(0.2, 0.8, 3)),
                              roughness=float(rng.uniform(0.05, 1.0)), metallic=float(rng.random() < 0.5),
                              clearcoat=float(rng.uniform(0, 1)), clearcoat_roughness=float(rng.uniform(0, 0.5)),
                              sheen_color=(float(rng.uniform(0, 1)),) * 3,
                              sheen_roughness=float(rng.uniform(0.2, 1.0)), **extra))
    return out


def _knot_scene(seed, tris, glass, blend, env_size, aperture):
    rng = _rng(seed + 31)
    pos, nrm = (x.cpu().numpy() for x in _knot(seed, tris, True))
    mats = _materials(rng, 16, glass, blend)
    cut = np.linspace(0, len(pos), 161).astype(int)  # bands along the tube
    pick = [b % 20 if b % 20 < 14 else 4 + b % 20 - 14 if b % 20 < 18 else b % 20 - 4 for b in range(160)]
    meshes = []
    for m in range(16):
        bands = [slice(cut[b], cut[b + 1]) for b in range(160) if pick[b] == m and cut[b + 1] > cut[b]]
        if bands:
            meshes.append(S.MeshInstance(M.Mesh(np.concatenate([pos[s] for s in bands]).reshape(-1),
                                                np.concatenate([nrm[s] for s in bands]).reshape(-1)), mats[m]))
    env = W.env_lognormal(rng, *env_size)
    y, x = int(env.height * 0.3), int(env.width * 0.6)
    env.data.reshape(env.height, env.width, 3)[y:y + 2, x:x + 2] = 5e4  # the sun's disk
    cam = S.Camera(position=(float(rng.uniform(-0.3, 0.3)), 0.4, 4.2), fov=40.0, aperture=aperture,
                   focus_distance=4.22)
    return S.Scene(name="knot", camera=cam, env=S.Environment(map=env, name="lognormal", background=True),
                   meshes=meshes)


def _scene(case, seed):
    kind = case["scene"]
    if kind == "box":
        return W.box_scene(seed)
    if kind == "sky":
        return W.sky_scene(seed)
    if kind == "textured":
        return W.textured_scene(seed)
    return _knot_scene(seed, case["tris"], 4, 2, (512, 256), 0.02)


class _State:
    def __init__(self, case, seed):
        self.case, self.seed = case, seed


def _pinned(r):
    return torch.empty((r.height, r.width, 4), dtype=torch.float32, pin_memory=True)


def _turn(cam, angle):
    """The camera moved a little around its target, as a viewer's drag moves it."""
    c, s = math.cos(angle), math.sin(angle)
    dx, dz = cam.position[0] - cam.target[0], cam.position[2] - cam.target[2]
    return S.Camera(position=(cam.target[0] + c * dx + s * dz, cam.position[1], cam.target[2] - s * dx + c * dz),
                    target=cam.target, fov=cam.fov, aperture=cam.aperture, focus_distance=cam.focus_distance)


def prepare(case, seed):
    st = _State(case, seed)
    kind = case["kind"]
    if kind == "pick":
        st.positions = _positions(case, seed).cpu().numpy().reshape(-1)
        st.bvh = B.build_bvh(st.positions)
        ray = _pick_ray(st.positions, seed)
        st.ray = {"origin": [float(x) for x in ray[:3]], "dir": [float(x) for x in ray[3:]]}
    elif kind == "rays":
        pos = _positions(case, seed)
        st.dev = B.build_device(pos.data_ptr(), pos.shape[0])
        rays = _rays(case, seed)
        if case["host"]:
            st.rays = rays.cpu().numpy()
        else:
            n = rays.shape[0]
            st.rays = rays
            st.prim = torch.empty(n, dtype=torch.int32, device="cuda")
            st.t, st.u, st.v = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3))
    elif kind == "build":
        st.positions = _positions(case, seed).cpu().numpy().reshape(-1)
        st.nodes = np.zeros((2 * (st.positions.size // 9) - 1) * 8, np.float32)  # the program's own scene buffer
    elif kind == "rebuild":
        st.positions = _positions(case, seed)
        st.rays = _rays(case, seed)
        n = st.rays.shape[0]
        st.prim = torch.empty(n, dtype=torch.int32, device="cuda")
        st.t, st.u, st.v = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3))
    elif kind == "frame":
        st.r = Renderer(case["width"], case["height"])
        st.r.settings.max_bounces = case["depth"]
        st.r.settings.samples_per_frame = case["spp"]
        st.r.load_scene(_scene(case, seed))
        st.color = _pinned(st.r)
        if case["view"]:
            st.cams = (st.r.scene.camera, _turn(st.r.scene.camera, 0.02))
    elif kind == "inverse":
        st.r = Renderer(case["width"], case["height"])
        st.r.settings.max_bounces = case["depth"]
        st.r.load_scene(W.adjoint_scene(seed))
        rng = _rng(seed + 5)
        st.theta = np.clip(AD.get_params(st.r.packed.materials) + rng.normal(0, 0.02, (st.r.packed.material_count, 6)),
                           0.0, 1.0).astype(np.float32)
        st.env = (st.r.scene.env.map.data * rng.uniform(0.9, 1.1, st.r.scene.env.map.data.size)).astype(np.float32)
        st.target = rng.uniform(0.0, 1.0, (case["height"], case["width"], 3)).astype(np.float32)
    else:
        st.rs, st.colors = [], []
        for k in range(case["scenes"]):
            r = Renderer(case["width"], case["height"])
            r.settings.max_bounces = case["depth"]
            r.load_scene(_knot_scene(seed * 64 + k, case["tris"], 0, 0, (256, 128), 0.0))
            st.rs.append(r)
            st.colors.append(_pinned(r))
        st.batch = Batch(st.rs)
    return st


def run(st):
    case = st.case
    kind = case["kind"]
    if kind == "pick":
        h = B.intersect_bvh(st.bvh, st.positions, st.ray)
        return [h.tri_index, np.array([h.t, h.u, h.v])] if h else [-1, np.zeros(3)]
    if kind == "rays":
        if case["host"]:
            return list(st.dev.intersect(st.rays))
        st.dev.intersect_device(st.rays.data_ptr(), st.rays.shape[0], st.prim.data_ptr(), st.t.data_ptr(),
                                st.u.data_ptr(), st.v.data_ptr())
        return [st.prim, st.t, st.u, st.v]
    if kind == "build":
        b = B.build_bvh(st.positions)
        st.nodes[:b.nodes.size] = b.nodes
        return [st.nodes, b.tri_indices, b.node_count, np.array(b.bounds.min + b.bounds.max)]
    if kind == "rebuild":
        dev = B.build_device(st.positions.data_ptr(), st.positions.shape[0])
        dev.intersect_device(st.rays.data_ptr(), st.rays.shape[0], st.prim.data_ptr(), st.t.data_ptr(),
                             st.u.data_ptr(), st.v.data_ptr())
        dev.check()
        count = dev.node_count
        dev.close()
        return [st.prim, st.t, st.u, st.v, count]
    if kind == "frame":
        r = st.r
        r.set_seed(st.seed * 1000)
        if not case["view"]:
            r.reset()
            r.trace_samples(case["spp"])
            r.read_color_async(st.color)
            return [st.color]
        r.upload_camera(st.cams[0])
        r.reset()
        canvases = [r.render()]  # the view at rest, then after a small move
        r.upload_camera(st.cams[1])
        canvases.append(r.render())
        r.read_color_async(st.color)
        return canvases + [st.color]
    if kind == "inverse":
        img = AD.forward(st.r, case["spp"], st.seed, st.theta, st.env)
        dl = 2.0 * (img - st.target)
        dm, de = AD.backward(st.r, case["spp"], st.seed, dl)
        return [img, dm, de]
    for r in st.rs:
        r.reset()
        r.set_seed(st.seed * 1000)
    st.batch.trace_samples(case["spp"])
    for r, c in zip(st.rs, st.colors):
        r.read_color_async(c)
    return list(st.colors)


def work(case):
    """Inputs read once, outputs written once; the operations of log2(triangles) box tests (20 each) and one triangle
    test (60) a ray, which no hierarchy does without."""
    kind = case["kind"]
    tris = case.get("tris", {"box": 81_960, "sky": 1_280, "textured": 1_300}.get(case.get("scene"), 81_960))
    per_ray = 60 + 20 * math.log2(max(2, tris))
    geometry = tris * 36
    if kind == "pick":
        return {"bytes": 48 + 28 + 64 * math.ceil(math.log2(tris)), "flops": per_ray}
    if kind == "rays":
        return {"bytes": case["rays"] * 40 + geometry, "flops": case["rays"] * per_ray}
    bounds = tris * 64 + tris * 4  # nodes (about one inner and one leaf for two triangles each) and indices
    sah = tris * max(1.0, math.log2(max(2, tris / 4))) * 30
    if kind == "build":
        return {"bytes": geometry + bounds, "flops": sah}
    if kind == "rebuild":
        return {"bytes": geometry + bounds + case["rays"] * 40, "flops": sah + case["rays"] * per_ray}
    pixels = case["width"] * case["height"]
    paths = pixels * case["spp"] * (case["scenes"] if kind == "batch" else 2 if case.get("view") else 1)
    # a path: two vertices, each with a closest-hit ray, a shadow ray and some 500 operations of shading
    flops = paths * 2 * (2 * per_ray + 500)
    if kind == "frame":
        frames = 2 if case["view"] else 1
        return {"bytes": tris * 100 + frames * pixels * (36 + (4 if case["view"] else 0)) + pixels * 16, "flops": flops}
    if kind == "inverse":
        return {"bytes": 3 * tris * 100 + pixels * (36 + 12 + 16) + 256 * 128 * 36, "flops": 3 * flops}
    return {"bytes": case["scenes"] * (tris * 100 + pixels * 52), "flops": flops}


# --------------------------------------------------------------------------- exact values
def _nearest(pos, rays, t_min):
    """Closest hits by brute force in binary64: t, u, v of each ray (inf, 0, 0 on a miss). Edge sides as 6-vectors
    (the ray's direction and moment against the edge's), so that pairs are matrix products; the winner's values by
    Moller and Trumbore's formulas."""
    v = pos.reshape(-1, 3, 3).double()
    a, b, c = v[:, 0], v[:, 1], v[:, 2]
    side = [torch.cat([torch.linalg.cross(p, q), q - p], 1) for p, q in ((a, b), (b, c), (c, a))]
    nrm = torch.linalg.cross(b - a, c - a)
    na = (nrm * a).sum(1)
    out = torch.zeros(rays.shape[0], 3, dtype=torch.float64, device=pos.device)
    out[:, 0] = math.inf
    step = max(1, (1 << 27) // max(1, a.shape[0]))
    for at in range(0, rays.shape[0], step):
        r = rays[at:at + step].double()
        o, d = r[:, :3], r[:, 3:]
        line = torch.cat([d, torch.linalg.cross(o, d)], 1)
        s0, s1, s2 = (line @ s.T for s in side)
        hit = ((s0 >= 0) & (s1 >= 0) & (s2 >= 0)) | ((s0 <= 0) & (s1 <= 0) & (s2 <= 0))
        del s0, s1, s2
        t = (na[None] - o @ nrm.T) / (d @ nrm.T)
        t = torch.where(hit & (t > t_min), t, math.inf)
        best, k = t.min(1)
        del t, hit
        e1, e2 = b[k] - a[k], c[k] - a[k]
        p = torch.linalg.cross(d, e2)
        inv = 1 / (e1 * p).sum(1)
        s = o - a[k]
        q = torch.linalg.cross(s, e1)
        got = torch.stack([(e2 * q).sum(1) * inv, (s * p).sum(1) * inv, (d * q).sum(1) * inv], 1)
        out[at:at + step] = torch.where((best < math.inf)[:, None], got, out[at:at + step])
    return out[:, 0], out[:, 1], out[:, 2]


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("pick", "rays", "rebuild"):
        return None  # images, gradients and trees: no plain formula short of another renderer or builder
    if case["tris"] * case.get("rays", 1) > 7e10:
        return None
    pos = _positions(case, seed)
    if kind == "pick":
        t, u, v = _nearest(pos, torch.from_numpy(_pick_ray(pos.cpu().numpy(), seed)[None]).cuda(), 1e-5)
        return [None, torch.stack([t[0], u[0], v[0]])]
    t, u, v = _nearest(pos, _rays(case, seed), 1e-5)
    return [None, t, u, v] if kind == "rays" else [None, t, u, v, None]
