"""What the backward's second replay takes over from its first one (triangles
and unoccluded next-event rays, per path and bounce), checked by the gradient's
homogeneity: without emitters every pixel is linear in the environment's
texels (paths, weights and clamp scales held fixed), so the environment
gradient times the environment is the weighted image itself.

Both sides are binary32 sums of the same terms: a texel's sum of some 1e3
atomic additions is off by at most 1e3 * 2^-24 = 6e-5, and a path that rounding
sends elsewhere in the forward kernel moves a sum over 851 pixels x 3 samples by
4e-4 of a typical sample; the bar is 2e-3.
"""
import numpy as np
import pytest

from lucent_gb300 import adjoint as AD
from lucent_gb300 import scene as S
from lucent_gb300 import workloads as W
from lucent_gb300.renderer import Renderer

pytestmark = pytest.mark.gpu


def _scene():
    sc = W.adjoint_scene(0, 3)
    mats = [S.material(albedo=(0.7, 0.6, 0.5), roughness=0.4),
            S.material(albedo=(0.9, 0.8, 0.9), roughness=0.0, transmission=1.0, ior=1.5),
            S.material(albedo=(0.8, 0.8, 0.3), roughness=0.2, metallic=1.0, clearcoat=0.5)]
    meshes = [S.MeshInstance(m.mesh, mats[i % 3]) for i, m in enumerate(sc.meshes)]
    return S.Scene(name="envonly", camera=sc.camera, env=sc.env, meshes=meshes)


@pytest.mark.parametrize("depth,w,h,spp", [(0, 37, 23, 3), (1, 37, 23, 3), (5, 37, 23, 3), (64, 37, 23, 3),
                                           (3, 1, 1, 40), (2, 1449, 1448, 1)])
def test_environment_gradient_is_homogeneous(depth, w, h, spp):
    r = Renderer(w, h)
    r.settings.max_bounces = depth
    r.load_scene(_scene())
    img = AD.forward(r, spp, 5)
    dl = np.random.default_rng(depth).uniform(0.5, 1.5, (h, w, 3)).astype(np.float32)
    dm, de = AD.backward(r, spp, 5, dl)
    want = float((dl.astype(np.float64) * img).sum())
    got = float((de.astype(np.float64).reshape(-1) * np.asarray(r.scene.env.map.data, np.float64).reshape(-1)).sum())
    assert want > 0 and abs(got - want) / want < 2e-3, (got, want)
    assert np.isfinite(dm).all() and np.isfinite(de).all()
    r.dispose()
