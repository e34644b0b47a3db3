"""Shading in two kernels (wavefronts of 2^18 paths and more) against the one
kernel that smaller wavefronts use: the same image from the same random
streams, in scenes of every shading class, with and without vertex attributes,
an environment, the three estimators, a path count that is no multiple of
anything, and as jobs of a batch. The films differ by the order of their
floating-point sums only: at most 2 * spp * depth contributions a pixel, each
rounded once."""
import numpy as np
import pytest

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu

SPLIT, SPP, DEPTH = 1 << 18, 9, 5
RTOL = 2 * SPP * DEPTH * 2.0 ** -24


def classes_scene(attr, env, emissive_lobe=False):
    """Spheres of every shading class over a plain floor under a quad light."""
    d = scenes.SceneDesc()
    mats = [[api.diffuse((0.6, 0.5, 0.4))], [api.microfacet("beckmann", 0.2), api.diffuse((0.3, 0.3, 0.3))],
            [api.conductor_ggx((0.9, 0.7, 0.5), 0.2)], [api.translucent((0.5, 0.5, 0.5)), api.diffuse((0.2, 0.2, 0.2))],
            [api.dielectric(1.5, 1.0)], [api.microfacet("beckmann", 0.3, eta=0.66, refract=2)], [],
            [api.diffuse((0.0, 0.0, 0.0))], [api.diffuse((0.4, 0.4, 0.4), (0.0, 0.8, 0.6))]]
    d.materials = [api.material(m) for m in mats] + [api.material([api.diffuse((0.2, 0.2, 0.2))], Le=(8.0, 7.0, 6.0))]
    if attr:
        d.textures = [api.checker_texture(6.0, 6.0)]
        d.materials[0] = api.material([api.textured(mats[0][0], 0)])
    v, i = scenes.quad((-1.0, 0.0, -1.0), (0, 0, 3.0), (3.0, 0, 0))
    d.add(v, i, 0, uv=np.array([[0, 0], [1, 0], [1, 1], [0, 1]], np.float32) if attr else None)
    sv, sf = scenes.icosphere(2)
    for k in range(1, len(d.materials) - 1):
        p = np.array([0.15 + 0.25 * (k % 4), 0.14, 0.2 + 0.3 * (k // 4)], np.float32)
        d.add(sv * np.float32(0.12) + p, sf, k, normals=sv if attr else None)
    v, i = scenes.quad((0.2, 1.2, 0.2), (0.6, 0, 0), (0, 0, 0.6))
    d.add(v, i, len(d.materials) - 1, is_light=True)
    d.point_lights = [((0.5, 0.9, -0.5), (0.1, 0.1, 0.1))]
    if env:
        d.env = (0.3, 0.35, 0.4)
    d.camera = api.Camera(eye=(0.5, 0.8, -1.2), lookat=(0.5, 0.1, 0.4), fov=45.0)
    return d


def agree(a, b):
    assert np.isfinite(a).all() and np.array_equal(a == 0, b == 0)
    assert (np.abs(a - b) <= RTOL * np.abs(b)).all(), np.abs(a - b).max()


@pytest.mark.parametrize("flags", [0, N.KZ_RENDER_FLAG_NEE_ONLY, N.KZ_RENDER_FLAG_BSDF_ONLY])
@pytest.mark.parametrize("attr,env", [(False, False), (False, True), (True, False), (True, True)])
def test_split_matches_one_kernel(gpu, attr, env, flags):
    d = classes_scene(attr, env)
    s = d.build()
    W, H = 211, 149  # 282,951 paths: the first wavefront is full, the second a ragged rest
    img = [api.Renderer(spp=SPP, max_depth=DEPTH, seed=3, wavefront_size=w, flags=flags).render(s, d.camera, W, H)
           for w in (SPLIT - 1, SPLIT)]
    agree(*img)


def test_split_batch_matches_renders(gpu):
    jobs = []
    for k, (attr, env) in enumerate([(False, False), (True, True), (False, True)]):
        d = classes_scene(attr, env)
        jobs.append({"scene": d.build(), "camera": d.camera, "width": 131 + k, "height": 97, "spp": SPP,
                     "max_depth": DEPTH, "seed": k})
    imgs, st = api.render_batch(jobs, api.batch_config(wavefront_size=SPLIT))
    assert st["threads"] == SPLIT
    for j, img in zip(jobs, imgs):
        r = api.Renderer(spp=SPP, max_depth=DEPTH, seed=j["seed"], wavefront_size=SPLIT - 1)
        agree(img, r.render(j["scene"], j["camera"], j["width"], j["height"]))
