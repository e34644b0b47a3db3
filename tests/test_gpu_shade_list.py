"""Plain paths listed per block before they are shaded, against the one-kernel
shading of smaller wavefronts: views in which almost every path stays plain,
almost every path leaves the scene, and all kinds mix, with one, several and a
ragged number of paths per thread. The films differ by the order of their
floating-point sums only."""
import numpy as np
import pytest

from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu

SPLIT, SPP, DEPTH = 1 << 18, 9, 4
RTOL = 2 * SPP * DEPTH * 2.0 ** -24  # at most 2 * spp * depth contributions a pixel, each rounded once


def scene(env):
    d = scenes.SceneDesc()
    d.materials = [api.material([api.diffuse((0.6, 0.5, 0.4))]), api.material([api.dielectric(1.5, 1.0)]),
                   api.material([api.diffuse((0.2, 0.2, 0.2))], Le=(8.0, 7.0, 6.0))]
    v, i = scenes.quad((-1.0, 0.0, -1.0), (0, 0, 3.0), (3.0, 0, 0))
    d.add(v, i, 0)
    sv, sf = scenes.icosphere(2)
    d.add(sv * np.float32(0.15) + np.array([0.5, 0.2, 0.5], np.float32), sf, 1)
    v, i = scenes.quad((0.2, 1.2, 0.2), (0.6, 0, 0), (0, 0, 0.6))
    d.add(v, i, 2, is_light=True)
    if env:
        d.env = (0.3, 0.35, 0.4)
    return d


@pytest.mark.parametrize("env", [False, True])
@pytest.mark.parametrize("eye,lookat,fov", [((0.5, 1.1, 0.4), (0.5, 0.0, 0.41), 60.0),   # floor everywhere
                                            ((0.5, 0.3, -6.0), (0.5, 3.0, 0.5), 70.0),  # nearly all miss
                                            ((0.5, 0.8, -1.2), (0.5, 0.1, 0.4), 45.0)])
@pytest.mark.parametrize("W,H", [(173, 169), (346, 150), (461, 307)])  # 263,133, 467,100 and 1,273,743 paths
def test_listed_paths_match_one_kernel(gpu, W, H, eye, lookat, fov, env):
    s = scene(env).build()
    cam = api.Camera(eye=eye, lookat=lookat, fov=fov)
    a, b = (api.Renderer(spp=SPP, max_depth=DEPTH, seed=5, wavefront_size=w).render(s, cam, W, H)
            for w in (SPLIT - 1, 1 << 21))
    assert np.isfinite(a).all() and np.array_equal(a == 0, b == 0)
    assert (np.abs(a - b) <= RTOL * np.abs(b)).all(), np.abs(a - b).max()
