"""Camera bundles whose rays part: in an image with pixels much coarser than the
triangles (a small image, or a scene seen from afar) a bundle gives up after a
bounded amount of work. The image and the ray counts are those of the paths
traced one by one (fetch counting keeps the single rays; the films differ by
the order of their sums), and the frame takes at most twice as long as those,
counting included; without the bound it took several to some hundred times as
long."""
import time

import numpy as np
import pytest

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def best_ms(f, n=5):
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return min(t) * 1e3


@pytest.mark.parametrize("w,h,spp,far", [(64, 64, 8, 1), (17, 33, 32, 1), (320, 180, 8, 200), (320, 180, 64, 20)])
def test_bundle_work_is_bounded(gpu, w, h, spp, far):
    d = scenes.terrain_scene(cells=256, n_spheres=16, subdiv=2)
    s, c, depth = d.build(), d.camera, 2
    eye, look = np.array(c.eye), np.array(c.lookat)
    cam = api.Camera(eye=tuple(look + (eye - look) * far), lookat=c.lookat, up=c.up, fov=c.fov)
    ref = api.Renderer(spp=spp, max_depth=depth, seed=4, flags=N.KZ_RENDER_FLAG_COUNT)
    r = api.Renderer(spp=spp, max_depth=depth, seed=4)
    want, got = ref.render(s, cam, w, h), r.render(s, cam, w, h)
    assert (np.abs(got - want) <= 2 * spp * depth * 2.0 ** -24 * np.abs(want)).all()
    for k in ("path_bounces", "shadow_rays", "paths"):
        assert r.last_stats[k] == ref.last_stats[k], k
    assert best_ms(lambda: r.render(s, cam, w, h)) <= 2.0 * best_ms(lambda: ref.render(s, cam, w, h))
