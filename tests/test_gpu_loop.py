"""The device-driven loop at its edges: every wavefront size (all paths at
once, several batches of iterations, one path at a time) and both ways of
tracing shadow rays (beside the next iteration's paths, and, with stage
timing, in a launch of their own) give the same image and the same ray counts.
The films differ by the order of their floating-point sums only: at most
2 * spp * depth contributions a pixel, each rounded once."""
import numpy as np
import pytest

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu

W, H, SPP = 23, 17, 3
TOTAL = W * H * SPP


@pytest.fixture(scope="module")
def box():
    d = scenes.box_scene()
    return d, d.build()


@pytest.mark.parametrize("depth", [1, 2, 5])
@pytest.mark.parametrize("size", [64, 1000, TOTAL - 1, TOTAL, TOTAL + 1, 0])
@pytest.mark.parametrize("flags", [0, N.KZ_RENDER_FLAG_TIMING])
def test_wavefront_sizes_agree(gpu, box, depth, size, flags):
    d, s = box
    ref = api.Renderer(spp=SPP, max_depth=depth, seed=2, flags=N.KZ_RENDER_FLAG_COUNT)
    want = ref.render(s, d.camera, W, H)
    r = api.Renderer(spp=SPP, max_depth=depth, seed=2, wavefront_size=size, flags=flags)
    got = r.render(s, d.camera, W, H)
    assert (np.abs(got - want) <= 2 * SPP * depth * 2.0 ** -24 * np.abs(want)).all()
    for k in ("path_bounces", "shadow_rays", "paths"):
        assert r.last_stats[k] == ref.last_stats[k], k


@pytest.mark.parametrize("n", [1, 7, 8, 9, 1215, 1216, 1217, 16383, 16384, 16385, 38911, 38912, 38913])
def test_few_rays_are_spread(gpu, oracle_mod, n):
    tv = scenes.triangle_soup(3000, seed=5)
    rays = scenes.soup_rays(n, seed=n)
    s, ob = scenes.soup_desc(tv).build(), oracle_mod.Bvh(tv)
    g, o = s.intersect(rays), ob.closest(rays)
    assert np.array_equal(g["prim_id"], o["prim"]) and np.array_equal(g["t"].view(np.uint32), o["t"].view(np.uint32))
    assert np.array_equal(s.occluded(rays), ob.any(rays))
