"""Camera paths traced in bundles against the same paths traced one by one
(fetch counting keeps the single rays): the same image and ray counts, with
bundles that straddle pixels and rows, end ragged, start after older paths in a
refilled wavefront, look along an axis (directions of both signs), and meet
more than their stack holds. The films differ by the order of their
floating-point sums only."""
import numpy as np
import pytest

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def agree(s, cam, w, h, spp, depth, size):
    ref = api.Renderer(spp=spp, max_depth=depth, seed=4, wavefront_size=size, flags=N.KZ_RENDER_FLAG_COUNT)
    want = ref.render(s, cam, w, h)
    r = api.Renderer(spp=spp, max_depth=depth, seed=4, wavefront_size=size)
    got = r.render(s, cam, w, h)
    assert np.isfinite(got).all()
    assert (np.abs(got - want) <= 2 * spp * depth * 2.0 ** -24 * np.abs(want)).all()
    for k in ("path_bounces", "shadow_rays", "paths"):
        assert r.last_stats[k] == ref.last_stats[k], k


@pytest.mark.parametrize("spp", [7, 8, 9, 17, 33, 64])
@pytest.mark.parametrize("size", [0, 1000, 31])
def test_bundles_match_single_rays(gpu, spp, size):
    d = scenes.box_scene()
    agree(d.build(), d.camera, 13, 7, spp, 4, size)


@pytest.mark.parametrize("n_tris", [1, 40, 3000, 60000])
def test_bundles_in_a_soup(gpu, n_tris):
    """Long, overlapping triangles and a wide field: many nodes per bundle."""
    r = np.random.default_rng(n_tris)
    tv = (r.random((n_tris, 1, 3)) + r.uniform(-0.3, 0.3, (n_tris, 3, 3))).astype(np.float32).reshape(-1, 9)
    d = scenes.soup_desc(tv)
    d.env = (0.5, 0.6, 0.7)
    views = ((0.5, 0.5, -2.0), (0.5, 0.5, 0.5)), ((0.4, 0.5, 0.6), (1.0, 0.2, 0.1)), ((2.0, 2.5, 3.0), (0.5, 0.5, 0.5))
    for eye, look in views:
        agree(d.build(), api.Camera(eye=eye, lookat=look, fov=100.0), 9, 8, 16, 2, 0)
