"""The persistent traversal loops with few rays: blocks beyond the queue's share
leave at once and a warp gives rays to some of its lanes only. Calls on rays
send so few to the warp-per-ray kernel; fetch counting and stage timing keep
the loops. The counts are those of the sequential traversal, the vertices' one
or two contributions add up to the same bits in either order."""
import ctypes as C

import numpy as np
import pytest
import torch

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def soup():
    d = scenes.soup_render_scene(3000, 5)
    d.env = (0.5, 0.6, 0.7)
    return d.build()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 255, 257, 1215, 1216, 1217, 16384, 16385, 38911, 38912, 38913])
def test_loops_with_few_rays(gpu, soup, n):
    rays = torch.from_numpy(scenes.soup_rays(n, seed=n).view(np.float32).reshape(n, 8)).cuda()
    rays[:, 3], rays[:, 7] = 1e-4, float("inf")  # the range that a path's own ray has
    out = {}
    for flags in (0, N.KZ_RENDER_FLAG_COUNT, N.KZ_RENDER_FLAG_TIMING):
        cfg, st, rgb = api.render_config(1, 1, 3, flags=flags), N.KzRenderStats(), torch.empty((n, 3), device="cuda")
        N.check(N.lib().kz_li_batch(soup.handle, C.c_void_p(rays.data_ptr()), n, C.byref(cfg),
                                    C.c_void_p(rgb.data_ptr()), N.KZ_MEM_DEVICE, C.byref(st)))
        torch.cuda.synchronize()
        out[flags] = rgb.cpu().numpy().view(np.uint32), st.path_bounces, st.shadow_rays
        if flags == N.KZ_RENDER_FLAG_COUNT:
            assert (st.closest_node_fetches, st.closest_tri_fetches) == soup.intersect_stats(rays)
    want = out[0]
    assert want[1] == n
    for flags, got in out.items():
        assert np.array_equal(got[0], want[0]) and got[1:] == want[1:], flags
