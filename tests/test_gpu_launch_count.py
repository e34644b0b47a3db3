"""kernel_launches of a render: generation, joint trace and shading in each
iteration, one shadow launch at the end of each batch of iterations, and from
the second batch on the kernel that carries the counters over."""
import pytest

from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,batches,iterations", [(0, 1, 1), (2048, 1, 8), (1000, 3, 8)])
def test_launches_are_counted(gpu, size, batches, iterations):
    d = scenes.box_scene()
    s, r = d.build(), api.Renderer(spp=4, max_depth=1, seed=1, wavefront_size=size)
    r.render(s, d.camera, 64, 64)  # 16,384 paths of one vertex: one wave, 8 and 17
    assert r.last_stats["kernel_launches"] == batches * (3 * iterations + 1) + batches - 1
