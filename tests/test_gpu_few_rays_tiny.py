"""Calls of rays through a handful of triangles: the limit of the warp-per-ray
kernel is lower there. Hits are the oracle's around it, and a call takes no
longer than one of more rays (within a tenth, timed in a row); with the limit of
larger scenes 16,384 rays through 36 triangles took 1.5 times as long as 20,000."""
import numpy as np
import pytest

from kazen_proto_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8191, 8192, 8193, 16384, 16385])
@pytest.mark.parametrize("tris", [1, 128, 129])
def test_hits_at_the_limit(gpu, oracle_mod, tris, n):
    tv = scenes.triangle_soup(tris, seed=5)
    rays = scenes.soup_rays(n, seed=n)
    s, ob = scenes.soup_desc(tv).build(), oracle_mod.Bvh(tv)
    g, o = s.intersect(rays), ob.closest(rays)
    assert np.array_equal(g["prim_id"], o["prim"]) and np.array_equal(g["t"].view(np.uint32), o["t"].view(np.uint32))
    assert np.array_equal(s.occluded(rays), ob.any(rays))


@pytest.mark.parametrize("query", ["closest", "any"])
def test_fewer_rays_take_no_longer(gpu, query):
    import torch
    d = scenes.box_scene()
    s, stream = d.build(), torch.cuda.Stream()
    s.set_stream(stream)
    r = np.random.default_rng(1)
    rays = scenes.api.make_rays(np.asarray(d.camera.eye, np.float32),
                                r.uniform((-0.3, -0.3, 1.0), (0.3, 0.3, 1.0), (20000, 3)).astype(np.float32))
    dev = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()

    def us(n):
        part, ts = dev[:n].contiguous(), []
        f = s.intersect if query == "closest" else s.occluded
        out = f(part)
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            for _ in range(20):
                f(part, out=out)
            b.record(stream)
            stream.synchronize()
            ts.append(a.elapsed_time(b) * 50)
        return min(ts)

    more = us(20000)
    for n in (12288, 14000, 16384):
        assert us(n) <= 1.1 * more, n
