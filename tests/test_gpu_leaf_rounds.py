"""The warp-shared leaf tests where their lists end: more pending (ray,
triangle) pairs than one or two rounds of a warp, ray counts that leave lanes
without a ray, nodes of every leaf size, and bounds that accept nothing. Hits
are compared bit for bit with the restatement's loop over every triangle."""
import numpy as np
import pytest

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import scenes

pytestmark = pytest.mark.gpu


def fan(n, seed):
    """n large triangles through one small region: most rays meet most of them."""
    r = np.random.default_rng(seed)
    c = r.uniform(0.45, 0.55, (n, 1, 3))
    return (c + r.uniform(-0.6, 0.6, (n, 3, 3))).astype(np.float32).reshape(n, 9)


@pytest.mark.parametrize("n_tris", [1, 2, 3, 4, 7, 8, 9, 23, 24, 25, 64, 193, 700])
@pytest.mark.parametrize("n_rays", [1, 31, 32, 33, 1000])
def test_leaf_rounds_match_every_triangle(gpu, oracle_mod, n_tris, n_rays):
    tv = fan(n_tris, n_tris)
    rays = scenes.soup_rays(n_rays, seed=n_tris + n_rays)
    rays["tmax"][::5] = np.float32(2.0)
    rays["tmax"][1::7] = np.float32(np.nan)
    s = scenes.soup_desc(tv).build()
    g, o = s.intersect(rays), oracle_mod.closest_brute(tv, rays)
    assert np.array_equal(g["prim_id"], o["prim"])
    hit = o["prim"] != N.KZ_INVALID_ID
    assert np.array_equal(g["t"][hit].view(np.uint32), o["t"][hit].view(np.uint32))
    assert np.array_equal(g["t"][~hit], rays["tmax"][~hit], equal_nan=True)
    o = oracle_mod.Bvh(tv).closest(rays)
    for k in ("u", "v"):
        assert np.array_equal(g[k][hit].view(np.uint32), o[k][hit].view(np.uint32))
    assert np.array_equal(s.occluded(rays), hit)
