"""Paths in flight of a guided render by default: a pass of up to
KZ_RENDER_DEFAULT_WAVEFRONT paths is one wave, while training (its records hold
the whole pass anyway) and frozen. One wave has at most max_depth iterations;
a pass cut into several has more."""
import pytest

from kazen_proto_gb300 import api, scenes

pytestmark = pytest.mark.gpu

DEPTH = 2


@pytest.mark.parametrize("w,h,spp,train", [(2304, 2048, 1, True), (2304, 2048, 1, False), (512, 512, 8, False)])
def test_a_pass_is_one_wave(gpu, w, h, spp, train):
    d = scenes.slit_room_scene()
    s, g = d.build(), api.Guide(seed=2)
    st = api.render_guided(s, g, d.camera, w, h, spp, DEPTH, seed=1, gcfg=api.guide_config(train=train))[2]
    assert st["paths"] == w * h * spp and st["iterations"] <= DEPTH
    g.close()
    s.close()
