"""Motion compensation with the strips of a launch whole, in halves and in quarters: pictures of few
strips and of many, blocks whose last strip is shorter than its parts, weighted prediction and
references outside the picture; every output byte equals the oracle's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(8, 8), (72, 40), (416, 240), (1280, 720), (2560, 1440), (3840, 2160)])
@pytest.mark.parametrize("kw", [dict(p_intra=0.0), dict(p_intra=0.1, p_wp=0.5, mv_range=4096)], ids=["plain", "weighted"])
def test_gpu_mc_parts(hb, gpu_ctx, port, w, h, kw):
    pic = hb.Picture(hb.default_cfg(w, h, w + h, **kw))
    refs = [hb.content(w, h, 1), hb.content(w, h, 2)]
    assert (gpu_ctx.reconstruct_picture(pic, refs) == port.reconstruct_picture(pic, refs)).all()
