"""The loop filter kernel at the sizes where its tiles (64x64) and its forms meet: one tile and
less, one sample block past a tile, CTBs smaller than a tile, pictures that take the form with
few tiles per SM, with many, and the one between; every output byte equals the oracle's."""
import pytest

import cases
from test_oracle import with_filter_edits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(8, 8), (64, 64), (72, 56), (136, 200), (2560, 1440), (4096, 2304)])
@pytest.mark.parametrize("log2_ctb", [4, 5, 6])
def test_gpu_loop_filter_tiles(hb, gpu_ctx, port, w, h, log2_ctb):
    cfg = dict(cases.FILTERS, log2_ctb=log2_ctb)
    pic = hb.Picture(hb.default_cfg(w, h, w + log2_ctb, **cfg))
    keep = with_filter_edits(hb, pic, w) if w == 136 else None   # slices, PCM and bypass CUs
    src = hb.content(w, h, h + log2_ctb)
    for db, sao in [(True, True), (True, False), (False, True)]:
        assert (gpu_ctx.loop_filter(pic, src, db, sao) == port.loop_filter(pic, src, db, sao)).all(), (db, sao)
    del keep
