"""The intra stage in its three forms (by the depth of the chain, the number of work items and the
CTUs' density) and bands of large TUs, at batches that take each form and at CTB sizes where a
CTU has few TUs; every output byte equals the oracle's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h,kw", [(1, 64, 64, dict(slice_type=2)), (1, 1280, 720, dict(slice_type=2)),
                                      (9, 640, 360, dict(slice_type=2)), (2, 640, 360, dict(slice_type=2, log2_ctb=5)),
                                      (2, 640, 360, dict(slice_type=2, log2_ctb=4)),
                                      (3, 1280, 720, dict(p_intra=0.1)), (12, 416, 240, dict(p_intra=0.05)),
                                      (70, 200, 136, dict(p_intra=0.5))])
def test_gpu_intra_forms(hb, gpu_ctx, port, n, w, h, kw):
    """(70 pictures: more than one launch holds, whose plan follows the first group's tickets.)"""
    refs = [hb.content(w, h, 1), hb.content(w, h, 2)]
    pics = [hb.Picture(hb.default_cfg(w, h, 500 + k, **kw)) for k in range(min(n, 4))]
    want = [port.reconstruct_picture(p, refs) for p in pics]
    streams, jobs = [], []
    for k in range(n):
        st = gpu_ctx.open_stream(w, h, 3)
        for slot, r in enumerate(refs):
            st.upload(slot, r)
        streams.append(st)
        jobs.append(st.prepare(pics[k % len(pics)]))
    for _ in range(2):   # the second launch finds the first one's border words
        hb.batch_launch(jobs, [2] * n)
    gpu_ctx.sync()
    for k, st in enumerate(streams):
        assert (st.download(2) == want[k % len(pics)]).all(), k
    for j in jobs:
        j.free()
    for st in streams:
        st.close()
