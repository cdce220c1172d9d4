"""Batched preparation says what is wrong with a picture's records before it takes or sends
anything for them: the first bad picture's own error, whatever the memory budget, and the context
then works as before."""
import ctypes as C

import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("bad_at", [0, 2])
def test_gpu_bad_picture_is_named_before_memory_is_taken(hb, gpu_ctx, port, pinned, bad_at):
    w, h = 416, 240
    refs = [hb.content(w, h, 1), hb.content(w, h, 2)]
    pics = [hb.Picture(hb.default_cfg(w, h, 60 + k, **cases.PICTURE)) for k in range(3)]
    if pinned:
        pics = [p.pin() for p in pics]
    streams = []
    for _ in pics:
        st = gpu_ctx.open_stream(w, h, 3)
        for slot, r in enumerate(refs):
            st.upload(slot, r)
        streams.append(st)
    t = pics[bad_at].syn.tus[0]
    size, t.log2_size = t.log2_size, 7
    try:
        if bad_at == 0:
            gpu_ctx.set_budget(1)   # nothing more: no picture's memory can be had
        with pytest.raises(hb.HevcGpuError) as e:
            hb.prepare_batch(streams, pics)
        assert e.value.code == hb.abi.HEVCGPU_EINVAL and f"picture {bad_at}: TU 0" in str(e.value)
    finally:
        gpu_ctx.set_budget((1 << 64) - 1)
        t.log2_size = size
    jobs = hb.prepare_batch(streams, pics)
    hb.batch_launch(jobs, [2] * 3)
    gpu_ctx.sync()
    for st, p in zip(streams, pics):
        assert (st.download(2) == port.reconstruct_picture(p, refs)).all()
    for j in jobs:
        j.free()
    for st in streams:
        st.close()


@pytest.mark.parametrize("n", [1, 5, 40])
def test_gpu_prepared_batches_of_any_length(hb, gpu_ctx, port, n):
    w, h = 200, 136
    refs = [hb.content(w, h, 1), hb.content(w, h, 2)]
    pics = [hb.Picture(hb.default_cfg(w, h, 70 + k, **cases.PICTURE)) for k in range(min(n, 7))]
    pics = [p.pin() if k % 2 else p for k, p in enumerate(pics)]
    want = [port.reconstruct_picture(p, refs) for p in pics]
    streams = []
    for _ in range(n):
        st = gpu_ctx.open_stream(w, h, 3)
        for slot, r in enumerate(refs):
            st.upload(slot, r)
        streams.append(st)
    jobs = hb.prepare_batch(streams, [pics[k % len(pics)] for k in range(n)])
    hb.batch_launch(jobs, [2] * n)
    gpu_ctx.sync()
    for k, st in enumerate(streams):
        assert (st.download(2) == want[k % len(pics)]).all(), k
    for j in jobs:
        j.free()
    for st in streams:
        st.close()
