"""Pictures whose intra TUs cover samples twice or are larger than their CTB: the records that
job preparation accepts but that the CTU form of the intra stage has no room for.  On the CPU,
which pictures go to which form, that the ones left to the CTU form stay within its sizes, and
that the others' order is decode order wherever one TU writes what another reads or covers.  On
the GPU, every output byte equals the oracle's, which goes through the TUs one by one."""
import ctypes as C
import random

import numpy as np
import pytest

import cases
from test_intra_schedule import CONFIGS

MAX_ITEMS, MAX_ENTRIES = 384, 2048   # work items and dependency entries of a CTU (intra.cuh)


class Records:
    """A generated picture with other TUs, given as dicts of hevc_tu_t fields."""

    def __init__(self, hb, pic, tus):
        self.base = pic
        self._syn = hb.abi.PictureSyntax()
        C.memmove(C.byref(self._syn), C.byref(pic.syn), C.sizeof(self._syn))
        self._tus = (hb.TU * max(1, len(tus)))()
        for t, d in zip(self._tus, tus):
            for k, v in d.items():
                setattr(t, k, v)
        self._syn.tus = C.cast(self._tus, type(self._syn.tus))
        self._syn.num_tus = len(tus)

    @property
    def syn(self):
        return self._syn

    @property
    def syn_ptr(self):
        return C.pointer(self._syn)


FIELDS = ("x", "y", "log2_size", "c_idx", "qp", "flags", "intra_mode", "coeff_offset")


def fields(pic):
    return [{k: getattr(pic.syn.tus[i], k) for k in FIELDS} for i in range(pic.syn.num_tus)]


def tu(hb, x, y, log2, c=0, mode=1):
    return dict(x=x, y=y, log2_size=log2, c_idx=c, intra_mode=mode, flags=hb.abi.HEVC_TU_INTRA)


def one_place(hb, n_large):
    """A 64x64 CTU: three quadrants of 4x4 TUs, then one TU of 32x32 coded again and again."""
    pic = hb.Picture(hb.default_cfg(64, 64, 5, slice_type=2))
    rng = random.Random(n_large)
    tus = [tu(hb, 32 * (q & 1) + 4 * x, 32 * (q >> 1) + 4 * y, 2, mode=rng.randrange(35))
           for q in range(3) for y in range(8) for x in range(8)]
    return Records(hb, pic, tus + [tu(hb, 32, 32, 5, mode=rng.randrange(35)) for _ in range(n_large)])


def repeated(hb, w, h, seed, share, **kw):
    """A generated picture in which some intra TUs are coded again, right away or some TUs
    later, at once or in quarters, with another mode."""
    pic = hb.Picture(hb.default_cfg(w, h, seed, **kw))
    rng = random.Random(seed)
    out, later = [], []
    for t in fields(pic):
        out.append(t)
        if t["flags"] & hb.abi.HEVC_TU_INTRA and not t["flags"] & hb.abi.HEVC_TU_PCM and rng.random() < share:
            again = dict(t, intra_mode=rng.randrange(35))
            if t["log2_size"] > 2 and rng.random() < 0.5:
                half = 1 << (t["log2_size"] - 1)
                again = dict(again, log2_size=t["log2_size"] - 1, x=t["x"] + half * rng.randrange(2),
                             y=t["y"] + half * rng.randrange(2))
            later.append((len(out) + rng.choice((0, 0, 3, 60)), again))
        while later and later[0][0] <= len(out):
            out.append(later.pop(0)[1])
    return Records(hb, pic, out + [t for _, t in later])


def large(hb, w, h, log2_ctb, c_log2):
    """TUs of 32x32 luma and of 1 << c_log2 chroma samples in smaller CTBs, with modes that do not
    read the row above past the TU (of which only the next CTB counts as available)."""
    pic = hb.Picture(hb.default_cfg(w, h, 9, slice_type=2, log2_ctb=log2_ctb))
    rng = random.Random(w)
    return Records(hb, pic, [tu(hb, x, y, lg, c, rng.choice((1, 2, 5, 8, 9, 10, 26)))
                             for c, lg in ((0, 5), (1, c_log2), (2, c_log2))
                             for y in range(0, h // (2 if c else 1), 1 << lg) for x in range(0, w // (2 if c else 1), 1 << lg)])


BY_LEVELS = {
    "one place, 2": lambda hb: one_place(hb, 2),
    "one place, 190": lambda hb: one_place(hb, 190),
    "repeated 64x64": lambda hb: repeated(hb, 64, 64, 11, 0.3, slice_type=2),
    "repeated 416x240": lambda hb: repeated(hb, 416, 240, 3, 0.02, slice_type=2),
    "repeated P/B 416x240, 32x32 CTBs": lambda hb: repeated(hb, 416, 240, 17, 0.1, log2_ctb=5, p_intra=0.4),
    "repeated tiles 200x136, 16x16 CTBs": lambda hb: repeated(hb, 200, 136, 23, 0.1, slice_type=2, log2_ctb=4, tile_cols=3,
                                                             tile_rows=2),
    "once, far apart": lambda hb: repeated(hb, 1280, 720, 7, 0.0002, slice_type=2),
    "large 128x96, 16x16 CTBs": lambda hb: large(hb, 128, 96, 4, 4),
    "large 128x64, 32x32 CTBs": lambda hb: large(hb, 128, 64, 5, 5),
}


def touched(s, t):
    """4x4 units that a TU covers and those around it (its reference array), in its plane."""
    n, sub = (1 << t.log2_size) // 4, 2 if t.c_idx else 1
    x, y, w, h = t.x // 4, t.y // 4, s.params.width // sub // 4, s.params.height // sub // 4
    around = {(x + k, y - 1) for k in range(-1, 2 * n)} | {(x - 1, y + k) for k in range(2 * n)}
    return ({(t.c_idx, x + i, y + j) for i in range(n) for j in range(n)},
            {(t.c_idx, i, j) for i, j in around if 0 <= i < w and 0 <= j < h})


@pytest.mark.parametrize("name", sorted(BY_LEVELS))
def test_levels_keep_decode_order(hb, name):
    pic = BY_LEVELS[name](hb)
    s = pic.syn
    order = hb.intra_levels(pic)
    intra = [i for i in range(s.num_tus) if s.tus[i].flags & hb.abi.HEVC_TU_INTRA]
    bands = {i: max(1, (1 << s.tus[i].log2_size) // 8) for i in intra}
    assert sorted(order[:, 0].tolist()) == [i for i in intra for _ in range(bands[i])]
    # the items to be complete before: all of the levels before
    before = order[:, 1]
    assert before[0] == 0 and (np.diff(before) >= 0).all() and (before <= np.arange(len(before))).all()
    assert all(before[k] == before[k - 1] or before[k] == k for k in range(1, len(before)))
    level = {int(i): int(b) for i, b in order}
    assert all(level[int(i)] == b for i, b in order), "a TU's bands are of one level"
    writer, readers = {}, {}
    for i in intra:
        covered, around = touched(s, s.tus[i])
        for u in around:
            assert u not in writer or level[writer[u]] < level[i], (i, u)
        for u in covered:
            assert u not in writer or level[writer[u]] < level[i], (i, u)
            assert all(level[r] < level[i] for r in readers.get(u, ())), (i, u)
        for u in around:
            readers.setdefault(u, []).append(i)
        for u in covered:
            writer[u] = i
            readers[u] = []


@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_pictures_coded_once_stay_with_the_ctu_form_and_in_its_sizes(hb, name):
    c = CONFIGS[name]
    pic = hb.Picture(hb.default_cfg(c["w"], c["h"], c["seed"], **c["cfg"]))
    assert len(hb.intra_levels(pic)) == 0
    sch = hb.intra_schedule(pic)
    for k in range(len(sch["ctu_addr"])):
        tasks = range(int(sch["ctu_first"][k]), int(sch["ctu_first"][k + 1]))
        sizes = [1 << pic.syn.tus[int(sch["task_tu"][j])].log2_size for j in tasks]
        assert sum(max(1, n // 8) if n > 8 else 1 for n in sizes) <= MAX_ITEMS
        assert sum(int(sch["task_deps"][j]) & 63 for j in tasks) <= MAX_ENTRIES


@pytest.mark.parametrize("n_large", [2, 190])
def test_records_past_the_ctu_form_are_accepted_and_leave_it(hb, n_large):
    """Past MAX_ITEMS and MAX_ENTRIES with 190, below both with 2."""
    pic = one_place(hb, n_large)
    sch = hb.intra_schedule(pic)
    assert len(sch["task_tu"]) == 192 + n_large
    assert (192 + 4 * n_large > MAX_ITEMS) == (n_large == 190) == (len(sch["deps"]) > MAX_ENTRIES)
    assert len(hb.intra_levels(pic)) == 192 + 4 * n_large


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(BY_LEVELS))
def test_gpu_levels(hb, gpu_ctx, port, name):
    pic = BY_LEVELS[name](hb)
    p = pic.syn.params
    content = hb.content(p.width, p.height, 4)
    assert (gpu_ctx.intra_recon(pic, content) == port.intra_recon(pic, content)).all()


@pytest.mark.gpu
def test_gpu_levels_beside_ctus(hb, gpu_ctx, port):
    """Both forms in one batch, twice, and the same pictures one by one."""
    w, h = 416, 240
    refs = [hb.content(w, h, 1), hb.content(w, h, 2)]
    pics = [repeated(hb, w, h, 31, 0.05, **cases.PICTURE), hb.Picture(hb.default_cfg(w, h, 32, **cases.PICTURE)),
            repeated(hb, w, h, 33, 0.05, slice_type=2), hb.Picture(hb.default_cfg(w, h, 34, slice_type=2))]
    assert [len(hb.intra_levels(p)) > 0 for p in pics] == [True, False, True, False]
    want = [port.reconstruct_picture(p, refs) for p in pics]
    streams, jobs = [], []
    for p in pics:
        st = gpu_ctx.open_stream(w, h, 3)
        for slot, r in enumerate(refs):
            st.upload(slot, r)
        streams.append(st)
        jobs.append(st.prepare(p))
    for _ in range(2):
        hb.batch_launch(jobs, [2] * 4)
    gpu_ctx.sync()
    for st, x in zip(streams, want):
        assert (st.download(2) == x).all()
    for job in jobs:
        job.launch(2)
    gpu_ctx.sync()
    for st, x in zip(streams, want):
        assert (st.download(2) == x).all()
    for j in jobs:
        j.free()
    for st in streams:
        st.close()


@pytest.mark.gpu
def test_gpu_levels_wait_gives_up(hb, gpu_ctx):
    pic = one_place(hb, 2)
    st = gpu_ctx.open_stream(64, 64, 3)
    job = st.prepare(pic)
    job.plant_unmet_wait()
    job.launch(2)
    with pytest.raises(hb.HevcGpuError) as e:
        gpu_ctx.sync()
    assert e.value.code == hb.abi.HEVCGPU_ETIMEOUT
    job.free()
    job = st.prepare(pic)   # the context stays usable
    job.launch(2)
    gpu_ctx.sync()
    job.free()
    st.close()
