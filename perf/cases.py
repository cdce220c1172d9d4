"""Performance cases of the reconstruction back end, through its public entry points.

Pictures are seeded synthetic syntax with the distributions of the repository's tests and
benchmark (CU quadtree split 0.5 down to 8x8, QP 22..37, MVs of +-256 quarter samples, 50 %
bi-prediction, 10 % explicit weights, SAO per CTU); reference pictures are the generator's
sinusoid content.  Every output is 8-bit samples, so outputs are compared byte for byte.

Kinds:
  launch    pictures whose records already lie in HBM (prepared jobs) into DPB slots: one
            launch per stage over the batch ("batch"), or picture by picture ("plain")
  gop       streams' groups of pictures: an I picture, then P/B pictures that each reference
            the two before, position by position in decode order
  decode    records in page-locked host memory -> prepared, uploaded, reconstructed, frames
            copied back into page-locked host buffers
  residual, inter, filters
            the stage calls on host buffers (dequantisation + inverse transform + add, motion
            compensation, deblocking + SAO)
"""
import ctypes as C
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from __graft_entry__ import load_package

hb = load_package()

PB = dict(p_intra=0.1, p_skip=0.2, p_merge=0.3)                          # a P/B picture
INTER = dict(p_intra=0.0, sao=0)                                         # motion compensation alone
FILTERS = dict(p_intra=0.1, p_merge=0.95, p_cbf_luma=0.15, p_skip=0.8)   # Bs 0/1/2 about 0.5/0.3/0.2
MIXED = ((416, 240), (416, 240), (416, 240), (416, 240), (1280, 720), (1280, 720), (1280, 720), (1920, 1080),
         (1920, 1080), (3840, 2160))
FRAME_OPTIONS = dict(log2_ctb=6, p_intra=0.1, p_pcm=0.0, scaling=False, tile_cols=1, tile_rows=1)


def listed():
    return [
        # 4096 independent residual blocks from host memory: the smallest unit a host decoder
        # hands over
        dict(name="residual_4096", kind="residual", blocks=4096, scaling=False),
        # motion compensation of one 1080p picture from two host reference pictures
        dict(name="inter_1080p", kind="inter", width=1920, height=1080),
        # deblocking and SAO of one 2160p picture in host memory
        dict(name="filters_2160p", kind="filters", width=3840, height=2160),
        # one small P/B picture, one launch per stage: the least work, where launches count
        dict(name="pb_416x240_1", kind="launch", form="plain", pictures="PB", width=416, height=240, streams=1,
             **FRAME_OPTIONS),
        # one 1080p P/B picture on its own: a single live stream
        dict(name="pb_1080p_1", kind="launch", form="plain", pictures="PB", width=1920, height=1080, streams=1,
             **FRAME_OPTIONS),
        # the steady state of a server: 16 streams' 1080p P/B pictures in one batch
        dict(name="pb_1080p_16", kind="launch", form="batch", pictures="PB", width=1920, height=1080, streams=16,
             **FRAME_OPTIONS),
        # segment starts: 8 streams' 1080p I pictures in one batch
        dict(name="i_1080p_8", kind="launch", form="batch", pictures="I", width=1920, height=1080, streams=8,
             **FRAME_OPTIONS),
        # 4 streams' 2160p P/B pictures in one batch
        dict(name="pb_2160p_4", kind="launch", form="batch", pictures="PB", width=3840, height=2160, streams=4,
             **FRAME_OPTIONS),
        # 4 streams' 720p groups of 8 pictures: consecutive batches depend on each other
        dict(name="gop_720p_4x8", kind="gop", width=1280, height=720, streams=4, frames=8, **FRAME_OPTIONS),
        # continuous batching: ten streams of four sizes (4:3:2:1) in one batch, every fifth one
        # at the I picture of a new segment
        dict(name="mixed_10", kind="launch", form="batch", pictures="mixed", width=0, height=0, streams=10,
             **FRAME_OPTIONS),
        # 8 streams' 1080p P/B pictures from records on the host to frames on the host
        dict(name="decode_1080p_8", kind="decode", width=1920, height=1080, streams=8, **FRAME_OPTIONS),
        # the optional tools at a ragged size: 32x32 CTBs, tiles, scaling lists, PCM, more intra
        dict(name="tools_1000x568_4", kind="launch", form="batch", pictures="PB", width=1000, height=568, streams=4,
             log2_ctb=5, p_intra=0.3, p_pcm=0.1, scaling=True, tile_cols=3, tile_rows=2),
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _size(rng, lo, hi):
    """A picture of lo..hi luma samples' width in one of the usual aspect ratios, a multiple of 8."""
    w = _log_uniform(rng, lo, hi)
    h = w * rng.uniform(0.5, 0.6)
    return max(64, int(w) // 8 * 8), max(40, int(h) // 8 * 8)


def _options(rng):
    log2_ctb = rng.choice((6, 6, 6, 5, 4))
    tiles = rng.random() < 0.2
    return dict(log2_ctb=log2_ctb, p_intra=round(rng.uniform(0.02, 0.3), 3), p_pcm=0.05 if rng.random() < 0.15 else 0.0,
                scaling=rng.random() < 0.2, tile_cols=2 if tiles else 1, tile_rows=2 if tiles else 1)


def draw(rng):
    kind = rng.choice(("launch",) * 6 + ("gop", "decode", "residual", "inter", "filters"))
    if kind == "residual":
        return dict(kind=kind, blocks=int(_log_uniform(rng, 256, 16384)), scaling=rng.random() < 0.3)
    if kind in ("inter", "filters"):
        w, h = _size(rng, 200, 1920 if kind == "inter" else 3840)
        return dict(kind=kind, width=w, height=h)
    if kind == "gop":
        w, h = _size(rng, 200, 1280)
        return dict(kind=kind, width=w, height=h, streams=rng.randint(1, 4), frames=rng.randint(3, 5), **_options(rng))
    if kind == "decode":
        w, h = _size(rng, 200, 1920)
        return dict(kind=kind, width=w, height=h, streams=rng.randint(1, 8), **_options(rng))
    pictures = rng.choice(("PB", "PB", "PB", "I"))
    w, h = _size(rng, 200, 3840 if pictures == "PB" else 1920)
    most = max(1, min(16 if pictures == "PB" else 8, 16 * 1920 * 1080 // (w * h)))
    n = max(1, min(most, int(_log_uniform(rng, 1, most + 1))))
    return dict(kind="launch", form="plain" if n == 1 else "batch", pictures=pictures, width=w, height=h, streams=n,
                **_options(rng))


# ------------------------------------------------------------------------------ inputs

_CTX = None


def _context():
    """The one context a decoding process has per device."""
    global _CTX
    if _CTX is None:
        torch.cuda.init()
        _CTX = hb.Context(0)
    return _CTX


def _syntax_options(case):
    return dict(log2_ctb=case["log2_ctb"], p_pcm=case["p_pcm"], scaling_lists=int(case["scaling"]),
                tile_cols=case["tile_cols"], tile_rows=case["tile_rows"])


def _picture(case, w, h, kind, seed):
    if kind == "I":
        return hb.Picture(hb.default_cfg(w, h, seed, slice_type=2, poc=0, **_syntax_options(case)))
    return hb.Picture(hb.default_cfg(w, h, seed, poc=8, **dict(PB, p_intra=case["p_intra"]), **_syntax_options(case)))


def _reference(pic, slots):
    """The DPB slots of the picture's two reference pictures, nearest first in list 0."""
    prm = pic.syn.params
    for i in range(prm.num_ref[0]):
        prm.ref_slot[0][i] = slots[i]
    for i in range(prm.num_ref[1]):
        prm.ref_slot[1][i] = slots[1 - i]


def _threads(f, items):
    with ThreadPoolExecutor(os.cpu_count() or 4) as ex:
        return list(ex.map(f, items))


class _Plane:
    def __init__(self, ptr, h, w, pitch):
        self.__cuda_array_interface__ = dict(shape=(h, w), typestr="|u1", data=(ptr, False), strides=(pitch, 1),
                                             version=3)


def _slot_views(stream, slot):
    """The samples of a DPB slot where they lie (the zero-copy output): one tensor when the
    planes follow each other without gaps, else one per plane."""
    p = [C.c_void_p() for _ in range(3)]
    py, pc = C.c_int32(), C.c_int32()
    rc = stream.lib.hevcgpu_slot_device_ptr(stream.h, slot, C.byref(p[0]), C.byref(p[1]), C.byref(p[2]), C.byref(py),
                                            C.byref(pc))
    if rc:
        raise RuntimeError("hevcgpu_slot_device_ptr")
    w, h = stream.width, stream.height
    if py.value == w and pc.value == w // 2:
        return [torch.as_tensor(_Plane(p[0].value, h * 3 // 2, w, w), device="cuda")]
    return [torch.as_tensor(_Plane(p[0].value, h, w, py.value), device="cuda")] + \
        [torch.as_tensor(_Plane(p[k].value, h // 2, w // 2, pc.value), device="cuda") for k in (1, 2)]


def _blocks(n, seed):
    """n blocks of the generator's mix with the share of each size fixed (50 % 4x4, 25 % 8x8,
    15 % 16x16, 10 % 32x32), so that every seed fills a pool of one length."""
    tus, drawn, coeffs, pred = hb.blocks(3 * n, seed)
    left = {2: n // 2, 3: n // 4, 4: n * 15 // 100}
    left[5] = n - sum(left.values())
    picked = []
    for i in range(drawn):
        if left[tus[i].log2_size]:
            left[tus[i].log2_size] -= 1
            picked.append(i)
    out = (hb.TU * n)()
    parts, end = [], 0
    for k, i in enumerate(picked):
        out[k] = tus[i]
        size = 1 << 2 * tus[i].log2_size
        parts.append(slice(tus[i].coeff_offset, tus[i].coeff_offset + size))
        out[k].coeff_offset = end
        end += size
    return out, n, np.concatenate([coeffs[p] for p in parts]), np.concatenate([pred[p] for p in parts])


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    if kind == "residual":
        tus, n, coeffs, pred = _blocks(case["blocks"], seed)
        return dict(case=case, ctx=ctx, tus=tus, n=n, coeffs=coeffs, pred=pred,
                    scaling=hb.scaling(seed) if case["scaling"] else None)
    if kind in ("inter", "filters"):
        w, h = case["width"], case["height"]
        pic = hb.Picture(hb.default_cfg(w, h, seed, **(INTER if kind == "inter" else FILTERS)))
        return dict(case=case, ctx=ctx, pic=pic,
                    content=_threads(lambda k: hb.content(w, h, 3 * seed + k), range(2 if kind == "inter" else 1)))
    if kind == "gop":
        return _prepare_gop(case, ctx, seed)
    n = case["streams"]
    sizes = MIXED[:n] if case.get("pictures") == "mixed" else ((case["width"], case["height"]),) * n
    kinds = [case.get("pictures", "PB")] * n
    if kinds[0] == "mixed":
        kinds = ["I" if i % 5 == 0 else "PB" for i in range(n)]

    def make(i):
        pic = _picture(case, *sizes[i], kinds[i], 1000 * seed + i)
        _reference(pic, (0, 1))
        refs = [hb.content(*sizes[i], 1000 * seed + 100 * i + k) for k in range(2)] if kinds[i] == "PB" else []
        return pic, refs

    made = _threads(make, range(n))
    streams = []
    for (w, h), (_, refs) in zip(sizes, made):
        st = ctx.open_stream(w, h, 3)
        for slot, plane in enumerate(refs):
            st.upload(slot, plane)
        streams.append(st)
    pics = [p for p, _ in made]
    if kind == "decode":
        frames = [torch.empty(hb.i420_size(w, h), dtype=torch.uint8).pin_memory().numpy() for w, h in sizes]
        return dict(case=case, ctx=ctx, streams=streams, pics=[p.pin() for p in pics], frames=frames, lane=hb.Lane(ctx),
                    slots=[2] * n)
    jobs = hb.prepare_batch(streams, pics)
    return dict(case=case, ctx=ctx, streams=streams, jobs=jobs, slots=[2] * n,
                out=[v for st in streams for v in _slot_views(st, 2)])


def _prepare_gop(case, ctx, seed):
    """Position k of a stream writes slot k; slot `frames` holds the picture before the group."""
    w, h, n, frames = case["width"], case["height"], case["streams"], case["frames"]

    def make(i):
        pic = _picture(case, w, h, "I" if i < n else "PB", 1000 * seed + i)
        if i >= n:
            k = i // n
            _reference(pic, (k - 1, k - 2 if k > 1 else frames))
        return pic

    pics = _threads(make, range(n * frames))
    before = _threads(lambda i: hb.content(w, h, 1000 * seed + 500 + i), range(n))
    streams = [ctx.open_stream(w, h, frames + 1) for _ in range(n)]
    for st, plane in zip(streams, before):
        st.upload(frames, plane)
    jobs = [hb.prepare_batch(streams, pics[n * k:n * (k + 1)]) for k in range(frames)]
    return dict(case=case, ctx=ctx, streams=streams, jobs=jobs,
                out=[v for k in range(frames) for st in streams for v in _slot_views(st, k)])


# ------------------------------------------------------------------------------ one pass

def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "residual":
        return ctx.residual_blocks(state["tus"], state["n"], state["coeffs"], state["pred"], state["scaling"])
    if kind == "inter":
        return ctx.inter_pred(state["pic"], state["content"])
    if kind == "filters":
        return ctx.loop_filter(state["pic"], state["content"][0])
    if kind == "gop":
        for k, jobs in enumerate(state["jobs"]):
            hb.batch_launch(jobs, [k] * len(jobs))
        return state["out"]
    if kind == "decode":
        jobs = hb.prepare_batch(state["streams"], state["pics"], wait_uploads=False)
        state["lane"].batch_launch(jobs, state["slots"])
        ticket = state["lane"].download_batch_async(state["streams"], state["slots"], state["frames"])
        state["lane"].wait(ticket)
        for job in jobs:
            job.free()
        return state["frames"]
    if case["form"] == "plain":
        for job in state["jobs"]:
            job.launch(2)
    else:
        hb.batch_launch(state["jobs"], state["slots"])
    return state["out"]


# ------------------------------------------------------------------------------ least work

def _record_bytes(pic):
    s = pic.syn
    return 16 * s.num_tus + 2 * s.num_coeffs + 20 * s.num_pus + (s.params.width // 4) * (s.params.height // 4) * 4


def _picture_bytes(case, w, h, kind):
    """Records and reference pictures read once, the picture written once; the records'
    density is that of a picture of at most 512x512 of the same kind."""
    sw, sh = min(w, 512), min(h, 512)
    frame = w * h * 3 // 2
    records = _record_bytes(_picture(case, sw, sh, kind, 1)) * (w * h) / (sw * sh)
    return records + frame * (1 if kind == "I" else 3)


def work(case):
    kind = case["kind"]
    if kind == "residual":
        _, n, coeffs, _ = _blocks(case["blocks"], 1)
        return dict(bytes=16 * n + 4 * coeffs.size, flops=0)
    if kind in ("inter", "filters"):
        w, h = case["width"], case["height"]
        grid = (w // 4) * (h // 4) * 4
        return dict(bytes=w * h * 3 // 2 * (3 if kind == "inter" else 2) + (0 if kind == "inter" else grid), flops=0)
    if kind == "gop":
        w, h = case["width"], case["height"]
        total = _picture_bytes(case, w, h, "I") + (case["frames"] - 1) * _picture_bytes(case, w, h, "PB")
        return dict(bytes=int(case["streams"] * total), flops=0)
    if case.get("pictures") == "mixed":
        return dict(bytes=int(sum(_picture_bytes(case, w, h, "I" if i % 5 == 0 else "PB")
                                  for i, (w, h) in enumerate(MIXED[:case["streams"]]))), flops=0)
    return dict(bytes=int(case["streams"] * _picture_bytes(case, case["width"], case["height"],
                                                           case.get("pictures", "PB"))), flops=0)
