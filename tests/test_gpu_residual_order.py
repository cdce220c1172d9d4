"""Blocks that cover samples of another block are added size by size, 4x4 first: in a picture (a
damaged stream can code a block twice) and in a caller's pool.  Every output byte equals the
oracle's, which goes through them in the order of the records, here with rising sizes where
they meet."""
import ctypes as C
import random

import numpy as np
import pytest

import cases
from test_intra_levels import Records, fields

pytestmark = pytest.mark.gpu


def over_smaller(hb, w, h, seed):
    """A P/B picture, then blocks of each size over coded blocks that are all smaller."""
    pic = hb.Picture(hb.default_cfg(w, h, seed, **dict(cases.PICTURE, p_intra=0.0)))
    rng = random.Random(seed)
    tus = fields(pic)
    of_size = {lg: [t for t in tus if t["log2_size"] == lg and t["flags"] & hb.abi.HEVC_TU_CODED] for lg in range(2, 6)}
    size = [np.zeros((h // (2 if c else 1) // 4, w // (2 if c else 1) // 4), np.int32) for c in range(3)]
    for t in tus:
        if t["flags"] & hb.abi.HEVC_TU_CODED:
            n = (1 << t["log2_size"]) // 4
            y, x = t["y"] // 4, t["x"] // 4
            size[t["c_idx"]][y:y + n, x:x + n] = t["log2_size"]
    added = 0
    for lg in (3, 4, 5):
        n = (1 << lg) // 4
        for c in range(3):
            for y in range(0, size[c].shape[0] - n + 1, n):
                for x in range(0, size[c].shape[1] - n + 1, n):
                    part = size[c][y:y + n, x:x + n]
                    if part.any() and part.max() < lg and rng.random() < 0.5 and of_size[lg]:
                        tus.append(dict(rng.choice(of_size[lg]), x=4 * x, y=4 * y, c_idx=c))
                        part[:] = lg
                        added += 1
    assert added > 20
    return Records(hb, pic, tus)


@pytest.mark.parametrize("w,h,seed", [(128, 64, 3), (416, 240, 4), (1280, 720, 5)])
def test_gpu_blocks_of_a_picture_over_others(hb, gpu_ctx, port, w, h, seed):
    pic = over_smaller(hb, w, h, seed)
    refs = [hb.content(w, h, 1), hb.content(w, h, 2)]
    want = port.reconstruct_picture(pic, refs)
    for _ in range(3):
        assert (gpu_ctx.reconstruct_picture(pic, refs) == want).all()


@pytest.mark.parametrize("static", [False, True])
def test_gpu_blocks_of_a_pool_over_others(hb, gpu_ctx, port, static):
    """Blocks of rising size over each other in a pool of 64 x 32x32."""
    import test_zz_no_alloc as no_alloc
    rng = np.random.default_rng(8)
    tus = []
    for lg in (2, 3, 4, 5):   # each size covers half of the places before it
        step = 1 << 2 * lg
        tus += [(lg, at) for at in range(0, 64 * 1024, step) if rng.random() < 0.5]
    arr = (hb.TU * len(tus))()
    for t, (lg, at) in zip(arr, tus):
        t.log2_size, t.coeff_offset, t.qp, t.flags = lg, at, int(rng.integers(20, 40)), hb.abi.HEVC_TU_CODED
    coeffs = rng.integers(-90, 91, 64 * 1024).astype(np.int16)
    pred = rng.integers(0, 256, 64 * 1024).astype(np.uint8)
    want = port.residual_blocks(arr, len(tus), coeffs, pred)
    covered = np.zeros(64 * 1024, bool)
    for lg, at in tus:
        covered[at:at + (1 << 2 * lg)] = True
    for _ in range(3):
        if static:
            got = no_alloc._run_static(hb, gpu_ctx, no_alloc._static_fn(hb)[1], arr, len(tus), coeffs, pred)
        else:
            got = gpu_ctx.residual_blocks(arr, len(tus), coeffs, pred)
        assert (got == want)[covered].all()
