"""The residual kernel where its CTAs end: counts of each size around a CTA's capacity (128, 16,
8 and 4 blocks), sizes that are missing, every QP, levels over the whole int16 range, transform
skip, bypass, and flat and drawn scaling lists; every output byte equals the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, 0, 0, 0), (127, 0, 0, 5), (128, 17, 0, 0), (129, 15, 9, 3), (0, 16, 7, 0),
                                    (0, 1, 8, 4), (300, 100, 50, 25), (0, 0, 1, 1)])
@pytest.mark.parametrize("scaled", [False, True])
def test_gpu_residual_sizes(hb, gpu_ctx, port, counts, scaled):
    rng = np.random.default_rng(sum(c * 10 ** k for k, c in enumerate(counts)) + scaled)
    sizes = rng.permutation(np.repeat([2, 3, 4, 5], counts))
    tus, at = (hb.TU * len(sizes))(), 0
    for t, lg in zip(tus, sizes):
        t.log2_size, t.coeff_offset, t.qp = int(lg), at, int(rng.integers(0, 100))
        t.c_idx = int(rng.integers(0, 3)) if lg < 5 else 0
        t.flags = hb.abi.HEVC_TU_CODED | int(rng.choice([0, hb.abi.HEVC_TU_INTRA]))
        t.flags |= int(rng.choice([0, 0, 0, hb.abi.HEVC_TU_BYPASS, hb.abi.HEVC_TU_TSKIP if lg == 2 else 0]))
        at += 1 << 2 * int(lg)
    kind = rng.random(at)
    coeffs = np.where(kind < 0.6, 0, np.where(kind < 0.9, rng.integers(-90, 91, at), rng.integers(-32768, 32768, at)))
    coeffs = coeffs.astype(np.int16)
    pred = rng.integers(0, 256, at).astype(np.uint8)
    sl = [hb.scaling(len(sizes))] if scaled else []
    got = gpu_ctx.residual_blocks(tus, len(sizes), coeffs, pred, *sl)
    assert (got == port.residual_blocks(tus, len(sizes), coeffs, pred, *sl)).all()
