"""dequant.h against the 64-bit formula it stands for (transform.cpp:360-365: product, shift by
qP / 6, rounding shift, narrowing modulo 2^32), on the CPU and with signed overflow trapped: at
every QP that validation accepts and every block size, levels at the ends of int16 and around 0,
scaling factors at the ends of a byte.  Then transform skip and bypass at every size on the GPU
against the oracle."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCALE = [40, 45, 51, 57, 64, 72]

WRAPPER = r"""
#include "dequant.h"
extern "C" void levels(int scale, int qp, int log2, int m, const int* in, int n, int* out) {
    const hevcgpu::Dequant q = hevcgpu::dequant_make(scale, qp, log2);
    for (int i = 0; i < n; i++) out[i] = hevcgpu::dequant_level(in[i], m, q);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("dequant")
    (d / "w.cpp").write_text(WRAPPER)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error",
                    "-I", os.path.join(ROOT, "hevc.js_b200", "csrc"), "-o", str(d / "w.so"), str(d / "w.cpp")], check=True)
    return C.CDLL(str(d / "w.so"))


@pytest.mark.parametrize("log2", [2, 3, 4, 5])
def test_dequant_is_the_64_bit_formula(lib, log2):
    edge = [-32768, -32767, -4097, -256, -91, -2, -1, 0, 1, 2, 63, 90, 255, 4096, 32766, 32767]
    c = np.array(edge + np.random.default_rng(log2).integers(-32768, 32768, 200).tolist(), np.int32)
    out = np.empty_like(c)
    p = C.POINTER(C.c_int)
    for qp in range(100):
        for m in (0, 1, 16, 115, 254, 255):
            lib.levels(SCALE[qp % 6], qp, log2, m, c.ctypes.data_as(p), len(c), out.ctypes.data_as(p))
            shift = 3 + log2
            want = [(((int(v) * m * SCALE[qp % 6] << (qp // 6)) + (1 << (shift - 1))) >> shift) & 0xFFFFFFFF for v in c]
            want = np.array([w - (1 << 32) if w >> 31 else w for w in want])
            assert (out == want)[c != 0].all(), (qp, m)
            assert (np.clip(out, -32768, 32767) == np.clip(want, -32768, 32767)).all(), (qp, m)


@pytest.mark.gpu
@pytest.mark.parametrize("scaled", [False, True])
def test_gpu_transform_skip_and_bypass_at_every_size(hb, gpu_ctx, port, scaled):
    rng = np.random.default_rng(40 + scaled)
    sizes = rng.permutation(np.repeat([2, 3, 4, 5], (130, 40, 20, 10)))
    tus, at = (hb.TU * len(sizes))(), 0
    for t, lg in zip(tus, sizes):
        t.log2_size, t.coeff_offset, t.qp = int(lg), at, int(rng.integers(0, 100))
        t.flags = hb.abi.HEVC_TU_CODED | int(rng.choice([hb.abi.HEVC_TU_TSKIP, hb.abi.HEVC_TU_TSKIP, hb.abi.HEVC_TU_BYPASS]))
        at += 1 << 2 * int(lg)
    coeffs = np.where(rng.random(at) < 0.5, rng.integers(-90, 91, at), rng.integers(-32768, 32768, at)).astype(np.int16)
    pred = rng.integers(0, 256, at).astype(np.uint8)
    sl = [hb.scaling(7)] if scaled else []
    got = gpu_ctx.residual_blocks(tus, len(sizes), coeffs, pred, *sl)
    assert (got == port.residual_blocks(tus, len(sizes), coeffs, pred, *sl)).all()
