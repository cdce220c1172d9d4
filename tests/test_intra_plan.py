"""intra_plan.h (what an intra TU reads, worked out from positions and its mode) against
per-sample definitions of its own, on the CPU: availability and substitution sample by sample
(intra_prediction.cpp:102-133, 177-197), the parts of the reference array a mode reads against
the samples its formulas touch, and the 4x4 and 8x8 weights against the prediction formulas
(:263-422).  All results are integers: equality."""
import ctypes as C
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ANGLE = [0, 0, 32, 26, 21, 17, 13, 9, 5, 2, 0, -2, -5, -9, -13, -17, -21, -26, -32, -26, -21, -17, -13, -9, -5, -2, 0,
         2, 5, 9, 13, 17, 21, 26, 32]
INV = [0] * 11 + [4096, 1638, 910, 630, 482, 390, 315, 256, 315, 390, 482, 630, 910, 1638, 4096] + [0] * 9

WRAPPER = r"""
#include "intra_plan.h"
using namespace hevcgpu;
extern "C" {
void subst(int x, int y, int n, int pw, int ph, int log2c, int sub, unsigned nb, int* out) {
    const unsigned w = avail_pack(intra_avail(x, y, n, pw, ph, log2c, sub, nb));
    for (int i = 0; i <= 4 * n; i++) out[i] = intra_substitute(avail_unpack(w, n), i);
}
int smoothed(int mode, int log2, int chroma, int disabled) { return intra_smoothed(mode, log2, chroma, disabled); }
unsigned need(int mode, int log2, int chroma, int pcm, int smooth, int bl, int tr, int l, int c, int t) {
    const IntraAvail a{1 << log2, bl, tr, l != 0, c != 0, t != 0};
    return intra_need(intra_parts(mode, log2, chroma, pcm, smooth), avail_segs(a));
}
int substitute(int log2, int bl, int tr, int l, int c, int t, int i) {
    return intra_substitute(IntraAvail{1 << log2, bl, tr, l != 0, c != 0, t != 0}, i);
}
int main_index(int vert, int inv, int n, int q) { return intra_main_index(vert, inv, n, q); }
void taps(int log2, int mode, int chroma, int x, int y, int lane, int* out) {
    static const IntraTapTable table = intra_tap_table();
    const IntraTaps k = log2 == 2 ? intra_taps_unpack(table.t[mode][chroma][lane][0], table.t[mode][chroma][lane][1])
                                  : intra_taps(log2, mode, chroma, x, y, lane, intra_angle(mode), intra_inv_angle(mode));
    for (int j = 0; j < 4; j++) { out[j] = k.i[j]; out[4 + j] = k.w[j]; }
    out[8] = k.add;
    out[9] = k.shift;
}
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "w.cpp").write_text(WRAPPER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "hevc.js_b200", "csrc"),
                    "-o", str(d / "w.so"), str(d / "w.cpp")], check=True)
    lib = C.CDLL(str(d / "w.so"))
    lib.need.restype = C.c_uint
    return lib


def zscan(x, y):
    return sum(((x >> b) & 1) << (2 * b) | ((y >> b) & 1) << (2 * b + 1) for b in range(5))


def position(x, y, n, i):
    return (x - 1, y + 2 * n - 1 - i) if i < 2 * n else (x + i - 2 * n - 1, y - 1)


def available(x, y, px, py, pw, ph, log2c, sub, nb):
    """One sample: in the picture, and in a usable neighbour CTB or at a lower z-scan address."""
    if px < 0 or py < 0 or px >= pw or py >= ph:
        return False
    dx, dy = (px >> log2c) - (x >> log2c), (py >> log2c) - (y >> log2c)
    if (dx, dy) == (0, 0):
        m = (1 << log2c) - 1
        return zscan((px & m) * sub >> 2, (py & m) * sub >> 2) < zscan((x & m) * sub >> 2, (y & m) * sub >> 2)
    bit = {(-1, 0): 1, (-1, -1): 2, (0, -1): 4, (1, -1): 8}.get((dx, dy), 0)
    return bool(nb & bit)


@pytest.mark.parametrize("log2_ctb", [4, 5, 6])
@pytest.mark.parametrize("sub", [1, 2])
def test_substitution_is_the_sample_by_sample_rule(plan, log2_ctb, sub):
    log2c = log2_ctb - (sub - 1)
    pw, ph = (2 * 64 + 24) // sub, (2 * 64 + 40) // sub    # ragged against every CTB and TU size
    rng = random.Random(log2_ctb * 10 + sub)
    seen = 0
    for log2 in range(2, min(5, log2c) + 1):
        n = 1 << log2
        for y in range(0, ph - n + 1, n):
            for x in range(0, pw - n + 1, n):
                for nb in (15, 0, rng.randrange(16), rng.randrange(16)):
                    out = (C.c_int * (4 * n + 1))()
                    plan.subst(x, y, n, pw, ph, log2c, sub, nb, out)
                    ok = [available(x, y, *position(x, y, n, i), pw, ph, log2c, sub, nb) for i in range(4 * n + 1)]
                    first = ok.index(True) if any(ok) else -1
                    last = -1
                    for i in range(4 * n + 1):
                        if ok[i]:
                            last = i
                        assert out[i] == (last if last >= 0 else first), (x, y, n, nb, i)
                    seen += 1
    assert seen > 300


def reads(mode, log2, chroma, smooth):
    """Reference array indices the prediction's result depends on (weight not 0)."""
    n = 1 << log2
    left, top = set(range(n, 2 * n)), set(range(2 * n + 1, 3 * n + 1))
    if smooth and log2 == 5:
        return set(range(4 * n + 1))    # the strong filter's decision
    if mode == 0:
        s = left | top | {n - 1, 3 * n + 1}
    elif mode == 1:
        s = left | top
    else:
        s = set()
        vert = mode >= 18
        for along in range(n):
            idx, fr = (along + 1) * ANGLE[mode] >> 5, (along + 1) * ANGLE[mode] & 31
            for q in range(1 + idx, n + 1 + idx + (1 if fr else 0)):
                k = q if q >= 0 else -min(2 * n, (-q * INV[mode] + 128) >> 8)
                s.add(2 * n + k if vert else 2 * n - k)
        if not chroma and n < 32 and mode in (10, 26):
            s |= {2 * n} | (left if mode == 26 else top)
    if smooth:
        s = {j for i in s for j in ((i,) if i in (0, 4 * n) else (i - 1, i, i + 1))}
    return s


@pytest.mark.parametrize("log2", [2, 3, 4, 5])
def test_needed_parts_hold_every_sample_read(plan, log2):
    n = 1 << log2
    part = [1 if i < n else 2 if i < 2 * n else 4 if i == 2 * n else 8 if i <= 3 * n else 16 for i in range(4 * n + 1)]
    shapes = [(bl, tr, l, c, t) for bl in (0, 4, n) for tr in (0, 4, n) for l in (0, 1) for c in (0, 1) for t in (0, 1)
              if l or not bl]
    for mode in range(35):
        for chroma in (0, 1):
            for disabled in (0, 1):
                smooth = plan.smoothed(mode, log2, chroma, disabled)
                dist = min(abs(mode - 26), abs(mode - 10))
                assert bool(smooth) == (not chroma and log2 > 2 and not disabled and mode != 1 and
                                        dist > {3: 7, 4: 1, 5: 0}.get(log2, 99))
                s = reads(mode, log2, chroma, smooth)
                for a in shapes:
                    src = {plan.substitute(log2, *a, i) for i in s} - {-1}
                    got = plan.need(mode, log2, chroma, 0, smooth, *a)
                    want = 0
                    for i in src:
                        want |= part[i]
                    assert want & ~got == 0, (mode, chroma, smooth, a, want, got)
                    if log2 == 2 and all(a) and a[:2] == (n, n):
                        assert want == got, (mode, chroma)    # 4x4: nothing waited for in vain
                    assert plan.need(mode, log2, chroma, 1, smooth, *a) == 0


@pytest.mark.parametrize("mode", range(35))
@pytest.mark.parametrize("chroma", [0, 1])
@pytest.mark.parametrize("log2", [2, 3])
def test_taps_of_a_block_are_its_prediction(plan, mode, chroma, log2):
    rng = random.Random(mode)
    n = 1 << log2
    for trial in range(24 if log2 == 2 else 6):
        R = [rng.choice((0, 255)) if trial < 2 * n else rng.randrange(256) for _ in range(4 * n + 1)]
        dc = (sum(R[n:2 * n]) + sum(R[2 * n + 1:3 * n + 1]) + n) >> (log2 + 1)
        for y in range(n):
            for x in range(n):
                left, top, corner = R[2 * n - 1 - y], R[2 * n + 1 + x], R[2 * n]
                if mode == 0:
                    want = ((n - 1 - x) * left + (x + 1) * R[3 * n + 1] + (n - 1 - y) * top + (y + 1) * R[n - 1] + n) >> \
                        (log2 + 1)
                elif mode == 1:
                    want = dc
                    if not chroma and x == 0 and y == 0:
                        want = (left + 2 * dc + top + 2) >> 2
                    elif not chroma and y == 0:
                        want = (top + 3 * dc + 2) >> 2
                    elif not chroma and x == 0:
                        want = (left + 3 * dc + 2) >> 2
                else:
                    vert = mode >= 18
                    main = (lambda q: R[2 * n + q] if vert else R[2 * n - q])
                    side = (lambda k: R[2 * n - k] if vert else R[2 * n + k])
                    ref = (lambda q: main(q) if q >= 0 else side(min(2 * n, (-q * INV[mode] + 128) >> 8)))
                    along, across = (y, x) if vert else (x, y)
                    idx, fr = (along + 1) * ANGLE[mode] >> 5, (along + 1) * ANGLE[mode] & 31
                    want = ref(across + 1 + idx)
                    if fr:
                        want = ((32 - fr) * want + fr * ref(across + 2 + idx) + 16) >> 5
                    if not chroma and mode == 26 and x == 0:
                        want = min(255, max(0, want + ((left - corner) >> 1)))
                    if not chroma and mode == 10 and y == 0:
                        want = min(255, max(0, want + ((top - corner) >> 1)))
                k = (C.c_int * 10)()
                plan.taps(log2, mode, chroma, x, y, y * n + x, k)
                v = [R[k[j]] for j in range(4)]
                if mode == 1:
                    total = 0
                    for other in range(2 * n):
                        k2 = (C.c_int * 10)()
                        plan.taps(log2, mode, chroma, x, y, other, k2)
                        total += R[k2[1]]
                    v[1] = (total + n) >> (log2 + 1)
                got = sum(v[j] * k[4 + j] for j in range(4)) + k[8] >> k[9]
                assert min(255, max(0, got)) == want, (x, y, trial)
