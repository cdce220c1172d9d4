// intra_plan.h — what an intra TU reads, from positions and its mode alone: which of its
// reference samples are available (build_reference_samples, intra_prediction.cpp:102-133),
// which sample stands in for one that is not (:177-197), which parts of the reference array
// the prediction reads, and for a 4x4 or 8x8 TU the samples and weights of each output
// sample
// (:263-422).  k_intra_ctus works all of it out before it waits for any sample.  Host and
// device code; no CUDA header is needed, so the rules are tested on the CPU.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define HEVC_HD constexpr __host__ __device__ __forceinline__
#else
#define HEVC_HD constexpr inline
#endif

namespace hevcgpu {

// Neighbour CTBs an intra TU may read from, as bits of a mask: they must precede the
// current CTB in raster order and share its slice and tile (intra_prediction.cpp:108-124).
enum : uint32_t { NB_LEFT = 1u, NB_ABOVE_LEFT = 2u, NB_ABOVE = 4u, NB_ABOVE_RIGHT = 8u };

// The reference array of an n x n TU has 4n + 1 samples: indices 0 .. 2n - 1 run up the left
// column (0 the lowest), 2n is the corner, 2n + 1 .. 4n run along the row above.  Its parts,
// in index order:
enum : uint32_t {
    SEG_BL = 1u,   // 0 .. n - 1: below-left
    SEG_L = 2u,    // n .. 2n - 1: left
    SEG_C = 4u,    // 2n: corner
    SEG_T = 8u,    // 2n + 1 .. 3n: top
    SEG_TR = 16u,  // 3n + 1 .. 4n: top-right
    SEG_ALL = 31u,
};

HEVC_HD int plan_min(int a, int b) { return a < b ? a : b; }
HEVC_HD int plan_max(int a, int b) { return a > b ? a : b; }

// 8-bit z-order address of a 4x4 unit inside a CTU (bit-interleave of 4-bit x, y).
HEVC_HD uint32_t zorder16(uint32_t bx, uint32_t by) {
    bx = (bx | (bx << 2)) & 0x33u;
    bx = (bx | (bx << 1)) & 0x55u;
    by = (by | (by << 2)) & 0x33u;
    by = (by | (by << 1)) & 0x55u;
    return bx | (by << 1);
}

// The available samples of a reference array.  A TU lies at a multiple of its size, so each
// of the five parts lies in one n x n block of one CTB: the block is available as a whole
// (an earlier CTB of the slice and tile, or a lower z-scan address in this CTB), except that
// the picture's bottom and right edges cut the below-left and top-right parts short.
struct IntraAvail {
    int n;         // TU size
    int bl, tr;    // available samples of the below-left and top-right parts (next to the TU)
    bool l, c, t;  // left, corner, top
};

// TU at (x, y) of a plane of pw x ph samples whose CTBs are 1 << log2c wide; sub is the
// plane's subsampling, nb the mask of usable neighbour CTBs.
HEVC_HD IntraAvail intra_avail(int x, int y, int n, int pw, int ph, int log2c, int sub, uint32_t nb) {
    const int cs = 1 << log2c, xi = x & (cs - 1), yi = y & (cs - 1);
    const uint32_t z = zorder16((uint32_t)(xi * sub) >> 2, (uint32_t)(yi * sub) >> 2);
    IntraAvail a{};
    a.n = n;
    a.l = x > 0 && (xi > 0 || (nb & NB_LEFT));
    a.t = y > 0 && (yi > 0 || (nb & NB_ABOVE));
    a.c = x > 0 && y > 0 && (xi > 0 ? (yi > 0 || (nb & NB_ABOVE)) : (nb & (yi > 0 ? NB_LEFT : NB_ABOVE_LEFT)) != 0);
    const bool bl = a.l && yi + n < cs &&
                    (xi == 0 || zorder16((uint32_t)((xi - 1) * sub) >> 2, (uint32_t)((yi + n) * sub) >> 2) < z);
    a.bl = bl ? plan_max(0, plan_min(n, ph - (y + n))) : 0;
    bool tr = false;
    if (yi > 0) tr = xi + n < cs && zorder16((uint32_t)((xi + n) * sub) >> 2, (uint32_t)((yi - 1) * sub) >> 2) < z;
    else tr = y > 0 && (nb & (xi + n < cs ? NB_ABOVE : NB_ABOVE_RIGHT));
    a.tr = tr ? plan_max(0, plan_min(n, pw - (x + n))) : 0;
    return a;
}

HEVC_HD uint32_t avail_segs(const IntraAvail& a) {
    return (a.bl ? SEG_BL : 0u) | (a.l ? SEG_L : 0u) | (a.c ? SEG_C : 0u) | (a.t ? SEG_T : 0u) | (a.tr ? SEG_TR : 0u);
}

// Packed form: bits 0-5 bl, 6-11 tr, 12 l, 13 c, 14 t.
HEVC_HD uint32_t avail_pack(const IntraAvail& a) {
    return (uint32_t)a.bl | ((uint32_t)a.tr << 6) | ((uint32_t)a.l << 12) | ((uint32_t)a.c << 13) | ((uint32_t)a.t << 14);
}
HEVC_HD IntraAvail avail_unpack(uint32_t w, int n) {
    return IntraAvail{n, (int)(w & 63u), (int)((w >> 6) & 63u), ((w >> 12) & 1u) != 0, ((w >> 13) & 1u) != 0,
                      ((w >> 14) & 1u) != 0};
}

// The index whose sample stands at index i: i itself when available, else the nearest
// available one below it, else the first available one (:177-197); -1 when none is.
HEVC_HD int intra_substitute(const IntraAvail& a, int i) {
    const int n = a.n;
    const int first = a.l ? n - a.bl : (a.c ? 2 * n : (a.t ? 2 * n + 1 : (a.tr ? 3 * n + 1 : -1)));
    if (i < 2 * n) return a.l ? plan_max(i, n - a.bl) : first;
    if (i > 3 * n && a.tr) return plan_min(i, 3 * n + a.tr);
    if (i > 2 * n && a.t) return plan_min(i, 3 * n);
    return a.c ? 2 * n : (a.l ? 2 * n - 1 : first);
}

// Whether the luma reference array is smoothed (:443-471): thresholds 7, 1 and 0 for 8x8,
// 16x16 and 32x32 on the mode's distance from vertical and horizontal.
HEVC_HD bool intra_smoothed(int mode, int log2, bool chroma, bool disabled) {
    if (chroma || log2 == 2 || disabled || mode == 1) return false;
    const int v = mode > 26 ? mode - 26 : 26 - mode, h = mode > 10 ? mode - 10 : 10 - mode;
    return plan_min(v, h) > (log2 == 3 ? 7 : (log2 == 4 ? 1 : 0));
}

// The parts of the reference array whose samples the prediction depends on, before
// substitution.  Horizontal modes 2..9 read down the left column, 27..34 along the row above,
// those between read left, corner and top (the projection of the side reference reaches at
// most n samples); planar reads one sample of each far part.  Smoothing reads one sample
// further on both sides of every sample read: into the corner, and for the modes that read a
// whole side into the far part (taken as all parts; the diagonal mode 18 stays one short).
// The strong smoothing of 32x32 decides on samples of all parts.
HEVC_HD uint32_t intra_parts(int mode, int log2, bool chroma, bool pcm, bool smooth) {
    if (pcm) return 0u;   // the PCM samples are the levels, with no prediction
    const bool edge = !chroma && log2 < 5;
    if (mode == 0) return smooth ? SEG_ALL : SEG_BL | SEG_L | SEG_T | SEG_TR;
    if (mode == 1) return SEG_L | SEG_T;
    if (smooth && log2 == 5) return SEG_ALL;
    if (mode < 10) return SEG_BL | SEG_L | (smooth ? SEG_C : 0u);
    if (mode == 10) return edge ? SEG_L | SEG_C | SEG_T : SEG_L;
    if (mode == 26) return edge ? SEG_L | SEG_C | SEG_T : SEG_T;
    if (mode > 26) return SEG_T | SEG_TR | (smooth ? SEG_C : 0u);
    if (smooth && mode != 18) return SEG_ALL;
    // angles -2 and -5 (next to 10 and 26): n rows times the angle stay above -32 in small TUs
    // and reach the corner only
    const int d = mode < 18 ? mode - 10 : 26 - mode;
    const bool side = !(d == 1 && log2 < 5) && !(d == 2 && log2 == 2);
    return (mode < 18 || side ? SEG_L : 0u) | SEG_C | (mode >= 18 || side ? SEG_T : 0u);
}

// The available parts those samples come from after substitution: a part without samples is
// filled from the nearest available part below it, else from the first available one.
HEVC_HD uint32_t intra_need(uint32_t parts, uint32_t avail) {
    uint32_t need = 0;
    for (uint32_t s = SEG_BL; s <= SEG_TR; s <<= 1) {
        if (!(parts & s)) continue;
        uint32_t below = avail & (2u * s - 1u);
        if (below) {
            while (below & (below - 1u)) below &= below - 1u;   // its highest bit
            need |= below;
        } else {
            need |= avail & (~avail + 1u);                      // the lowest available part
        }
    }
    return need;
}

// intraPredAngle and invAngle of the angular modes (intra_prediction.cpp:263-422).
HEVC_HD int intra_angle(int mode) {
    constexpr int8_t t[35] = {0,   0,   32,  26,  21,  17,  13,  9,   5,  2,  0,  -2, -5, -9, -13, -17, -21, -26,
                              -32, -26, -21, -17, -13, -9,  -5,  -2,  0,  2,  5,  9,  13, 17, 21,  26,  32};
    return t[mode];
}
HEVC_HD int intra_inv_angle(int mode) {
    constexpr int16_t t[35] = {0,    0,   256, 315, 390, 482, 630, 910, 1638, 4096, 0,    4096, 1638, 910, 630, 482, 390, 315,
                               256,  315, 390, 482, 630, 910, 1638, 4096, 0,  4096, 1638, 910,  630,  482, 390, 315, 256};
    return t[mode];
}

struct IntraAngles {
    int8_t angle[35];
    int16_t inv[35];
};
HEVC_HD IntraAngles intra_angles() {
    IntraAngles r{};
    for (int mode = 0; mode < 35; mode++) {
        r.angle[mode] = (int8_t)intra_angle(mode);
        r.inv[mode] = (int16_t)intra_inv_angle(mode);
    }
    return r;
}

// Main reference entry q of an angular mode as a reference array index: q >= 0 runs along
// the main side, q < 0 is the side reference projected through invAngle (:346-368).  Entries
// past the end are read only with weight 0.
HEVC_HD int intra_main_index(bool vert, int inv, int n, int q) {
    const int k = q >= 0 ? q : -plan_min(2 * n, ((-q) * inv + 128) >> 8);
    return plan_max(0, plan_min(4 * n, vert ? 2 * n + k : 2 * n - k));
}

// The prediction of sample (x, y) of an unsmoothed 4x4 or 8x8 TU as one form over four samples
// of the (substituted) reference array:
//   clip((i[0] * w[0] + i[1] * w[1] + i[2] * w[2] + i[3] * w[3] + add) >> shift)
// covers planar (:263-289), angular (:323-422) and the boundary filters of modes 26 and 10
// (p + ((side - corner) >> 1) = (2p + side - corner) >> 1).  DC (:295-317): i[1] is one of
// the 2n samples of the sum, by `lane`, and the rounded mean takes its place.
struct IntraTaps {
    int i[4], w[4], add, shift;
};
HEVC_HD IntraTaps intra_taps(int log2, int mode, bool chroma, int x, int y, int lane, int ang, int inv) {
    const int n = 1 << log2;
    if (mode == 0)
        return IntraTaps{{2 * n - 1 - y, 3 * n + 1, 2 * n + 1 + x, n - 1}, {n - 1 - x, x + 1, n - 1 - y, y + 1}, n, log2 + 1};
    if (mode == 1) {
        const bool ex = !chroma && x == 0, ey = !chroma && y == 0;
        const int k = lane & (2 * n - 1);
        return IntraTaps{{2 * n + 1 + x, k < n ? n + k : n + 1 + k, 2 * n - 1 - y, 2 * n},
                         {ey ? 1 : 0, 4 - (ex ? 1 : 0) - (ey ? 1 : 0), ex ? 1 : 0, 0},
                         ex || ey ? 2 : 0,
                         2};
    }
    const bool vert = mode >= 18;
    const int along = vert ? y : x, across = vert ? x : y;
    const int idx = ((along + 1) * ang) >> 5, fr = ((along + 1) * ang) & 31, q = across + 1 + idx;
    const int a = intra_main_index(vert, inv, n, q), b = intra_main_index(vert, inv, n, q + 1);
    const int side = vert ? 2 * n - 1 - along : 2 * n + 1 + along;
    if (ang == 0 && !chroma && across == 0) return IntraTaps{{a, b, side, 2 * n}, {2, 0, 1, -1}, 0, 1};
    return IntraTaps{{a, b, side, 2 * n}, {32 - fr, fr, 0, 0}, 16, 5};
}

// The taps of every mode, plane kind and lane of a 4x4 TU, 8 bytes each: word 0 the four
// indices (5 bits each), w[0] and w[1] (6 bits each); word 1 w[2] (bits 0-2), w[3] + 1 (3-5),
// add (6-10), shift (11-13).  "Mode" MODE_PCM predicts nothing (weights 0): a PCM TU's samples
// are its levels.
constexpr int MODE_PCM = 35;
struct IntraTapTable {
    uint32_t t[36][2][16][2];
};
HEVC_HD IntraTapTable intra_tap_table() {
    IntraTapTable r{};
    for (int i = 0; i < 32; i++) r.t[MODE_PCM][i / 16][i % 16][1] = 1u << 3;
    for (int mode = 0; mode < 35; mode++)
        for (int c = 0; c < 2; c++)
            for (int lane = 0; lane < 16; lane++) {
                const IntraTaps k = intra_taps(2, mode, c != 0, lane & 3, lane >> 2, lane, intra_angle(mode),
                                               intra_inv_angle(mode));
                r.t[mode][c][lane][0] = (uint32_t)k.i[0] | (uint32_t)k.i[1] << 5 | (uint32_t)k.i[2] << 10 |
                                        (uint32_t)k.i[3] << 15 | (uint32_t)k.w[0] << 20 | (uint32_t)k.w[1] << 26;
                r.t[mode][c][lane][1] =
                    (uint32_t)k.w[2] | (uint32_t)(k.w[3] + 1) << 3 | (uint32_t)k.add << 6 | (uint32_t)k.shift << 11;
            }
    return r;
}
HEVC_HD IntraTaps intra_taps_unpack(uint32_t a, uint32_t b) {
    return IntraTaps{{(int)(a & 31u), (int)(a >> 5 & 31u), (int)(a >> 10 & 31u), (int)(a >> 15 & 31u)},
                      {(int)(a >> 20 & 63u), (int)(a >> 26), (int)(b & 7u), (int)(b >> 3 & 7u) - 1},
                      (int)(b >> 6 & 31u),
                      (int)(b >> 11)};
}

}  // namespace hevcgpu
