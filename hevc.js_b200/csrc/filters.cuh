// filters.cuh — the in-loop filters: deblocking (deblocking.cpp:50-614) and SAO (sao.cpp:20-243)
// of a picture in one kernel, from the reconstruction buffer into the DPB slot.
//
// One CTA per 64x64 luma tile (and its two 32x32 chroma tiles).  The tile comes into shared
// memory once, with 4 luma and 2 chroma samples around it; both edge directions and SAO run
// there, and the result is written once.  The edges around the tile are filtered by the CTAs
// on both sides (27 % more segments), which is what it costs that nothing between the stages
// goes through memory.
//   1. Which 4-sample segments are filtered, vertical and horizontal: it follows from the
//      records alone, while the samples are on their way.  They go to lists, so that what
//      comes next runs in full warps (a thread per segment left 10 to 14 of 32 lanes working):
//      those whose motion decides to one that is gone through first, those to filter to lists
//      by plane and direction.
//   2. vertical edges, 3. horizontal edges: one segment per thread, on 16-bit lanes.
//   4. SAO on 16-bit lanes, 8 samples per thread and step, and the store.
// Bound by instructions: 16 1080p P/B pictures issue 67 million warp instructions in 104 us, at
// 0.6 per scheduler and cycle; their bytes take 19 us.  Before, as three kernels through memory
// (vertical edges, horizontal edges, SAO), 93 million in 163 us.  No load is waited for where the
// next one could be issued: 108 us with grid words and SAO records read one after the other.
#pragma once

#include "device_common.cuh"

namespace hevcgpu {

__device__ const uint8_t c_beta[52] = {0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  6,  7,
                                   8,  9,  10, 11, 12, 13, 14, 15, 16, 17, 18, 20, 22, 24, 26, 28, 30, 32,
                                   34, 36, 38, 40, 42, 44, 46, 48, 50, 52, 54, 56, 58, 60, 62, 64};
__device__ const uint8_t c_tc[54] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1,  1,  1,  1,  1,  1,  1,  1,  1,
                                 2, 2, 2, 2, 3, 3, 3, 3, 4, 4, 4, 5, 5, 6, 6, 7, 8, 9, 10, 11, 13, 14, 16, 18, 20, 22, 24};
__device__ const uint8_t c_qpc[58] = {0,  1,  2,  3,  4,  5,  6,  7,  8,  9,  10, 11, 12, 13, 14, 15, 16, 17, 18, 19,
                                  20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 29, 30, 31, 32, 33, 33, 34, 34, 35, 35,
                                  36, 36, 37, 37, 38, 39, 40, 41, 42, 43, 44, 45, 46, 47, 48, 49, 50, 51};

// Bs 1 of two inter sides whose residual does not decide it (deblocking.cpp:166-247): other
// references, another number of vectors, or vectors a whole sample or more apart.  Motion entries
// as their words: the vectors of the two lists, the reference indices (-1: none) in the third.
// poc: POC by list and index, 16 for an index past the list's end.
__device__ __forceinline__ bool mv_near(uint32_t a, uint32_t b) {
    a ^= 0x80008000u;
    b ^= 0x80008000u;
    return ((__vmaxu2(a, b) - __vminu2(a, b)) & 0xFFFCFFFCu) == 0u;
}
__device__ __forceinline__ bool bs_motion(const int32_t (&poc)[2][17], const MotionEnt* gp, const MotionEnt* gq) {
    const uint32_t *wp = reinterpret_cast<const uint32_t*>(gp), *wq = reinterpret_cast<const uint32_t*>(gq);
    const uint32_t p0 = wp[0], p1 = wp[1], pr = wp[2], q0 = wq[0], q1 = wq[1], qr = wq[2];
    const int pr0 = (int8_t)pr, pr1 = (int8_t)(pr >> 8), qr0 = (int8_t)qr, qr1 = (int8_t)(qr >> 8);
    const int np = (pr0 >= 0) + (pr1 >= 0), nq = (qr0 >= 0) + (qr1 >= 0);
    if (np != nq) return true;
    if (np == 0) return false;
    // a one-list side gives that list's picture and vector
    const int a0 = pr0 >= 0 ? poc[0][min(pr0, 16)] : poc[1][min(pr1, 16)];
    const int b0 = qr0 >= 0 ? poc[0][min(qr0, 16)] : poc[1][min(qr1, 16)];
    if (np == 1) return a0 != b0 || !mv_near(pr0 >= 0 ? p0 : p1, qr0 >= 0 ? q0 : q1);
    const int a1 = poc[1][min(pr1, 16)], b1 = poc[1][min(qr1, 16)];
    // the same two pictures in the same order with near vectors, or in the other order
    return !((a0 == b0 && a1 == b1 && mv_near(p0, q0) && mv_near(p1, q1)) ||
             (a0 == b1 && a1 == b0 && mv_near(p0, q1) && mv_near(p1, q0)));
}

__device__ __forceinline__ const hevc_slice_t& slice_at(const PicDesc& P, int addr) {
    int s = P.ctb_slice ? P.ctb_slice[addr] : 0;
    return P.slices[s < P.num_slices ? s : 0];
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// Two samples per word as 16-bit lanes: the even bytes of a word, the odd ones, and back.
__device__ __forceinline__ uint32_t lanes_even(uint32_t w) { return prmt(w, 0u, 0x4240u); }
__device__ __forceinline__ uint32_t lanes_odd(uint32_t w) { return prmt(w, 0u, 0x4341u); }
__device__ __forceinline__ uint32_t lanes_join(uint32_t even, uint32_t odd) { return prmt(even, odd, 0x6240u); }
__device__ __forceinline__ uint32_t both(int v) { return (uint32_t)v * 0x00010001u; }
__device__ __forceinline__ uint32_t lane_clamp(uint32_t v, uint32_t lo, uint32_t hi) { return __vmins2(__vmaxs2(v, lo), hi); }
__device__ __forceinline__ uint32_t lane_absdiff(uint32_t a, uint32_t b) { return __vmaxs2(a, b) - __vmins2(a, b); }
__device__ __forceinline__ int lane_max(uint32_t v) { return max((int)(v & 0xFFFFu), (int)(v >> 16)); }

// Transposes a 4x4 block of bytes held as four words.
__device__ __forceinline__ void transpose4(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
    const uint32_t t0 = prmt(a, b, 0x5140u), t1 = prmt(c, d, 0x5140u), t2 = prmt(a, b, 0x7362u), t3 = prmt(c, d, 0x7362u);
    a = prmt(t0, t1, 0x5410u);
    b = prmt(t0, t1, 0x7632u);
    c = prmt(t2, t3, 0x5410u);
    d = prmt(t2, t3, 0x7632u);
}

// Strong filter of one side on lanes (:444-470): x0..x3 the side's samples from the edge on,
// y0, y1 the other side's; t2 = 2 tc lanes, nt2 its negative.
__device__ __forceinline__ void luma_strong(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t y0, uint32_t y1,
                                            uint32_t t2, uint32_t nt2, uint32_t (&o)[3]) {
    const uint32_t a = x1 + x0 + y0;
    const uint32_t v[3] = {((x2 + 2 * a + y1 + 0x00040004u) >> 3) & 0x1FFF1FFFu, ((x2 + a + 0x00020002u) >> 2) & 0x3FFF3FFFu,
                           ((2 * x3 + 3 * x2 + a + 0x00040004u) >> 3) & 0x1FFF1FFFu};
    const uint32_t x[3] = {x0, x1, x2};
#pragma unroll
    for (int i = 0; i < 3; i++) o[i] = lane_clamp(v[i], __viaddmax_s16x2(x[i], nt2, 0u), x[i] + t2);   // (v >= 0)
}

// Filter of one 4-sample luma segment (:404-520) held as words of 4 lines: w[0..3] = p3 .. p0,
// w[4..7] = q0 .. q3.  Arithmetic on 16-bit lanes, lines 0 and 2, then 1 and 3; values that can
// be negative carry a bias (256 for the normal filter's deltas), so that lanes stay apart.
__device__ __forceinline__ void luma_segment(uint32_t (&w)[8], int beta, int tc, bool noP, bool noQ) {
    // decisions on lines 0 and 3
    uint32_t d[8];
#pragma unroll
    for (int i = 0; i < 8; i++) d[i] = prmt(w[i], 0u, 0x4340u);
    const uint32_t dp = lane_absdiff(d[1] + d[3], 2 * d[2]), dq = lane_absdiff(d[6] + d[4], 2 * d[5]), dpq = dp + dq;
    if ((int)((dpq & 0xFFFFu) + (dpq >> 16)) >= beta) return;
    const bool strong = 2 * lane_max(dpq) < (beta >> 2) &&
                        lane_max(lane_absdiff(d[0], d[3]) + lane_absdiff(d[4], d[7])) < (beta >> 3) &&
                        lane_max(lane_absdiff(d[3], d[4])) < ((5 * tc + 1) >> 1);
    uint32_t n[2][8];   // the lanes, then the filtered ones
#pragma unroll
    for (int i = 0; i < 8; i++) {
        n[0][i] = lanes_even(w[i]);
        n[1][i] = lanes_odd(w[i]);
    }
    if (strong) {
        const uint32_t t2 = both(2 * tc), nt2 = (uint32_t)(uint16_t)(-2 * tc) * 0x00010001u;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t(&v)[8] = n[h];
            uint32_t po[3], qo[3];
            luma_strong(v[3], v[2], v[1], v[0], v[4], v[5], t2, nt2, po);
            luma_strong(v[4], v[5], v[6], v[7], v[3], v[2], t2, nt2, qo);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                v[3 - i] = po[i];
                v[4 + i] = qo[i];
            }
        }
    } else {
        const int thr = (beta + (beta >> 1)) >> 3;
        const bool dEp = (int)((dp & 0xFFFFu) + (dp >> 16)) < thr, dEq = (int)((dq & 0xFFFFu) + (dq >> 16)) < thr;
        const uint32_t lo10 = both(257 - 10 * tc), hi10 = both(255 + 10 * tc), lo = both(256 - tc), hi = both(256 + tc);
        const uint32_t lo2 = both(256 - (tc >> 1)), hi2 = both(256 + (tc >> 1));
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t(&v)[8] = n[h];
            const uint32_t p0 = v[3], p1 = v[2], p2 = v[1], q0 = v[4], q1 = v[5], q2 = v[6];
            // 256 + delta (4096 = 16 * 256, and the rounding 8)
            const uint32_t dl = ((9 * q0 + 3 * p1 + 0x10081008u - (9 * p0 + 3 * q1)) >> 4) & 0x0FFF0FFFu;
            // lanes with |delta| >= 10 tc keep their samples
            const uint32_t out = ((lane_clamp(dl, lo10, hi10) ^ dl) + 0x7FFF7FFFu) & 0x80008000u;
            const uint32_t keep = (out >> 15) * 0xFFFFu;
            const uint32_t de = lane_clamp(dl, lo, hi), nd = 0x02000200u - de;   // 256 + delta, 256 - delta
            auto side = [&](uint32_t x0, uint32_t x1, uint32_t x2, uint32_t e, bool second, uint32_t& o0, uint32_t& o1) {
                o0 = (lane_clamp(x0 + e, 0x01000100u, 0x01FF01FFu) & ~keep) | (x0 & keep);   // the low byte counts
                if (second) {
                    const uint32_t avg = ((x2 + x0 + 0x00010001u) >> 1) & 0x01FF01FFu;
                    const uint32_t f = lane_clamp(((avg + e + 0x01000100u - x1) >> 1) & 0x7FFF7FFFu, lo2, hi2);
                    o1 = (lane_clamp(x1 + f, 0x01000100u, 0x01FF01FFu) & ~keep) | (x1 & keep);
                }
            };
            side(p0, p1, p2, de, dEp, v[3], v[2]);
            side(q0, q1, q2, nd, dEq, v[4], v[5]);
        }
    }
#pragma unroll
    for (int i = 1; i < 4; i++) {
        if (!noP) w[i] = lanes_join(n[0][i], n[1][i]);
        if (!noQ) w[3 + i] = lanes_join(n[0][3 + i], n[1][3 + i]);
    }
}

constexpr int LF_T = 64;                              // luma tile
constexpr int LF_X = 16;                              // column of the tile's first sample in its rows
constexpr int LF_LP = LF_T + 32, LF_LR = LF_T + 8;    // luma rows' pitch, rows (4 above)
constexpr int LF_CP = LF_T / 2 + 32, LF_CR = LF_T / 2 + 4;   // chroma (2 above)
constexpr int LF_U = LF_T / 4 + 2;                    // 4x4 units across, with one around the tile
constexpr int LF_E = LF_T / 8 + 1;                    // edges of one direction
constexpr int LF_SEGS = LF_E * LF_U;                  // their 4-sample segments
constexpr int LF_TASKS = (LF_SEGS + 31) / 32;         // warps' worth of them
constexpr int LF_CTBS = (LF_T / 16) * (LF_T / 16);    // CTBs of a tile, at most

// SAO of one CTB and plane (type, cls: the record's): edge offset for type 2, else band offset with k = the lanes of
// -band_position; a0 the tile offset of neighbour a (b lies opposite); the offsets as bytes
// of lo, hi in the order of the index each form computes.
struct LfSao {
    uint32_t lo, hi, k;
    int16_t a0;
    uint8_t type, cls;
};

// CTAs per SM that the register budget is sized for, by the CTA's threads.  More and smaller CTAs
// hide each other's barriers: 16 1080p P/B pictures 139 us with 256 threads (127 with room for
// 5), 108 with 128 (112 with room for 8, 110 for 12).  But a tile takes longer with 128, which
// counts when every tile is resident at once: four 1000x568 pictures' batch 118 us with 256,
// 124 with 128.
constexpr int lf_ctas(int threads) { return threads > 128 ? 1024 / threads : 10; }

struct LfSmem {
    alignas(16) uint8_t y[LF_LR * LF_LP];
    alignas(16) uint8_t c[2][LF_CR * LF_CP];
    uint32_t blk[LF_U * LF_U];
    LfSao sao[LF_CTBS * 3];
    // segments to filter, by direction: index | (Bs - 1) << 8; those whose motion decides
    uint16_t luma[2][LF_SEGS], chroma[2][LF_SEGS], motion[2 * LF_SEGS];
    int n_luma[2], n_chroma[2], n_motion;
    uint8_t beta[52], tc[54], qpc[58];
    int32_t poc[2][17];
    hevc_slice_t slice;   // the picture's, when it has one
};

// Appends the entries of the lanes with `on` to a list.
__device__ __forceinline__ void lf_append(bool on, int entry, uint16_t* list, int* n, int lane) {
    const uint32_t m = __ballot_sync(0xffffffffu, on);
    if (m == 0u) return;
    int at = 0;
    if (lane == 0) at = atomicAdd(n, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (on) list[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)entry;
}

// Segment i of a direction: its first sample in the tile (4 along the edge, -4 .. 64) and its
// side q in the grid words.
struct LfSeg {
    int x, y, at;
};
__device__ __forceinline__ LfSeg lf_segment(int i, int dir) {
    const int e = i / LF_U, u = i - e * LF_U - 1;
    LfSeg g;
    g.x = dir ? 4 * u : 8 * e;
    g.y = dir ? 8 * e : 4 * u;
    g.at = (g.y / 4 + 1) * LF_U + g.x / 4 + 1;
    return g;
}
// Slice header of a sample's CTB.
__device__ __forceinline__ hevc_slice_t lf_slice(const PicDesc& P, int x, int y) {
    return slice_at(P, (y >> P.log2_ctb) * P.wctb + (x >> P.log2_ctb));
}
// Whether the edge at (x, y) is filtered, in a picture whose slice or tile boundaries may not be.
__device__ __noinline__ bool lf_crosses(const PicDesc& P, int x, int y, int dir) {
    const int xp = dir ? x : x - 1, yp = dir ? y - 1 : y;
    const int aq = (y >> P.log2_ctb) * P.wctb + (x >> P.log2_ctb), ap = (yp >> P.log2_ctb) * P.wctb + (xp >> P.log2_ctb);
    const hevc_slice_t sl = slice_at(P, aq);
    if (sl.deblocking_disabled) return false;
    if (P.tiles_check && P.ctb_tile && P.ctb_tile[aq] != P.ctb_tile[ap]) return false;
    return !(P.slice_check && P.ctb_slice && P.ctb_slice[aq] != P.ctb_slice[ap] && !sl.lf_across_slices);
}
// The two sides of a segment: QP, and whether a side keeps its samples (PCM with
// pcm_loop_filter_disabled, transquant bypass).
struct LfSides {
    int qp;
    bool no_p, no_q;
};
__device__ __forceinline__ LfSides lf_sides(uint32_t bp, uint32_t bq, bool pcm_off) {
    const uint32_t off = HEVC_BLK_BYPASS | (pcm_off ? HEVC_BLK_PCM : 0u);
    return LfSides{((int8_t)(bp >> HEVC_BLK_QP_SHIFT) + (int8_t)(bq >> HEVC_BLK_QP_SHIFT) + 1) >> 1, (bp & off) != 0u,
                   (bq & off) != 0u};
}

// 255 + sign(a - c) per lane, from a and 255 - c.
__device__ __forceinline__ uint32_t lane_sign(uint32_t a, uint32_t nc) {
    return __vmaxs2(__viaddmin_s16x2(a, nc, 0x01000100u), 0x00FE00FEu);
}
// Samples c plus the offsets that the lanes' indices (0..4, even and odd samples) pick.
__device__ __forceinline__ uint32_t lanes_offset(uint32_t c, uint32_t ie, uint32_t io, uint32_t lo, uint32_t hi) {
    const uint32_t off = prmt(lo, hi, prmt(ie + (io << 4), 0u, 0x4420u));   // the four nibbles, then their bytes
    return lanes_join(__viaddmin_s16x2_relu(lanes_even(c), prmt(off, 0u, 0xA280u), 0x00FF00FFu),   // sign-extended
                      __viaddmin_s16x2_relu(lanes_odd(c), prmt(off, 0u, 0xB391u), 0x00FF00FFu));
}

// Samples of a word (x .. x + 3, y) of plane ci that SAO leaves as they are although its CTB
// has it on, as a mask of bytes: PCM with pcm_loop_filter_disabled and transquant bypass, and,
// for edge offset, a neighbour across a slice or tile boundary that filtering may not cross.
__device__ __noinline__ uint32_t lf_keep(const PicDesc& P, int ci, int x, int y, bool neighbours, int dx, int dy) {
    const int sub = ci ? 2 : 1, gw = P.width >> 2, pw = P.width / sub, ph = P.height / sub;
    uint32_t keep = 0;
    for (int i = 0; i < 4; i++) {
        const int xs = x + i;
        bool k = false;
        if (P.pcm_bypass_any) {
            const uint32_t b = P.blk[(int64_t)((y * sub) >> 2) * gw + ((xs * sub) >> 2)];
            k = (P.pcm_lf_disabled && (b & HEVC_BLK_PCM)) || (b & HEVC_BLK_BYPASS);
        }
        if (neighbours && (P.slice_check || P.tiles_check)) {
            const int cur = ((y * sub) >> P.log2_ctb) * P.wctb + ((xs * sub) >> P.log2_ctb);
            for (int nk = 0; nk < 2; nk++) {
                const int nx = xs + (nk ? -dx : dx), ny = y + (nk ? -dy : dy);
                if (nx < 0 || nx >= pw || ny < 0 || ny >= ph) continue;   // kept anyway
                const int na = ((ny * sub) >> P.log2_ctb) * P.wctb + ((nx * sub) >> P.log2_ctb);
                const int sc = P.ctb_slice ? P.ctb_slice[cur] : 0, sn = P.ctb_slice ? P.ctb_slice[na] : 0;
                k = k || (sc != sn && !slice_at(P, sn < sc ? cur : na).lf_across_slices) ||
                    (P.tiles_check && P.ctb_tile && P.ctb_tile[cur] != P.ctb_tile[na]);
            }
        }
        if (k) keep |= 0xFFu << (8 * i);
    }
    return keep;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, lf_ctas(THREADS)) k_loop_filter(const __grid_constant__ SegTable st,
                                                                         int deblock) {
    __shared__ LfSmem S;
    const PicDesc& P = *st.s[blockIdx.y].pic;
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    pdl_next();
    const int W = P.width, H = P.height, gw = W >> 2, tw = (W + LF_T - 1) / LF_T;
    const int x0 = (blockIdx.x % tw) * LF_T, y0 = (blockIdx.x / tw) * LF_T;
    if (y0 >= H) return;
    const int pitch_y = P.pitch_y, pitch_c = P.pitch_c, lctb = P.log2_ctb;
    const uint8_t* const rec = P.rec;
    const int64_t off_cb = P.off_cb, off_cr = P.off_cr;
    // ---- the records: grid words, filter tables, SAO parameters
    if (deblock) {
#pragma unroll 1
        for (int q = tid; q < LF_U * LF_U; q += THREADS) {
            const int ux = (x0 >> 2) - 1 + q % LF_U, uy = (y0 >> 2) - 1 + q / LF_U;
            if (ux >= 0 && ux < gw && uy >= 0 && uy < H >> 2) cp_async4(S.blk + q, P.blk + (int64_t)uy * gw + ux);
            else S.blk[q] = 0u;
        }
        cp_async_commit();
        if (tid < 52) S.beta[tid] = c_beta[tid];
        if (tid < 54) S.tc[tid] = c_tc[tid];
        if (tid < 58) S.qpc[tid] = c_qpc[tid];
        if (tid < 2) S.n_luma[tid] = S.n_chroma[tid] = 0;
        if (tid >= 64 && tid < 98) {
            const int l = (tid - 64) / 17, k = (tid - 64) % 17;
            S.poc[l][k] = k < 16 && k < P.num_ref[l] ? P.ref_poc[l][k] : -999999;
        }
        if (tid == 98) S.n_motion = 0;
        if (tid == 99) S.slice = slice_at(P, 0);
    }
    const int cpt = lctb >= 6 ? 1 : LF_T >> lctb;   // CTBs across the tile
    pdl_wait();
    // ---- the samples, in 16-byte pieces (one that starts inside the picture ends inside the
    // row's pitch, a multiple of 64): 6 of 8 threads per luma row, 4 per chroma row
    {
        const int k = tid & 7, x = x0 - LF_X + 16 * k;
        if (k < LF_LP / 16 && x >= 0 && x < W) {
#pragma unroll
            for (int i = 0; i < (LF_LR + THREADS / 8 - 1) / (THREADS / 8); i++) {
                const int r = (tid >> 3) + THREADS / 8 * i, y = y0 - 4 + r;
                if (r < LF_LR && y >= 0 && y < H) cp_async16(S.y + r * LF_LP + 16 * k, rec + (int64_t)y * pitch_y + x);
            }
        }
        const int kc = tid & 3, xc = (x0 >> 1) - LF_X + 16 * kc;
        if (xc >= 0 && xc < W >> 1) {
#pragma unroll
            for (int i = 0; i < (2 * LF_CR + THREADS / 4 - 1) / (THREADS / 4); i++) {
                const int q = (tid >> 2) + THREADS / 4 * i, c = q >= LF_CR, r = q - c * LF_CR, y = (y0 >> 1) - 2 + r;
                if (q < 2 * LF_CR && y >= 0 && y < H >> 1)
                    cp_async16(S.c[c] + r * LF_CP + 16 * kc, rec + (c ? off_cr : off_cb) + (int64_t)y * pitch_c + xc);
            }
        }
    }
    cp_async_commit();
    if (deblock) {
        cp_async_wait<1>();
        __syncthreads();   // grid words, tables, counts
        // ---- 1. the segments to filter
        const bool boundaries = P.tiles_check || P.slice_check;
#pragma unroll 1
        for (int task = warp; task < 2 * LF_TASKS; task += THREADS / 32) {
            const int dir = task >= LF_TASKS, i = (task - dir * LF_TASKS) * 32 + lane;
            const LfSeg g = lf_segment(i, dir);
            const int x = x0 + g.x, y = y0 + g.y, q = dir ? y : x;
            const bool in = i < LF_SEGS && x >= 0 && y >= 0 && x < W && y < H && q > 0;
            const uint32_t bq = in ? S.blk[g.at] : 0u, bp = in ? S.blk[g.at - (dir ? LF_U : 1)] : 0u;
            bool on = bq & (dir ? HEVC_BLK_EDGE_H : HEVC_BLK_EDGE_V);
            if (boundaries) {
                if (on) on = lf_crosses(P, x, y, dir);
            } else if (S.slice.deblocking_disabled) {
                on = false;
            }
            // the edge is a TU's when a multiple of the TU size of either side
            const int tp = (1 << ((bp >> HEVC_BLK_TU_SHIFT) & 0xFF)) - 1, tq = (1 << ((bq >> HEVC_BLK_TU_SHIFT) & 0xFF)) - 1;
            const bool intra = (bp | bq) & HEVC_BLK_INTRA;
            const bool known = intra || (((bp | bq) & HEVC_BLK_CBF) && ((q & tp) == 0 || (q & tq) == 0));
            lf_append(on && known, i | (int)intra << 8, S.luma[dir], &S.n_luma[dir], lane);
            lf_append(on && !known, i | dir << 8, S.motion, &S.n_motion, lane);
            // chroma: Bs 2 on the 8-sample chroma grid (:538-609)
            lf_append(on && intra && (q & 15) == 0, i, S.chroma[dir], &S.n_chroma[dir], lane);
        }
        __syncthreads();
        const MotionEnt* const mot = P.mot;
#pragma unroll 1
        for (int k0 = tid - lane; k0 < S.n_motion; k0 += THREADS) {
            const int k = k0 + lane, en = k < S.n_motion ? S.motion[k] : 0, dir = en >> 8, i = en & 255;
            const LfSeg g = lf_segment(i, dir);
            const MotionEnt* const m = mot + (int64_t)((y0 + g.y) >> 2) * gw + ((x0 + g.x) >> 2);
            const bool on = k < S.n_motion && bs_motion(S.poc, m - (dir ? gw : 1), m);
            lf_append(on && dir == 0, i, S.luma[0], &S.n_luma[0], lane);
            lf_append(on && dir == 1, i, S.luma[1], &S.n_luma[1], lane);
        }
    }
    // SAO parameters, while the samples are on their way: a CTB and plane per thread, the record's
    // bytes in one round of loads
    if (THREADS - 1 - tid < cpt * cpt * 3) {
        const int ci = (THREADS - 1 - tid) % 3, k = (THREADS - 1 - tid) / 3;
        const int cx = (x0 >> lctb) + k % cpt, cy = (y0 >> lctb) + k / cpt;
        LfSao s = {0, 0, 0, 0, 0, 0};
        if (P.sao_enabled && cx < P.wctb && cy < P.hctb) {
            const hevc_sao_t& sp = P.sao[cy * P.wctb + cx];
            const int8_t* const off = sp.offset[ci];
            const int band = sp.band_pos[ci];
            s.type = sp.type[ci];
            s.cls = sp.eo_class[ci];
            s.lo = (uint8_t)off[0] | (uint32_t)(uint8_t)off[1] << 8 | (uint32_t)(uint8_t)off[2] << 16 |
                   (uint32_t)(uint8_t)off[3] << 24;
            s.hi = (uint8_t)off[4];
            if (s.type == 2) {   // the index computed is 4 - edgeIdx
                const int pitch = ci ? LF_CP : LF_LP, dx = s.cls == 1 ? 0 : (s.cls == 3 ? 1 : -1), dy = s.cls == 0 ? 0 : -1;
                s.a0 = (int16_t)(dy * pitch + dx);
                const uint32_t lo = s.lo;
                s.lo = __byte_perm(lo, s.hi, 0x1234);
                s.hi = lo & 0xFFu;
            } else {             // index 4 outside the four bands: no offset
                s.k = (uint32_t)(uint16_t)(-band) * 0x00010001u;
                s.hi = 0u;
            }
        }
        S.sao[ci * LF_CTBS + k] = s;
    }
    cp_async_wait<0>();
    __syncthreads();
    // ---- 2., 3. vertical, then horizontal edges.  A segment writes only words (luma) or samples
    // (chroma) that no other of its direction touches.  Chroma segments go to the last warps,
    // which the luma ones leave free.
    if (deblock) {
        const bool by_ctb = P.tiles_check || P.slice_check, pcm_off = P.pcm_lf_disabled != 0;
        const int c_off[2] = {P.cb_qp_offset, P.cr_qp_offset};
#pragma unroll 1
        for (int dir = 0; dir < 2; dir++) {
            const int n_luma = S.n_luma[dir], n_chroma = S.n_chroma[dir];
#pragma unroll 1
            for (int q = tid; q < n_luma; q += THREADS) {
                const int en = S.luma[dir][q];
                const LfSeg g = lf_segment(en & 255, dir);
                const LfSides sd = lf_sides(S.blk[g.at - (dir ? LF_U : 1)], S.blk[g.at], pcm_off);
                const hevc_slice_t sl = by_ctb ? lf_slice(P, x0 + g.x, y0 + g.y) : S.slice;
                const int beta = S.beta[clip3(0, 51, sd.qp + 2 * sl.beta_offset_div2)];
                const int tc = S.tc[clip3(0, 53, sd.qp + 2 * (en >> 8) + 2 * sl.tc_offset_div2)];
                if (beta == 0 || tc == 0) continue;   // nothing changes
                // the 8 rows across a horizontal edge; of a vertical one the p and q words of its
                // 4 rows, transposed to the same form
                uint32_t w[8];
                uint8_t* const o = S.y + (4 + g.y - 4 * dir) * LF_LP + LF_X + g.x - 4 * (1 - dir);
                const int row = LF_LP, half = dir ? 4 * LF_LP : 4;
#pragma unroll
                for (int k = 0; k < 8; k++) w[k] = *reinterpret_cast<const uint32_t*>(o + (k & 3) * row + (k >> 2) * half);
                if (dir == 0) {
                    transpose4(w[0], w[1], w[2], w[3]);
                    transpose4(w[4], w[5], w[6], w[7]);
                }
                luma_segment(w, beta, tc, sd.no_p, sd.no_q);
                if (dir == 0) {
                    transpose4(w[0], w[1], w[2], w[3]);
                    transpose4(w[4], w[5], w[6], w[7]);
                }
#pragma unroll
                for (int k = 0; k < 8; k++) *reinterpret_cast<uint32_t*>(o + (k & 3) * row + (k >> 2) * half) = w[k];
            }
#pragma unroll 1
            for (int q = THREADS - 1 - tid; q < 2 * n_chroma; q += THREADS) {
                const int ci = q & 1;
                const LfSeg g = lf_segment(S.chroma[dir][q >> 1], dir);
                const LfSides sd = lf_sides(S.blk[g.at - (dir ? LF_U : 1)], S.blk[g.at], pcm_off);
                const hevc_slice_t sl = by_ctb ? lf_slice(P, x0 + g.x, y0 + g.y) : S.slice;
                const int tc = S.tc[clip3(0, 53, S.qpc[clip3(0, 57, sd.qp + c_off[ci])] + 2 + 2 * sl.tc_offset_div2)];
                const int stp = dir ? LF_CP : 1, along = dir ? 1 : LF_CP;   // across the edge, along it
                uint8_t* const s0 = S.c[ci] + (2 + g.y / 2) * LF_CP + LF_X + g.x / 2;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    uint8_t* const t = s0 + k * along;
                    const int p1 = t[-2 * stp], p0 = t[-stp], q0 = t[0], q1 = t[stp];
                    const int delta = clip3(-tc, tc, ((((q0 - p0) * 4) + p1 - q1 + 4) >> 3));
                    if (!sd.no_p) t[-stp] = (uint8_t)clip_u8(p0 + delta);
                    if (!sd.no_q) t[0] = (uint8_t)clip_u8(q0 - delta);
                }
            }
            __syncthreads();
        }
    }
    // ---- 4. SAO and the store
    uint8_t* const dst = static_cast<uint8_t*>(const_cast<void*>(st.s[blockIdx.y].items));
    const bool rare = P.pcm_bypass_any || P.slice_check || P.tiles_check;
    // the 8 samples at tile offset o of plane ci, sample (x, y) of a pw x ph plane
    auto sao_pair = [&](int ci, const uint8_t* plane, int o, int x, int y, int pw, int ph, const LfSao& s) -> uint2 {
        uint2 v = *reinterpret_cast<const uint2*>(plane + o);
        if (s.type == 0) return v;
        const uint32_t c[2] = {v.x, v.y};
        uint32_t r[2], keep[2] = {0u, 0u};
        if (s.type == 2) {
            const int da = o + s.a0, db = o - s.a0, sa = 8 * (da & 3), sb = 8 * (db & 3);
            const uint32_t* const wa = reinterpret_cast<const uint32_t*>(plane) + (da >> 2);
            const uint32_t* const wb = reinterpret_cast<const uint32_t*>(plane) + (db >> 2);
            const uint32_t a[3] = {wa[0], wa[1], wa[2]}, b[3] = {wb[0], wb[1], wb[2]};
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const uint32_t na = __funnelshift_r(a[k], a[k + 1], sa), nb = __funnelshift_r(b[k], b[k + 1], sb);
                const uint32_t ce = lanes_even(~c[k]), co = lanes_odd(~c[k]);
                // 510 + sign(a - c) + sign(b - c) = 512 - edgeIdx
                const uint32_t ie = lane_sign(lanes_even(na), ce) + lane_sign(lanes_even(nb), ce) - 0x01FC01FCu;
                const uint32_t io = lane_sign(lanes_odd(na), co) + lane_sign(lanes_odd(nb), co) - 0x01FC01FCu;
                r[k] = lanes_offset(c[k], ie, io, s.lo, s.hi);
            }
            if (s.cls != 1) {   // picture edges keep theirs (in a row's second word past its end, any)
                if (x == 0) keep[0] = 0xFFu;
                if (x + 4 >= pw) keep[0] |= 0xFF000000u;
                if (x + 8 >= pw) keep[1] = 0xFF000000u;
            }
            if (s.cls != 0 && (y == 0 || y == ph - 1)) keep[0] = keep[1] = 0xFFFFFFFFu;
        } else {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                // (c >> 3) - band_position mod 2^16, or 4 outside the four bands (no wrap-around,
                // sao.cpp:229-230)
                const uint32_t ie = __viaddmin_u16x2((lanes_even(c[k]) >> 3) & 0x001F001Fu, s.k, 0x00040004u);
                const uint32_t io = __viaddmin_u16x2((lanes_odd(c[k]) >> 3) & 0x001F001Fu, s.k, 0x00040004u);
                r[k] = lanes_offset(c[k], ie, io, s.lo, s.hi);
            }
        }
        if (rare) {
            const int dx = s.cls == 1 ? 0 : (s.cls == 3 ? 1 : -1), dy = s.cls == 0 ? 0 : -1;
            keep[0] |= lf_keep(P, ci, x, y, s.type == 2, dx, dy);
            if (x + 4 < pw) keep[1] |= lf_keep(P, ci, x + 4, y, s.type == 2, dx, dy);
        }
        v.x = (c[0] & keep[0]) | (r[0] & ~keep[0]);
        v.y = (c[1] & keep[1]) | (r[1] & ~keep[1]);
        return v;
    };
    {
        constexpr int ROWS = THREADS / 8;   // rows of the tile a step covers
        const int col = 8 * (tid & 7), row0 = tid >> 3, x = x0 + col;
        if (x < W) {
#pragma unroll
            for (int i = 0; i < LF_T / ROWS; i++) {
                const int row = row0 + ROWS * i, y = y0 + row;
                if (y < H)
                    *reinterpret_cast<uint2*>(dst + (int64_t)y * pitch_y + x) =
                        sao_pair(0, S.y, (4 + row) * LF_LP + LF_X + col, x, y, W, H,
                                 S.sao[(row >> lctb) * cpt + (col >> lctb)]);
            }
        }
    }
    {
        constexpr int ROWS = THREADS / 4;   // of Cb, then Cr
        const int col = 8 * (tid & 3), x = (x0 >> 1) + col, pw = W >> 1, lc = lctb - 1;
        if (x < pw) {
#pragma unroll
            for (int i = 0; i < (LF_T + ROWS - 1) / ROWS; i++) {
                const int q = (tid >> 2) + ROWS * i, c = q >= LF_T / 2, row = q % (LF_T / 2), y = (y0 >> 1) + row;
                if (q < LF_T && y < H >> 1) {
                    uint8_t* const d = dst + (c ? off_cr : off_cb) + (int64_t)y * pitch_c + x;
                    const uint2 v = sao_pair(1 + c, S.c[c], (2 + row) * LF_CP + LF_X + col, x, y, pw, H >> 1,
                                             S.sao[(1 + c) * LF_CTBS + (row >> lc) * cpt + (col >> lc)]);
                    if (x + 4 < pw)
                        *reinterpret_cast<uint2*>(d) = v;
                    else   // half a pair: planes are a multiple of 4 wide
                        *reinterpret_cast<uint32_t*>(d) = v.x;
                }
            }
        }
    }
}

}  // namespace hevcgpu
