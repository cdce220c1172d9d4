// kernels.cuh — the reconstruction kernels (sm_100a).
//
//   k_residual        dequant + inverse DST/DCT + add-and-clip of coded TUs
//                     (transform.cpp:293-394, coding_tree.cpp:371-396)
//   (motion compensation: mc.cuh; intra prediction: intra.cuh)
//   k_motion_grid     4x4 motion grid of the PUs (store_pu_motion's grid)
//   (in-loop filters: filters.cuh)
//   k_picture_checksum  per-plane checksum of a frame (H.265 picture hash SEI, D.3.19)
#pragma once

#include "dequant.h"
#include "device_common.cuh"

namespace hevcgpu {

// ======================================================================================
// Inverse transform.  The N-point inverse DCT is computed by the even/odd recursion of
// the HEVC basis: out[k] = E[k] + O[k], out[N-1-k] = E[k] - O[k], with E the N/2-point
// inverse of the even inputs and O[k] the odd-input dot products, two products per
// instruction (dp2a).  The basis entries
// are integer cosines of pi*i*(2k+1)/64 (H.265 eq. 8-315); cos_mag lists the 33
// magnitudes for angles 0..pi/2 and every coefficient below is a compile-time constant.
// Integer sums are exact, so any summation order reproduces the reference's butterflies.
// ======================================================================================
__host__ __device__ constexpr int cos_mag(int m) {
    constexpr int t[33] = {64, 90, 90, 90, 89, 88, 87, 85, 83, 82, 80, 78, 75, 73, 70, 67, 64,
                           61, 57, 54, 50, 46, 43, 38, 36, 31, 25, 22, 18, 13, 9,  4,  0};
    return t[m];
}
__host__ __device__ constexpr int cos_entry(int m) {
    return (m & 127) <= 32 ? cos_mag(m & 127)
           : (m & 127) <= 64 ? -cos_mag(64 - (m & 127))
           : (m & 127) <= 96 ? -cos_mag((m & 127) - 64)
                             : cos_mag(128 - (m & 127));
}
// weight of input n in output k of the N-point inverse DCT
template <int N>
__host__ __device__ constexpr int dct_w(int n, int k) { return cos_entry(n * (32 / N) * (2 * k + 1)); }

// Two products of a word of int16 pairs with bytes 0, 1 (lo) or 2, 3 (hi) of the weights.
__device__ __forceinline__ int dp2_lo(uint32_t x, uint32_t w, int c) {
    int d;
    asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(w), "r"(c));
    return d;
}
__device__ __forceinline__ int dp2_hi(uint32_t x, uint32_t w, int c) {
    int d;
    asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(w), "r"(c));
    return d;
}
// lo, hi clipped to int16, as a word
__device__ __forceinline__ uint32_t pack_sat_s16x2(int lo, int hi) {
    uint32_t d;
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(d) : "r"(hi), "r"(lo));
    return d;
}
__host__ __device__ constexpr uint32_t pack_w(int a, int b, int c, int d) {
    return (uint32_t)(uint8_t)a | (uint32_t)(uint8_t)b << 8 | (uint32_t)(uint8_t)c << 16 | (uint32_t)(uint8_t)d << 24;
}

// The inputs of an N-point transform come as N/2 words of two, paired as the recursion adds them
// up: the odd ones (1,3), (5,7) .., then the odd ones of the N/2-point transform of the even
// ones, (2,6), (10,14) .., and so on, at last (0, N/2).  Input n of level l (n an odd multiple of
// 1 << l) lies in word m_l + (n >> l) / 4, m_l = N/2 - (N/2 >> l).
// The two inputs of word m:
template <int N>
__device__ __forceinline__ void pair_inputs(int m, int& a, int& b) {
    const int x = N / 2 - m, top = 31 - __clz(N / 4);
    const int l = x == 1 ? top + 1 : top - (31 - __clz(x - 1));
    const int i = m - (N / 2 - (N / 2 >> l));
    a = x == 1 ? 0 : (4 * i + 1) << l;
    b = x == 1 ? N / 2 : a + (2 << l);
}
// The half word of input n.
template <int N>
__device__ __forceinline__ int pair_place(int n) {
    if (n == 0) return N - 2;
    const int l = __ffs(n) - 1, q = n >> l;
    return n == N / 2 ? N - 1 : 2 * (N / 2 - (N / 2 >> l) + (q >> 2)) + ((q >> 1) & 1);
}

// M-point inverse DCT of the M/2 words at x, each output plus `round`.
template <int M>
__device__ __forceinline__ void idct_pairs(const uint32_t* x, int round, int* dst) {
    if constexpr (M == 2) {
        dst[0] = dp2_lo(x[0], pack_w(64, 64, 0, 0), round);
        dst[1] = dp2_lo(x[0], pack_w(64, -64, 0, 0), round);
    } else {
        int E[M / 2];
        idct_pairs<M / 2>(x + M / 4, round, E);
#pragma unroll
        for (int k = 0; k < M / 2; k++) {
            int o = 0;
#pragma unroll
            for (int t = 0; t < (M + 7) / 8; t++) {
                const uint32_t w = pack_w(dct_w<M>(8 * t + 1, k), dct_w<M>(8 * t + 3, k),
                                          M > 4 ? dct_w<M>(8 * t + 5, k) : 0, M > 4 ? dct_w<M>(8 * t + 7, k) : 0);
                o = dp2_lo(x[2 * t], w, o);
                if (M > 4) o = dp2_hi(x[2 * t + 1], w, o);
            }
            dst[k] = E[k] + o;
            dst[M - 1 - k] = E[k] - o;
        }
    }
}

__constant__ int c_level_scale[6] = {40, 45, 51, 57, 64, 72};
__device__ __forceinline__ Dequant dequant_of(int qp, int log2) { return dequant_make(c_level_scale[qp % 6], qp, log2); }
// Levels of one column in two rows, each row's two columns in a word: the columns' pairs.
__device__ __forceinline__ void dequant_pairs(uint32_t a, uint32_t b, const Dequant& q, int ma0, int ma1, int mb0, int mb1,
                                              uint32_t& p0, uint32_t& p1) {
    p0 = pack_sat_s16x2(dequant_level((int16_t)a, ma0, q), dequant_level((int16_t)b, mb0, q));
    p1 = pack_sat_s16x2(dequant_level((int)a >> 16, ma1, q), dequant_level((int)b >> 16, mb1, q));
}

// Scaling factors m (transform.cpp:320-358): matrixId is the plane plus 3 for a non-intra CU
// below 32x32, 0 or 3 at 32x32; a 4x4 block reads its list at j*4 + i, larger ones the 8x8 list
// at (j/r)*8 + i/r (r = N/8), and 16x16 and 32x32 blocks take the DC value (0 read as 16) at
// (0,0).  The lists sit 16-byte aligned.
template <int LOG2>
__device__ __forceinline__ const uint8_t* scaling_list(const hevc_scaling_t* S, int c_idx, bool intra) {
    constexpr int SIZE_ID = LOG2 - 2;
    return S->list[SIZE_ID][(SIZE_ID < 3 ? c_idx : 0) + (intra ? 0 : 3)];
}

// A TU of a residual launch: its record, where its levels lie, and for an intra TU (its residual
// goes to the intra stage) where the residual goes.
struct ResTu {
    hevc_tu_t t;
    uint32_t from, to;
    bool live, intra, bypass, tskip;
};
__device__ __forceinline__ ResTu res_tu(const PicDesc& P, const uint32_t* items, int item, int n) {
    ResTu r;
    r.live = item < n;
    const uint32_t id = r.live ? items[item] : 0u, at = id & ~RES_INTRA_ITEM;
    r.intra = (id & RES_INTRA_ITEM) != 0;
    r.t = r.live ? (r.intra ? P.itu_rec[at] : P.tus[at]) : hevc_tu_t{};
    const int2 ft = r.intra ? P.itu_res[at] : make_int2((int)r.t.coeff_offset, 0);
    r.from = (uint32_t)ft.x;
    r.to = (uint32_t)ft.y;
    r.bypass = r.t.flags & (HEVC_TU_BYPASS | HEVC_TU_PCM);   // levels are the residual
    r.tskip = (r.t.flags & HEVC_TU_TSKIP) && !r.bypass;
    return r;
}
// 4 predicted samples plus their residuals, clipped (reconstruct_block).
__device__ __forceinline__ uint32_t add_clip4(uint32_t pred, uint32_t r01, uint32_t r23) {
    // residuals above 256 saturate the same, and the sum then stays in int16
    const uint32_t a = __viaddmin_s16x2_relu(__byte_perm(pred, 0u, 0x4140), __vmins2(r01, 0x01000100u), 0x00FF00FFu);
    const uint32_t b = __viaddmin_s16x2_relu(__byte_perm(pred, 0u, 0x4342), __vmins2(r23, 0x01000100u), 0x00FF00FFu);
    return __byte_perm(a, b, 0x6420);
}

// Row j of a TU's prediction and output, and the pitch of their rows (n: of packed blocks).
struct ResAt {
    const uint8_t* pred;
    uint8_t* out;
    int pitch;
};
__device__ __forceinline__ ResAt res_at(const PicDesc& P, const ResTu& u, int j, int n, int mode) {
    if (mode == RES_PACKED) return ResAt{P.rec + u.t.coeff_offset + j * n, P.dst + u.t.coeff_offset + j * n, n};
    const int pitch = u.t.c_idx ? P.pitch_c : P.pitch_y;
    uint8_t* const out =
        P.rec + (u.t.c_idx == 0 ? 0 : (u.t.c_idx == 1 ? P.off_cb : P.off_cr)) + (int64_t)(u.t.y + j) * pitch + u.t.x;
    return ResAt{out, out, pitch};
}

// ---- 4x4: a thread per TU, in registers.  Row of inputs -> outputs k: word k of `w` holds the
// four weights, DCT or DST-VII (transform.cpp:22-43) alike, so the two mix in a warp.
__device__ __forceinline__ void residual_4x4(const PicDesc& P, const ResTu& u, int mode) {
    uint32_t r[8];   // residuals, two words a row
    uint32_t x[2][4];   // words of rows (0, 1) and (2, 3), by column
    if (u.live) {
        const int4* src = reinterpret_cast<const int4*>(P.coeffs + u.from);
        const int4 c0 = src[0], c1 = src[1];
        const uint32_t c[8] = {(uint32_t)c0.x, (uint32_t)c0.y, (uint32_t)c0.z, (uint32_t)c0.w,
                               (uint32_t)c1.x, (uint32_t)c1.y, (uint32_t)c1.z, (uint32_t)c1.w};
        if (u.bypass) {
#pragma unroll
            for (int i = 0; i < 8; i++) r[i] = c[i];
        } else {
            const Dequant q = dequant_of(u.t.qp, 2);
            uint4 m = make_uint4(0x10101010u, 0x10101010u, 0x10101010u, 0x10101010u);
            if (P.scaling)
                m = *reinterpret_cast<const uint4*>(scaling_list<2>(P.scaling, u.t.c_idx, u.t.flags & HEVC_TU_INTRA));
            const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const uint32_t ma = mw[2 * h] >> 16 * i, mb = mw[2 * h + 1] >> 16 * i;
                    dequant_pairs(c[4 * h + i], c[4 * h + 2 + i], q, ma & 255, ma >> 8 & 255, mb & 255, mb >> 8 & 255,
                                  x[h][2 * i], x[h][2 * i + 1]);
                }
        }
    }
    pdl_wait();   // what is above needs only the records; the predictions come from the kernels before
    if (!u.live) return;
    const ResAt at = res_at(P, u, 0, 4, mode);
    uint32_t pv[4];
    if (!u.intra) {
#pragma unroll
        for (int k = 0; k < 4; k++) pv[k] = *reinterpret_cast<const uint32_t*>(at.pred + k * at.pitch);
    }
    if (u.tskip) {
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t a = x[h][2 * i], b = x[h][2 * i + 1];
                r[4 * h + i] = pack_sat_s16x2(((int)(int16_t)a + 64) >> 7, ((int)(int16_t)b + 64) >> 7);
                r[4 * h + 2 + i] = pack_sat_s16x2((((int)a >> 16) + 64) >> 7, (((int)b >> 16) + 64) >> 7);
            }
    } else if (!u.bypass) {
        const bool dst = (u.t.flags & HEVC_TU_INTRA) && u.t.c_idx == 0;
        const uint32_t w[4] = {dst ? pack_w(29, 74, 84, 55) : pack_w(64, 83, 64, 36),
                               dst ? pack_w(55, 74, -29, -84) : pack_w(64, 36, -64, -83),
                               dst ? pack_w(74, 0, -74, 74) : pack_w(64, -36, -64, 83),
                               dst ? pack_w(84, -74, 55, -29) : pack_w(64, -83, 64, -36)};
#pragma unroll
        for (int k = 0; k < 4; k++) {   // first pass gives row k, the second its residuals
            int y[4];
#pragma unroll
            for (int i = 0; i < 4; i++) y[i] = dp2_hi(x[1][i], w[k], dp2_lo(x[0][i], w[k], 64)) >> 7;
            const uint32_t y01 = pack_sat_s16x2(y[0], y[1]), y23 = pack_sat_s16x2(y[2], y[3]);
            int z[4];
#pragma unroll
            for (int i = 0; i < 4; i++) z[i] = dp2_hi(y23, w[i], dp2_lo(y01, w[i], 2048)) >> 12;
            r[2 * k] = pack_sat_s16x2(z[0], z[1]);
            r[2 * k + 1] = pack_sat_s16x2(z[2], z[3]);
        }
    }
    if (u.intra) {
        uint4* dst = reinterpret_cast<uint4*>(P.resid + u.to);
        dst[0] = make_uint4(r[0], r[1], r[2], r[3]);
        dst[1] = make_uint4(r[4], r[5], r[6], r[7]);
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        *reinterpret_cast<uint32_t*>(at.out + k * at.pitch) = add_clip4(pv[k], r[2 * k], r[2 * k + 1]);
}

// ---- 8x8 to 32x32: N threads per TU, all in one warp.  Thread j dequantises half of two rows
// into words of two inputs, transforms column j and then row j.  Shared memory of a TU: the words
// [N/2][N], then, over them, the intermediate's rows, inputs in the order of the words, at a
// pitch that keeps 16-byte reads of rows free of bank conflicts; TUs of a warp start in banks
// that keep its column accesses so.
__host__ __device__ constexpr int res_pitch(int n) { return n == 8 ? 16 : (n == 16 ? 48 : 80); }        // bytes
__host__ __device__ constexpr int res_slot(int n) { return n == 8 ? 160 : (n == 16 ? 832 : 2560); }     // bytes
constexpr int RES_THREADS = 128;
__host__ __device__ constexpr int res_tus(int log2) { return log2 == 2 ? RES_THREADS : RES_THREADS >> log2; }   // of a CTA

template <int LOG2>
__device__ __forceinline__ void residual_nxn(const PicDesc& P, const ResTu& u, int j, uint8_t* slot, int mode) {
    constexpr int N = 1 << LOG2;
    uint32_t* const words = reinterpret_cast<uint32_t*>(slot);
    if (u.live) {
        const int m = j / 2, h = j % 2;
        int ra, rb;
        pair_inputs<N>(m, ra, rb);
        const int16_t* const src = P.coeffs + u.from + h * (N / 2);
        constexpr int W = N / 4;   // words of half a row
        uint32_t a[W], b[W], x[N / 2];
        if constexpr (N == 8) {
            const uint2 va = *reinterpret_cast<const uint2*>(src + ra * N), vb = *reinterpret_cast<const uint2*>(src + rb * N);
            a[0] = va.x, a[1] = va.y, b[0] = vb.x, b[1] = vb.y;
        } else {
#pragma unroll
            for (int q = 0; q < W / 4; q++) {
                const uint4 va = reinterpret_cast<const uint4*>(src + ra * N)[q];
                const uint4 vb = reinterpret_cast<const uint4*>(src + rb * N)[q];
                a[4 * q] = va.x, a[4 * q + 1] = va.y, a[4 * q + 2] = va.z, a[4 * q + 3] = va.w;
                b[4 * q] = vb.x, b[4 * q + 1] = vb.y, b[4 * q + 2] = vb.z, b[4 * q + 3] = vb.w;
            }
        }
        if (u.bypass) {
#pragma unroll
            for (int i = 0; i < W; i++) {
                x[2 * i] = __byte_perm(a[i], b[i], 0x5410);
                x[2 * i + 1] = __byte_perm(a[i], b[i], 0x7632);
            }
        } else {
            const Dequant q = dequant_of(u.t.qp, LOG2);
            if (P.scaling) {
                constexpr int R = N / 8;
                const uint8_t* const list = scaling_list<LOG2>(P.scaling, u.t.c_idx, u.t.flags & HEVC_TU_INTRA);
                const uint32_t ma = *reinterpret_cast<const uint32_t*>(list + 8 * (ra / R) + 4 * h);
                const uint32_t mb = *reinterpret_cast<const uint32_t*>(list + 8 * (rb / R) + 4 * h);
                int dc = ma & 255;
                if (LOG2 >= 4 && ra == 0 && h == 0) {
                    constexpr int SIZE_ID = LOG2 - 2;
                    dc = P.scaling->dc[LOG2 >= 4 ? SIZE_ID - 2 : 0]
                                      [(SIZE_ID < 3 ? u.t.c_idx : 0) + (u.t.flags & HEVC_TU_INTRA ? 0 : 3)];
                    dc = dc ? dc : 16;
                }
#pragma unroll
                for (int i = 0; i < W; i++) {
                    const int s0 = 8 * (2 * i / R), s1 = 8 * ((2 * i + 1) / R);
                    dequant_pairs(a[i], b[i], q, i == 0 ? dc : (int)(ma >> s0 & 255), ma >> s1 & 255, mb >> s0 & 255,
                                  mb >> s1 & 255, x[2 * i], x[2 * i + 1]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < W; i++) dequant_pairs(a[i], b[i], q, 16, 16, 16, 16, x[2 * i], x[2 * i + 1]);
            }
        }
        uint4* const d = reinterpret_cast<uint4*>(words + j * (N / 2));   // row m, half h
#pragma unroll
        for (int q = 0; q < N / 8; q++) d[q] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
    }
    __syncwarp();
    // first pass: column j, shift 7, int16 clip
    const bool transform = u.live && !u.bypass && !u.tskip;
    uint32_t x[N / 2], r[N / 2];
    int d[N];
    if (transform) {
#pragma unroll
        for (int m = 0; m < N / 2; m++) x[m] = words[m * N + j];
    }
    __syncwarp();
    if (transform) {
        idct_pairs<N>(x, 64, d);
        uint8_t* const col = slot + 2 * pair_place<N>(j);
#pragma unroll
        for (int k = 0; k < N; k += 2) {
            const uint32_t v = pack_sat_s16x2(d[k] >> 7, d[k + 1] >> 7);
            *reinterpret_cast<uint16_t*>(col + k * res_pitch(N)) = (uint16_t)v;
            *reinterpret_cast<uint16_t*>(col + (k + 1) * res_pitch(N)) = (uint16_t)(v >> 16);
        }
    }
    __syncwarp();
    pdl_wait();   // what is above needs only the records; the predictions come from the kernels before
    const ResAt at = res_at(P, u, j, N, mode);
    uint32_t pv[N / 4];   // the prediction's row
    if (u.live && !u.intra) {
        if constexpr (N == 8) {
            const uint2 v = *reinterpret_cast<const uint2*>(at.pred);
            pv[0] = v.x, pv[1] = v.y;
        } else {
#pragma unroll
            for (int q = 0; q < N / 16; q++) {
                const uint4 v = reinterpret_cast<const uint4*>(at.pred)[q];
                pv[4 * q] = v.x, pv[4 * q + 1] = v.y, pv[4 * q + 2] = v.z, pv[4 * q + 3] = v.w;
            }
        }
    }
    // second pass: row j, shift 12 (20 - BitDepth), int16 clip; r: words of residuals in order
    if (transform) {
        const uint4* const row = reinterpret_cast<const uint4*>(slot + j * res_pitch(N));
#pragma unroll
        for (int q = 0; q < N / 8; q++) {
            const uint4 v = row[q];
            x[4 * q] = v.x, x[4 * q + 1] = v.y, x[4 * q + 2] = v.z, x[4 * q + 3] = v.w;
        }
        idct_pairs<N>(x, 2048, d);
#pragma unroll
        for (int k = 0; k < N / 2; k++) r[k] = pack_sat_s16x2(d[2 * k] >> 12, d[2 * k + 1] >> 12);
    } else if (u.live) {   // the levels of row j, or with transform skip what they dequantise to
        const int place = pair_place<N>(j);
        const int16_t* const row = reinterpret_cast<const int16_t*>(words + place / 2 * N) + place % 2;
#pragma unroll
        for (int k = 0; k < N / 2; k++) {
            int v0 = row[4 * k], v1 = row[4 * k + 2];
            if (u.tskip) v0 = (v0 + 64) >> 7, v1 = (v1 + 64) >> 7;
            r[k] = pack_sat_s16x2(v0, v1);
        }
    }

    if (!u.live) return;
    if (u.intra) {
        uint4* const dst = reinterpret_cast<uint4*>(P.resid + u.to + j * N);
#pragma unroll
        for (int q = 0; q < N / 8; q++) dst[q] = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
        return;
    }
#pragma unroll
    for (int q = 0; q < N / 4; q++) pv[q] = add_clip4(pv[q], r[2 * q], r[2 * q + 1]);
    if constexpr (N == 8) {
        *reinterpret_cast<uint2*>(at.out) = make_uint2(pv[0], pv[1]);
    } else {
#pragma unroll
        for (int q = 0; q < N / 16; q++)
            reinterpret_cast<uint4*>(at.out)[q] = make_uint4(pv[4 * q], pv[4 * q + 1], pv[4 * q + 2], pv[4 * q + 3]);
    }
}

// The coded TUs of a launch's pictures, all sizes.  Per picture the items lie by size, largest
// first, and so do its blocks.
struct ResSeg {
    const uint32_t* items;
    const PicDesc* pic;
    int32_t n[4];    // 4x4, 8x8, 16x16, 32x32
    int32_t block0;
    int32_t pad;
};
struct ResTable {
    int32_t n;
    int32_t pad;
    ResSeg s[MAX_SEGS];
};
__host__ __device__ constexpr int res_blocks(int n, int log2) { return (n + res_tus(log2) - 1) / res_tus(log2); }

// Bound by latency: a block's chain of dependent loads (item, record, levels, prediction) at 10
// CTAs per SM, 0.5 warp instructions per scheduler and cycle; 16 1080p P/B pictures 50 us (9
// CTAs 52, 12 CTAs 50), their bytes 18 us.  As four launches, N threads per TU also for
// 4x4, products of single levels and 64-bit dequantisation, it issued 41 million warp
// instructions in 61 us, now 26; for one picture four launches' latency counted: 23 us, now 11.
// The prediction is read before the second pass, which hides its latency (57 us when read after).
__global__ void __launch_bounds__(RES_THREADS, 10) k_residual(const __grid_constant__ ResTable st, int mode) {
    __shared__ __align__(16) uint8_t s_tu[res_tus(5) * res_slot(32)];
    static_assert(res_tus(3) * res_slot(8) <= sizeof(s_tu) && res_tus(4) * res_slot(16) <= sizeof(s_tu));
    pdl_next();
    int k = 0, b = blockIdx.x;
    while (k + 1 < st.n && st.s[k + 1].block0 <= b) k++;
    const ResSeg& sg = st.s[k];
    b -= sg.block0;
    const PicDesc& P = *sg.pic;
    const uint32_t* items = sg.items;
    const int tid = threadIdx.x;
    if (b < res_blocks(sg.n[3], 5)) {
        const ResTu u = res_tu(P, items, b * res_tus(5) + tid / 32, sg.n[3]);
        residual_nxn<5>(P, u, tid % 32, s_tu + tid / 32 * res_slot(32), mode);
        return;
    }
    b -= res_blocks(sg.n[3], 5);
    items += sg.n[3];
    if (b < res_blocks(sg.n[2], 4)) {
        const ResTu u = res_tu(P, items, b * res_tus(4) + tid / 16, sg.n[2]);
        residual_nxn<4>(P, u, tid % 16, s_tu + tid / 16 * res_slot(16), mode);
        return;
    }
    b -= res_blocks(sg.n[2], 4);
    items += sg.n[2];
    if (b < res_blocks(sg.n[1], 3)) {
        const ResTu u = res_tu(P, items, b * res_tus(3) + tid / 8, sg.n[1]);
        residual_nxn<3>(P, u, tid % 8, s_tu + tid / 8 * res_slot(8), mode);
        return;
    }
    b -= res_blocks(sg.n[1], 3);
    items += sg.n[1];
    residual_4x4(P, res_tu(P, items, b * res_tus(2) + tid, sg.n[0]), mode);
}

// ======================================================================================
// Motion grid: one warp per PU writes its 4x4 entries (used by the Bs derivation).
// ======================================================================================
__global__ void k_motion_grid(const __grid_constant__ SegTable st) {
    pdl_next();
    pdl_wait();
    const PicDesc& P = *st.s[blockIdx.y].pic;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
    if (warp >= P.num_pus) return;
    const hevc_pu_t pu = P.pus[warp];
    MotionEnt m;
    m.mv[0][0] = pu.mv[0][0]; m.mv[0][1] = pu.mv[0][1];
    m.mv[1][0] = pu.mv[1][0]; m.mv[1][1] = pu.mv[1][1];
    m.ref[0] = pu.ref_idx[0]; m.ref[1] = pu.ref_idx[1];
    m.pad = 0;
    const int bw = pu.w / 4, n = bw * (pu.h / 4), gw = P.width / 4;
    for (int e = lane; e < n; e += 32) {
        int gy = pu.y / 4 + e / bw, gx = pu.x / 4 + e % bw;
        P.mot[(int64_t)gy * gw + gx] = m;
    }
}

// Frame output: the conformance window of a slot's three planes widened to 16-bit
// samples (the HEVCFrame planes of hevc_decoder_get_frame).  Plane p covers rows
// [0, h[p]) of its window; each thread writes 8 samples (one 16-byte store) of a staged
// row whose pitch is the window width rounded up to 8 samples, so every store is aligned;
// the bytes are read one by one (the window may start on any even column).
// The checksum of the H.265 decoded picture hash SEI (Rec. ITU-T H.265 D.3.19) of each
// plane of a frame, for 8-bit samples: the sum modulo 2^32 of sample ^ xorMask over the
// plane, xorMask = (x & 0xFF) ^ (y & 0xFF) ^ (x >> 8) ^ (y >> 8).  A sum, so the planes'
// rows are shared out over the CTAs (grid.y = plane) and the partial sums added atomically
// (32-bit wrap-around is the modulo).
struct ChecksumArgs {
    const uint8_t* src[3];
    int32_t pitch[3], w[3], h[3];
    uint32_t* out;   // three words, zero before the launch
};
__global__ void __launch_bounds__(256) k_picture_checksum(const __grid_constant__ ChecksumArgs a) {
    const int p = blockIdx.y;
    const int w = a.w[p], h = a.h[p];
    uint32_t sum = 0;
    for (int y = blockIdx.x; y < h; y += gridDim.x) {
        const uint8_t* row = a.src[p] + (int64_t)y * a.pitch[p];
        const uint32_t ym = (uint32_t)(y & 0xFF) ^ (uint32_t)(y >> 8);
        for (int x = threadIdx.x; x < w; x += blockDim.x)
            sum += (uint32_t)row[x] ^ ym ^ (uint32_t)(x & 0xFF) ^ (uint32_t)(x >> 8);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&a.out[p], sum);
}

struct WidenArgs {
    const uint8_t* src[3];   // first sample of the window in each plane of the slot
    int32_t src_pitch[3];
    uint16_t* dst[3];        // staged planes
    int32_t w[3], h[3], vecs[3];   // window size; 8-sample vectors per staged row
    int64_t first[3];              // first vector index of each plane (first[0] = 0)
    int64_t total;
};

__global__ void __launch_bounds__(256) k_widen_frame(const __grid_constant__ WidenArgs a) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.total) return;
    const int p = i >= a.first[2] ? 2 : (i >= a.first[1] ? 1 : 0);
    const int64_t k = i - a.first[p];
    const int row = (int)(k / a.vecs[p]), x0 = (int)(k % a.vecs[p]) * 8;
    const uint8_t* s = a.src[p] + (int64_t)row * a.src_pitch[p];
    uint32_t v[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int x = x0 + 2 * q;
        const uint32_t lo = x < a.w[p] ? s[x] : 0u, hi = x + 1 < a.w[p] ? s[x + 1] : 0u;
        v[q] = lo | (hi << 16);
    }
    *reinterpret_cast<uint4*>(a.dst[p] + (int64_t)row * a.vecs[p] * 8 + x0) = make_uint4(v[0], v[1], v[2], v[3]);
}

}  // namespace hevcgpu
