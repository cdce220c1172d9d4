// kernels.cuh — the reconstruction kernels (sm_100a).
//
//   k_residual<LOG2>  dequant + inverse DST/DCT + add-and-clip of coded TUs
//                     (transform.cpp:293-394, coding_tree.cpp:371-396)
//   (motion compensation: mc.cuh; intra prediction: intra.cuh)
//   k_motion_grid     4x4 motion grid of the PUs (store_pu_motion's grid)
//   (in-loop filters: filters.cuh)
//   k_picture_checksum  per-plane checksum of a frame (H.265 picture hash SEI, D.3.19)
#pragma once

#include "device_common.cuh"

namespace hevcgpu {

// ======================================================================================
// Inverse transform.  The N-point inverse DCT is computed by the even/odd recursion of
// the HEVC basis: out[k] = E[k] + O[k], out[N-1-k] = E[k] - O[k], with E the N/2-point
// inverse of the even inputs and O[k] the odd-input dot products.  The basis entries
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

template <int N>
__device__ __forceinline__ void idct_1d(const int* src, int* dst) {
    if constexpr (N == 2) {
        dst[0] = 64 * src[0] + 64 * src[1];
        dst[1] = 64 * src[0] - 64 * src[1];
    } else {
        int ev[N / 2], E[N / 2];
#pragma unroll
        for (int n = 0; n < N / 2; n++) ev[n] = src[2 * n];
        idct_1d<N / 2>(ev, E);
#pragma unroll
        for (int k = 0; k < N / 2; k++) {
            int o = 0;
#pragma unroll
            for (int n = 0; n < N / 2; n++) o += dct_w<N>(2 * n + 1, k) * src[2 * n + 1];
            dst[k] = E[k] + o;
            dst[N - 1 - k] = E[k] - o;
        }
    }
}

// DST-VII 4x4 (transform.cpp:22-43): out[k] = sum_n D[n][k] * src[n]
__device__ __forceinline__ void idst4_1d(const int* s, int* d) {
    d[0] = 29 * s[0] + 74 * s[1] + 84 * s[2] + 55 * s[3];
    d[1] = 55 * s[0] + 74 * s[1] - 29 * s[2] - 84 * s[3];
    d[2] = 74 * s[0] - 74 * s[2] + 74 * s[3];
    d[3] = 84 * s[0] - 74 * s[1] + 55 * s[2] - 29 * s[3];
}

template <int N>
__device__ __forceinline__ void inv_1d(const int* s, int* d, bool dst4) {
    if constexpr (N == 4) {
        if (dst4) { idst4_1d(s, d); return; }
    }
    idct_1d<N>(s, d);
}

// Dequantisation of one level (transform.cpp:360-365) with ms = m * levelScale[qP % 6]:
// the product, the shift by qP / 6 and the rounding shift in int64, narrowing to int
// (modulo 2^32), int16 clip.  |c * ms| <= 32768 * 255 * 72 fits an int.
__device__ __forceinline__ int16_t dequant1(int c, int ms, int qp_per, int bd_shift) {
    if (c == 0) return 0;
    long long v = (long long)(c * ms);
    v = v * (1ll << qp_per) + (1ll << (bd_shift - 1));
    v >>= bd_shift;
    return (int16_t)clip3(-32768, 32767, (int)(unsigned)(unsigned long long)v);
}

// Scaling factors m of row j of an N x N block (transform.cpp:320-358): matrixId is the
// plane plus 3 for a non-intra CU below 32x32, 0 or 3 at 32x32; a 4x4 block reads its
// list at j*4 + i, larger ones the 8x8 list at (j/r)*8 + i/r (r = N/8), and 16x16 and
// 32x32 blocks take the DC value (0 read as 16) at (0,0).  The lists sit 16-byte aligned,
// so a row is one 4- or 8-byte load.
template <int LOG2>
__device__ __forceinline__ void scaling_row(const hevc_scaling_t* S, int c_idx, bool intra, int j,
                                            int (&m)[1 << LOG2]) {
    constexpr int N = 1 << LOG2, SIZE_ID = LOG2 - 2;
    const int matrix = (SIZE_ID < 3 ? c_idx : 0) + (intra ? 0 : 3);
    const uint8_t* list = S->list[SIZE_ID][matrix];
    if constexpr (LOG2 == 2) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(list + 4 * j);
#pragma unroll
        for (int i = 0; i < 4; i++) m[i] = (w >> (8 * i)) & 255;
    } else {
        constexpr int R = N / 8;
        const uint2 w = *reinterpret_cast<const uint2*>(list + 8 * (j / R));
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int k = i / R;
            m[i] = ((k < 4 ? w.x : w.y) >> (8 * (k & 3))) & 255;
        }
        if constexpr (LOG2 >= 4) {
            if (j == 0) {
                const int dc = S->dc[SIZE_ID - 2][matrix];
                m[0] = dc ? dc : 16;
            }
        }
    }
}

__constant__ int c_level_scale[6] = {40, 45, 51, 57, 64, 72};

// Residual kernel: N threads per TU (thread j owns column j in the first pass and row j
// in the second), 128 threads per CTA.  Coefficients are staged through shared memory;
// the intermediate has a padded row pitch (N + 2 int16) so that row reads by different
// threads hit distinct banks.
template <int LOG2>
__global__ void __launch_bounds__(128) k_residual(const __grid_constant__ SegTable st, int mode) {
    constexpr int N = 1 << LOG2;
    constexpr int TUS = 128 / N;
    constexpr int TP = N + 2;
    __shared__ __align__(16) int16_t s_coef[TUS][N * N];
    __shared__ int16_t s_tmp[TUS][N * TP];

    pdl_next();
    const int slot = threadIdx.x / N;
    const int j = threadIdx.x % N;
    const Seg& sg = st.s[find_seg(st, blockIdx.x)];
    const int item = (blockIdx.x - sg.block0) * TUS + slot;
    const bool live = item < sg.n_items;
    const PicDesc& P = *sg.pic;
    const uint32_t id = live ? static_cast<const uint32_t*>(sg.items)[item] : 0u;
    const bool intra_item = (id & RES_INTRA_ITEM) != 0;   // residual into resid, for the intra stage
    const uint32_t at = id & ~RES_INTRA_ITEM;
    hevc_tu_t t = live ? (intra_item ? P.itu_rec[at] : P.tus[at]) : hevc_tu_t{};
    const int2 from_to = intra_item ? P.itu_res[at] : make_int2((int)t.coeff_offset, 0);
    const bool bypass = t.flags & (HEVC_TU_BYPASS | HEVC_TU_PCM);   // levels are the residual
    const bool tskip = (t.flags & HEVC_TU_TSKIP) && !bypass;
    const bool dst4 = (LOG2 == 2) && (t.flags & HEVC_TU_INTRA) && t.c_idx == 0;

    // load row j of the levels and dequantise it
    if (live) {
        const int16_t* src = P.coeffs + (uint32_t)from_to.x + j * N;
        int16_t v[N];
        if constexpr (N >= 8) {
#pragma unroll
            for (int q = 0; q < N / 8; q++) {
                int4 w = reinterpret_cast<const int4*>(src)[q];
                *reinterpret_cast<int4*>(&v[q * 8]) = w;
            }
        } else {
            int2 w = *reinterpret_cast<const int2*>(src);
            *reinterpret_cast<int2*>(&v[0]) = w;
        }
        if (!bypass) {
            const int scale = c_level_scale[t.qp % 6], qp_per = t.qp / 6, bd_shift = 8 + LOG2 - 5;
            if (P.scaling) {
                int m[N];
                scaling_row<LOG2>(P.scaling, t.c_idx, t.flags & HEVC_TU_INTRA, j, m);
#pragma unroll
                for (int i = 0; i < N; i++) v[i] = dequant1(v[i], m[i] * scale, qp_per, bd_shift);
            } else {
#pragma unroll
                for (int i = 0; i < N; i++) v[i] = dequant1(v[i], 16 * scale, qp_per, bd_shift);
            }
        }
#pragma unroll
        for (int i = 0; i < N; i++) s_coef[slot][j * N + i] = v[i];
    }
    __syncthreads();

    // first pass: column j, shift 7, int16 clip
    if (live && !tskip && !bypass) {
        int s[N], d[N];
#pragma unroll
        for (int n = 0; n < N; n++) s[n] = s_coef[slot][n * N + j];
        inv_1d<N>(s, d, dst4);
#pragma unroll
        for (int k = 0; k < N; k++) s_tmp[slot][k * TP + j] = (int16_t)clip3(-32768, 32767, (d[k] + 64) >> 7);
    }
    __syncthreads();
    // second pass: row j, shift 12 (20 - BitDepth), int16 clip
    int r[N];
    if (!live) {
    } else if (bypass) {
#pragma unroll
        for (int k = 0; k < N; k++) r[k] = s_coef[slot][j * N + k];
    } else if (tskip) {
#pragma unroll
        for (int k = 0; k < N; k++) r[k] = (s_coef[slot][j * N + k] + 64) >> 7;
    } else {
        int s[N], d[N];
#pragma unroll
        for (int n = 0; n < N; n++) s[n] = s_tmp[slot][j * TP + n];
        inv_1d<N>(s, d, dst4);
#pragma unroll
        for (int k = 0; k < N; k++) r[k] = clip3(-32768, 32767, (d[k] + 2048) >> 12);
    }

    pdl_wait();   // the transforms need only the records; the predictions come from the kernels before
    if (!live) return;
    if (intra_item) {
        // residual of an intra TU: the wavefront adds it to its prediction.  A row goes out in
        // 16-byte words (8-byte ones for 4x4): residuals lie at multiples of 16 samples
        uint32_t w[N / 2];
#pragma unroll
        for (int k = 0; k < N / 2; k++) w[k] = __byte_perm((uint32_t)r[2 * k], (uint32_t)r[2 * k + 1], 0x5410);
        int16_t* dst = P.resid + from_to.y + j * N;
        if constexpr (N >= 8) {
#pragma unroll
            for (int q = 0; q < N / 8; q++)
                reinterpret_cast<uint4*>(dst)[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        } else {
            *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
        }
        return;
    }
    const uint8_t* pred;
    uint8_t* out;
    if (mode == RES_PACKED) {
        pred = P.rec + t.coeff_offset + j * N;
        out = P.dst + t.coeff_offset + j * N;
    } else {
        int pitch = t.c_idx ? P.pitch_c : P.pitch_y;
        int64_t base = t.c_idx == 0 ? 0 : (t.c_idx == 1 ? P.off_cb : P.off_cr);
        out = P.rec + base + (int64_t)(t.y + j) * pitch + t.x;
        pred = out;
    }
    // add the prediction row and clip (reconstruct_block)
    if constexpr (N >= 16) {
#pragma unroll
        for (int q = 0; q < N / 16; q++) {
            uint4 pv = reinterpret_cast<const uint4*>(pred)[q];
            const uint8_t* pb = reinterpret_cast<const uint8_t*>(&pv);
            uint4 ov;
            uint8_t* ob = reinterpret_cast<uint8_t*>(&ov);
#pragma unroll
            for (int i = 0; i < 16; i++) ob[i] = (uint8_t)clip_u8(pb[i] + r[q * 16 + i]);
            reinterpret_cast<uint4*>(out)[q] = ov;
        }
    } else if constexpr (N == 8) {
        uint2 pv = *reinterpret_cast<const uint2*>(pred);
        const uint8_t* pb = reinterpret_cast<const uint8_t*>(&pv);
        uint2 ov;
        uint8_t* ob = reinterpret_cast<uint8_t*>(&ov);
#pragma unroll
        for (int i = 0; i < 8; i++) ob[i] = (uint8_t)clip_u8(pb[i] + r[i]);
        *reinterpret_cast<uint2*>(out) = ov;
    } else {
        uint32_t pv = *reinterpret_cast<const uint32_t*>(pred);
        uint32_t ov = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) ov |= (uint32_t)clip_u8((int)((pv >> (8 * i)) & 0xFF) + r[i]) << (8 * i);
        *reinterpret_cast<uint32_t*>(out) = ov;
    }
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
