// intra.cuh — intra prediction (perform_intra_prediction, intra_prediction.cpp:428-481,
// with build_reference_samples :44-211, filtering :217-257, planar/DC/angular :263-422).
//
// Every intra TU reads reference samples left of and above it.  Those samples are final
// when this stage runs, except where an earlier intra TU writes them (MC and the inter
// residuals ran before).  The host turns that into a dependency list per intra TU: the
// TUs that own samples of its reference array, in its own CTU (local) or in an earlier CTU
// (external), and orders each CTU's TUs by their depth in the picture's dependency DAG.
// k_intra_ctus runs one CTA per CTU with intra TUs: it stages the CTU with the samples
// around it, its TU records, dependency lists and residuals in shared memory; its warps take
// the TUs in order and run each one once the TUs whose samples its mode reads are complete
// (one-arrival barriers in shared memory for local ones; the CTA's watcher warp follows the
// flags that other CTUs publish and brings their samples in).  Every wait gives up after
// WAIT_LIMIT_NS of the GPU's global timer (or SPIN_LIMIT polls, should the timer not
// advance), sets ST_TIMEOUT in the context's sticky status word (the host turns it into
// HEVCGPU_ETIMEOUT) and returns.
//
// What bounds it: the chain of dependent TUs, not bytes.  So everything that needs no sample
// comes before a TU's wait (intra_plan.h: availability, substitution, sample addresses and
// weights), every sample is read from shared memory after it, and a TU does not wait for
// samples that its mode does not read (a 1080p I picture's longest chain: 860 TUs instead of
// 2167).  Batch of 8 1080p I pictures: 1.18 ms, 2.18 ms with the waits on every owner and the
// work after the wait.
#pragma once

#include <cuda/atomic>

#include "device_common.cuh"
#include "intra_plan.h"

namespace hevcgpu {

__constant__ int8_t c_intra_angle[35] = {0,   0,   32,  26,  21,  17,  13,  9,  5,  2,  0,  -2,
                                         -5,  -9,  -13, -17, -21, -26, -32, -26, -21, -17, -13, -9,
                                         -5,  -2,  0,   2,   5,   9,   13,  17,  21,  26,  32};
__constant__ int16_t c_inv_angle[35] = {0,    0,    256, 315, 390, 482,  630,  910,  1638, 4096, 0,   4096,
                                        1638, 910,  630, 482, 390, 315,  256,  315,  390,  482,  630, 910,
                                        1638, 4096, 0,   4096, 1638, 910, 630, 482,  390,  315,  256};


// The picture fields a TU reads, copied into shared memory once per CTA: reads of the
// descriptor in global memory would go through L1, which every GPU-scope acquire on the SM
// invalidates, and sit in each TU's chain of dependent loads.
struct IntraPic {
    uint8_t* rec;
    int64_t off_cb, off_cr;
    int32_t width, height, log2_ctb, pitch_y, pitch_c, intra_smoothing_disabled, strong_intra;
};

// A warp's reference samples of an 8x8..32x32 TU, in main order (mirrored for the
// horizontal modes, so that the main side always runs upwards from index 2n): as read, and
// smoothed and / or projected.
struct alignas(4) IntraWarpSmem {
    uint8_t raw[132];   // 4n + 1 samples
    uint8_t ref[132];   // the smoothed array, or main entries q = -n .. 2n + 1 at [q + n]
};

// One plane of the CTU in shared memory with the samples around it that its TUs read: the
// column left of it, the corner, and the row above as far as the end of the above-right
// CTU.  Sample (x, y) counted from the CTU's origin is at t[y * pitch + x]; only row -1
// reaches past the CTU's width.
struct CtuTile {
    uint8_t* t;
    int pitch, x0, y0;
};

// Address (offset from the CTU's origin in its tile) of reference sample k of a TU whose
// origin is at offset o.
__device__ __forceinline__ int ref_offset(int o, int pitch, int n, int k) {
    return k < 2 * n ? o - 1 + (2 * n - 1 - k) * pitch : o - pitch + (k - 2 * n - 1);
}

__device__ __forceinline__ uint32_t dp4a_uu(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// The 4x4 TU (most TUs, and most of a picture's dependency chain): one output sample per lane
// (x = lane & 3, y = lane >> 2; the upper half of the warp repeats the lower), each from four
// samples of the tile whose addresses and weights are known before the wait (IntraTaps4), so
// that what follows it is four shared loads, a weighted sum and a store.  4x4 references are
// never smoothed (:217-230 and :443-445).  done() completes the TU: the tile holds its
// samples; the store to the picture follows it, off the chain.
// In a 1080p I picture a TU takes 150 cycles after its wait; 980 when samples were fetched by
// lane and moved by shuffles, other CTUs' samples read through L2, and the substitution found
// with ballots.
template <typename Wait, typename Done>
__device__ __forceinline__ bool intra_tu4(const IntraPic& P, const hevc_tu_t& t, uint32_t av_word, int lane,
                                          const CtuTile& tile, const int16_t* res, Wait&& wait, Done&& done) {
    const bool chroma = t.c_idx != 0;
    const int x = lane & 3, y = (lane >> 2) & 3, mode = t.intra_mode;
    const IntraAvail av = avail_unpack(av_word, 4);
    const IntraTaps4 k = intra_taps4(mode, chroma, x, y, lane, c_intra_angle[mode], c_inv_angle[mode]);
    const int o = (t.y - tile.y0) * tile.pitch + (t.x - tile.x0);
    const bool none = avail_segs(av) == 0u;   // no reference sample: every one is 128
    int at[4];
#pragma unroll
    for (int j = 0; j < 4; j++) at[j] = none ? 0 : ref_offset(o, tile.pitch, 4, intra_substitute(av, k.i[j]));
    const int r = res != nullptr ? res[lane & 15] : 0;
    const bool pcm = (t.flags & HEVC_TU_PCM) != 0;
    uint8_t* const plane = P.rec + (t.c_idx == 0 ? 0 : (t.c_idx == 1 ? P.off_cb : P.off_cr));
    const int pitch = chroma ? P.pitch_c : P.pitch_y;
    if (!wait()) return false;
    int v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = none ? 128 : (int)tile.t[at[j]];
    if (mode == 1) v[1] = (int)(__reduce_add_sync(0xffffffffu, lane < 8 ? v[1] : 0) + 4) >> 3;
    int p = clip_u8((v[0] * k.w[0] + v[1] * k.w[1] + v[2] * k.w[2] + v[3] * k.w[3] + k.add) >> k.shift);
    if (pcm) p = 0;   // the PCM samples are the levels, with no prediction
    const uint8_t out = (uint8_t)clip_u8(p + r);
    if (lane < 16) tile.t[o + y * tile.pitch + x] = out;
    done();
    if (lane < 16) plane[(int64_t)(t.y + y) * pitch + t.x + x] = out;
    return true;
}

// The 8x8, 16x16 and 32x32 TU (perform_intra_prediction, then reconstruct_block's add and
// clip), one copy of the code for the three sizes to keep the kernel small in the instruction
// cache.  After the wait the substituted reference array goes from the tile to the warp's
// shared memory in main order; smoothing and the projection of the side reference, where the
// mode has them, make one more pass over it; then each lane predicts groups of 4 samples of a
// row (its column is the same for all its groups).  done() as in intra_tu4, after the stores.
template <typename Wait, typename Done>
__device__ __forceinline__ bool intra_tu(const IntraPic& P, const hevc_tu_t& t, uint32_t av_word, int lane,
                                         IntraWarpSmem& W, const CtuTile& tile, const int16_t* res, Wait&& wait,
                                         Done&& done) {
    constexpr int RMAX = 5;   // lane rounds of the largest reference array
    const int log2 = t.log2_size, n = 1 << log2, total = 4 * n + 1, mode = t.intra_mode;
    const bool chroma = t.c_idx != 0, vert = mode >= 18 || mode < 2;
    const IntraAvail av = avail_unpack(av_word, n);
    const bool none = avail_segs(av) == 0u;
    const bool smooth = intra_smoothed(mode, log2, chroma, P.intra_smoothing_disabled != 0);
    const int ang = c_intra_angle[mode], inv = c_inv_angle[mode];
    const int o = (t.y - tile.y0) * tile.pitch + (t.x - tile.x0);
    int at[RMAX];   // where sample i = lane + 32 r of the array in main order lies
#pragma unroll
    for (int r = 0; r < RMAX; r++) {
        const int i = plan_min(lane + 32 * r, 4 * n);
        at[r] = none ? 0 : ref_offset(o, tile.pitch, n, intra_substitute(av, vert ? i : 4 * n - i));
    }
    const int gpr = n >> 2, x0 = 4 * (lane & (gpr - 1)), ystep = 32 >> (log2 - 2);
    int cidx[4], cw[4];   // horizontal modes: the columns' offsets and weights
#pragma unroll
    for (int j = 0; j < 4; j++) {
        cidx[j] = ((x0 + j + 1) * ang) >> 5;
        cw[j] = ((x0 + j + 1) * ang) & 31;
    }
    const bool edge = !chroma && n < 32, pcm = (t.flags & HEVC_TU_PCM) != 0;
    uint8_t* const plane = P.rec + (t.c_idx == 0 ? 0 : (t.c_idx == 1 ? P.off_cb : P.off_cr));
    const int pitch = chroma ? P.pitch_c : P.pitch_y;
    if (!wait()) return false;

    // 1. the substituted reference array (:177-197)
#pragma unroll
    for (int r = 0; r < RMAX; r++) {
        const int i = lane + 32 * r;
        if (i < total) W.raw[i] = none ? (uint8_t)128 : tile.t[at[r]];
    }
    __syncwarp();
    // 2. smoothing of luma references (:217-257, :443-471): [1 2 1] over the array, ends
    //    kept, or the bilinear strong smoothing of 32x32; and for the modes with a negative
    //    angle the main reference with the side reference projected (:346-368)
    int ro = 0, mo = 2 * n;   // offsets from W.raw: the array in main order, main reference entry 0
    if (smooth || ang < 0) {
        const int c = W.raw[2 * n], e0 = W.raw[0], e1 = W.raw[4 * n];
        const bool strong = smooth && n == 32 && P.strong_intra && abs(c + e1 - 2 * W.raw[3 * n]) < 8 &&
                            abs(c + e0 - 2 * W.raw[n]) < 8;
        const int count = ang < 0 ? 3 * n + 2 : total;
        for (int e = lane; e < count; e += 32) {
            const int i = ang < 0 ? intra_main_index(true, inv, n, e - n) : e;
            int f = W.raw[i];
            if (smooth && i != 0 && i != 4 * n) {
                if (strong) {
                    const int d = i > 2 * n ? i - 2 * n : 2 * n - i;   // from the corner (0: the corner itself)
                    f = ((2 * n - d) * c + d * (i > 2 * n ? e1 : e0) + n) >> (log2 + 1);
                } else {
                    f = (W.raw[i - 1] + 2 * f + W.raw[i + 1] + 2) >> 2;
                }
            }
            W.ref[e] = (uint8_t)f;
        }
        __syncwarp();
        ro = (int)sizeof(W.raw);
        mo = ro + (ang < 0 ? n : 2 * n);   // with a negative angle only the main entries are read
    }
    const uint8_t* const R = W.raw + ro;
    const uint8_t* const M = W.raw + mo;
    // 3. prediction + residual, clip, store
    int dc = 0;
    if (mode == 1) {   // predict_dc :295-317
        int sum = 0;
        if (lane < n) sum = R[2 * n + 1 + lane] + R[2 * n - 1 - lane];
        sum = __reduce_add_sync(0xffffffffu, sum);
        dc = (sum + n) >> (log2 + 1);
    }
    const int corner = M[0];
    for (int y = lane >> (log2 - 2); y < n; y += ystep) {
        int p[4];
        if (mode == 0) {   // predict_planar :263-289
            const int left = R[2 * n - 1 - y], tr = R[3 * n + 1], bl = R[n - 1];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int x = x0 + j;
                p[j] = ((n - 1 - x) * left + (x + 1) * tr + (n - 1 - y) * R[2 * n + 1 + x] + (y + 1) * bl + n) >>
                       (log2 + 1);
            }
        } else if (mode == 1) {
            const int left = R[2 * n - 1 - y];
#pragma unroll
            for (int j = 0; j < 4; j++) p[j] = edge && y == 0 ? (R[2 * n + 1 + x0 + j] + 3 * dc + 2) >> 2 : dc;
            if (edge && x0 == 0) p[0] = y == 0 ? (R[2 * n + 1] + left + 2 * dc + 2) >> 2 : (left + 3 * dc + 2) >> 2;
        } else if (vert) {   // predict_angular :323-422, main reference on top
            // entries q .. q + 4 of the main reference as bytes of two realigned words; sample j
            // weighs bytes j and j + 1
            const int idx = ((y + 1) * ang) >> 5, fr = ((y + 1) * ang) & 31;
            const int a = mo + x0 + 1 + idx;
            const uint32_t* const words = reinterpret_cast<const uint32_t*>(W.raw) + (a >> 2);
            const uint32_t w0 = words[0], w1 = words[1];
            const uint32_t lo = __funnelshift_r(w0, w1, 8 * (a & 3)), hi = w1 >> (8 * (a & 3));
            const uint32_t wt = (uint32_t)(32 - fr) | ((uint32_t)fr << 8);
            p[0] = (int)(dp4a_uu(lo, wt, 16u) >> 5);
            p[1] = (int)(dp4a_uu(lo, wt << 8, 16u) >> 5);
            p[2] = (int)(dp4a_uu(lo, wt << 16, 16u) >> 5);
            p[3] = (int)(dp4a_uu(__funnelshift_r(lo, hi, 24), wt, 16u) >> 5);
            if (edge && mode == 26 && x0 == 0) p[0] = clip_u8(p[0] + ((R[2 * n - 1 - y] - corner) >> 1));
        } else {   // main reference on the left
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint8_t* m = M + y + 1 + cidx[j];
                p[j] = ((32 - cw[j]) * m[0] + cw[j] * m[1] + 16) >> 5;
            }
            if (edge && mode == 10 && y == 0) {
#pragma unroll
                for (int j = 0; j < 4; j++) p[j] = clip_u8(p[j] + ((R[2 * n - 1 - x0 - j] - corner) >> 1));
            }
        }
        if (pcm) {   // the PCM samples are the levels, with no prediction
#pragma unroll
            for (int j = 0; j < 4; j++) p[j] = 0;
        }
        // residual (four int16 in one 8-byte load), clip, one word to the tile and the picture
        if (res != nullptr) {
            const int2 rw = *reinterpret_cast<const int2*>(res + y * n + x0);
            p[0] = clip_u8(p[0] + (int)(int16_t)(rw.x & 0xFFFF));
            p[1] = clip_u8(p[1] + (rw.x >> 16));
            p[2] = clip_u8(p[2] + (int)(int16_t)(rw.y & 0xFFFF));
            p[3] = clip_u8(p[3] + (rw.y >> 16));
        }
        const uint32_t w = (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
        *reinterpret_cast<uint32_t*>(tile.t + o + y * tile.pitch + x0) = w;
        *reinterpret_cast<uint32_t*>(plane + (int64_t)(t.y + y) * pitch + t.x + x0) = w;
    }
    done();
    return true;
}

// ---------------------------------------------------------------------------------------
// CTU tasks.  One CTA per CTU that holds intra TUs.  CTAs take CTUs by ticket in wavefront
// order per picture (2 * row + column: the diagonal band along which a picture's
// dependencies advance), the pictures of a launch side by side.  The CTA stages the CTU with
// the samples around it, its TU records and their residuals in shared memory; then its warps
// take the TUs one at a time in task order (by depth in the picture's DAG, so every TU comes
// after the TUs it depends on) and run each as soon as the TUs whose samples it reads are
// complete: a TU of the same CTU through its one-arrival barrier in shared memory, a TU of
// an earlier CTU through that TU's published completion in global memory.  No barrier ties
// the warps together, so the critical path is the chain of dependent TUs itself.  Every wait
// is for a TU taken earlier, by this CTA or by a CTA holding an earlier ticket, which is
// already running; every wait is bounded.  The CTA's last warp is its watcher: it alone
// polls the global flags of the TUs of other CTUs and copies their samples into the tile's
// border, so the workers only read shared memory and wait on shared-memory barriers, which
// suspend them without taking issue slots.
// ---------------------------------------------------------------------------------------
constexpr int IC_WARPS = 8;
constexpr int IC_THREADS = 32 * IC_WARPS;
constexpr int IC_MIN_BLOCKS = 3;
// Tiles: a margin of 16 bytes (its last byte is the column left of the CTU; 16 keeps the
// CTU's rows on 16-byte boundaries for the asynchronous copies), the CTU, the CTU to the
// right (row -1 only); row -1 first.  Pitches that are odd multiples of 16 spread a column
// over the banks.
constexpr int IC_MARGIN = 16;
constexpr int IC_LP = IC_MARGIN + 2 * 64, IC_LH = 65;    // luma: pitch, rows
constexpr int IC_CP = IC_MARGIN + 2 * 32, IC_CH = 33;    // chroma
constexpr int IC_MAX_TUS = 256 + 2 * 64;             // 4x4 TUs of a 64x64 CTU, all planes
constexpr int IC_MAX_RES = 64 * 64 + 2 * 32 * 32;    // residual samples of a 64x64 CTU
constexpr int IC_DEP_STAGE = 2048;                   // dependency entries staged per CTU
constexpr int IC_MAX_WATCH = 128;                    // TUs of other CTUs a CTU waits for
constexpr int IC_WORKERS = IC_WARPS - 1;             // worker warps; the last warp watches
constexpr unsigned long long WAIT_LIMIT_NS = 1000000000ull;   // a wait gives up after a second
constexpr unsigned SPIN_LIMIT = 1u << 26;            // backstop: polls of at least 64 ns

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// 16-byte asynchronous global -> shared copy (through L2 only, so that samples other
// CTUs wrote are seen), and the wait for all of a thread's copies.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(gmem));
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// One-arrival barriers in shared memory, one per TU of the CTU: the warp that completes
// the TU arrives (release), the warps whose TUs read its samples wait on phase 0 (acquire).
// A waiting thread is suspended by the hardware until the phase completes or the time hint
// runs out, so waiting warps take no issue slots from the working ones.
__device__ __forceinline__ void mbar_init1(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n\t}" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(bar))
                 : "memory");
}
// whether phase 0 of the barrier has completed, without waiting
__device__ __forceinline__ bool mbar_test0(uint64_t* bar) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cta.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"((uint32_t)__cvta_generic_to_shared(bar))
        : "memory");
    return ok != 0;
}
// true once phase 0 of the barrier has completed; false when the time hint ran out first
__device__ __forceinline__ bool mbar_try_wait0(uint64_t* bar) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], 0, %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(20000u)
        : "memory");
    return ok != 0;
}

// Copy plane c of CTU (rx, ry) and the samples around it into its tile (16-byte copies are
// issued, not waited for).  Samples of other CTUs that an intra TU still has to write come
// again with that TU's completion (the watcher); all others are final.
__device__ __forceinline__ void stage_tile(const PicDesc& P, int c, int rx, int ry, uint8_t* origin, int tid,
                                           int threads) {
    const int sub = c ? 2 : 1, ctbc = (1 << P.log2_ctb) / sub;
    const int pw = P.width / sub, ph = P.height / sub, pitch = c ? P.pitch_c : P.pitch_y;
    const uint8_t* plane = P.rec + (c == 0 ? 0 : (c == 1 ? P.off_cb : P.off_cr));
    const int tp = c ? IC_CP : IC_LP;
    const int x0 = rx * ctbc, y0 = ry * ctbc;
    if (ctbc >= 16) {
        // rows 0 .. ctbc - 1, then the row above over two CTUs (a 16-byte piece that starts
        // inside the picture ends inside the row's pitch, a multiple of 64)
        const int row_chunks = ctbc / 16, own = ctbc * row_chunks;
        for (int e = tid; e < own + 2 * row_chunks; e += threads) {
            const int r = e < own ? e / row_chunks : -1, q = e < own ? e % row_chunks : e - own;
            const int y = y0 + r, x = x0 + 16 * q;
            if (y < 0 || y >= ph || x >= pw) continue;
            cp_async16(origin + r * tp + 16 * q, plane + (int64_t)y * pitch + x);
        }
    } else {  // 8-sample chroma CTBs (16x16 CTUs): words
        for (int e = tid; e < ctbc * 2 + 4; e += threads) {
            const int r = e < ctbc * 2 ? e / 2 : -1, q = e < ctbc * 2 ? e % 2 : e - ctbc * 2;
            const int y = y0 + r, x = x0 + 4 * q;
            if (y < 0 || y >= ph || x >= pw) continue;
            *reinterpret_cast<uint32_t*>(origin + r * tp + 4 * q) =
                __ldcg(reinterpret_cast<const uint32_t*>(plane + (int64_t)y * pitch + x));
        }
    }
    if (rx > 0)   // the corner and the column to the left
        for (int r = tid - 1; r < ctbc; r += threads) {
            const int y = y0 + r;
            if (y >= 0 && y < ph) origin[r * tp - 1] = __ldcg(plane + (int64_t)y * pitch + x0 - 1);
        }
}

// The state one worker's wait for a TU's dependencies reads.
struct IntraWait {
    const uint32_t* s_dep;      // the CTU's staged dependency entries
    const uint32_t* dep_list;   // all entries (those past the staged ones)
    uint64_t* s_bar;            // completion barriers of the CTU's TUs, then its watch barriers
    int32_t* itu_done;          // published completions (direct external entries)
    uint32_t* sticky;
    volatile int* s_abort;
    int dfirst, doff, dcount, staged, task, n_watch, n_itu, epoch, lane;
    uint32_t need;              // the parts of the reference array the TU reads (SEG_*)
};

// True while the wait that began at t0 may go on (t0 = 0: it begins now).
__device__ __forceinline__ bool wait_goes_on(unsigned long long& t0, unsigned polls, uint32_t* sticky,
                                             volatile int* s_abort) {
    if (*s_abort) return false;
    const unsigned long long now = global_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 <= WAIT_LIMIT_NS && polls < SPIN_LIMIT) return true;
    atomicOr(sticky, ST_TIMEOUT);
    return false;
}

// A direct external entry: polls the published completion (only a planted test wait has one).
__device__ __noinline__ bool wait_published(int32_t* flag, int epoch, uint32_t* sticky, volatile int* s_abort) {
    cuda::atomic_ref<int32_t, cuda::thread_scope_device> f(*flag);
    unsigned long long t0 = 0;
    for (unsigned polls = 0; f.load(cuda::memory_order_relaxed) != epoch; polls++) {
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> status(*sticky);
        if (!wait_goes_on(t0, polls, sticky, s_abort) || (status.load(cuda::memory_order_relaxed) & ST_TIMEOUT))
            return false;
        __nanosleep(64);
    }
    cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
    return true;
}

// The wait for a TU's dependencies, between the position work and the loads of a TU path:
// each lane tests one entry's barrier, entries whose TU wrote nothing the mode reads are
// passed over, and while some are pending the warp is suspended as a whole on the pending one
// with the greatest index (watched TUs come after local ones, local ones by depth), which
// is mostly the last to complete.  Testing the entries one after the other cost 130 cycles
// each.  Every wait reads the global timer and gives up after WAIT_LIMIT_NS (SPIN_LIMIT tries
// as a backstop), marking the sticky status; a wait also ends when another warp of the CTA
// gave up (s_abort) or, for external waits, when a wait anywhere did (the status word).
__device__ __forceinline__ bool intra_wait(const IntraWait& w) {
    constexpr uint32_t FULL = 0xffffffffu;
    bool gave_up = false;
    for (int base = 0; base < w.dcount && !gave_up; base += 32) {
        const int q = base + w.lane, at = w.doff + q;
        uint32_t bar = 0;   // 1 + index of the barrier this lane's entry waits for, 0 when it does not
        if (q < w.dcount) {
            const uint32_t e = at >= 0 && at < w.staged ? w.s_dep[at] : __ldg(&w.dep_list[w.dfirst + at]);
            const uint32_t k = e & INTRA_DEP_INDEX;
            if (e & INTRA_DEP_EXTERNAL) {
                if (k < (uint32_t)w.n_itu) {
                    gave_up = !wait_published(&w.itu_done[k], w.epoch, w.sticky, w.s_abort);
                } else {
                    atomicOr(w.sticky, ST_BAD_RECORD);
                    gave_up = true;
                }
            } else if ((e >> INTRA_DEP_SEG_SHIFT) & w.need) {
                if (k < (uint32_t)((e & INTRA_DEP_WATCH) ? w.n_watch : w.task)) {
                    bar = 1 + ((e & INTRA_DEP_WATCH) ? IC_MAX_TUS + k : k);
                    if (mbar_test0(&w.s_bar[bar - 1])) bar = 0;
                } else {
                    atomicOr(w.sticky, ST_BAD_RECORD);   // not an earlier TU, or no such watch slot: refused
                    gave_up = true;
                }
            }
        }
        gave_up = __any_sync(FULL, gave_up);
        unsigned long long t0 = 0;
        uint32_t last = __reduce_max_sync(FULL, bar);
        for (unsigned polls = 0; last != 0u && !gave_up; polls++) {
            if (!mbar_try_wait0(&w.s_bar[last - 1])) gave_up = !wait_goes_on(t0, polls, w.sticky, w.s_abort);
            if (bar != 0u && mbar_test0(&w.s_bar[bar - 1])) bar = 0;
            last = __reduce_max_sync(FULL, bar);
            // the lanes may have seen the barrier, the abort word or the clock at different moments
            gave_up = __any_sync(FULL, gave_up);
        }
    }
    // the warp barrier orders each lane's acquires before every lane's reads of the samples
    __syncwarp();
    return !gave_up;
}

// A CTA's shared memory (dynamic: more than 48 KB).
struct IntraSmem {
    alignas(16) uint8_t t_luma[IC_LH * IC_LP];
    alignas(16) uint8_t t_chroma[2][IC_CH * IC_CP];
    alignas(16) hevc_tu_t tu[IC_MAX_TUS];
    alignas(16) int16_t res[IC_MAX_RES];
    alignas(16) hevc_tu_t wtu[IC_MAX_WATCH];   // records of the watched TUs of other CTUs
    uint64_t bar[IC_MAX_TUS + IC_MAX_WATCH];   // completion of the CTU's TUs, by task index, then of the watched ones
    IntraWarpSmem ws[IC_WORKERS];
    uint32_t av[IC_MAX_TUS];        // available and needed reference samples (avail_pack)
    uint32_t itu_dep[IC_MAX_TUS];   // dependency lists: (offset << 6) | count
    uint32_t dep[IC_DEP_STAGE];     // the CTU's dependency entries
    uint32_t watch[IC_MAX_WATCH];   // the watched TUs' task indices in the picture
    uint32_t wneed[IC_MAX_WATCH / 32];   // those whose samples some TU reads
    IntraPic pic;
    uint32_t nb;
    int ticket, pic_index, next;
    volatile int abort;
};

__global__ void __launch_bounds__(IC_THREADS, IC_MIN_BLOCKS) k_intra_ctus(const __grid_constant__ SegTable st,
                                                                       int32_t* tickets, int total, uint32_t* sticky) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    IntraSmem& S = *reinterpret_cast<IntraSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    if (tid == 0) {
        // Each picture hands out its CTUs by ticket in wavefront order.  CTAs start at picture
        // blockIdx.x % n, so the pictures of a launch progress side by side; a picture whose
        // tickets are used up passes the CTA on.  There are as many CTAs as CTUs, so every
        // CTA finds one.
        int k = blockIdx.x % st.n, got = -1;
        for (int tries = 0; tries < st.n && got < 0; tries++) {
            const int n_k = (k + 1 < st.n ? st.s[k + 1].aux0 : total) - st.s[k].aux0;
            const int v = atomicAdd(&tickets[k], 1);
            if (v < n_k) got = v;
            else k = k + 1 == st.n ? 0 : k + 1;
        }
        // a wait of this launch (or an earlier one not yet read) gave up: the CTU could only
        // wait for work that will not come, so the CTA ends at once
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> status(*sticky);
        S.ticket = (status.load(cuda::memory_order_relaxed) & ST_TIMEOUT) ? -1 : got;
        S.pic_index = k;
        S.abort = 0;
        S.next = 0;
    }
    if (tid < IC_MAX_WATCH / 32) S.wneed[tid] = 0;
    __syncthreads();
    if (S.ticket < 0) return;
    const int k = S.pic_index;
    const PicDesc& P = *st.s[k].pic;
    const int32_t epoch = st.s[k].aux1;
    const int idx = S.ticket;
    const int a = P.ictu_addr[idx], rx = a % P.wctb, ry = a / P.wctb;

    if (tid == 32) {
        S.pic.rec = P.rec;
        S.pic.off_cb = P.off_cb;
        S.pic.off_cr = P.off_cr;
        S.pic.width = P.width;
        S.pic.height = P.height;
        S.pic.log2_ctb = P.log2_ctb;
        S.pic.pitch_y = P.pitch_y;
        S.pic.pitch_c = P.pitch_c;
        S.pic.intra_smoothing_disabled = P.intra_smoothing_disabled;
        S.pic.strong_intra = P.strong_intra;
    }
    if (tid == 4) {  // which neighbour CTBs share this CTB's slice and tile
        const int sl = P.ctb_slice ? P.ctb_slice[a] : 0, ti = P.ctb_tile ? P.ctb_tile[a] : 0;
        auto same = [&](int nx, int ny) {
            if (nx < 0 || ny < 0 || nx >= P.wctb) return false;
            const int b = ny * P.wctb + nx;
            return (P.ctb_slice ? P.ctb_slice[b] : 0) == sl && (P.ctb_tile ? P.ctb_tile[b] : 0) == ti;
        };
        S.nb = (same(rx - 1, ry) ? NB_LEFT : 0u) | (same(rx - 1, ry - 1) ? NB_ABOVE_LEFT : 0u) |
               (same(rx, ry - 1) ? NB_ABOVE : 0u) | (same(rx + 1, ry - 1) ? NB_ABOVE_RIGHT : 0u);
    }

    // stage the CTU's tiles, TU records and residuals (packed in task order, one thread per
    // TU) in one round of asynchronous copies
    const int off = P.ictu_tu_off[idx], n_tu = P.ictu_tu_off[idx + 1] - off;
    for (int i = tid; i < n_tu; i += IC_THREADS) {
        cp_async16(&S.tu[i], &P.itu_rec[off + i]);
        mbar_init1(&S.bar[i]);
        S.itu_dep[i] = __ldg(&P.itu_dep[off + i]);
    }
    // the CTU's dependency entries are contiguous in task order
    const uint32_t dfirst = __ldg(&P.itu_dep[off]) >> 6, dlast_e = __ldg(&P.itu_dep[off + n_tu - 1]);
    const int n_dep = (int)((dlast_e >> 6) + (dlast_e & 63u)) - (int)dfirst;
    const int staged = max(0, min(n_dep, IC_DEP_STAGE));
    for (int q = tid; q < staged; q += IC_THREADS) S.dep[q] = __ldg(&P.dep_list[dfirst + q]);
    const uint32_t wd = __ldg(&P.ictu_watch[idx]);
    const int n_watch = min((int)(wd & 0xFFu), IC_MAX_WATCH);
    for (int q = tid; q < n_watch; q += IC_THREADS) {
        const uint32_t w = __ldg(&P.watch[(wd >> 8) + q]);
        S.watch[q] = w;
        if (w < (uint32_t)P.n_itu) cp_async16(&S.wtu[q], &P.itu_rec[w]);
        mbar_init1(&S.bar[IC_MAX_TUS + q]);
    }
    // the CTU's origin in each plane's tile
    auto origin = [&](int c) {
        return c == 0 ? S.t_luma + IC_LP + IC_MARGIN : S.t_chroma[0] + (c - 1) * (IC_CH * IC_CP) + IC_CP + IC_MARGIN;
    };
    for (int c = 0; c < 3; c++) stage_tile(P, c, rx, ry, origin(c), tid, IC_THREADS);
    for (int i = tid; i < n_tu; i += IC_THREADS) {
        const int4 r = __ldg(&P.itu_res[off + i]);
        for (int c = 0; c < r.z; c++) cp_async16(S.res + r.y + 8 * c, P.resid + r.x + 8 * c);
    }
    cp_async_wait_all();
    __syncthreads();

    // what each TU reads, and the watched TUs that write some of it
    const int ctbl = 1 << P.log2_ctb;
    for (int i = tid; i < n_tu; i += IC_THREADS) {
        const hevc_tu_t t = S.tu[i];
        const int c = t.c_idx != 0;
        const IntraAvail av = intra_avail(t.x, t.y, 1 << t.log2_size, P.width >> c, P.height >> c, P.log2_ctb - c, 1 + c,
                                          S.nb);
        const bool smooth = intra_smoothed(t.intra_mode, t.log2_size, c, P.intra_smoothing_disabled != 0);
        const uint32_t need = intra_need(
            intra_parts(t.intra_mode, t.log2_size, c, (t.flags & HEVC_TU_PCM) != 0, smooth), avail_segs(av));
        S.av[i] = avail_pack(av, need);
        const uint32_t dd = S.itu_dep[i];
        for (int q = 0; q < (int)(dd & 63u); q++) {
            const int at = (int)(dd >> 6) - (int)dfirst + q;
            const uint32_t e = at >= 0 && at < staged ? S.dep[at] : __ldg(&P.dep_list[(dd >> 6) + q]);
            const uint32_t j = e & INTRA_DEP_INDEX;
            if ((e & INTRA_DEP_WATCH) && ((e >> INTRA_DEP_SEG_SHIFT) & need) && j < (uint32_t)n_watch)
                atomicOr(&S.wneed[j / 32], 1u << (j % 32));
        }
    }
    __syncthreads();

    if (warp == IC_WORKERS) {
        // The watcher: each lane follows the published completions of up to 4 watched TUs of
        // other CTUs that some TU here reads from, all of them polled at once through L2
        // (the wait is bounded like every other).  When some are seen, the warp copies
        // each one's samples along this CTU into the tile's border and arrives on its
        // watch barrier.  The acquire fence orders the other CTU's samples before the copies,
        // the release arrival the copies before every read of a worker that waits on the
        // barrier.
        constexpr int R = IC_MAX_WATCH / 32;
        bool pend[R], bad = false;
        int32_t* flag[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int j = lane + 32 * r;
            pend[r] = j < n_watch && ((S.wneed[r] >> lane) & 1u);
            if (pend[r] && S.watch[j] >= (uint32_t)P.n_itu) bad = true;   // no such TU: refused
            flag[r] = P.itu_done + (pend[r] && !bad ? S.watch[j] : 0);
        }
        if (__any_sync(0xffffffffu, bad)) {
            if (bad) atomicOr(sticky, ST_BAD_RECORD);
            S.abort = 1;
            return;
        }
        unsigned long long t0 = 0;
        for (unsigned polls = 0;; polls++) {
            int32_t v[R];
            // relaxed polls (a GPU-scope acquire invalidates the SM's L1), one acquire fence
            // once flags are seen
#pragma unroll
            for (int r = 0; r < R; r++) {
                cuda::atomic_ref<int32_t, cuda::thread_scope_device> f(*flag[r]);
                v[r] = pend[r] ? f.load(cuda::memory_order_relaxed) : epoch;
            }
            uint32_t seen[R], some = 0, left = 0;
#pragma unroll
            for (int r = 0; r < R; r++) {
                seen[r] = __ballot_sync(0xffffffffu, pend[r] && v[r] == epoch);
                left |= __ballot_sync(0xffffffffu, pend[r] && v[r] != epoch);
                some |= seen[r];
            }
            if (some) {
                cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
                __syncwarp();
#pragma unroll
                for (int r = 0; r < R; r++) {
                    pend[r] = pend[r] && v[r] != epoch;
                    for (uint32_t m = seen[r]; m; m &= m - 1u) {
                        const int j = 32 * r + __ffs(m) - 1;
                        const hevc_tu_t t = S.wtu[j];
                        const int c = t.c_idx != 0, n = 1 << t.log2_size, ctbc = ctbl >> c;
                        const int x = t.x - rx * ctbc, y = t.y - ry * ctbc;   // counted from this CTU
                        const int pitch = c ? P.pitch_c : P.pitch_y, tp = c ? IC_CP : IC_LP;
                        uint8_t* const o = origin(t.c_idx);
                        const uint8_t* const src =
                            P.rec + (t.c_idx == 0 ? 0 : (t.c_idx == 1 ? P.off_cb : P.off_cr)) + (int64_t)t.y * pitch + t.x;
                        if (lane < n) {
                            // its last row along this CTU's top, its last column along the left side
                            if (y + n == 0 && x + lane >= -1 && x + lane < 2 * ctbc)
                                o[x + lane - tp] = __ldcg(src + (int64_t)(n - 1) * pitch + lane);
                            if (x + n == 0 && y + lane >= 0 && y + lane < ctbc)
                                o[(y + lane) * tp - 1] = __ldcg(src + (int64_t)lane * pitch + n - 1);
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&S.bar[IC_MAX_TUS + j]);
                    }
                }
                t0 = 0;
                polls = 0;
            }
            if (!left) break;
            if (some) continue;
            cuda::atomic_ref<uint32_t, cuda::thread_scope_device> status(*sticky);
            const bool stop = !wait_goes_on(t0, polls, sticky, &S.abort) ||
                              (status.load(cuda::memory_order_relaxed) & ST_TIMEOUT);
            if (__any_sync(0xffffffffu, stop)) {
                S.abort = 1;
                break;
            }
            __nanosleep(32);
        }
        return;
    }
    for (;;) {
        int i = 0;
        if (lane == 0) i = S.abort ? n_tu : atomicAdd(&S.next, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= n_tu) break;
        const hevc_tu_t tu = S.tu[i];
        const uint32_t dd = S.itu_dep[i], av = S.av[i];
        const int dcount = (int)(dd & 63u), doff = (int)(dd >> 6) - (int)dfirst;
        const IntraWait wc{S.dep,  P.dep_list, S.bar, P.itu_done, sticky, &S.abort, (int)dfirst,   doff, dcount,
                           staged, i,          n_watch, P.n_itu,  epoch,  lane,     avail_need(av)};
        auto wait = [&]() -> bool { return intra_wait(wc); };
        // after the warp barrier, lane 0's release arrival orders the warp's samples in the
        // tile before the completion
        auto done = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.bar[i]);
        };
        const int ctbc = tu.c_idx ? ctbl / 2 : ctbl;
        CtuTile tile;
        tile.t = origin(tu.c_idx);
        tile.pitch = tu.c_idx ? IC_CP : IC_LP;
        tile.x0 = rx * ctbc;
        tile.y0 = ry * ctbc;
        const int16_t* res = (tu.flags & HEVC_TU_CODED) ? S.res + tu.coeff_offset : nullptr;
        const bool ok = tu.log2_size == 2 ? intra_tu4(S.pic, tu, av, lane, tile, res, wait, done)
                                          : intra_tu(S.pic, tu, av, lane, S.ws[warp], tile, res, wait, done);
        if (!ok) {
            if (lane == 0) S.abort = 1;
            break;
        }
        if (tu.reserved[0] & ITU_PUBLISH) {
            // the release store orders the warp's samples in the picture before the flag
            __syncwarp();
            if (lane == 0) {
                cuda::atomic_ref<int32_t, cuda::thread_scope_device> g(P.itu_done[off + i]);
                g.store(epoch, cuda::memory_order_release);
            }
        }
    }
}

}  // namespace hevcgpu
