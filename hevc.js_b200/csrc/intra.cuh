// intra.cuh — intra prediction (perform_intra_prediction, intra_prediction.cpp:428-481,
// with build_reference_samples :44-211, filtering :217-257, planar/DC/angular :263-422).
//
// Every intra TU reads reference samples left of and above it.  Those samples are final
// when this stage runs, except where an earlier intra TU writes them (MC and the inter
// residuals ran before).  The host turns that into a dependency list per intra TU: the
// TUs that own samples of its reference array, in its own CTU (local) or in an earlier CTU
// (external), and orders each CTU's TUs by their depth in the picture's dependency DAG.
// k_intra_plan turns that into work items with everything positions and modes tell; then
// k_intra_ctus runs one CTA per CTU with intra TUs: it stages the CTU with the samples
// around it, its items and residuals in shared memory; its warps take the items in order and
// run each one once the TUs whose samples its mode reads are complete (a barrier in shared
// memory per TU, which counts them; the CTA's watcher warp follows the border words that
// other CTUs write and brings their samples in).  Every wait gives up after WAIT_LIMIT_NS of
// the GPU's global timer (or SPIN_LIMIT polls, should the timer not advance), sets ST_TIMEOUT
// in the context's sticky status word (the host turns it into HEVCGPU_ETIMEOUT) and returns.
//
// What bounds it: the chain of dependent TUs and, in P/B pictures, the instructions per TU;
// not bytes.  So
//   - a TU waits only for TUs whose samples its mode reads (a 1080p I picture's longest chain
//     is 860 TUs; 2167 with every owner of its reference array);
//   - everything that needs no sample comes before its wait (intra_plan.h: availability,
//     substitution, sample addresses and weights), every sample is read from shared memory;
//   - a completed TU arrives at the TUs that wait for it, so a wait is one barrier (185 cycles
//     when it is met already, 97 from the last arrival; 550 and 270 when each TU tested the
//     barriers of all it depends on);
//   - samples cross CTU borders with their flag in one 64-bit word, with no fence on either
//     side;
//   - the code is small: what does not run per TU is a kernel of its own, since instruction
//     cache misses were half of all stalls with it inside.
// With the plan, 1 and 8 1080p I pictures take 0.42 and 0.59 ms (the eight 2.18 with waits on every
// owner and the work after the wait), 1 and 16 1080p P/B pictures 43 and 129 us, 107 and 276 then.
#pragma once

#include <cuda/atomic>

#include "device_common.cuh"
#include "intra_plan.h"

namespace hevcgpu {

__device__ const IntraTapTable c_intra_taps = intra_tap_table();
__constant__ IntraAngles c_intra = intra_angles();

// A warp's reference samples of an 8x8..32x32 TU, in main order: mirrored for the horizontal
// modes, so that the main side always runs upwards from index 2n.
struct alignas(4) IntraWarpSmem {
    uint8_t ref[136];   // 4n + 1 samples, and what aligned reads of them reach past the end
};

// A plane of the CTU lies in shared memory as a tile with the samples around it that its TUs
// read: the column left of it, the corner, and the row above as far as the end of the
// above-right CTU.  Sample (x, y) counted from the CTU's origin is at origin[y * pitch + x];
// only row -1 reaches past the CTU's width.

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

// A work item as k_intra_plan lays it down for the warp that runs it (32 bytes), a TU or one
// band of it: where its samples lie, what stands in for reference samples that are not
// available, what it waits for and who waits for it.
struct alignas(16) IntraTask {
    uint32_t pic;          // offset of the TU's first sample in the picture buffer
    uint32_t source;       // (first << 16) | count of the TUs that wait for the TU, in rev
    uint16_t tile;         // offset of its first sample in the CTU's tiles
    uint16_t res;          // offset of its residual in the CTU's residuals (zeros for a 4x4 TU without one)
    int16_t first, corner; // the first available reference sample and the one that stands at
                           // the corner, as tile offsets from its first sample
    uint8_t mode, flags;   // 0..34 or MODE_PCM; TASK_*
    uint8_t log2, y0;      // the TU's size; first row of the band
    int8_t angle;
    uint8_t waits;         // arrivals the TU's barrier takes
    uint8_t bl, tr;        // available samples below-left and top-right
    uint8_t row, column;   // its first border word along the CTU's bottom / right, or TASK_NO_EDGE
    int16_t inv_angle;
    uint16_t bar, pad;     // its barrier: the task index
};
static_assert(sizeof(IntraTask) == 32, "IntraTask is copied as two 16-byte words");
constexpr uint8_t TASK_NO_EDGE = 0xFF;
enum : uint8_t {
    TASK_CHROMA = 1, TASK_CODED = 2, TASK_SMOOTH = 4, TASK_LEFT = 8, TASK_TOP = 16,   // left / top available
    TASK_STARTED = 32,   // waits for nothing: its barrier starts complete
};

// Tile offset, from the TU's first sample, of the sample that stands at index i of its
// reference array (intra_substitute; the constant 128 when none is available).
__device__ __forceinline__ int task_where(const IntraTask& t, int n, int pitch, int i) {
    const bool top = t.flags & TASK_TOP;
    const int left = t.flags & TASK_LEFT ? (2 * n - 1 - plan_max(i, n - t.bl)) * pitch - 1 : t.first;
    const int along = plan_min(i, 3 * n + t.tr) - 2 * n - 1 - pitch;
    return i < 2 * n ? left : (i > (top ? 2 * n : 3 * n) && (top || t.tr) ? along : t.corner);
}

// Rows y0 .. y0 + rows - 1 of an 8x8 (smoothed), 16x16 or 32x32 TU (perform_intra_prediction,
// then reconstruct_block's add and clip) into the tile, one copy of the code for the three
// sizes.  The substituted reference array comes from the tile into registers, sample
// lane + 32 r in lane `lane` and the last one in every lane, is smoothed there and goes to the
// warp's shared memory in main order; for a negative angle the side reference is projected in
// front of the main one, in place; then each lane predicts groups of 4 samples of a row.
// at[r]: where sample lane + 32 r lies (r < 2); at_end: where sample 4n lies.
__device__ __forceinline__ void intra_predict(const IntraTask& task, int strong_intra, int lane, uint8_t* ref,
                                              int at0, int at1, int at_end, uint8_t* t, int pitch, int y0, int rows,
                                              const int16_t* res, bool coded) {
    constexpr uint32_t FULL = 0xffffffffu;
    const int log2 = task.log2, n = 1 << log2, mode = task.mode, ang = task.angle;
    const bool vert = mode >= 18 || mode < 2, smooth = task.flags & TASK_SMOOTH;
    const bool edge = !(task.flags & TASK_CHROMA) && log2 < 5;
    // 1. the substituted reference array (:177-197)
    int v[4], end = t[at_end];
    v[0] = t[at0];
    v[1] = v[2] = v[3] = 0;
    if (log2 > 3) v[1] = t[at1];
    if (log2 > 4) {
#pragma unroll
        for (int r = 2; r < 4; r++)
            v[r] = t[task_where(task, n, pitch, vert ? lane + 32 * r : 4 * n - lane - 32 * r)];
    }
    // 2. smoothing of luma references (:217-257, :443-471): [1 2 1] over the array, ends
    //    kept, or the bilinear strong smoothing of 32x32
    if (smooth) {
        const int rounds = 1 << (log2 - 3);
        int f[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            f[r] = v[r];
            if (r >= rounds) continue;
            const int down = __shfl_sync(FULL, v[r], (lane + 31) & 31), up = __shfl_sync(FULL, v[r], (lane + 1) & 31);
            const int below = r > 0 ? __shfl_sync(FULL, v[r > 0 ? r - 1 : 0], 31) : v[0];
            const int above = r + 1 < rounds ? __shfl_sync(FULL, v[r < 3 ? r + 1 : 3], 0) : end;
            if (r > 0 || lane > 0) f[r] = ((lane ? down : below) + 2 * v[r] + (lane < 31 ? up : above) + 2) >> 2;
        }
        if (log2 == 5 && strong_intra) {
            const int e0 = __shfl_sync(FULL, v[0], 0), c = __shfl_sync(FULL, v[2], 0);
            if (abs(c + end - 2 * __shfl_sync(FULL, v[3], 0)) < 8 && abs(c + e0 - 2 * __shfl_sync(FULL, v[1], 0)) < 8) {
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int i = lane + 32 * r, d = abs(i - 64);   // from the corner
                    if (i > 0) f[r] = ((64 - d) * c + d * (i > 64 ? end : e0) + 32) >> 6;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) v[r] = f[r];
    }
    ref[lane] = (uint8_t)v[0];
    if (log2 > 3) ref[lane + 32] = (uint8_t)v[1];
    if (log2 > 4) {
        ref[lane + 64] = (uint8_t)v[2];
        ref[lane + 96] = (uint8_t)v[3];
    }
    if (lane == 0) ref[4 * n] = (uint8_t)end;
    __syncwarp();
    // 3. for a negative angle, main entries -1 .. -n: the side reference projected through
    //    invAngle (:346-368)
    if (ang < 0) {
        const int side = ref[2 * n - plan_min(2 * n, ((lane + 1) * task.inv_angle + 128) >> 8)];
        __syncwarp();
        if (lane < n) ref[2 * n - 1 - lane] = (uint8_t)side;
        __syncwarp();
    }
    // 4. prediction + residual, clip, store
    int dc = 0;
    if (mode == 1) {   // predict_dc :295-317
        dc = (int)__reduce_add_sync(FULL, lane < n ? ref[2 * n + 1 + lane] + ref[2 * n - 1 - lane] : 0);
        dc = (dc + n) >> (log2 + 1);
    }
    const int x0 = 4 * (lane & ((n >> 2) - 1));
#pragma unroll 1
    for (int y = y0 + (lane >> (log2 - 2)); y < y0 + rows; y += 128 >> log2) {
        int2 rw = make_int2(0, 0);   // residual: four int16 in one 8-byte load
        if (coded) rw = *reinterpret_cast<const int2*>(res + y * n + x0);
        int p[4];
        if (mode < 2) {   // planar (:263-289) or DC with its edge rows
            const int left = ref[2 * n - 1 - y], tr = ref[3 * n + 1], bl = ref[n - 1];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int x = x0 + j, top = ref[2 * n + 1 + x];
                p[j] = mode == 0 ? ((n - 1 - x) * left + (x + 1) * tr + (n - 1 - y) * top + (y + 1) * bl + n) >> (log2 + 1)
                       : edge && y == 0 ? (top + 3 * dc + 2) >> 2
                                        : dc;
            }
            if (mode == 1 && edge && x0 == 0)
                p[0] = y == 0 ? (ref[2 * n + 1] + left + 2 * dc + 2) >> 2 : (left + 3 * dc + 2) >> 2;
        } else if (vert) {   // predict_angular :323-422, main reference on top
            // entries q .. q + 4 of the main reference as bytes of two realigned words; sample j
            // weighs bytes j and j + 1
            const int idx = ((y + 1) * ang) >> 5, fr = ((y + 1) * ang) & 31;
            const int a = 2 * n + x0 + 1 + idx;
            const uint32_t* const words = reinterpret_cast<const uint32_t*>(ref) + (a >> 2);
            const uint32_t w0 = words[0], w1 = words[1];
            const uint32_t lo = __funnelshift_r(w0, w1, 8 * (a & 3)), hi = w1 >> (8 * (a & 3));
            const uint32_t wt = (uint32_t)(32 - fr) | ((uint32_t)fr << 8);
            p[0] = (int)(dp4a_uu(lo, wt, 16u) >> 5);
            p[1] = (int)(dp4a_uu(lo, wt << 8, 16u) >> 5);
            p[2] = (int)(dp4a_uu(lo, wt << 16, 16u) >> 5);
            p[3] = (int)(dp4a_uu(__funnelshift_r(lo, hi, 24), wt, 16u) >> 5);
            if (edge && mode == 26 && x0 == 0) p[0] = clip_u8(p[0] + ((ref[2 * n - 1 - y] - ref[2 * n]) >> 1));
        } else {   // main reference on the left
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int idx = ((x0 + j + 1) * ang) >> 5, fr = ((x0 + j + 1) * ang) & 31;
                const uint8_t* m = ref + 2 * n + y + 1 + idx;
                p[j] = ((32 - fr) * m[0] + fr * m[1] + 16) >> 5;
                if (edge && mode == 10 && y == 0) p[j] = clip_u8(p[j] + ((ref[2 * n - 1 - x0 - j] - ref[2 * n]) >> 1));
            }
        }
        if (mode == MODE_PCM) p[0] = p[1] = p[2] = p[3] = 0;
        *reinterpret_cast<uint32_t*>(t + y * pitch + x0) =
            pack_sat_u8x4(p[0] + (int)(int16_t)(rw.x & 0xFFFF), p[1] + (rw.x >> 16), p[2] + (int)(int16_t)(rw.y & 0xFFFF),
                          p[3] + (rw.y >> 16));
    }
}

// ---------------------------------------------------------------------------------------
// CTU tasks.  One CTA per CTU that holds intra TUs.  CTAs take CTUs by ticket in wavefront
// order per picture (2 * row + column: the diagonal band along which a picture's
// dependencies advance), the pictures of a launch side by side.  The CTA's warps take the
// items one at a time in task order (by depth in the picture's DAG, so every TU comes after
// the TUs it depends on).  No barrier ties the warps together, so the critical path is the
// chain of dependent TUs itself.  Every wait is for a TU taken earlier, by this CTA or by a
// CTA holding an earlier ticket, which is already running.  The CTA's last warp is its
// watcher: it alone polls words of other CTUs, so the workers only read shared memory and
// wait on shared-memory barriers, which suspend them without taking issue slots.
// ---------------------------------------------------------------------------------------
// Warps of a CTA (the last one watches): the more, the more the chains decide and not the number
// of TUs (intra_warps).
constexpr int IC_NARROW = 8, IC_WIDE = 16, IC_FULL = 24;
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
constexpr int IC_SOURCES = IC_MAX_TUS + IC_MAX_WATCH;   // what a TU can wait for: TUs here, watched TUs
// These hold because intra TUs cover no sample twice and lie within their CTB (pictures for which
// that is not so go to k_intra_levels): a work item covers a 4x4 unit or more, and a TU of u x u
// units has at most 4u + 1 owners around it, five a unit at most.
static_assert(5 * IC_MAX_TUS <= IC_DEP_STAGE, "a CTU's dependency entries fit");
// Border words (4 samples) a CTU's TUs can read, per plane: the corner, the row above over two
// CTUs, the column to the left.
constexpr int IC_EDGE_L = 1 + 3 * 16, IC_EDGE_C = 1 + 3 * 8;
constexpr int IC_EDGES = 128;                        // >= IC_EDGE_L + 2 * IC_EDGE_C, 4 per watcher lane
constexpr int IC_TILES = IC_LH * IC_LP + 2 * IC_CH * IC_CP;   // bytes of the three tiles; then a byte 128
constexpr unsigned long long WAIT_LIMIT_NS = 1000000000ull;   // a wait gives up after a second
constexpr unsigned SPIN_LIMIT = 1u << 26;            // polls, should the timer not advance

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Barriers in shared memory, one per TU of the CTU that waits for others, with as many
// arrivals as the TUs it waits for: each arrives when it completes (release), the TU's warp
// waits on phase 0 (acquire).  A waiting thread is suspended by the hardware until the phase
// completes or the time hint runs out, so waiting warps take no issue slots from the working
// ones.
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(arrivals)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n\t}" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(bar))
                 : "memory");
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

// Copy plane c of CTU (rx, ry) and the samples around it into its tile (copies issued, not
// waited for).  Samples of other CTUs that an intra TU still has to write come again as
// border words (the watcher); all others are final.
template <int THREADS>
__device__ __forceinline__ void stage_tile(const PicDesc& P, int c, int rx, int ry, uint8_t* origin, int tid) {
    const int sub = c ? 1 : 0, log2c = P.log2_ctb - sub, cs = 1 << log2c;
    const int pw = P.width >> sub, ph = P.height >> sub, pitch = c ? P.pitch_c : P.pitch_y;
    const uint8_t* const plane = P.rec + (c == 0 ? 0 : (c == 1 ? P.off_cb : P.off_cr));
    const int tp = c ? IC_CP : IC_LP;
    const int x0 = rx << log2c, y0 = ry << log2c;
    if (log2c >= 4) {
        // rows 0 .. cs - 1, then the row above over two CTUs (a 16-byte piece that starts
        // inside the picture ends inside the row's pitch, a multiple of 64)
        const int per_row = log2c - 4, own = cs << per_row;
#pragma unroll 1
        for (int e = tid; e < own + (2 << per_row); e += THREADS) {
            const int r = e < own ? e >> per_row : -1, q = e < own ? e & ((1 << per_row) - 1) : e - own;
            const int y = y0 + r, x = x0 + 16 * q;
            if (y >= 0 && y < ph && x < pw) cp_async16(origin + r * tp + 16 * q, plane + (int64_t)y * pitch + x);
        }
    } else {  // 8-sample chroma CTBs (16x16 CTUs): words
#pragma unroll 1
        for (int e = tid; e < 8 * 2 + 4; e += THREADS) {
            const int r = e < 16 ? e >> 1 : -1, q = e < 16 ? e & 1 : e - 16;
            const int y = y0 + r, x = x0 + 4 * q;
            if (y >= 0 && y < ph && x < pw) cp_async4(origin + r * tp + 4 * q, plane + (int64_t)y * pitch + x);
        }
    }
    // the corner and the column to the left, as the words that end there
    if (rx > 0 && tid <= cs) {
        const int y = y0 + tid - 1;
        if (y >= 0 && y < ph) cp_async4(origin + (tid - 1) * tp - 4, plane + (int64_t)y * pitch + x0 - 4);
    }
}

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

// Lane 0's claim of the next work item, one instruction with no branch around it; the other
// lanes get 0.
__device__ __forceinline__ uint32_t claim_item(int* next, int lane) {
    uint32_t v;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %2, 0;\n\tmov.u32 %0, 0;\n\t@p atom.shared.add.u32 %0, [%1], 1;\n\t}"
        : "=&r"(v)
        : "r"((uint32_t)__cvta_generic_to_shared(next)), "r"(lane)
        : "memory");
    return v;
}

// Border words of one CTU in the picture's edge buffer, ctb of them per CTU in raster order:
// the bottom row's words (Y, Cb, Cr), then the right column's.  A word holds 4 samples and
// the epoch of the launch that wrote them, stored and read whole: a reader that finds its
// epoch has the samples too, with no fence on either side and no second read.
__device__ __forceinline__ int edge_word(int ctb, int c, bool column, int i) {
    return (column ? ctb >> 1 : 0) + (c == 0 ? 0 : (c == 1 ? ctb >> 2 : (ctb >> 2) + (ctb >> 3))) + i;
}

// Offset of the CTU's origin in each plane's tile (IntraSmem: luma, Cb, Cr tiles one after
// the other).
__device__ __forceinline__ int tile_origin(int c) {
    return c == 0 ? IC_LP + IC_MARGIN : IC_LH * IC_LP + (c - 1) * (IC_CH * IC_CP) + IC_CP + IC_MARGIN;
}

// ---------------------------------------------------------------------------------------
// The plan of a CTU's tasks, one CTA per CTU: which samples each TU can and does read, for
// how many TUs it waits, and for each TU and watched TU ("source") the TUs that wait for it.
// It follows from the records alone, so it is a launch of its own before the samples are
// needed: inside k_intra_ctus it took 5,500 to 16,000 of a CTU's cycles and its code pushed
// the TU paths out of the instruction caches (no_instruction 5.5 of 11 stall cycles per
// instruction; 0.7 of 6 now).
//   itu_task[item]    the work items
//   watch_plan[...]   per watched TU: its waiting TUs as in IntraTask::source, and its border words
//   rev[...]          task indices counted from the CTU's first, at dep_first
//   ictu_edge[...]    per border word the watch slot whose sample it awaits, or 0xFF
// ---------------------------------------------------------------------------------------
constexpr int AV_WAITS_SHIFT = 16;           // s_av: avail_pack; bits 16-21 the arrivals the TU waits for
constexpr uint32_t AV_UNMET = 1u << 22;      // a planted test wait: an arrival that never comes
constexpr int AV_NEED_SHIFT = 23;            // bits 23-27 the parts of its reference array it reads
constexpr int AV_BANDS_SHIFT = 28;           // bits 28-30 its bands
constexpr int IP_THREADS = 128;

__global__ void __launch_bounds__(IP_THREADS) k_intra_plan(const __grid_constant__ SegTable st, int32_t* tickets,
                                                             int later, uint32_t* sticky) {
    __shared__ uint32_t s_av[IC_MAX_TUS], s_count[IC_SOURCES], s_fill[IC_SOURCES], s_total, s_bad;
    __shared__ __align__(4) uint8_t s_edge[IC_EDGES];
    const int tid = threadIdx.x, lane = tid % 32;
    pdl_next();   // MC and the residuals' transforms need nothing of the plan
    if (later) pdl_wait();   // the tickets are in use by the group before
    if (blockIdx.x == 0 && tid < st.n) tickets[tid] = 0;
    const int k = find_seg(st, blockIdx.x);
    const PicDesc& P = *st.s[k].pic;
    const int idx = blockIdx.x - st.s[k].block0;
    const IntraCtu C = static_cast<const IntraCtu*>(st.s[k].items)[idx];
    const int n_tu = min(C.n_tu, IC_MAX_TUS), n_watch = min(C.n_watch, IC_MAX_WATCH);
    auto source = [&](int q) { return q < n_tu ? q : IC_MAX_TUS + q - n_tu; };   // the CTU's TUs, then those it watches
#pragma unroll 1
    for (int q = tid; q < n_tu + n_watch; q += IP_THREADS) s_count[source(q)] = 0;
    if (tid < IC_EDGES / 4) reinterpret_cast<uint32_t*>(s_edge)[tid] = 0xFFFFFFFFu;
    if (tid == 0) {
        s_total = 0;
        s_bad = C.n_tu > IC_MAX_TUS || C.n_watch > IC_MAX_WATCH || C.n_dep > IC_DEP_STAGE || C.n_item > IC_MAX_TUS;
    }
#pragma unroll 1
    for (int i = tid; i < n_tu; i += IP_THREADS) {
        const hevc_tu_t t = P.itu_rec[C.tu_first + i];
        const uint32_t dd = P.itu_dep[C.tu_first + i], at = dd >> 6;
        const int c = t.c_idx != 0;
        const IntraAvail av =
            intra_avail(t.x, t.y, 1 << t.log2_size, P.width >> c, P.height >> c, P.log2_ctb - c, 1 + c, C.nb);
        const bool smooth = intra_smoothed(t.intra_mode, t.log2_size, c, P.intra_smoothing_disabled != 0);
        const uint32_t need =
            intra_need(intra_parts(t.intra_mode, t.log2_size, c, (t.flags & HEVC_TU_PCM) != 0, smooth), avail_segs(av));
        // a list outside the CTU's entries is a planted one
        const bool planted = (dd & 63u) && (at < C.dep_first || at >= C.dep_first + (uint32_t)C.n_dep) &&
                             (P.dep_list[at] & INTRA_DEP_EXTERNAL);
        s_av[i] = avail_pack(av) | (planted ? AV_UNMET : 0u) | (need << AV_NEED_SHIFT) |
                  ((uint32_t)intra_bands(t.log2_size) << AV_BANDS_SHIFT);
    }
    __syncthreads();
    // the entries whose TU wrote something the waiting TU's mode reads.  Refused: an entry that
    // names no earlier TU and no watch slot, or no task of the CTU
    auto read = [&](int q, int& i, int& s) {
        const uint32_t e = __ldg(&P.dep_list[C.dep_first + q]);
        s = (int)(e & INTRA_DEP_SOURCE);
        i = (int)((e >> INTRA_DEP_TASK_SHIFT) & INTRA_DEP_SOURCE);
        if (i >= n_tu || s >= (s < IC_MAX_TUS ? i : IC_MAX_TUS + n_watch)) {
            s_bad = 1;
            return false;
        }
        return ((e >> INTRA_DEP_SEG_SHIFT) & (s_av[i] >> AV_NEED_SHIFT) & SEG_ALL) != 0;
    };
#pragma unroll 1
    for (int q = tid; q < C.n_dep; q += IP_THREADS) {
        int i, s;
        if (read(q, i, s)) {
            atomicAdd(&s_count[s], 1u);
            atomicAdd(&s_av[i], (s < IC_MAX_TUS ? s_av[s] >> AV_BANDS_SHIFT : 1u) << AV_WAITS_SHIFT);   // one per band
        }
    }
    __syncthreads();
    // room in rev for each source's waiting TUs (sources in any order: a warp takes its
    // sources' room at once), and the border words the watched TUs stand for
#pragma unroll 1
    for (int q = tid; q - lane < n_tu + n_watch; q += IP_THREADS) {
        const bool live = q < n_tu + n_watch;
        const int s = source(live ? q : 0);
        const uint32_t count = live ? s_count[s] : 0u;
        uint32_t end = count;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, end, d);
            if (lane >= d) end += v;
        }
        uint32_t first = 0;
        if (lane == 31 && end) first = atomicAdd(&s_total, end);
        first = __shfl_sync(0xffffffffu, first, 31) + end - count;
        if (!live) continue;
        s_fill[s] = first;
        s_count[s] = (first << 16) | count;
        const int j = s - IC_MAX_TUS;
        if (j >= 0) {
            const IntraWatch w = intra_watch_unpack(P.watch[C.watch_first + j]);
            const int cw = (1 << (P.log2_ctb - (w.c ? 1 : 0))) / 4;   // words across the CTU
            uint8_t* const edge = s_edge + (w.c == 0 ? 0 : IC_EDGE_L + (w.c - 1) * IC_EDGE_C);
            const int left0 = 1 + 2 * (w.c ? 8 : 16);
            uint32_t n = 0;
#pragma unroll 1
            for (int u = 0; u < w.n4 && count; u++) {
                if (w.y4 + w.n4 == 0 && w.x4 + u >= -1 && w.x4 + u < 2 * cw) {
                    edge[1 + w.x4 + u] = (uint8_t)j;
                    n++;
                }
                if (w.x4 + w.n4 == 0 && w.y4 + u >= 0 && w.y4 + u < cw) {
                    edge[left0 + w.y4 + u] = (uint8_t)j;
                    n++;
                }
            }
            P.watch_plan[C.watch_first + j] = make_uint2((first << 16) | count, n);
            if (count && n == 0) s_bad = 1;   // not beside this CTU: refused
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int q = tid; q < C.n_dep; q += IP_THREADS) {
        int i, s;
        if (read(q, i, s)) P.rev[C.dep_first + atomicAdd(&s_fill[s], 1u)] = (uint16_t)i;
    }
#pragma unroll 1
    for (int q = tid; q < C.n_item; q += IP_THREADS) {
        const int item = P.itu_item[C.item_first + q], i = item & (int)INTRA_DEP_SOURCE, band = item >> INTRA_DEP_TASK_SHIFT;
        const hevc_tu_t t = P.itu_rec[C.tu_first + i];
        const int c = t.c_idx, sub = c ? 1 : 0, n = 1 << t.log2_size, cs = 1 << (P.log2_ctb - sub);
        const int x = t.x & (cs - 1), y = t.y & (cs - 1), tp = c ? IC_CP : IC_LP, pitch = c ? P.pitch_c : P.pitch_y;
        const IntraAvail a = avail_unpack(s_av[i], n);
        const bool coded = t.flags & HEVC_TU_CODED, publish = t.reserved[0] & ITU_PUBLISH, pcm = t.flags & HEVC_TU_PCM;
        const bool none = avail_segs(a) == 0u;
        const int waits = (int)(s_av[i] >> AV_WAITS_SHIFT & 63u) + (s_av[i] & AV_UNMET ? 1 : 0), ctb = 1 << P.log2_ctb;
        IntraTask k;
        k.pic = (uint32_t)((c == 0 ? 0 : (c == 1 ? P.off_cb : P.off_cr)) + (int64_t)t.y * pitch + t.x);
        k.source = s_count[i];
        k.tile = (uint16_t)(tile_origin(c) + y * tp + x);
        k.res = coded ? (uint16_t)t.coeff_offset : (uint16_t)IC_MAX_RES;
        k.first = (int16_t)(none ? IC_TILES - k.tile : ref_offset(0, tp, n, intra_substitute(a, 0)));
        k.corner = (int16_t)(none ? IC_TILES - k.tile : ref_offset(0, tp, n, intra_substitute(a, 2 * n)));
        k.mode = pcm ? (uint8_t)MODE_PCM : t.intra_mode;
        const bool smooth = !pcm && intra_smoothed(t.intra_mode, t.log2_size, c != 0, P.intra_smoothing_disabled != 0);
        k.flags = (uint8_t)((c ? TASK_CHROMA : 0) | (coded ? TASK_CODED : 0) | (smooth ? TASK_SMOOTH : 0) |
                            (a.l ? TASK_LEFT : 0) | (a.t ? TASK_TOP : 0) | (waits ? 0 : TASK_STARTED));
        k.log2 = t.log2_size;
        k.y0 = (uint8_t)(band * IC_BAND);
        k.angle = pcm ? 0 : c_intra.angle[t.intra_mode];
        k.inv_angle = pcm ? 0 : c_intra.inv[t.intra_mode];
        k.waits = (uint8_t)plan_max(waits, 1);
        k.bl = (uint8_t)a.bl;
        k.tr = (uint8_t)a.tr;
        k.row = publish && y + n == cs ? (uint8_t)edge_word(ctb, c, false, x / 4) : TASK_NO_EDGE;
        k.column = publish && x + n == cs ? (uint8_t)edge_word(ctb, c, true, y / 4) : TASK_NO_EDGE;
        k.bar = (uint16_t)i;
        k.pad = 0;
        P.itu_task[C.item_first + q] = k;
    }
    if (tid < IC_EDGES / 4)
        reinterpret_cast<uint32_t*>(P.ictu_edge)[idx * (IC_EDGES / 4) + tid] = reinterpret_cast<const uint32_t*>(s_edge)[tid];
    if (tid == 0 && s_bad) atomicOr(sticky, ST_BAD_RECORD);   // k_intra_ctus then does nothing
    pdl_wait();
}

// ---------------------------------------------------------------------------------------
// The CTU tasks themselves.
// ---------------------------------------------------------------------------------------
// A CTA's shared memory (dynamic: more than 48 KB).
struct IntraSmem {
    alignas(16) uint8_t tiles[IC_TILES + 16];   // and the constant 128, for TUs with no reference sample
    alignas(16) IntraTask task[IC_MAX_TUS];     // the CTU's part of PicDesc::itu_task
    alignas(16) int16_t res[IC_MAX_RES + 16];   // and the residual of 4x4 TUs without one
    alignas(16) uint8_t edge[IC_EDGES];     // PicDesc::ictu_edge
    alignas(16) uint16_t rev[IC_DEP_STAGE + 2];   // the CTU's part of PicDesc::rev
    uint64_t bar[IC_MAX_TUS];               // what each TU waits for
    uint2 watch[IC_MAX_WATCH];              // PicDesc::watch_plan, y counted down as border words come
    IntraWarpSmem ws[IC_FULL - 1];
    int ticket, pic_index, next;
    volatile int abort;
};
static_assert(IC_LH * IC_LP % 16 == 0 && IC_CH * IC_CP % 16 == 0, "the tiles' rows lie on 16-byte boundaries");

// CTAs per SM that the register budget is sized for.  Four narrow ones take the register file whole:
// a batch of 16 1080p P/B pictures alone 393 us instead of 398, but on two lanes, whose kernels
// share the SMs, 38,000 frames/s instead of 42,400.
constexpr int ic_ctas(int warps) { return warps == IC_NARROW ? 3 : 32 / warps; }

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, ic_ctas(WARPS)) k_intra_ctus(const __grid_constant__ SegTable st,
                                                                                 int32_t* tickets, int total,
                                                                                 uint32_t* sticky) {
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr int THREADS = 32 * WARPS;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    IntraSmem& S = *reinterpret_cast<IntraSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    pdl_next();
    pdl_wait();
    if (tid == 0) {
        // Each picture hands out its CTUs by ticket in wavefront order.  CTAs start at picture
        // blockIdx.x % n, so the pictures of a launch progress side by side; a picture whose
        // tickets are used up passes the CTA on.  There are as many CTAs as CTUs, so every
        // CTA finds one.
        int k = blockIdx.x % st.n, got = -1;
        for (int tries = 0; tries < st.n && got < 0; tries++) {
            const int n_k = (k + 1 < st.n ? st.s[k + 1].block0 : total) - st.s[k].block0;
            const int v = atomicAdd(&tickets[k], 1);
            if (v < n_k) got = v;
            else k = k + 1 == st.n ? 0 : k + 1;
        }
        S.ticket = got;
        S.pic_index = k;
        S.next = 0;
    }
    if (tid == 32) {
        // a wait of this launch (or an earlier one not yet read) gave up, or the plan was
        // refused: the CTU could only wait for work that will not come, so the CTA ends at once
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> status(*sticky);
        S.abort = status.load(cuda::memory_order_relaxed) != 0;
    }
    __syncthreads();
    if (S.ticket < 0 || S.abort) {
        cp_async_wait_all();
        return;
    }
    const int k = S.pic_index;
    const PicDesc& P = *st.s[k].pic;
    const int32_t epoch = st.s[k].epoch;
    // the CTU's record: the same 16-byte loads by every thread, and no chain of loads after it
    const int4* const cp = reinterpret_cast<const int4*>(static_cast<const IntraCtu*>(st.s[k].items) + S.ticket);
    const int4 c0 = __ldg(cp), c1 = __ldg(cp + 1), c2 = __ldg(cp + 2);
    const int a = c0.x, n_dep = min(c0.w, IC_DEP_STAGE), n_watch = min(c1.z, IC_MAX_WATCH);
    const int n_res = min(c2.y, IC_MAX_RES), n_item = min(c2.w, IC_MAX_TUS);
    const int rx = a % P.wctb, ry = a / P.wctb, ctbl = 1 << P.log2_ctb;

    // Everything the CTU's tasks read, in one round of asynchronous copies: its tiles,
    // residuals and plan.
#pragma unroll 1
    for (int q = tid; q < 2 * n_item; q += THREADS)
        cp_async16(reinterpret_cast<uint4*>(S.task) + q, reinterpret_cast<const uint4*>(P.itu_task + c2.z) + q);
#pragma unroll 1
    for (int q = tid; q < 2 * n_watch; q += THREADS)
        cp_async4(reinterpret_cast<uint32_t*>(S.watch) + q, reinterpret_cast<const uint32_t*>(P.watch_plan + c1.y) + q);
    const int odd = c1.x & 1;   // rev goes in words
#pragma unroll 1
    for (int q = tid; q < (n_dep + odd + 1) / 2; q += THREADS)
        cp_async4(S.rev + 2 * q, P.rev + c1.x - odd + 2 * q);
    if (tid < IC_EDGES / 16) cp_async16(S.edge + 16 * tid, P.ictu_edge + S.ticket * IC_EDGES + 16 * tid);
#pragma unroll 1
    for (int q = tid; q < n_res / 8; q += THREADS) cp_async16(S.res + 8 * q, P.resid + c2.x + 8 * q);
#pragma unroll 1
    for (int c = 0; c < 3; c++) stage_tile<THREADS>(P, c, rx, ry, S.tiles + tile_origin(c), tid);
    uint8_t* const rec = P.rec;
    const int pitch_y = P.pitch_y, pitch_c = P.pitch_c, strong_intra = P.strong_intra;
    uint64_t* const edge = P.edge;
    cp_async_wait_all();
    __syncthreads();
#pragma unroll 1
    for (int q = tid; q < n_item; q += THREADS) {
        const IntraTask& k = S.task[q];
        if (k.y0 == 0) {
            mbar_init(&S.bar[k.bar], k.waits);
            if (k.flags & TASK_STARTED) mbar_arrive(&S.bar[k.bar]);
        }
    }
    if (tid < 16) S.res[IC_MAX_RES + tid] = 0;
    if (tid == 32) S.tiles[IC_TILES] = 128;
    __syncthreads();

    // TU or watched TU s is complete: arrive at the TUs that wait for it, the first'th and every
    // step'th after it
    auto complete = [&](uint32_t source, int first, int step) {
#pragma unroll 1
        for (int q = first; q < (int)(source & 0xFFFFu); q += step) mbar_arrive(&S.bar[S.rev[odd + (source >> 16) + q]]);
    };
    if (warp == WARPS - 1) {
        // The watcher: each lane follows up to 4 border words that TUs of other CTUs write and
        // some TU here reads, all of them polled at once through L2 (the wait is bounded like
        // every other).  A word that has come goes into the tile's border; with its last one
        // a watched TU is complete.  The warp barrier and the release arrivals order the
        // border's samples before every read of a TU that waits.
        constexpr int R = IC_EDGES / 32;
        const uint64_t* word[R];
        uint8_t* to[R];       // where its 4 samples go
        int step[R], slot[R]; // 1 along a row; the tile's pitch down the column
        uint32_t pend = 0;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int l = lane + 32 * r;
            slot[r] = S.edge[l];
            const bool live = slot[r] < n_watch;
            pend |= live ? 1u << r : 0u;
            const int c = l < IC_EDGE_L ? 0 : (l < IC_EDGE_L + IC_EDGE_C ? 1 : 2);
            const int i = l - (c == 0 ? 0 : IC_EDGE_L + (c - 1) * IC_EDGE_C), left0 = 1 + 2 * (c ? 8 : 16);
            const int cw = (c ? ctbl / 2 : ctbl) / 4, tp = c ? IC_CP : IC_LP;
            const bool column = i >= left0;
            const int x4 = i - 1, y4 = i - left0;
            const int from = column ? a - 1 : a - P.wctb + (x4 < 0 ? -1 : (x4 < cw ? 0 : 1));
            const int at = column ? y4 : (x4 < 0 ? cw - 1 : (x4 < cw ? x4 : x4 - cw));
            word[r] = edge + (live ? (int64_t)from * ctbl + edge_word(ctbl, c, column, at) : 0);
            to[r] = S.tiles + tile_origin(c) + (column ? 4 * y4 * tp - 1 : 4 * x4 - tp);
            step[r] = column ? tp : 1;
        }
        unsigned long long t0 = 0;
        for (unsigned polls = 0; __any_sync(FULL, pend != 0u); polls++) {
            uint64_t v[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                cuda::atomic_ref<const uint64_t, cuda::thread_scope_device> w(*word[r]);
                v[r] = pend >> r & 1u ? w.load(cuda::memory_order_relaxed) : 0;
            }
            uint32_t seen = 0;
#pragma unroll
            for (int r = 0; r < R; r++)
                if ((pend >> r & 1u) && (int32_t)(v[r] >> 32) == epoch) {
                    seen |= 1u << r;
                    for (int b = 0; b < 4; b++) to[r][b * step[r]] = (uint8_t)(v[r] >> (8 * b));
                }
            pend &= ~seen;
            if (__any_sync(FULL, seen != 0u)) {
                __syncwarp();
#pragma unroll
                for (int r = 0; r < R; r++)
                    if ((seen >> r & 1u) && atomicSub(&S.watch[slot[r]].y, 1u) == 1u)
                        complete(S.watch[slot[r]].x, 0, 1);
                t0 = 0;
                polls = 0;
                continue;
            }
            cuda::atomic_ref<uint32_t, cuda::thread_scope_device> status(*sticky);
            const bool stop = !wait_goes_on(t0, polls, sticky, &S.abort) ||
                              (status.load(cuda::memory_order_relaxed) & ST_TIMEOUT);
            if (__any_sync(FULL, stop)) {
                S.abort = 1;
                break;
            }
            __nanosleep(20);
        }
        return;
    }
    // Waits until all TUs that the TU of barrier `bar` waits for are complete; every lane acquires.
    auto wait = [&](uint64_t* bar) {
        unsigned long long t0 = 0;
#pragma unroll 1
        for (unsigned polls = 0;; polls++) {
            // the lanes may see the barrier, the abort word or the clock at different moments
            const bool over = mbar_try_wait0(bar);
            if (__all_sync(FULL, over)) return true;
            if (!__all_sync(FULL, over || wait_goes_on(t0, polls, sticky, &S.abort))) {
                S.abort = 1;
                return false;
            }
        }
    };
    // Border words of rows y0 .. y0 + rows - 1 of a TU along the CTU's bottom and right.
    auto publish = [&](const IntraTask& task, const uint8_t* t, int pitch, int y0, int rows, int n) {
        uint64_t* const words = edge + (int64_t)a * ctbl + lane;
        const uint64_t tag = (uint64_t)(uint32_t)epoch << 32;
        if (task.row != TASK_NO_EDGE && y0 + rows == n && lane < n / 4) {
            cuda::atomic_ref<uint64_t, cuda::thread_scope_device> w(words[task.row]);
            w.store(tag | *reinterpret_cast<const uint32_t*>(t + (n - 1) * pitch + 4 * lane), cuda::memory_order_relaxed);
        }
        if (task.column != TASK_NO_EDGE && lane < rows / 4) {
            const uint8_t* const col = t + (y0 + 4 * lane) * pitch + n - 1;
            cuda::atomic_ref<uint64_t, cuda::thread_scope_device> w(words[task.column + y0 / 4]);
            w.store(tag | (uint32_t)col[0] | (uint32_t)col[pitch] << 8 | (uint32_t)col[2 * pitch] << 16 |
                        (uint32_t)col[3 * pitch] << 24,
                    cuda::memory_order_relaxed);
        }
    };
    uint32_t claim = claim_item(&S.next, lane);
#pragma unroll 1
    for (;;) {
        const int item = (int)__shfl_sync(FULL, claim, 0);
        if (item >= n_item) break;
        // ---- before the wait: all that positions and the mode tell
        const IntraTask task = S.task[item];
        const bool chroma = task.flags & TASK_CHROMA;
        const int pitch = chroma ? IC_CP : IC_LP, ppitch = chroma ? pitch_c : pitch_y;
        uint8_t* const t = S.tiles + task.tile;   // the TU in its tile
        const int count = (int)(task.source & 0xFFFFu);
        // the first of the TUs that wait for this one, by lane
        int next = lane < count ? S.rev[odd + (task.source >> 16) + lane] : -1;
        if (task.log2 == 2) {
            // 4x4 (most TUs, and most of a picture's dependency chain): one output sample per
            // lane (the upper half of the warp repeats the lower), weighed from four samples of
            // the tile (IntraTaps); lane k finds where index k of the reference array lies.
            // No branch but DC's between the wait and the completion: one cost a lone warp
            // some 25 cycles.
            const uint2 taps = __ldg(reinterpret_cast<const uint2*>(c_intra_taps.t) + (task.mode * 2 + (chroma ? 1 : 0)) * 16 + (lane & 15));
            const int w = task_where(task, 4, pitch, plan_min(lane, 16));
            IntraTaps k = intra_taps_unpack(taps.x, taps.y);
            int at[4];
#pragma unroll
            for (int j = 0; j < 4; j++) at[j] = __shfl_sync(FULL, w, k.i[j]);
            int r = S.res[task.res + (lane & 15)];
            const int x = lane & 3, y = (lane >> 2) & 3;
            uint8_t* const to = t + y * pitch + x;
            uint8_t* const pic = rec + (task.pic + (uint32_t)(y * ppitch + x));
            // (keeps the compiler from moving this work behind the wait)
#pragma unroll
            for (int j = 0; j < 4; j++) asm volatile("" : "+r"(at[j]), "+r"(k.w[j]));
            asm volatile("" : "+r"(k.add), "+r"(k.shift), "+r"(r), "+r"(next));
            if (!wait(&S.bar[task.bar])) break;
            claim = claim_item(&S.next, lane);   // the warp's next item: its latency hides here
            int v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = t[at[j]];
            if (task.mode == 1) v[1] = (int)(__reduce_add_sync(FULL, lane < 8 ? v[1] : 0) + 4) >> 3;   // predict_dc :295-317
            const int p = clip_u8((v[0] * k.w[0] + v[1] * k.w[1] + v[2] * k.w[2] + v[3] * k.w[3] + k.add) >> k.shift);
            const uint8_t out = (uint8_t)clip_u8(p + r);
            if (lane < 16) *to = out;
            // complete: after the warp barrier, each lane's release arrival orders the warp's
            // samples in the tile before it
            __syncwarp();
            if (next >= 0) mbar_arrive(&S.bar[next]);
            if (lane < 16) *pic = out;
            if ((task.row & task.column) != TASK_NO_EDGE) publish(task, t, pitch, 0, 4, 4);
            if (count > 32) complete(task.source, 32 + lane, 32);
            continue;
        }
        // 8x8 and up.  Unsmoothed 8x8: two output samples per lane, (x, y) and (x, y + 4), in the
        // same way.  Others: at[0] and at[1] samples lane and lane + 32 of the reference array
        // in main order (mirrored for the horizontal modes), at[2] the last.
        const int log2 = task.log2, n = 1 << log2, rows = plan_min(n, IC_BAND), y0 = task.y0;
        const bool coded = task.flags & TASK_CODED, direct = log2 == 3 && !(task.flags & TASK_SMOOTH);
        const int16_t* const res = S.res + (coded ? task.res : 0);
        int at[4], at_b[4], r_a = 0, r_b = 0;
        IntraTaps ka, kb;
        if (direct) {
            const int x = lane & 7, y = lane >> 3;
            const int w = task_where(task, 8, pitch, lane), w32 = task_where(task, 8, pitch, 32);
            const int mode = plan_min(task.mode, 34);
            ka = intra_taps(3, mode, chroma, x, y, lane, task.angle, task.inv_angle);
            kb = intra_taps(3, mode, chroma, x, y + 4, lane, task.angle, task.inv_angle);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int a32 = __shfl_sync(FULL, w, ka.i[j] & 31), b32 = __shfl_sync(FULL, w, kb.i[j] & 31);
                at[j] = ka.i[j] == 32 ? w32 : a32;
                at_b[j] = kb.i[j] == 32 ? w32 : b32;
                if (task.mode == MODE_PCM) ka.w[j] = kb.w[j] = 0;
                asm volatile("" : "+r"(at[j]), "+r"(at_b[j]), "+r"(ka.w[j]), "+r"(kb.w[j]));
            }
            if (task.mode == MODE_PCM) ka.add = kb.add = 0;
            if (coded) {
                r_a = res[lane];
                r_b = res[lane + 32];
            }
        } else {
            const bool vert = task.mode >= 18 || task.mode < 2;
            at[0] = task_where(task, n, pitch, vert ? lane : 4 * n - lane);
            at[1] = task_where(task, n, pitch, vert ? lane + 32 : 4 * n - lane - 32);
            at[2] = task_where(task, n, pitch, vert ? 4 * n : 0);
        }
        if (!wait(&S.bar[task.bar])) break;
        claim = claim_item(&S.next, lane);
        if (direct) {
            auto weigh = [&](const int (&v)[4], const IntraTaps& k, int r) {
                return (uint8_t)clip_u8(
                    clip_u8((v[0] * k.w[0] + v[1] * k.w[1] + v[2] * k.w[2] + v[3] * k.w[3] + k.add) >> k.shift) + r);
            };
            int v[4], u[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                v[j] = t[at[j]];
                u[j] = t[at_b[j]];
            }
            if (task.mode == 1) v[1] = u[1] = (int)(__reduce_add_sync(FULL, lane < 16 ? v[1] : 0) + 8) >> 4;
            uint8_t* const to = t + (lane >> 3) * pitch + (lane & 7);
            to[0] = weigh(v, ka, r_a);
            to[4 * pitch] = weigh(u, kb, r_b);
        } else {
            intra_predict(task, strong_intra, lane, S.ws[warp].ref, at[0], at[1], at[2], t, pitch, y0, rows, res, coded);
        }
        __syncwarp();
        if (next >= 0) mbar_arrive(&S.bar[next]);
        if (count > 32) complete(task.source, 32 + lane, 32);
        if ((task.row & task.column) != TASK_NO_EDGE) publish(task, t, pitch, y0, rows, n);
        // then the picture gets the band, off the chain
#pragma unroll 1
        for (int e = lane; e < rows * n / 4; e += 32) {
            const int r = y0 + (e >> (log2 - 2)), c = 4 * (e & (n / 4 - 1));
            *reinterpret_cast<uint32_t*>(rec + task.pic + r * ppitch + c) =
                *reinterpret_cast<const uint32_t*>(t + r * pitch + c);
        }
    }
}

}  // namespace hevcgpu
