// intra_levels.cuh — the intra stage of pictures whose records no bitstream that codes every
// block once has: intra TUs that cover samples of other intra TUs (a damaged stream that codes
// a block twice), or that are larger than their CTB.
//
// k_intra_ctus relies on neither happening: with every 4x4 unit written once, a CTU has at most
// IC_MAX_TUS work items and IC_DEP_STAGE dependencies, and a border word has one writer.  Here
// the host sorts a picture's TUs into levels by what decode order asks for (build_intra_levels):
// a TU comes after the writers of every sample it reads or covers and after the readers of every
// sample it covers.  Warps take the TUs (those of 16x16 and 32x32 in bands of 8 rows) level by
// level, and start one when all of the levels before have completed, which one counter per
// picture tells.  So nothing is sized by how often a block is coded.  Reference samples come from
// the picture, each with its own availability, since a TU may reach past its CTB.
//
// Bound by the levels, one after another: a counter's round trip through L2, reference samples
// from L2, one item's work and its release, 5 us a level (a 1080p I picture with a few blocks coded
// twice: 2,158 levels, 11 ms; 14.8 ms with TUs not in bands).  64 to 256 warps a picture make no
// difference to it; a P/B picture (87 levels) takes 0.86 ms with 64, 0.68 with 128, 0.61 with 256.
// Every wait is bounded as in intra.cuh.
#pragma once

#include "intra.cuh"

namespace hevcgpu {

constexpr int IL_WARPS = 8, IL_CTAS = 32;   // per picture

__global__ void __launch_bounds__(32 * IL_WARPS) k_intra_levels(const __grid_constant__ SegTable st, uint32_t* sticky) {
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr int R = 5;   // rounds of 32 that cover the 4n + 1 reference samples
    __shared__ uint8_t s_ref[IL_WARPS][4 * 32 + 4];
    const int lane = threadIdx.x % 32;
    uint8_t* const ref = s_ref[threadIdx.x / 32];
    pdl_next();
    pdl_wait();
    const Seg& sg = st.s[blockIdx.y];
    const PicDesc& P = *sg.pic;
    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> status(*sticky);
    cuda::atomic_ref<int32_t, cuda::thread_scope_device> done(P.level_state[IL_DONE]);
    for (;;) {
        int q = 0;
        if (lane == 0) q = atomicAdd(&P.level_state[0], 1);
        q = __shfl_sync(FULL, q, 0);
        if (q >= sg.n_items) return;
        const int2 task = P.level_task[q];
        const int tu = task.x & IL_TASK, y0 = (task.x >> IL_BAND_SHIFT) * IC_BAND;
        const hevc_tu_t t = P.itu_rec[tu];
        const int16_t* const res = t.flags & HEVC_TU_CODED ? P.resid + P.itu_res[tu].y : nullptr;
        const int chroma = t.c_idx != 0, log2 = t.log2_size, n = 1 << log2, total = 4 * n + 1;
        const int pitch = chroma ? P.pitch_c : P.pitch_y, pw = P.width >> chroma, ph = P.height >> chroma;
        const int log2c = P.log2_ctb - chroma, m = (1 << log2c) - 1, rx = t.x >> log2c, ry = t.y >> log2c;
        uint8_t* const plane = P.rec + (t.c_idx == 0 ? 0 : (t.c_idx == 1 ? P.off_cb : P.off_cr));
        const uint32_t z = zorder16((uint32_t)((t.x & m) << chroma) >> 2, (uint32_t)((t.y & m) << chroma) >> 2);
        // availability (intra_prediction.cpp:102-133) of sample i of the reference array, counted
        // up the left column, over the corner and along the row above: this CTB's by z-scan
        // address, and those of the CTBs left, above-left, above and above-right that share its
        // slice and tile
        auto place = [&](int i, int& x, int& y) {
            x = i <= 2 * n ? t.x - 1 : t.x + i - 2 * n - 1;
            y = i < 2 * n ? t.y + 2 * n - 1 - i : t.y - 1;
        };
        auto usable = [&](int i) {
            int x, y;
            place(i, x, y);
            if (i >= total || x < 0 || y < 0 || x >= pw || y >= ph) return false;
            const int dx = (x >> log2c) - rx, dy = (y >> log2c) - ry;
            if (dx == 0 && dy == 0)
                return zorder16((uint32_t)((x & m) << chroma) >> 2, (uint32_t)((y & m) << chroma) >> 2) < z;
            if (!(dy == 0 ? dx == -1 : dy == -1 && dx >= -1 && dx <= 1)) return false;
            const int a = ry * P.wctb + rx, b = a + dy * P.wctb + dx;
            return (!P.ctb_slice || P.ctb_slice[a] == P.ctb_slice[b]) && (!P.ctb_tile || P.ctb_tile[a] == P.ctb_tile[b]);
        };
        uint32_t mask[R];
        int first = -1;
#pragma unroll
        for (int r = 0; r < R; r++) {
            mask[r] = __ballot_sync(FULL, usable(lane + 32 * r));
            if (first < 0 && mask[r]) first = 32 * r + __ffs(mask[r]) - 1;
        }
        // the sample that stands at each index (:177-197): the nearest available one below, else
        // the first available one
        int at[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            int k = -1;
#pragma unroll
            for (int w = r; w >= 0; w--) {
                const uint32_t below = w == r ? mask[w] & ((2u << lane) - 1u) : mask[w];
                if (k < 0 && below) k = 32 * w + 31 - __clz(below);
            }
            int x, y;
            place(k < 0 ? first : k, x, y);
            at[r] = y * pitch + x;
        }
        int go = 1;
        if (lane == 0) {
            unsigned long long t0 = 0;
            for (unsigned polls = 0; done.load(cuda::memory_order_relaxed) < task.y; polls++) {
                const unsigned long long now = global_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > WAIT_LIMIT_NS || polls >= SPIN_LIMIT) atomicOr(sticky, ST_TIMEOUT);
                if (status.load(cuda::memory_order_relaxed) & ST_TIMEOUT) {
                    go = 0;
                    break;
                }
                __nanosleep(20);
            }
            cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
        }
        if (!__shfl_sync(FULL, go, 0)) return;   // (and orders lane 0's acquire before every lane's loads)
        __syncwarp();
        int v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] = 128;
            if (lane + 32 * r >= total) continue;
            if (first >= 0) v[r] = __ldcg(plane + at[r]);
            ref[lane + 32 * r] = (uint8_t)v[r];
        }
        __syncwarp();
        // smoothing (:217-257, :443-471)
        const int mode = t.intra_mode;
        if (intra_smoothed(mode, log2, chroma != 0, P.intra_smoothing_disabled != 0)) {
            const int c = ref[2 * n], e0 = ref[0], e1 = ref[4 * n];
            const bool strong = log2 == 5 && P.strong_intra && abs(c + e1 - 2 * ref[3 * n]) < 8 &&
                                abs(c + e0 - 2 * ref[n]) < 8;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int i = lane + 32 * r, d = abs(i - 2 * n);
                if (i == 0 || i >= 4 * n) continue;
                v[r] = strong ? ((64 - d) * c + d * (i > 64 ? e1 : e0) + 32) >> 6
                              : (ref[i - 1] + 2 * v[r] + ref[i + 1] + 2) >> 2;
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < R; r++)
                if (lane + 32 * r < total) ref[lane + 32 * r] = (uint8_t)v[r];
            __syncwarp();
        }
        // prediction (:263-422) plus residual, clipped
        const int dc = ((int)__reduce_add_sync(FULL, lane < n ? ref[2 * n + 1 + lane] + ref[2 * n - 1 - lane] : 0) + n) >>
                       (log2 + 1);
        const int ang = c_intra.angle[mode], inv = c_intra.inv[mode];
        const bool vert = mode >= 18, edge = !chroma && log2 < 5, pcm = t.flags & HEVC_TU_PCM;
#pragma unroll 1
        for (int e = y0 * n + lane; e < min(n, y0 + IC_BAND) * n; e += 32) {
            const int x = e & (n - 1), y = e >> log2, left = ref[2 * n - 1 - y], top = ref[2 * n + 1 + x];
            int p = dc;
            if (mode == 0) {
                p = ((n - 1 - x) * left + (x + 1) * ref[3 * n + 1] + (n - 1 - y) * top + (y + 1) * ref[n - 1] + n) >>
                    (log2 + 1);
            } else if (mode == 1) {
                if (edge && y == 0) p = x == 0 ? (top + left + 2 * dc + 2) >> 2 : (top + 3 * dc + 2) >> 2;
                else if (edge && x == 0) p = (left + 3 * dc + 2) >> 2;
            } else {
                const int along = vert ? y : x, k = (vert ? x : y) + 1 + (((along + 1) * ang) >> 5);
                const int fr = ((along + 1) * ang) & 31;
                p = ((32 - fr) * ref[intra_main_index(vert, inv, n, k)] + fr * ref[intra_main_index(vert, inv, n, k + 1)] + 16) >> 5;
                if (edge && mode == 26 && x == 0) p = clip_u8(p + ((left - ref[2 * n]) >> 1));
                if (edge && mode == 10 && y == 0) p = clip_u8(p + ((top - ref[2 * n]) >> 1));
            }
            plane[(int64_t)(t.y + y) * pitch + t.x + x] = (uint8_t)clip_u8((pcm ? 0 : p) + (res ? res[e] : 0));
        }
        // complete: the warp's samples, then the release
        __syncwarp();
        if (lane == 0) done.fetch_add(1, cuda::memory_order_release);
    }
}

}  // namespace hevcgpu
