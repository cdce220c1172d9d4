// device_common.cuh — device-side picture descriptors, tables and helpers shared by the
// reconstruction kernels.
#pragma once

#include <cstdint>

#include "hevcgpu.h"

namespace hevcgpu {

// ---------------------------------------------------------------------------------------
// Per-picture descriptor.  Kernels take an array of these and work items that carry the
// index of their picture, so one launch can serve one picture (plain form) or many
// pictures of many streams (batched form).  All three planes of a picture buffer live in
// one allocation: Cb at y + off_cb, Cr at y + off_cr, with row pitches pitch_y / pitch_c.
// ---------------------------------------------------------------------------------------
struct MotionEnt {           // 4x4 motion grid entry (PUMotionInfo, inter_prediction.h:16)
    int16_t mv[2][2];
    int8_t  ref[2];          // refIdxLX, -1 when predFlagLX is 0
    int16_t pad;
};
static_assert(sizeof(MotionEnt) == 12, "MotionEnt is written as three words by the MC kernel");

// Intra schedule entries.  Each intra TU in task order has a dependency list: an entry names
// a TU of the same CTU by its task index counted from the CTU's first, or, with
// INTRA_DEP_WATCH, a slot of the CTU's watch list, the TUs of earlier CTUs it waits for.
// (INTRA_DEP_EXTERNAL: a planted test wait.)  A TU that some other CTU depends on carries
// ITU_PUBLISH in reserved[0] of its task-order record and writes its samples along the CTU's
// bottom and right into the picture's edge buffer.
constexpr uint32_t INTRA_DEP_EXTERNAL = 0x80000000u;
constexpr uint32_t INTRA_DEP_WATCH = 0x40000000u;   // | watch slot of the CTU: the form handed out
// The form uploaded: bits 0-8 the source (task index, or IC_MAX_TUS + watch slot), bits 9-17
// the task that depends on it, bits 24-28 the parts of that task's reference array that hold
// samples of the source (SEG_*, intra_plan.h): the task does not wait for sources of which
// its mode reads no part.
constexpr uint32_t INTRA_DEP_SOURCE = 0x1FFu;
constexpr int INTRA_DEP_TASK_SHIFT = 9;
constexpr int INTRA_DEP_SEG_SHIFT = 24;
constexpr uint8_t ITU_PUBLISH = 1u;
// A 16x16 or 32x32 TU is done in bands of 8 rows, each by a warp of its own (1,310 and 2,340
// cycles a band): one warp took 1,770 and 4,200 cycles for the whole TU, a good part of a
// CTU's chain.
constexpr int IC_BAND = 8;
__host__ __device__ constexpr int intra_bands(int log2) { return log2 > 3 ? (1 << log2) / IC_BAND : 1; }

constexpr int IL_BAND_SHIFT = 24, IL_TASK = (1 << IL_BAND_SHIFT) - 1;   // of PicDesc::level_task
constexpr int IL_DONE = 64, IL_STATE = IL_DONE + 1;   // words of PicDesc::level_state: taken (0), complete (in another line)

// An intra CTU: its raster address, its TUs in the task order arrays, its entries in the
// dependency lists and the watch list, its residuals in the residual buffer, its work items,
// and which neighbour CTUs its TUs may read (NB_*).  Three 16-byte loads.
struct IntraCtu {
    int32_t addr, tu_first, n_tu, n_dep;
    uint32_t dep_first, watch_first;
    int32_t n_watch;
    uint32_t nb;
    int32_t res_first, n_res, item_first, n_item;
};
static_assert(sizeof(IntraCtu) == 48, "IntraCtu is read as three 16-byte words");

// Geometry of a watched TU, in units of 4 samples counted from the watching CTU's origin in
// the TU's plane.
struct IntraWatch {
    int c, n4, x4, y4;
};
__host__ __device__ __forceinline__ uint32_t intra_watch_pack(const IntraWatch& w) {
    return (uint32_t)w.c | (uint32_t)w.n4 << 2 | (uint32_t)(w.x4 + 128) << 8 | (uint32_t)(w.y4 + 128) << 16;
}
__host__ __device__ __forceinline__ IntraWatch intra_watch_unpack(uint32_t v) {
    return IntraWatch{(int)(v & 3u), (int)(v >> 2 & 15u), (int)(v >> 8 & 255u) - 128, (int)(v >> 16 & 255u) - 128};
}

struct IntraTask;   // intra.cuh

struct PicDesc {
    int32_t width, height;               // luma
    int32_t pitch_y, pitch_c;
    int64_t off_cb, off_cr;
    uint8_t* rec;                        // reconstruction / deblocking buffer
    uint8_t* dst;                        // packed output of independent blocks (RES_PACKED)
    const uint8_t* ref[2][16];           // reference pictures by list entry (Y base)
    int32_t num_ref[2];
    int32_t ref_poc[2][16];
    const hevc_tu_t* tus;
    const int16_t* coeffs;
    int16_t* resid;                      // residuals of coded intra TUs, CTU by CTU in task order
    const hevc_pu_t* pus;
    const hevc_wp_t* wp;
    const uint32_t* blk;                 // (W/4)*(H/4)
    MotionEnt* mot;                      // (W/4)*(H/4), built on the device from pus
    const hevc_sao_t* sao;
    const uint8_t* ctb_slice;            // may be null
    const uint16_t* ctb_tile;            // may be null
    const hevc_slice_t* slices;
    const hevc_scaling_t* scaling;       // scaling lists, or null for flat scaling
    // intra CTU tasks (intra.cuh): the CTUs that hold intra TUs (IntraCtu, handed to the launch)
    // in wavefront order (key 2 * row + column), and their TUs ordered by depth in the picture's
    // dependency DAG (task order)
    const hevc_tu_t* itu_rec;            // TU records in task order; coeff_offset holds the
                                         // offset of the TU's residual in the CTU's, reserved[0]
                                         // ITU_PUBLISH
    const int2* itu_res;                 // per task entry of a coded TU: its levels' offset in
                                         // coeffs, its residual's offset in resid
    const uint32_t* itu_dep;             // per task entry: (offset in dep_list << 6) | count
    const uint32_t* dep_list;            // dependency entries
    const uint16_t* itu_item;            // work items of each CTU: task | band << INTRA_DEP_TASK_SHIFT
    const uint32_t* watch;               // TUs of other CTUs each CTU waits for (intra_watch_pack)
    // the plan k_intra_plan makes of them for k_intra_ctus
    IntraTask* itu_task;
    uint2* watch_plan;
    uint16_t* rev;
    uint8_t* ictu_edge;
    uint64_t* edge;                      // border words of every CTU, 1 << log2_ctb each
    // or, in a picture that k_intra_levels does: its work items in the order they are taken, task
    // index | band << IL_BAND_SHIFT, and the number of items in the levels before; items taken,
    // items complete
    const int2* level_task;
    int32_t* level_state;
    int32_t num_pus;
    int32_t num_slices;
    int32_t log2_ctb, wctb, hctb;
    int32_t sao_enabled;
    int32_t pcm_lf_disabled;
    int32_t strong_intra;
    int32_t intra_smoothing_disabled;
    int32_t cb_qp_offset, cr_qp_offset;
    int32_t tiles_check;                 // tiles enabled and no filtering across tiles
    int32_t slice_check;                 // more than one slice in the picture
    int32_t pcm_bypass_any;              // some CU is PCM or transquant-bypass
};

// Programmatic dependent launch.  The kernels of a batch follow each other on one stream, and
// each lets the next one start as soon as all its own CTAs have (pdl_next), so that the next
// one's launch and whatever it can do by itself fill this one's last wave.  pdl_wait returns
// when the kernel before has completed; every kernel calls it, at the latest before it ends,
// so a kernel that has passed it knows that all kernels before it are done.  The first kernel
// of a batch is launched without the attribute: it starts when everything before it is done,
// and pdl_wait returns at once.  One 416x240 P/B picture 93 -> 57 us, one 1080p 128 -> 95,
// 16 in a batch 503 -> 485.
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// 16-byte asynchronous global -> shared copy (through L2 only, so that samples other
// CTUs wrote are seen), and the wait for all of a thread's copies.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(gmem));
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Until at most N of the thread's groups of copies are under way.
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Work items ----------------------------------------------------------------------------
// Residual items are TU indices (int32), or RES_INTRA_ITEM | task index for intra TUs;
// motion-compensation items are packed strips (mc_item, mc.cuh).

// A launch covers up to MAX_SEGS pictures.  Segment k owns the blocks
// [block0, next block0) of an item-list launch, or blockIdx.y == k of a per-picture
// launch (whose items field is the picture the loop filter writes).  The table is a kernel
// parameter, so a batched launch needs no device-side bookkeeping.  (A graph that held one would
// replay the epoch of its intra launch, and take the border words of the launch before for new.)
constexpr int MAX_SEGS = 64;
struct Seg {
    const void* items;
    const PicDesc* pic;
    int32_t n_items;
    int32_t block0;
    int32_t epoch;   // of an intra launch
    int32_t pad;
};
struct SegTable {
    int32_t n;
    int32_t pad;
    Seg s[MAX_SEGS];
};

__device__ __forceinline__ int find_seg(const SegTable& st, int b) {
    int k = 0;
    while (k + 1 < st.n && st.s[k + 1].block0 <= b) k++;
    return k;
}

constexpr uint32_t RES_INTRA_ITEM = 0x80000000u;

// Residual destinations.
enum ResMode : int32_t {
    RES_PACKED = 0,   // pred/out packed per TU at coeff_offset (config-1 form)
    RES_PICTURE = 1,  // inter TUs: add to rec; intra TUs: int16 residual into resid
};

// Device status word bits (written with atomicOr; read by the host after a sync).
enum : uint32_t {
    ST_BAD_RECORD = 1u,   // a record pointed outside its picture; the item was skipped
    ST_TIMEOUT = 2u,      // a bounded wait gave up; the kernel returned early
};

// Header of a flow area (the intra launches' state of a context or lane): 16 bytes kept
// free; the sticky status word (ST_* bits) follows it, then one CTU ticket counter per
// picture of a launch.
struct FlowState {
    int32_t reserved[4];
};

__device__ __forceinline__ int clip3(int lo, int hi, int v) { return v < lo ? lo : (v > hi ? hi : v); }
// v0..v3 saturated to 0..255 and packed as bytes 0..3 (PTX cvt.pack.sat: the low 16 bits
// of c move up by 16 and a, b take bits 15..8 and 7..0).
__device__ __forceinline__ uint32_t pack_sat_u8x4(int v0, int v1, int v2, int v3) {
    uint32_t t, d;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, 0;" : "=r"(t) : "r"(v3), "r"(v2));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(v1), "r"(v0), "r"(t));
    return d;
}
__device__ __forceinline__ int clip_u8(int v) { return v < 0 ? 0 : (v > 255 ? 255 : v); }

}  // namespace hevcgpu
