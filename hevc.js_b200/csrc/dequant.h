// dequant.h — dequantisation of a level (transform.cpp:360-365) in 32 bits.  Host and device
// code; no CUDA header is needed, so it is tested on the CPU.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define HEVC_HD_INLINE __host__ __device__ __forceinline__
#else
#define HEVC_HD_INLINE inline
#endif

namespace hevcgpu {

// The product with m * levelScale[qP % 6], the shift by qP / 6 and the rounding shift by
// s = 3 + log2 size, modulo 2^32 (an int16 clip follows).  With qP / 6 < s the two shifts are one
// rounding shift by the difference (the product has as many zeros at its end as the first put
// there, and |level * 255 * 72| stays below 2^30); else the second undoes a part of the first.
// Both forms: (level * (m * scale) + add) >> rs, where at high QPs the product wraps around:
// unsigned, since signed overflow is undefined.
struct Dequant {
    uint32_t scale, add;
    int rs;
};
HEVC_HD_INLINE Dequant dequant_make(int level_scale, int qp, int log2) {
    const int d = 3 + log2 - qp / 6;
    Dequant q;
    q.scale = (uint32_t)level_scale << (d < 0 ? -d : 0);
    q.rs = d > 0 ? d : 0;
    q.add = d > 0 ? 1u << (d - 1) : 0u;
    return q;
}
HEVC_HD_INLINE int dequant_level(int level, int m, const Dequant& q) {
    return (int)((uint32_t)level * ((uint32_t)m * q.scale) + q.add) >> q.rs;
}

}  // namespace hevcgpu
