// Smallest and largest voxel value over 16-byte chunks of bricks, kept in packed
// form: two 16-bit lanes per word (8-bit voxels as even and odd bytes), so that a
// chunk of 8- or 16-bit voxels costs one instruction per word and bound.
#pragma once

#include <cstdint>

namespace gc {

__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Values of EB bytes each (1, 2: unsigned integers; 4: floats, NaNs ignored).
template <int EB>
struct ValueRange {
    uint32_t mn0 = 0xffffffffu, mx0 = 0u;
    uint32_t mn1 = 0xffffffffu, mx1 = 0u;  // EB 1: the odd bytes
    __device__ __forceinline__ void add(uint32_t w) {
        if constexpr (EB == 1) {
            const uint32_t e = w & 0x00ff00ffu, o = (w >> 8) & 0x00ff00ffu;
            mn0 = min_u16x2(mn0, e);
            mx0 = max_u16x2(mx0, e);
            mn1 = min_u16x2(mn1, o);
            mx1 = max_u16x2(mx1, o);
        } else {
            mn0 = min_u16x2(mn0, w);
            mx0 = max_u16x2(mx0, w);
        }
    }
    __device__ __forceinline__ void add(uint4 c) {
        add(c.x);
        add(c.y);
        add(c.z);
        add(c.w);
    }
    __device__ __forceinline__ uint32_t lowest() const {
        const uint32_t m = EB == 1 ? min_u16x2(mn0, mn1) : mn0;
        return min(m & 0xffffu, m >> 16);
    }
    __device__ __forceinline__ uint32_t highest() const {
        const uint32_t m = EB == 1 ? max_u16x2(mx0, mx1) : mx0;
        return max(m & 0xffffu, m >> 16);
    }
    // EB 1, two interleaved 8-bit channels (even and odd bytes): the bounds of
    // channel 0 in the low 16 bits, of channel 1 in the high ones
    __device__ __forceinline__ uint32_t mn_channels() const {
        return min(mn0 & 0xffffu, mn0 >> 16) | min(mn1 & 0xffffu, mn1 >> 16) << 16;
    }
    __device__ __forceinline__ uint32_t mx_channels() const {
        return max(mx0 & 0xffffu, mx0 >> 16) | max(mx1 & 0xffffu, mx1 >> 16) << 16;
    }
    // as the ray caster's samplers normalize them (monotone, so the range of the
    // normalized values)
    __device__ __forceinline__ void normalized(float &lo, float &hi) const {
        const float s = EB == 1 ? 1.0f / 255.0f : 1.0f / 65535.0f;
        lo = static_cast<float>(lowest()) * s;
        hi = static_cast<float>(highest()) * s;
    }
};
template <>
struct ValueRange<4> {
    float lo_ = 3.4e38f, hi_ = -3.4e38f;
    __device__ __forceinline__ void add(uint32_t w) {
        lo_ = fminf(lo_, __uint_as_float(w));
        hi_ = fmaxf(hi_, __uint_as_float(w));
    }
    __device__ __forceinline__ void add(uint4 c) {
        add(c.x);
        add(c.y);
        add(c.z);
        add(c.w);
    }
    __device__ __forceinline__ void normalized(float &lo, float &hi) const {
        lo = lo_;
        hi = hi_;
    }
};

}  // namespace gc
