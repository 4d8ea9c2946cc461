// Visible value bins of a view (empty-space skipping).
#pragma once

#include "cache.cuh"

namespace gc {

// A sample whose value lies in bin b reads transfer-function entries within
// [floor(b/64 w - 1/2) - 1, floor((b+1)/64 w - 1/2) + 2]; its opacity after the
// correction 1 - (1 - a)^k is below k a / (1 - a) <= 1.05 k a for a <= 0.04,
// so with a the largest alpha of those entries and k the largest exponent of
// the view's levels, a bin with 1.05 k a < 0.0009 never reaches the
// compositing threshold 0.001.  Two bins per lane; every lane gets the result.
// (Rounded operations throughout: the exact and the fast build agree.)
__device__ __forceinline__ unsigned long long visible_bins(const ViewParams &vp, uint32_t lane) {
    if (!vp.skip_empty) return ~0ull;
    float kmax = 0.f;
    for (uint32_t l = 0; l < vp.nlevels; ++l) kmax = fmaxf(kmax, vp.kexp[l]);
    const int w = static_cast<int>(vp.tfw);
    const float wf = static_cast<float>(w);
    unsigned long long mine = 0;
#pragma unroll
    for (uint32_t b = lane; b < kValueBins; b += 32) {
        const float lo = static_cast<float>(b) / kValueBins, hi = static_cast<float>(b + 1) / kValueBins;
        int i0 = static_cast<int>(floorf(__fadd_rn(__fmul_rn(lo, wf), -0.5f))) - 1;
        int i1 = static_cast<int>(floorf(__fadd_rn(__fmul_rn(hi, wf), -0.5f))) + 2;
        i0 = max(i0, 0);
        i1 = min(i1, w - 1);
        float amax = 0.f;
#pragma unroll 4
        for (int i = i0; i <= i1; ++i) amax = fmaxf(amax, __ldg(vp.tf + 4 * i + 3));
        const bool visible = !(amax <= 0.04f && __fmul_rn(__fmul_rn(1.05f, kmax), amax) < 0.0009f);
        if (visible) mine |= 1ull << b;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine |= __shfl_xor_sync(0xffffffffu, mine, o);
    return mine;
}

// Two 8-bit channels and a 2D transfer function of at most kTwoBinRows rows: rows[b]
// gets the bins of channel 1 that are visible with bin b of channel 0 (32 bins
// each, the install's), by a block of 256 threads for each b.  A sample with its
// channels in bins b and c reads table entries within the same margins on either
// axis; the bound is the one above.  (The skip: a 777x555 frame of 256^3 x 2 voxels
// 1.90 -> 1.62 ms.)
constexpr uint32_t kTwoBinRows = 64;  // table rows at most (more: nothing is skipped)
__device__ __forceinline__ void visible_row_of_two(const ViewParams &vp, uint32_t b, uint32_t *rows) {
    __shared__ float s_row[kTwoBinRows];  // the largest alpha of b's columns in every row of the table
    const uint32_t lane = threadIdx.x & 31u;
    const int w = static_cast<int>(vp.tfw), h = static_cast<int>(vp.tfh);
    auto first = [](uint32_t bin, int n) {
        return max(static_cast<int>(floorf(__fadd_rn(__fmul_rn(static_cast<float>(bin) / 32.0f, static_cast<float>(n)), -0.5f))) - 1, 0);
    };
    auto last = [](uint32_t bin, int n) {
        return min(static_cast<int>(floorf(__fadd_rn(__fmul_rn(static_cast<float>(bin + 1u) / 32.0f, static_cast<float>(n)), -0.5f))) + 2, n - 1);
    };
    const int i0 = first(b, w), i1 = last(b, w);
#pragma unroll 4
    for (int j = static_cast<int>(threadIdx.x >> 5); j < h; j += 8) {
        float a = 0.f;
        for (int i = i0 + static_cast<int>(lane); i <= i1; i += 32) a = fmaxf(a, __ldg(vp.tf + 4 * (j * w + i) + 3));
        // (not negative, so the order of the bits is the order of the values)
        const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(a));
        if (lane == 0) s_row[j] = __uint_as_float(m);
    }
    __syncthreads();
    if (threadIdx.x >= 32u) return;
    float kmax = 0.f, a = 0.f;
    for (uint32_t l = 0; l < vp.nlevels; ++l) kmax = fmaxf(kmax, vp.kexp[l]);
    const int j1 = last(lane, h);
    for (int j = first(lane, h); j <= j1; ++j) a = fmaxf(a, s_row[j]);
    const bool visible = !(a <= 0.04f && __fmul_rn(__fmul_rn(1.05f, kmax), a) < 0.0009f);
    const uint32_t seen = __ballot_sync(0xffffffffu, visible);
    if (lane == 0) rows[b] = seen;
}

}  // namespace gc
