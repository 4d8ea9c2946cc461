// Device side of tests/test_gpu_exact_math.py: the branch-free divisions of
// csrc/exact_math.cuh against the compiler's IEEE division, over every operand
// the ray caster can pass.  counts[i] = operands whose quotient differs.
#include <cuda_runtime.h>

#include "exact_math.cuh"

__device__ void tally(unsigned long long *count, float a, float b) {
    if (__float_as_uint(a) != __float_as_uint(b)) atomicAdd(count, 1ull);
}

template <uint32_t D>
__device__ void constant(unsigned long long *count, uint32_t i) {
    // every significand, at the exponents of the smallest and largest samples
    for (uint32_t e : {127u - 72u, 127u - 24u, 127u, 127u + 19u}) {
        const float x = __uint_as_float(e << 23 | i);
        tally(count, gc::div_exact<D>(x), __fdiv_rn(x, static_cast<float>(D)));
        tally(count, gc::div_exact<D>(-x), __fdiv_rn(-x, static_cast<float>(D)));
    }
    if (i <= 8u * 65535u)  // every sum of eight voxels
        tally(count, gc::div_exact<D>(static_cast<float>(i)), __fdiv_rn(static_cast<float>(i), static_cast<float>(D)));
}

__global__ void check(unsigned long long *counts) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 significands
    constant<255u>(counts + 0, i);
    constant<65535u>(counts + 1, i);
    constant<2040u>(counts + 2, i);
    constant<524280u>(counts + 3, i);
    // gc_log2's quotient (m - 1) / (m + 1) for every float m in [0.5, 2)
    for (uint32_t e : {126u, 127u}) {
        const float m = __uint_as_float(e << 23 | i);
        if (m >= 0.70710678f && m < 1.4142136f)
            tally(counts + 4, gc::div_near_two(m - 1.0f, m + 1.0f), __fdiv_rn(m - 1.0f, m + 1.0f));
    }
}

extern "C" int exact_math_check(unsigned long long *counts, void *stream) {
    check<<<(1u << 23) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(counts);
    return static_cast<int>(cudaGetLastError());
}
