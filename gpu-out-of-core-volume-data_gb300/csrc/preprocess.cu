// Preprocessor kernels: mip pyramid (2x2x2 box reduction), bricking with a
// covering border, and empty-brick flags.  Everything stays resident in HBM;
// the reference streams 512 MB chunks through cudaMalloc/H2D/kernel/D2H/free
// per chunk (GcCore/src/cuda/libPreprocessor/Mipmapper.cu:401-578) and bricks
// on the CPU with one seek+read per brick row
// (GcCore/src/libPreprocessor/Bricker_v2.cpp:79-252).
#include <algorithm>
#include <cstring>

#include "cache.cuh"
#include "gc_internal.h"
#include "value_range.cuh"

namespace gc {

// ---------------------------------------------------------------------------
// mip_reduce: one 2x2x2 pass.
//
// Reference arithmetic (down_sampling_inner, Mipmapper.cu:29-105):
//   8-bit channels : uint64 sum of the 8 inputs, integer division by 8;
//   16-bit, 1 ch.  : double sum (its initial value is uninitialised in the
//                    reference; zero here), / 8.0, truncating conversion;
//                    the sum of 8 u16 is exact so this is floor(sum / 8);
//   f32            : double sum in (z, y, x) loop order, / 8.0, rounded to float.
// The reference handles interleaved channels only on the 8-bit path; here every
// integer channel width uses the per-channel floor mean.
//
// Vector kernel: one thread per 16-byte chunk of each of the 4 input rows
// (y0,z0), (y1,z0), (y0,z1), (y1,z1); it writes the 8 output bytes that chunk
// reduces to.  Every input byte is read once, with 128-bit loads.
template <int CB, int NC>
__device__ inline void reduce_chunk(const uint4 (&r)[4], uint2 &out) {
    if constexpr (CB == 1) {
        const uint8_t *b0 = reinterpret_cast<const uint8_t *>(&r[0]);
        const uint8_t *b1 = reinterpret_cast<const uint8_t *>(&r[1]);
        const uint8_t *b2 = reinterpret_cast<const uint8_t *>(&r[2]);
        const uint8_t *b3 = reinterpret_cast<const uint8_t *>(&r[3]);
        uint8_t *o = reinterpret_cast<uint8_t *>(&out);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = j / NC, c = j % NC;
            const int a = (2 * i) * NC + c, b = (2 * i + 1) * NC + c;
            uint32_t s = b0[a] + b0[b] + b1[a] + b1[b] + b2[a] + b2[b] + b3[a] + b3[b];
            o[j] = static_cast<uint8_t>(s / 8u);
        }
    } else if constexpr (CB == 2) {
        const uint16_t *h0 = reinterpret_cast<const uint16_t *>(&r[0]);
        const uint16_t *h1 = reinterpret_cast<const uint16_t *>(&r[1]);
        const uint16_t *h2 = reinterpret_cast<const uint16_t *>(&r[2]);
        const uint16_t *h3 = reinterpret_cast<const uint16_t *>(&r[3]);
        uint16_t *o = reinterpret_cast<uint16_t *>(&out);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = j / NC, c = j % NC;
            const int a = (2 * i) * NC + c, b = (2 * i + 1) * NC + c;
            uint32_t s = h0[a] + h0[b] + h1[a] + h1[b] + h2[a] + h2[b] + h3[a] + h3[b];
            o[j] = static_cast<uint16_t>(s / 8u);
        }
    } else {
        const float *f0 = reinterpret_cast<const float *>(&r[0]);
        const float *f1 = reinterpret_cast<const float *>(&r[1]);
        const float *f2 = reinterpret_cast<const float *>(&r[2]);
        const float *f3 = reinterpret_cast<const float *>(&r[3]);
        float *o = reinterpret_cast<float *>(&out);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            double s = 0.0;
            s += f0[2 * i];
            s += f0[2 * i + 1];
            s += f1[2 * i];
            s += f1[2 * i + 1];
            s += f2[2 * i];
            s += f2[2 * i + 1];
            s += f3[2 * i];
            s += f3[2 * i + 1];
            o[i] = static_cast<float>(s / 8.0);
        }
    }
}

struct MipParams {
    uint32_t X, Y, Z;            // source dims
    uint32_t oX, oY, oZ;         // output dims
    uint64_t in_row, out_row;    // bytes per row
    uint32_t chunks;             // 16-byte chunks per input row that produce output
    uint64_t total;              // chunks * oY * oZ
};

template <int CB, int NC>
__global__ void __launch_bounds__(256) mip_vec_kernel(const uint8_t *__restrict__ src,
                                                      uint8_t *__restrict__ dst, MipParams p) {
    for (uint64_t t = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; t < p.total;
         t += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t chunk = static_cast<uint32_t>(t % p.chunks);
        const uint64_t orow = t / p.chunks;
        const uint32_t oy = static_cast<uint32_t>(orow % p.oY), oz = static_cast<uint32_t>(orow / p.oY);
        const uint64_t r00 = (static_cast<uint64_t>(2 * oz) * p.Y + 2 * oy) * p.in_row;
        const uint64_t plane = static_cast<uint64_t>(p.Y) * p.in_row;
        const uint64_t off = static_cast<uint64_t>(chunk) * 16;
        uint4 r[4];
        r[0] = __ldcs(reinterpret_cast<const uint4 *>(src + r00 + off));
        r[1] = __ldcs(reinterpret_cast<const uint4 *>(src + r00 + p.in_row + off));
        r[2] = __ldcs(reinterpret_cast<const uint4 *>(src + r00 + plane + off));
        r[3] = __ldcs(reinterpret_cast<const uint4 *>(src + r00 + plane + p.in_row + off));
        uint2 o;
        reduce_chunk<CB, NC>(r, o);
        *reinterpret_cast<uint2 *>(dst + (static_cast<uint64_t>(oz) * p.oY + oy) * p.out_row + chunk * 8) = o;
    }
}

// Bytes [s, s + 16) of the 32-byte pair (a, b) for a per-lane s in 0..15: a
// two-level select by whole words, then a funnel shift by the byte remainder.
__device__ __forceinline__ uint4 window16(uint4 a, uint4 b, uint32_t s) {
    const bool w2 = (s & 8u) != 0u, w1 = (s & 4u) != 0u;
    const uint32_t u0 = w2 ? a.z : a.x, u1 = w2 ? a.w : a.y, u2 = w2 ? b.x : a.z, u3 = w2 ? b.y : a.w,
                   u4 = w2 ? b.z : b.x, u5 = w2 ? b.w : b.y;
    const uint32_t v0 = w1 ? u1 : u0, v1 = w1 ? u2 : u1, v2 = w1 ? u3 : u2, v3 = w1 ? u4 : u3, v4 = w1 ? u5 : u4;
    const uint32_t r = (s & 3u) * 8u;
    return make_uint4(__funnelshift_r(v0, v1, r), __funnelshift_r(v1, v2, r), __funnelshift_r(v2, v3, r),
                      __funnelshift_r(v3, v4, r));
}

// Levels whose rows start anywhere (odd sizes, rows of no whole 16 bytes): as
// mip_vec_kernel, but a thread cuts its 16 bytes of each of the four rows out of
// two aligned 16-byte loads (the second mostly in L1) and stores its up to eight
// bytes as wide as their place allows.  A load that would pass the level's end is
// taken byte by byte.  381x347x291 u8 -> its second level: 34 us (a thread per
// value, eight byte loads) -> 19 us.
template <int CB, int NC>
__global__ void __launch_bounds__(256) mip_window_kernel(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst,
                                                         MipParams p) {
    constexpr uint32_t vb = CB * NC, per = 8u / vb;  // output voxels of a thread
    const uint64_t level = static_cast<uint64_t>(p.Z) * p.Y * p.in_row;
    for (uint64_t t = blockIdx.x * 256ull + threadIdx.x; t < p.total; t += gridDim.x * 256ull) {
        const uint32_t c = static_cast<uint32_t>(t % p.chunks);
        const uint64_t orow = t / p.chunks;
        const uint32_t oy = static_cast<uint32_t>(orow % p.oY), oz = static_cast<uint32_t>(orow / p.oY);
        const uint32_t n = min(per, p.oX - c * per) * vb;  // output bytes
        uint4 r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t a = ((2ull * oz + (k >> 1)) * p.Y + 2u * oy + (k & 1)) * p.in_row + 16ull * c;
            const uint32_t s = static_cast<uint32_t>(a) & 15u;
            const uint64_t lo = a - s;
            const bool two = s + 2u * n > 16u;
            if (lo + (two ? 32u : 16u) <= level) {
                const uint4 q0 = __ldg(reinterpret_cast<const uint4 *>(src + lo));
                r[k] = window16(q0, two ? __ldg(reinterpret_cast<const uint4 *>(src + lo + 16)) : q0, s);
            } else {
                uint32_t v[4] = {0u, 0u, 0u, 0u};
                for (uint32_t i = 0; i < 2u * n; ++i) v[i >> 2] |= static_cast<uint32_t>(src[a + i]) << (8u * (i & 3u));
                r[k] = make_uint4(v[0], v[1], v[2], v[3]);
            }
        }
        uint2 o;
        reduce_chunk<CB, NC>(r, o);
        uint8_t *d = dst + (static_cast<uint64_t>(oz) * p.oY + oy) * p.out_row + 8ull * c;
        const uint32_t at = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(d));
        if (n == 8u && (at & 7u) == 0u) {
            *reinterpret_cast<uint2 *>(d) = o;
        } else if (n == 8u && (at & 3u) == 0u) {
            reinterpret_cast<uint32_t *>(d)[0] = o.x;
            reinterpret_cast<uint32_t *>(d)[1] = o.y;
        } else if (vb >= 2u || (at & 1u) == 0u) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t h = ((i & 2u ? o.y : o.x) >> (16u * (i & 1u))) & 0xffffu;
                if (2u * i + 2u <= n)
                    reinterpret_cast<uint16_t *>(d)[i] = static_cast<uint16_t>(h);
                else if (2u * i < n)
                    d[2 * i] = static_cast<uint8_t>(h);
            }
        } else {
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i)
                if (i < n) d[i] = static_cast<uint8_t>((i & 4u ? o.y : o.x) >> (8u * (i & 3u)));
        }
    }
}

// Generic path (any width, odd sizes): one thread per output channel value.
__global__ void mip_scalar_kernel(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst,
                                  MipParams p, uint32_t cb, uint32_t nc) {
    const uint64_t n = static_cast<uint64_t>(p.oX) * p.oY * p.oZ * nc;
    for (uint64_t t = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; t < n;
         t += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t c = static_cast<uint32_t>(t % nc);
        const uint64_t v = t / nc;
        const uint32_t ox = static_cast<uint32_t>(v % p.oX);
        const uint64_t r = v / p.oX;
        const uint32_t oy = static_cast<uint32_t>(r % p.oY), oz = static_cast<uint32_t>(r / p.oY);
        const uint64_t eb = static_cast<uint64_t>(cb) * nc;
        uint64_t isum = 0;
        double dsum = 0.0;
        for (int dz = 0; dz < 2; ++dz)
            for (int dy = 0; dy < 2; ++dy)
                for (int dx = 0; dx < 2; ++dx) {
                    const uint64_t vox = (static_cast<uint64_t>(2 * oz + dz) * p.Y + (2 * oy + dy)) * p.X + (2 * ox + dx);
                    const uint8_t *ptr = src + vox * eb + c * cb;
                    if (cb == 1)
                        isum += *ptr;
                    else if (cb == 2)
                        isum += *reinterpret_cast<const uint16_t *>(ptr);
                    else
                        dsum += *reinterpret_cast<const float *>(ptr);
                }
        uint8_t *o = dst + ((static_cast<uint64_t>(oz) * p.oY + oy) * p.oX + ox) * eb + c * cb;
        if (cb == 1)
            *o = static_cast<uint8_t>(isum / 8u);
        else if (cb == 2)
            *reinterpret_cast<uint16_t *>(o) = static_cast<uint16_t>(isum / 8u);
        else
            *reinterpret_cast<float *>(o) = static_cast<float>(dsum / 8.0);
    }
}

static void launch_mip(const void *src, void *dst, const uint32_t d[3], uint32_t eb, uint32_t nc,
                       cudaStream_t s) {
    GC_REQUIRE(eb % nc == 0, "encoded bytes must be a multiple of channels");
    const uint32_t cb = eb / nc;
    GC_REQUIRE(cb == 1 || cb == 2 || cb == 4, "bytes per channel must be 1, 2 or 4");
    MipParams p;
    p.X = d[0];
    p.Y = d[1];
    p.Z = d[2];
    p.oX = d[0] / 2;
    p.oY = d[1] / 2;
    p.oZ = d[2] / 2;
    GC_REQUIRE(p.oX && p.oY && p.oZ, "level too small to down-sample");
    p.in_row = static_cast<uint64_t>(p.X) * eb;
    p.out_row = static_cast<uint64_t>(p.oX) * eb;
    const int grid = sm_count() * 8;
    const bool aligned = (reinterpret_cast<uintptr_t>(src) % 16 == 0) &&
                         (reinterpret_cast<uintptr_t>(dst) % 8 == 0) && (p.X % 2 == 0) &&
                         (p.in_row % 16 == 0);
    if (aligned) {
        p.chunks = static_cast<uint32_t>(p.in_row / 16);
        p.total = static_cast<uint64_t>(p.chunks) * p.oY * p.oZ;
        auto *in = static_cast<const uint8_t *>(src);
        auto *out = static_cast<uint8_t *>(dst);
        if (cb == 1 && nc == 1)
            mip_vec_kernel<1, 1><<<grid, 256, 0, s>>>(in, out, p);
        else if (cb == 1 && nc == 2)
            mip_vec_kernel<1, 2><<<grid, 256, 0, s>>>(in, out, p);
        else if (cb == 1 && nc == 4)
            mip_vec_kernel<1, 4><<<grid, 256, 0, s>>>(in, out, p);
        else if (cb == 2 && nc == 1)
            mip_vec_kernel<2, 1><<<grid, 256, 0, s>>>(in, out, p);
        else if (cb == 2 && nc == 2)
            mip_vec_kernel<2, 2><<<grid, 256, 0, s>>>(in, out, p);
        else if (cb == 4 && nc == 1)
            mip_vec_kernel<4, 1><<<grid, 256, 0, s>>>(in, out, p);
        else
            mip_scalar_kernel<<<grid, 256, 0, s>>>(in, out, p, cb, nc);
        GC_CUDA(cudaGetLastError());
        count_launch();
        return;
    }
    // windows of 16 bytes from a number of threads on, below which a thread per value
    // fills the SMs better.  Windows / a thread per value, at threads of eight bytes
    // out: u8 17k 6.1 / 4.2 us, 28k 6.0 / 4.3, 38k 6.1 / 6.2, 80k 6.3 / 8.2; u16 31k 5.4 /
    // 4.1, 41k 6.0 / 4.3, 49k 6.1 / 5.2, 54k 6.1 / 6.0, 158k 6.3 / 8.2; two 16-bit channels
    // 45k 5.6 / 4.3, 61k 5.6 / 6.2; two 8-bit channels, whose values are smaller and twice
    // as many, 17k 4.7 / 4.1, 23k 5.7 / 4.3, 32k 5.2 / 6.0, 72k 6.2 / 7.0; four 32k 4.6 /
    // 6.1.  Floats (a voxel is a load either way) a thread per value at every size: 500k
    // 41 / 39 us.
    p.chunks = static_cast<uint32_t>((p.out_row + 7) / 8);
    p.total = static_cast<uint64_t>(p.chunks) * p.oY * p.oZ;
    if (p.total >= (cb == 1 && nc > 1 ? 28672u : 53248u) && reinterpret_cast<uintptr_t>(src) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(dst) % eb == 0 &&
        ((cb == 1 && (nc == 1 || nc == 2 || nc == 4)) || (cb == 2 && nc <= 2))) {
        const auto go = [&](auto kernel) {
            kernel<<<static_cast<unsigned>(std::min<uint64_t>((p.total + 255) / 256, static_cast<uint64_t>(grid))), 256, 0,
                     s>>>(static_cast<const uint8_t *>(src), static_cast<uint8_t *>(dst), p);
        };
        if (cb == 1)
            nc == 1 ? go(mip_window_kernel<1, 1>) : nc == 2 ? go(mip_window_kernel<1, 2>) : go(mip_window_kernel<1, 4>);
        else
            nc == 1 ? go(mip_window_kernel<2, 1>) : go(mip_window_kernel<2, 2>);
    } else {
        mip_scalar_kernel<<<grid, 256, 0, s>>>(static_cast<const uint8_t *>(src),
                                                static_cast<uint8_t *>(dst), p, cb, nc);
    }
    GC_CUDA(cudaGetLastError());
    count_launch();
}

// One 2x2x2 pass over the four rows' W words each: W / 2 words out.  Integer
// widths sum pairs of values in packed halves or words; floats as reduce_chunk
// does.
template <int CB, int NC, int W>
__device__ __forceinline__ void reduce_rows(const uint32_t (&r)[4][W], uint32_t (&out)[W / 2]) {
    if constexpr (CB == 1 && NC <= 2) {
        uint32_t h[W];  // two result bytes of each word
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uint32_t e = 0, o = 0;  // sums of the even and the odd bytes, 16 bits each
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                e += r[k][w] & 0x00ff00ffu;
                o += (r[k][w] >> 8) & 0x00ff00ffu;
            }
            if constexpr (NC == 1) {
                const uint32_t s = e + o;  // voxel pairs: byte 0 + 1, byte 2 + 3
                h[w] = ((s & 0xffffu) >> 3) | ((s >> 19) << 8);
            } else {
                h[w] = (((e & 0xffffu) + (e >> 16)) >> 3) | ((((o & 0xffffu) + (o >> 16)) >> 3) << 8);
            }
        }
#pragma unroll
        for (int w = 0; w < W / 2; ++w) out[w] = h[2 * w] | (h[2 * w + 1] << 16);
    } else if constexpr (CB == 2 && NC == 1) {
        uint32_t h[W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uint32_t s = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) s += (r[k][w] & 0xffffu) + (r[k][w] >> 16);
            h[w] = s >> 3;
        }
#pragma unroll
        for (int w = 0; w < W / 2; ++w) out[w] = h[2 * w] | (h[2 * w + 1] << 16);
    } else {  // one voxel a word: words 2 w and 2 w + 1
        static_assert(CB * NC == 4, "voxels of 4 bytes");
#pragma unroll
        for (int w = 0; w < W / 2; ++w) {
            if constexpr (CB == 4) {
                double d = 0.0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    d += __uint_as_float(r[k][2 * w]);
                    d += __uint_as_float(r[k][2 * w + 1]);
                }
                out[w] = __float_as_uint(static_cast<float>(d / 8.0));
            } else if constexpr (CB == 2) {
                uint32_t lo = 0, hi = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    lo += (r[k][2 * w] & 0xffffu) + (r[k][2 * w + 1] & 0xffffu);
                    hi += (r[k][2 * w] >> 16) + (r[k][2 * w + 1] >> 16);
                }
                out[w] = (lo >> 3) | ((hi >> 3) << 16);
            } else {
                uint32_t e = 0, o = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    e += (r[k][2 * w] & 0x00ff00ffu) + (r[k][2 * w + 1] & 0x00ff00ffu);
                    o += ((r[k][2 * w] >> 8) & 0x00ff00ffu) + ((r[k][2 * w + 1] >> 8) & 0x00ff00ffu);
                }
                out[w] = ((e >> 3) & 0x00ff00ffu) | (((o >> 3) & 0x00ff00ffu) << 8);
            }
        }
    }
}

// Two levels in one pass: a thread reduces a 16-byte chunk of four rows of four
// slices to 8 bytes a row of the first level and 4 of the second, the second from
// the rounded values of the first.  Bound by HBM: the source is read once and the
// first level not at all (a pass a level: 1.29 instead of 1.17 times the source),
// and a small pyramid takes half the launches.  Lanes are neighbours along x, so
// that a warp reads 512 bytes of a row at a time, eight loads in flight a lane.
// A 1024^3 u16 pyramid 450 -> 363 us (6.8 TB/s), a 64^3 one 6.4 -> 5.2 us.  Three
// levels in one pass measured slower at every size (420 us; 7.3 us): 124 registers.
struct FusedMip {
    const uint8_t *src;
    uint8_t *dst[2];             // levels 1 and 2
    uint32_t Y;                  // source rows per slice
    uint32_t oY[2], oZ[2];       // of each level
    uint64_t row;                // source bytes per row; level l has row >> l
    uint32_t chunks, yb, zb;     // threads along x, y, z
};
template <int CB, int NC>
__global__ void __launch_bounds__(128) mip_fused_kernel(const FusedMip m) {
    const uint64_t t = blockIdx.x * 128ull + threadIdx.x;
    if (t >= static_cast<uint64_t>(m.chunks) * m.yb * m.zb) return;
    const uint32_t c = static_cast<uint32_t>(t % m.chunks), g = static_cast<uint32_t>(t / m.chunks);
    const uint32_t by = g % m.yb, bz = g / m.yb;
    const uint64_t plane = m.row * m.Y;
    uint32_t v[2][2][2];  // level 1: [slice][row] words
#pragma unroll
    for (uint32_t dz = 0; dz < 2; ++dz) {
        const uint32_t z1 = 2u * bz + dz;
        uint32_t r[2][4][4];
#pragma unroll
        for (uint32_t y = 0; y < 2; ++y) {
            const uint32_t y1 = 2u * by + y;
            if (z1 < m.oZ[0] && y1 < m.oY[0]) {
                const uint8_t *p = m.src + 2ull * z1 * plane + 2ull * y1 * m.row + 16ull * c;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 q = __ldcs(reinterpret_cast<const uint4 *>(p + (k & 1) * m.row + (k >> 1) * plane));
                    r[y][k][0] = q.x, r[y][k][1] = q.y, r[y][k][2] = q.z, r[y][k][3] = q.w;
                }
            }
        }
#pragma unroll
        for (uint32_t y = 0; y < 2; ++y) {
            const uint32_t y1 = 2u * by + y;
            if (z1 < m.oZ[0] && y1 < m.oY[0]) {
                reduce_rows<CB, NC, 4>(r[y], v[dz][y]);
                *reinterpret_cast<uint2 *>(m.dst[0] + (static_cast<uint64_t>(z1) * m.oY[0] + y1) * (m.row >> 1) +
                                           8ull * c) = make_uint2(v[dz][y][0], v[dz][y][1]);
            }
        }
    }
    if (bz < m.oZ[1] && by < m.oY[1]) {
        uint32_t q[4][2], o[1];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int w = 0; w < 2; ++w) q[k][w] = v[k >> 1][k & 1][w];
        reduce_rows<CB, NC, 2>(q, o);
        *reinterpret_cast<uint32_t *>(m.dst[1] + (static_cast<uint64_t>(bz) * m.oY[1] + by) * (m.row >> 2) + 4ull * c) = o[0];
    }
}

// The two levels after a level of dims d in one pass.  False where the pass does
// not apply: rows of no whole 16-byte chunks, levels off their chunks' grid, other
// voxel types, a level of no rows.
static bool launch_mip_fused(const uint8_t *src, uint8_t *const dst[2], const uint32_t d[3], uint32_t eb, uint32_t nc,
                             cudaStream_t s) {
    const uint32_t cb = eb / nc;
    const bool typed = (cb == 1 && (nc == 1 || nc == 2 || nc == 4)) || (cb == 2 && nc <= 2) || (cb == 4 && nc == 1);
    if (eb % nc || !typed || (static_cast<uint64_t>(d[0]) * eb) % 16 || reinterpret_cast<uintptr_t>(src) % 16 ||
        reinterpret_cast<uintptr_t>(dst[0]) % 8 || reinterpret_cast<uintptr_t>(dst[1]) % 4 || d[1] < 4 || d[2] < 4)
        return false;
    FusedMip m{};
    m.src = src;
    m.Y = d[1];
    m.row = static_cast<uint64_t>(d[0]) * eb;
    for (uint32_t l = 0; l < 2; ++l) {
        m.dst[l] = dst[l];
        m.oY[l] = d[1] >> (l + 1);
        m.oZ[l] = d[2] >> (l + 1);
    }
    m.chunks = static_cast<uint32_t>(m.row / 16);
    m.yb = (m.oY[0] + 1) / 2;
    m.zb = (m.oZ[0] + 1) / 2;
    const uint64_t blocks = (static_cast<uint64_t>(m.chunks) * m.yb * m.zb + 127) / 128;
    if (blocks >= (1ull << 31)) return false;
    auto go = [&](auto kernel) { kernel<<<static_cast<unsigned>(blocks), 128, 0, s>>>(m); };
    if (cb == 1)
        nc == 1 ? go(mip_fused_kernel<1, 1>) : nc == 2 ? go(mip_fused_kernel<1, 2>) : go(mip_fused_kernel<1, 4>);
    else if (cb == 2)
        nc == 1 ? go(mip_fused_kernel<2, 1>) : go(mip_fused_kernel<2, 2>);
    else
        go(mip_fused_kernel<4, 1>);
    GC_CUDA(cudaGetLastError());
    count_launch();
    return true;
}

// ---------------------------------------------------------------------------
// Bricking: small brick (bx, by, bz) of level dims D covers voxels
// [b * (B - 2c) - c, b * (B - 2c) - c + B) per axis; voxels outside the level
// are zero (Bricker_v2.cpp:145-200), and so is every small brick whose start
// b * (B - 2c) is outside the level on some axis.  Output layout: big bricks in (z, y, x)
// raster order, each (BB*B)^3 voxels x-fastest; small brick (i, j, k) of a big
// brick at voxel offset (i*B, j*B, k*B) (Bricker_v2.cpp:149-152, 295-299).

// One voxel of a small brick the slow way (bricks on the level's edge, odd
// voxel widths): zero outside the level or in an unvisited brick.
__device__ __forceinline__ void brick_voxel(const uint8_t *__restrict__ level, uint8_t *__restrict__ dptr,
                                            const BrickParams &p, bool visited, int64_t gx, int64_t gy, int64_t gz) {
    const bool inside = visited && gx >= 0 && gy >= 0 && gz >= 0 && gx < p.D[0] && gy < p.D[1] && gz < p.D[2];
    const uint8_t *sptr = level + ((static_cast<uint64_t>(gz) * p.D[1] + gy) * p.D[0] + gx) * p.eb;
    switch (p.eb) {
        case 1:
            *dptr = inside ? __ldg(sptr) : uint8_t(0);
            break;
        case 2:
            *reinterpret_cast<uint16_t *>(dptr) = inside ? __ldg(reinterpret_cast<const uint16_t *>(sptr)) : uint16_t(0);
            break;
        case 4:
            *reinterpret_cast<uint32_t *>(dptr) = inside ? __ldg(reinterpret_cast<const uint32_t *>(sptr)) : 0u;
            break;
        default:
            for (uint32_t b = 0; b < p.eb; ++b) dptr[b] = inside ? sptr[b] : 0;
    }
}

// 16 bytes of a source row starting at byte `s` (0..15) of the aligned pair (a, b).
__device__ __forceinline__ uint4 row_bytes16(uint4 a, uint4 b, uint32_t s) {
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const uint32_t r = (s & 3u) * 8u;
    uint32_t o[4];
    // s / 4 is the same for every thread of a brick: a uniform branch with
    // constant register indices in each arm
    switch (s >> 2) {
#define GC_ROW_CASE(Q)                                                                  \
    case Q:                                                                             \
        _Pragma("unroll") for (int k = 0; k < 4; ++k) o[k] = __funnelshift_r(w[Q + k], w[Q + k + 1], r); \
        break;
        GC_ROW_CASE(0)
        GC_ROW_CASE(1)
        GC_ROW_CASE(2)
        GC_ROW_CASE(3)
#undef GC_ROW_CASE
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// Copies small brick (sx, sy, sz) of a level into its place in a big brick
// (big_base; (ix, iy, iz) = its position among the big brick's BB bricks),
// with the 32 lanes of a warp.  p.fast (B a power of two, whole 16-byte
// chunks per row, rows 16 bytes apart in the level, 16-byte aligned buffers):
// the brick goes in 16-byte output chunks.  A chunk whose source row lies
// inside the level and whose voxels all lie inside the row -- all chunks of an
// interior brick -- starts at the same byte offset s modulo 16 as every other
// such chunk of the brick, so it is two aligned 16-byte loads and a funnel
// shift by s, stored with one 16-byte store.  A row outside the level, or an
// unvisited brick, stores zeros; a chunk straddling the level's x edge is
// assembled voxel by voxel.  Otherwise the brick is copied voxel by voxel.
__device__ __forceinline__ void copy_small_brick(const uint8_t *__restrict__ level, const BrickParams &p,
                                                 uint32_t sx, uint32_t sy, uint32_t sz, uint8_t *big_base,
                                                 uint32_t ix, uint32_t iy, uint32_t iz, uint32_t lane) {
    const uint32_t B = p.B;
    const uint32_t bvx = p.BB[0] * B, bvy = p.BB[1] * B;
    const int64_t ox = static_cast<int64_t>(sx) * p.Beff - p.c;
    const int64_t oy = static_cast<int64_t>(sy) * p.Beff - p.c;
    const int64_t oz = static_cast<int64_t>(sz) * p.Beff - p.c;
    // The reference visits a small brick only if its start lies inside the
    // level on every axis (Bricker_v2.cpp:203-221); the others stay zero even
    // where their covering border reaches into the volume.
    const bool visited = static_cast<uint64_t>(sx) * p.Beff < p.D[0] &&
                         static_cast<uint64_t>(sy) * p.Beff < p.D[1] && static_cast<uint64_t>(sz) * p.Beff < p.D[2];
    if (p.fast) {
        const uint32_t k = 16u / p.eb;                  // voxels per chunk
        const uint32_t nchunks = 1u << (2u * p.b_shift + p.cpr_shift);
        const uint64_t row_stride = static_cast<uint64_t>(p.D[0]) * p.eb;
        // byte offset modulo 16 of the brick's first voxel in any row (rows
        // are multiples of 16 bytes apart; ox may be negative)
        const uint32_t s = static_cast<uint32_t>(ox * static_cast<int64_t>(p.eb)) & 15u;
        uint8_t *obase = big_base + ((static_cast<uint64_t>(iz) * B * bvy + iy * B) * bvx + ix * B) * p.eb;
        const uint64_t drow = static_cast<uint64_t>(bvx) * p.eb;  // output row stride
        if (visited && ox >= 0 && oy >= 0 && oz >= 0 && ox + B <= p.D[0] && oy + B <= p.D[1] && oz + B <= p.D[2]) {
            // Interior brick (the common case, the same branch for the whole
            // warp): no per-chunk tests; each lane issues the loads of 4 chunks
            // before it stores them.  The second load of a pair ends at or
            // before the end of its row: the chunk's first voxel byte plus 16
            // lies inside the row, and rows end on 16-byte boundaries.
            const uint8_t *sbase = level + (static_cast<uint64_t>(oz) * p.D[1] + static_cast<uint64_t>(oy)) * row_stride +
                                   static_cast<uint64_t>(ox) * p.eb - s;
            const uint32_t cmask = (1u << p.cpr_shift) - 1u;
            for (uint32_t c0 = lane; c0 < nchunks; c0 += 128u) {
                uint4 a[4], b[4] = {};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t c = c0 + 32u * u;
                    if (c < nchunks) {
                        const uint32_t row = c >> p.cpr_shift;
                        const uint8_t *src = sbase + (static_cast<uint64_t>(row >> p.b_shift) * p.D[1] + (row & (B - 1u))) *
                                                         row_stride + (c & cmask) * 16u;
                        a[u] = __ldg(reinterpret_cast<const uint4 *>(src));
                        if (s) b[u] = __ldg(reinterpret_cast<const uint4 *>(src + 16));
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t c = c0 + 32u * u;
                    if (c < nchunks) {
                        const uint32_t row = c >> p.cpr_shift;
                        uint8_t *dst = obase + (static_cast<uint64_t>(row >> p.b_shift) * bvy + (row & (B - 1u))) * drow +
                                       (c & cmask) * 16u;
                        *reinterpret_cast<uint4 *>(dst) = s ? row_bytes16(a[u], b[u], s) : a[u];
                    }
                }
            }
            return;
        }
#pragma unroll 4
        for (uint32_t c = lane; c < nchunks; c += 32u) {
            const uint32_t cx = c & ((1u << p.cpr_shift) - 1u), row = c >> p.cpr_shift;
            const uint32_t ly = row & (B - 1u), lz = row >> p.b_shift;
            uint8_t *dst = obase + (static_cast<uint64_t>(lz) * bvy + ly) * drow + cx * 16u;
            const int64_t ry = oy + ly, rz = oz + lz, x0 = ox + static_cast<int64_t>(cx) * k;
            const bool row_in = visited && ry >= 0 && rz >= 0 && ry < p.D[1] && rz < p.D[2];
            if (!row_in) {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(0u, 0u, 0u, 0u);
            } else if (x0 >= 0 && x0 + k <= p.D[0]) {
                const uint64_t src = (static_cast<uint64_t>(rz) * p.D[1] + ry) * row_stride +
                                     static_cast<uint64_t>(x0) * p.eb - s;
                const uint4 a = __ldg(reinterpret_cast<const uint4 *>(level + src));
                *reinterpret_cast<uint4 *>(dst) =
                    s ? row_bytes16(a, __ldg(reinterpret_cast<const uint4 *>(level + src + 16)), s) : a;
            } else {
                for (uint32_t v = 0; v < k; ++v)
                    brick_voxel(level, dst + v * p.eb, p, true, x0 + v, ry, rz);
            }
        }
        return;
    }
    const uint32_t nvox = B * B * B;
    for (uint32_t v = lane; v < nvox; v += 32u) {
        const uint32_t lx = v % B, ly = (v / B) % B, lz = v / (B * B);
        uint8_t *dptr = big_base + ((static_cast<uint64_t>(iz * B + lz) * bvy + (iy * B + ly)) * bvx + (ix * B + lx)) * p.eb;
        brick_voxel(level, dptr, p, visited, ox + lx, oy + ly, oz + lz);
    }
}

// The bricker of one level: one warp per small brick (grid-stride over
// bricks); the per-brick index arithmetic is done once per warp and brick
// (16 chunks per lane for B16 u16), the per-chunk one with shifts.
__global__ void __launch_bounds__(256) brick_kernel(const uint8_t *__restrict__ level,
                                                    uint8_t *__restrict__ out, BrickParams p) {
    const uint64_t big_bytes = static_cast<uint64_t>(p.BB[0] * p.B) * (p.BB[1] * p.B) * (p.BB[2] * p.B) * p.eb;
    const uint32_t nsx = p.nbig[0] * p.BB[0], nsy = p.nbig[1] * p.BB[1];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t nsmall = static_cast<uint32_t>(p.nsmall);  // < 2^32 (checked on the host)
    for (uint32_t sb = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; sb < nsmall; sb += nwarps) {
        // small brick grid = nbig * BB per axis, x fastest
        const uint32_t sx = sb % nsx, rest = sb / nsx;
        const uint32_t sy = rest % nsy, sz = rest / nsy;
        const uint32_t gx = sx / p.BB[0], gy = sy / p.BB[1], gz = sz / p.BB[2];
        const uint64_t big = (static_cast<uint64_t>(gz) * p.nbig[1] + gy) * p.nbig[0] + gx;
        copy_small_brick(level, p, sx, sy, sz, out + big * big_bytes, sx - gx * p.BB[0], sy - gy * p.BB[1],
                         sz - gz * p.BB[2], lane);
    }
}

// Bytes [s, s + 8) of the 16-byte pair (a, b) for a per-lane s in 0..7.
__device__ __forceinline__ uint2 window8(uint2 a, uint2 b, uint32_t s) {
    const bool w1 = (s & 4u) != 0u;
    const uint32_t v0 = w1 ? a.y : a.x, v1 = w1 ? b.x : a.y, v2 = w1 ? b.y : b.x;
    const uint32_t r = (s & 3u) * 8u;
    return make_uint2(__funnelshift_r(v0, v1, r), __funnelshift_r(v1, v2, r));
}

// x / d for x, d < 2^16: a shift, or a multiply-high by ceil(2^32 / d).
struct SmallDiv {
    uint32_t m = 0, shift = 0;
    SmallDiv() = default;
    explicit SmallDiv(uint32_t d) {
        if ((d & (d - 1u)) == 0u)
            while ((1u << shift) < d) ++shift;
        else
            m = static_cast<uint32_t>(((1ull << 32) + d - 1u) / d);
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t x) const { return m ? __umulhi(x, m) : x >> shift; }
};

// One launch of the slab bricker.
struct SlabParams {
    BrickParams p;
    uint32_t nb;             // bricks of a slab, adjacent along x
    uint32_t ngx;            // slabs along x
    uint32_t zparts, zlen;   // blocks that share a slab's slices, and slices of each
    uint32_t cprow;          // 16-byte chunks copied of each source row
    uint32_t pitch;          // bytes between the rows of a slice in shared memory
    uint32_t stages;
    uint32_t cpr;            // output chunks per brick row
    uint64_t items;
    SmallDiv by_cprow, by_brick, by_cpr;  // / cprow, / (B cpr), / cpr
};

// A 16-byte asynchronous copy of n <= 16 source bytes, the rest zeros.
__device__ __forceinline__ void copy16_async(uint32_t dst, const uint8_t *src, uint32_t n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits until at most `left` (0 to 3) of this thread's newest copy groups are in flight.
__device__ __forceinline__ void copies_wait(uint32_t left) {
    if (left == 0)
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    else if (left == 1)
        asm volatile("cp.async.wait_group 1;" ::: "memory");
    else if (left == 2)
        asm volatile("cp.async.wait_group 2;" ::: "memory");
    else
        asm volatile("cp.async.wait_group 3;" ::: "memory");
}

// Slab bricker, for brick rows of whole CH-byte chunks (16, or 8 for 8-byte rows)
// and levels of any row length.  A block takes a slab of nb bricks adjacent along
// x and walks the slab's slices (one z of the level each): the B source rows of a
// slice come into shared memory as aligned 16-byte asynchronous copies, several
// slices ahead, and go out as whole brick rows -- consecutive lanes write
// consecutive chunks of one brick, each cut out of its row at any byte offset
// (rows of a level need not be multiples of 16 bytes apart: every row has its own
// offset in its first chunk).  Copies are cut at the end of the row (zeros follow,
// the bricker's value there), rows outside the level are zeros, bytes left of the
// row are masked on the way out, unvisited bricks are zeros.
//
// Bound by HBM: the level is read once (slab edges again from L2) and the bricks,
// (B / (B - 2c))^3 times its size, written once.  A slab is about 512 output
// chunks a slice, so that a row's copies are several hundred bytes; small levels
// share a slab's slices among blocks until the SMs are filled, because a block's
// slices follow one another.  768^3 u16, 16^3 bricks, level 0 (2.27 GB): 450 us with
// a warp per run of bricks straight from the level (32-byte pieces of 16 bricks a
// store) -> 347 us, 6.5 TB/s; its level of 8 bricks 51 -> 4.4 us; level 0 of a
// 381x347x291 u8 volume (rows of odd length) 310 us voxel by voxel -> 25 us.
template <int CH, uint32_t NT>
__global__ void __launch_bounds__(NT) brick_slab_kernel(const uint8_t *__restrict__ level, uint8_t *__restrict__ out,
                                                         const SlabParams sp) {
    extern __shared__ __align__(128) uint8_t slab_smem[];
    const BrickParams &p = sp.p;
    const uint32_t B = p.B, eb = p.eb, tid = threadIdx.x;
    const uint32_t nsx = p.nbig[0] * p.BB[0], nsy = p.nbig[1] * p.BB[1];
    const uint32_t bvx = p.BB[0] * B, bvy = p.BB[1] * B;
    const uint64_t big_bytes = static_cast<uint64_t>(bvx) * bvy * (p.BB[2] * B) * eb;
    const uint64_t drow = static_cast<uint64_t>(bvx) * eb;  // output row stride
    const int64_t row_bytes = static_cast<int64_t>(p.D[0]) * eb, plane = row_bytes * p.D[1];
    const uint32_t slice_bytes = B * sp.pitch, ncopy = B * sp.cprow;
    const uint32_t smem = static_cast<uint32_t>(__cvta_generic_to_shared(slab_smem));
    for (uint64_t item = blockIdx.x; item < sp.items; item += gridDim.x) {
        const uint32_t zp = static_cast<uint32_t>(item % sp.zparts);
        const uint64_t slab = item / sp.zparts;
        const uint32_t g = static_cast<uint32_t>(slab % sp.ngx);
        const uint32_t rest = static_cast<uint32_t>(slab / sp.ngx), sy = rest % nsy, sz = rest / nsy;
        const uint32_t sx0 = g * sp.nb, nbx = min(sp.nb, nsx - sx0);
        const bool yz_vis = static_cast<uint64_t>(sy) * p.Beff < p.D[1] && static_cast<uint64_t>(sz) * p.Beff < p.D[2];
        // the slab's first byte in any row (negative in the covering left of x = 0)
        const int64_t o0 = (static_cast<int64_t>(sx0) * p.Beff - p.c) * eb;
        const int64_t y0 = static_cast<int64_t>(sy) * p.Beff - p.c;
        const uint32_t lz0 = zp * sp.zlen, nz = min(sp.zlen, B - lz0);
        const int64_t z0 = static_cast<int64_t>(sz) * p.Beff - p.c + lz0;  // of the block's first slice
        const uint32_t nchunks = nbx * B * sp.cpr;
        const uint32_t gy = sy / p.BB[1], gz = sz / p.BB[2];
        uint8_t *const out0 = out + (static_cast<uint64_t>(gz) * p.nbig[1] + gy) * p.nbig[0] * big_bytes +
                              (static_cast<uint64_t>((sz - gz * p.BB[2]) * B + lz0) * bvy + (sy - gy * p.BB[1]) * B) * drow;

        // A thread's copies and chunks are the same in every slice up to the slice's
        // offset: the first kPre of each are worked out once per slab.
        struct Copy {
            int64_t rb;    // the row's first byte in the level, in the block's first slice
            uint32_t to;   // its place in a stage
            uint32_t q;    // chunk of the row
            bool in;       // the row lies inside the level's y range
        };
        auto copy_of = [&](uint32_t t) {
            Copy c;
            const uint32_t row = sp.by_cprow(t);
            const int64_t y = y0 + row;
            c.q = t - row * sp.cprow;
            c.to = row * sp.pitch + 16u * c.q;
            c.in = yz_vis && y >= 0 && y < p.D[1];
            c.rb = z0 * plane + y * row_bytes;
            return c;
        };
        auto copy_chunk = [&](const Copy &c, uint32_t i, uint32_t stage) {
            const int64_t z = z0 + i, rb = c.rb + plane * i;
            // inside the row from a chunk that reaches it on: the address is not negative
            // there (the level is 16-byte aligned), and the cut copy ends at the row's end
            int64_t a = ((rb + o0) & ~static_cast<int64_t>(15)) + 16 * static_cast<int64_t>(c.q);
            const bool some = c.in && z >= 0 && z < p.D[2] && a + 16 > rb && a < rb + row_bytes;
            const uint32_t n = some ? static_cast<uint32_t>(min(static_cast<int64_t>(16), rb + row_bytes - a)) : 0u;
            copy16_async(stage + c.to, level + (some ? a : 0), n);
        };
        struct Chunk {
            uint8_t *dst;     // in the block's first slice
            uint32_t s;       // the row's offset in its first chunk, in the block's first slice
            uint32_t row;     // the row's place in a stage
            uint32_t at;      // the chunk's bytes after the row's offset
            uint32_t zeros;   // leading zero bytes (the covering left of the row; all in an unvisited brick)
        };
        auto chunk_of = [&](uint32_t t) {
            Chunk c;
            const uint32_t j = sp.by_brick(t), r = t - j * (B * sp.cpr);
            const uint32_t ly = sp.by_cpr(r), k = r - ly * sp.cpr;
            const uint32_t sx = sx0 + j, gx = sx / p.BB[0];
            c.dst = out0 + gx * big_bytes + ly * drow + (sx - gx * p.BB[0]) * B * eb + k * CH;
            c.s = static_cast<uint32_t>(z0 * plane + (y0 + ly) * row_bytes + o0);
            c.row = ly * sp.pitch;
            c.at = j * p.Beff * eb + k * CH;
            c.zeros = 0;
            if (!yz_vis || static_cast<uint64_t>(sx) * p.Beff >= p.D[0])
                c.zeros = CH;
            else if (sx * p.Beff < p.c && k * CH < (p.c - sx * p.Beff) * eb)
                c.zeros = (p.c - sx * p.Beff) * eb - k * CH;
            return c;
        };
        // The chunk whose bytes start at byte `at` of the row `w`, to dst.
        auto put_bytes = [&](const uint8_t *row, uint32_t at, uint32_t zeros, uint8_t *dst) {
            const uint8_t *w = row + (at & ~static_cast<uint32_t>(CH - 1));
            uint32_t v[CH / 4];
            if constexpr (CH == 16) {
                const uint4 x = window16(reinterpret_cast<const uint4 *>(w)[0], reinterpret_cast<const uint4 *>(w)[1],
                                         at & 15u);
                v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
            } else {
                const uint2 x =
                    window8(reinterpret_cast<const uint2 *>(w)[0], reinterpret_cast<const uint2 *>(w)[1], at & 7u);
                v[0] = x.x, v[1] = x.y;
            }
            if (zeros) {
#pragma unroll
                for (uint32_t q = 0; q < CH / 4; ++q) {
                    const uint32_t z = zeros > 4u * q ? zeros - 4u * q : 0u;
                    v[q] = z >= 4u ? 0u : v[q] & (0xffffffffu << (8u * z));
                }
            }
            if constexpr (CH == 16)
                *reinterpret_cast<uint4 *>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
            else
                *reinterpret_cast<uint2 *>(dst) = make_uint2(v[0], v[1]);
        };
        const uint64_t dslice = static_cast<uint64_t>(bvy) * drow;  // output slice stride
        auto put_chunk = [&](const Chunk &c, uint32_t i, const uint8_t *stage) {
            put_bytes(stage + c.row, ((c.s + static_cast<uint32_t>(plane) * i) & 15u) + c.at, c.zeros, c.dst + i * dslice);
        };
        constexpr uint32_t kPre = 2;
        Copy cp[kPre];
        Chunk ck[kPre];
#pragma unroll
        for (uint32_t u = 0; u < kPre; ++u) {
            cp[u] = copy_of(min(tid + NT * u, ncopy - 1u));
            ck[u] = chunk_of(min(tid + NT * u, nchunks - 1u));
        }
        if ((plane & 15) == 0 && ncopy <= NT * kPre && nchunks <= NT * kPre) {
            // Planes whole 16-byte chunks apart: a row starts at the same byte of its
            // first chunk in every slice, so a thread's copies and chunks only advance
            // by a plane and an output slice.
            const uint8_t *src[kPre];
            uint32_t n[kPre];
#pragma unroll
            for (uint32_t u = 0; u < kPre; ++u) {
                const int64_t a = ((cp[u].rb + o0) & ~static_cast<int64_t>(15)) + 16 * static_cast<int64_t>(cp[u].q);
                const bool some = cp[u].in && a + 16 > cp[u].rb && a < cp[u].rb + row_bytes;
                n[u] = some ? static_cast<uint32_t>(min(static_cast<int64_t>(16), cp[u].rb + row_bytes - a)) : 0u;
                src[u] = level + a;  // read only in slices inside the level
                ck[u].at += ck[u].s & 15u;
            }
            uint32_t to_stage = 0, from_stage = 0;
            auto next = [&](uint32_t st) { return st + slice_bytes == sp.stages * slice_bytes ? 0u : st + slice_bytes; };
            auto copy_slice = [&](uint32_t i) {
                if (i < nz) {
                    const bool z_in = z0 + i >= 0 && z0 + i < p.D[2];  // the same for the block
#pragma unroll
                    for (uint32_t u = 0; u < kPre; ++u) {
                        if (tid + NT * u < ncopy) {
                            const uint32_t k = z_in ? n[u] : 0u;
                            copy16_async(smem + to_stage + cp[u].to, k ? src[u] : level, k);
                        }
                        src[u] += plane;
                    }
                    to_stage = next(to_stage);
                }
                copies_commit();
            };
            for (uint32_t i = 0; i + 1 < sp.stages; ++i) copy_slice(i);
            for (uint32_t i = 0; i < nz; ++i) {
                copies_wait(sp.stages - 2u);
                __syncthreads();  // slice i is here for all, and slice i - 1 has been read by all
                copy_slice(i + sp.stages - 1u);
#pragma unroll
                for (uint32_t u = 0; u < kPre; ++u) {
                    if (tid + NT * u < nchunks)
                        put_bytes(slab_smem + from_stage + ck[u].row, ck[u].at, ck[u].zeros, ck[u].dst);
                    ck[u].dst += dslice;
                }
                from_stage = next(from_stage);
            }
        } else {
            auto copy_slice = [&](uint32_t i) {
                if (i < nz) {
                    const uint32_t stage = smem + (i % sp.stages) * slice_bytes;
#pragma unroll
                    for (uint32_t u = 0; u < kPre; ++u)
                        if (tid + NT * u < ncopy) copy_chunk(cp[u], i, stage);
                    for (uint32_t t = tid + NT * kPre; t < ncopy; t += NT) copy_chunk(copy_of(t), i, stage);
                }
                copies_commit();
            };
            for (uint32_t i = 0; i + 1 < sp.stages; ++i) copy_slice(i);
            for (uint32_t i = 0; i < nz; ++i) {
                copies_wait(sp.stages - 2u);
                __syncthreads();
                copy_slice(i + sp.stages - 1u);
                const uint8_t *stage = slab_smem + (i % sp.stages) * slice_bytes;
#pragma unroll
                for (uint32_t u = 0; u < kPre; ++u)
                    if (tid + NT * u < nchunks) put_chunk(ck[u], i, stage);
                for (uint32_t t = tid + NT * kPre; t < nchunks; t += NT) put_chunk(chunk_of(t), i, stage);
            }
        }
        __syncthreads();  // the last slices have been read before the next slab's copies
    }
}

constexpr uint32_t kSlabShared = 200u << 10;  // shared memory of a slab's slices, at most

// Launches the slab bricker where it applies: brick rows of whole 16- or 8-byte
// chunks, a 16-byte aligned level, a store aligned to the chunks, and at least two
// slices in shared memory.
static bool launch_brick_slabs(const uint8_t *level, uint8_t *out, const BrickParams &p, cudaStream_t s) {
    const uint32_t row = p.B * p.eb;
    const uint32_t ch = row % 16 == 0 ? 16u : (row % 8 == 0 ? 8u : 0u);
    if (!ch || reinterpret_cast<uintptr_t>(level) % 16 || reinterpret_cast<uintptr_t>(out) % ch) return false;
    SlabParams sp;
    sp.p = p;
    sp.cpr = row / ch;
    const uint32_t nsx = p.nbig[0] * p.BB[0];
    // about 512 output chunks a slice (two per thread), fewer of the smallest bricks,
    // whose slabs have few slices; at most 1 KiB of a row, and of the smallest bricks
    // no more than the copies of a slice are two per thread too
    const uint32_t chunks = p.B <= 4 ? 128u : p.B <= 8 ? 256u : 512u;
    const uint32_t in_row = p.B > 8 ? 1024u / (p.Beff * p.eb) : (16u * (chunks / p.B) - 15u - row) / (p.Beff * p.eb) + 1u;
    sp.nb = std::max(1u, std::min(std::min(nsx, chunks / std::max(1u, p.B * sp.cpr)), in_row));
    sp.ngx = (nsx + sp.nb - 1) / sp.nb;
    sp.nb = (nsx + sp.ngx - 1) / sp.ngx;  // slabs of about the same size
    const uint32_t span = (sp.nb - 1) * p.Beff * p.eb + row;
    sp.cprow = (15u + span + 15u) / 16u;
    // the lanes of a quarter warp read 16-byte words of rows a pitch apart: cpr
    // words on from row to row modulo the 8 words of a bank line
    uint32_t words = sp.cprow + 1u;
    if (sp.cpr < 8u)
        while (words % 8u != (ch == 16 ? sp.cpr : 1u) % 8u) ++words;
    sp.pitch = words * 16u;
    const uint32_t slice = p.B * sp.pitch;
    sp.stages = std::min(4u, (96u << 10) / slice);
    if (sp.stages < 2u) sp.stages = std::min(2u, kSlabShared / slice);
    if (sp.stages < 2u || p.B * sp.cprow >= 65536u) return false;
    const uint64_t slabs = static_cast<uint64_t>(sp.ngx) * (p.nbig[1] * p.BB[1]) * (p.nbig[2] * p.BB[2]);
    // two copies and two chunks a thread: blocks of 64 or 128 threads where those fill no
    // more, so that more slabs are in flight.  Blocks of 256 / these: floats in 4^3
    // bricks, covering 1, 64^3 12.8 / 7.2 us, 384^3 577 / 440 (a warp per run of bricks
    // 8.3 and 596); u8 in 8^3 bricks 128^3 10.6 / 6.6, in 16^3 bricks 160^3 11.1 / 7.1
    const uint32_t work = std::max(sp.nb * p.B * sp.cpr, p.B * sp.cprow);
    const uint32_t threads = work <= 128u ? 64u : work <= 256u ? 128u : 256u;
    // four blocks per SM, as far as a slab has slices: at most with the small blocks, which
    // pay more for starting than for their slices, at least with those of 256 threads
    // (at most: B 32 u16 of 381x347x291 50 -> 60 us)
    const uint64_t want = static_cast<uint64_t>(sm_count()) * 4u;
    uint32_t parts = 1;
    while (parts < p.B && (threads < 256u ? slabs * parts * 2u <= want : slabs * parts < want)) parts *= 2u;
    sp.zlen = (p.B + parts - 1) / parts;
    sp.zparts = (p.B + sp.zlen - 1) / sp.zlen;
    sp.items = slabs * sp.zparts;
    sp.by_cprow = SmallDiv(sp.cprow);
    sp.by_brick = SmallDiv(p.B * sp.cpr);
    sp.by_cpr = SmallDiv(sp.cpr);
    const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>(sp.items, 1u << 30));
    const uint32_t bytes = sp.stages * slice;
    auto go = [&](auto kernel) {
        // always to the same limit: the attribute belongs to the kernel, not to the
        // call, and another thread's smaller slab must not lower it before this launch
        if (bytes > (48u << 10))
            GC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSlabShared));
        kernel<<<grid, threads, bytes, s>>>(level, out, sp);
    };
    if (ch == 16)
        threads == 64    ? go(brick_slab_kernel<16, 64>)
        : threads == 128 ? go(brick_slab_kernel<16, 128>)
                         : go(brick_slab_kernel<16, 256>);
    else
        threads == 64    ? go(brick_slab_kernel<8, 64>)
        : threads == 128 ? go(brick_slab_kernel<8, 128>)
                         : go(brick_slab_kernel<8, 256>);
    GC_CUDA(cudaGetLastError());
    count_launch();
    return true;
}

// Bricks cut on demand from a device-resident pyramid (the device-levels
// brick source): job j = big brick (x, y, z) of level `lvl` of volume `vol`
// into staging slot `slot`; one block per job, its warps over the job's small
// bricks, each by the level bricker's rule.
// list: the jobs are the elements of a miss list instead, j into slot j (volumes
// whose big bricks are one brick each; elements of other volumes are skipped).
__global__ void __launch_bounds__(256) cut_bricks_kernel(const CutSources srcs, const uint4 *__restrict__ jobs,
                                                         const uint4 *__restrict__ list, const StoreMap m, uint32_t n,
                                                         uint8_t *__restrict__ staging, uint64_t stride) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t j = blockIdx.x; j < n; j += gridDim.x) {
        uint4 job;
        if (list) {
            job = list[j];
            const StoreLevel &l = m.level[job.w];
            if (l.cut == 0u) continue;
            job.w = (j << 8) | (l.cut - 1u);
        } else {
            job = jobs[j];
        }
        const uint32_t lvl = job.w & 63u, vol = (job.w >> 6) & 3u, slot = job.w >> 8;
        const CutSource &cs = srcs.vol[vol];
        BrickParams p = cs.p;
        for (int a = 0; a < 3; ++a) p.D[a] = cs.dims[lvl][a];
        p.fast = cs.fast[lvl];
        const uint32_t nsub = p.BB[0] * p.BB[1] * p.BB[2];
        for (uint32_t sub = warp; sub < nsub; sub += nw) {
            const uint32_t ix = sub % p.BB[0], iy = (sub / p.BB[0]) % p.BB[1], iz = sub / (p.BB[0] * p.BB[1]);
            copy_small_brick(cs.pyramid + cs.offset[lvl], p, job.x * p.BB[0] + ix, job.y * p.BB[1] + iy,
                             job.z * p.BB[2] + iz, staging + static_cast<uint64_t>(slot) * stride, ix, iy, iz,
                             lane);
        }
    }
}

void launch_cut_bricks(const CutSources &srcs, const uint4 *jobs, const uint4 *list, const StoreMap &m, uint32_t n,
                       uint8_t *staging, uint64_t stride, cudaStream_t s) {
    if (n == 0) return;
    cut_bricks_kernel<<<std::min<uint32_t>(n, static_cast<uint32_t>(sm_count()) * 8), 256, 0, s>>>(srcs, jobs, list, m, n,
                                                                                                 staging, stride);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

// Empty flags: 1 if every channel value of the big brick is < threshold
// (DefaultBrickProcessorPredicate: (float)value < threshold).
__global__ void __launch_bounds__(256) empty_kernel(const uint8_t *__restrict__ bricks, uint64_t nbig,
                                                    uint64_t big_values, uint32_t cb, float threshold,
                                                    uint8_t *__restrict__ flags) {
    __shared__ int s_nonempty;
    for (uint64_t b = blockIdx.x; b < nbig; b += gridDim.x) {
        if (threadIdx.x == 0) s_nonempty = 0;
        __syncthreads();
        const uint8_t *base = bricks + b * big_values * cb;
        int nonempty = 0;
        for (uint64_t i = threadIdx.x; i < big_values && !nonempty; i += blockDim.x) {
            float v;
            if (cb == 1)
                v = static_cast<float>(base[i]);
            else if (cb == 2)
                v = static_cast<float>(reinterpret_cast<const uint16_t *>(base)[i]);
            else
                v = reinterpret_cast<const float *>(base)[i];
            if (!(v < threshold)) nonempty = 1;
        }
        if (__syncthreads_or(nonempty) && threadIdx.x == 0) s_nonempty = 1;
        __syncthreads();
        if (threadIdx.x == 0) flags[b] = s_nonempty ? 0 : 1;
        __syncthreads();
    }
}

// One turn of G threads over a big brick, four 16-byte loads in flight a thread, from
// chunk c0 on: true where a value of the thread's chunks reaches the threshold.
template <int CB, int G>
__device__ __forceinline__ bool reaches(const uint4 *__restrict__ p, uint64_t c0, uint32_t lane, uint64_t chunks,
                                        float threshold) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const uint64_t c = c0 + u * G + lane;
        if (c < chunks) v[u] = __ldcs(p + c);
    }
    ValueRange<CB> range;
    bool over = false, any = false;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (c0 + u * G + lane < chunks) {
            any = true;
            if constexpr (CB == 4) {
                over = over || !(__uint_as_float(v[u].x) < threshold) || !(__uint_as_float(v[u].y) < threshold) ||
                       !(__uint_as_float(v[u].z) < threshold) || !(__uint_as_float(v[u].w) < threshold);
            } else {
                range.add(v[u]);
            }
        }
    }
    if constexpr (CB != 4) over = any && !(static_cast<float>(range.highest()) < threshold);
    return over;
}

// The same for big bricks of whole 16-byte chunks, 16-byte aligned, a warp each, 16
// bytes a lane with four loads in flight, ended by a vote once a value reaches the
// threshold (an integer brick is empty when its largest value is below it).  Bound
// by the read of the bricks that are empty; the first 2 KiB are read of every
// brick.  The bricks of a 768^3 u16 volume (16^3, 1.36 GB): 712 -> 66 us; 16,384 big
// bricks of 32 KiB dense / half of them empty / all empty, value by value 13 / 450 /
// 777, a block each 42 / 61 / 77, a warp each 9 / 56 / 87 us.
template <int CB>
__global__ void __launch_bounds__(256) empty_warp_kernel(const uint4 *__restrict__ bricks, uint64_t nbig,
                                                         uint64_t chunks, float threshold,
                                                         uint8_t *__restrict__ flags) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t b = static_cast<uint64_t>(blockIdx.x) * 8u + threadIdx.x / 32u; b < nbig;
         b += static_cast<uint64_t>(gridDim.x) * 8u) {
        const uint4 *p = bricks + b * chunks;
        bool nonempty = false;
        for (uint64_t c0 = 0; c0 < chunks && !nonempty; c0 += 128u)
            nonempty = __any_sync(0xffffffffu, reaches<CB, 32>(p, c0, lane, chunks, threshold)) != 0;
        if (lane == 0) flags[b] = nonempty ? 0 : 1;
    }
}

// Big bricks of 32 KiB and more that are no warps enough: a block takes `per` of them
// (up to 8, as far as the bricks fill the SMs), a warp first looks at the first 512
// bytes of each, and the whole block reads those that this leaves open.  4,854 big
// bricks of 108 KiB dense / half of them empty / all empty, value by value 6.6 / 433 /
// 760, a block each without the look (16 KiB of every brick) 15 / 46 / 79, with it 5.6 /
// 46 / 82 us; 1,024 of 32 KiB 4.5 / 27 / 27, 5.6 / 6.5 / 6.8, 4.4 / 6.8 / 8.5 us.  Up to
// four per SM no look (kLook): 16 KiB of each cost nothing there, the look 1 us.
template <int CB, bool kLook>
__global__ void __launch_bounds__(256) empty_block_kernel(const uint4 *__restrict__ bricks, uint64_t nbig,
                                                          uint64_t chunks, uint32_t per, float threshold,
                                                          uint8_t *__restrict__ flags) {
    __shared__ uint32_t s_open[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint64_t b0 = static_cast<uint64_t>(blockIdx.x) * per;
    bool open = !kLook && warp < per && b0 + warp < nbig;
    if (kLook && warp < per && b0 + warp < nbig) {
        open = !__any_sync(0xffffffffu, reaches<CB, 32>(bricks + (b0 + warp) * chunks, 0, lane, 32, threshold));
        if (!open && lane == 0) flags[b0 + warp] = 0;
    }
    if (lane == 0) s_open[warp] = open;
    __syncthreads();
    for (uint32_t w = 0; w < per; ++w) {
        if (!s_open[w]) continue;  // the same for the block
        const uint4 *p = bricks + (b0 + w) * chunks;
        bool nonempty = false;
        for (uint64_t c0 = 0; c0 < chunks && !nonempty; c0 += 1024u)
            nonempty = __syncthreads_or(reaches<CB, 256>(p, c0, tid, chunks, threshold)) != 0;
        if (tid == 0) flags[b0 + w] = nonempty ? 0 : 1;
    }
}

}  // namespace gc

using namespace gc;

extern "C" {

int gc_mip_level(const void *src, void *dst, const uint32_t src_dims[3], uint32_t encoded_bytes,
                 uint32_t channels, void *stream) {
    return guard([&] {
        GC_REQUIRE(src && dst && src_dims, "null argument");
        GC_REQUIRE(channels >= 1, "channels must be >= 1");
        launch_mip(src, dst, src_dims, encoded_bytes, channels, as_stream(stream));
    });
}

int gc_mip_build(void *pyramid, const gc_layout *layout, const uint64_t *level_offsets,
                 uint32_t encoded_bytes, uint32_t channels, void *stream) {
    return guard([&] {
        GC_REQUIRE(pyramid && layout && level_offsets, "null argument");
        GC_REQUIRE(layout->nb_levels >= 1 && layout->nb_levels <= GC_MAX_LEVELS, "bad layout");
        GC_REQUIRE(level_offsets[0] == 0, "level 0 must start at offset 0");
        uint8_t *base = static_cast<uint8_t *>(pyramid);
        for (uint32_t l = 1; l < layout->nb_levels; ++l)
            for (int a = 0; a < 3; ++a)
                GC_REQUIRE(layout->mip[l][a] == layout->mip[l - 1][a] / 2,
                           "level sizes that stop halving (dimension <= 2) are not supported");
        for (uint32_t l = 1; l < layout->nb_levels;) {
            const uint32_t *d = layout->mip[l - 1];
            uint8_t *dst[2] = {base + level_offsets[l], nullptr};
            if (l + 1 < layout->nb_levels) {
                dst[1] = base + level_offsets[l + 1];
                if (launch_mip_fused(base + level_offsets[l - 1], dst, d, encoded_bytes, channels, as_stream(stream))) {
                    l += 2;
                    continue;
                }
            }
            launch_mip(base + level_offsets[l - 1], dst[0], d, encoded_bytes, channels, as_stream(stream));
            ++l;
        }
    });
}

int gc_bricks_build(const void *level, const uint32_t level_dims[3], const gc_volume_desc *vol,
                    const uint32_t nb_big_bricks[3], void *out, void *stream) {
    return guard([&] {
        GC_REQUIRE(level && level_dims && vol && nb_big_bricks && out, "null argument");
        validate_volume(*vol);
        BrickParams p;
        for (int a = 0; a < 3; ++a) {
            p.D[a] = level_dims[a];
            p.BB[a] = vol->big_brick_size[a];
            p.nbig[a] = nb_big_bricks[a];
            GC_REQUIRE(p.nbig[a] > 0, "nb_big_bricks must be > 0");
        }
        p.B = vol->brick_size;
        p.c = vol->covering;
        p.Beff = p.B - 2 * p.c;
        p.eb = vol->encoded_bytes;
        p.nsmall = static_cast<uint64_t>(p.nbig[0] * p.BB[0]) * (p.nbig[1] * p.BB[1]) * (p.nbig[2] * p.BB[2]);
        // 16-byte row chunks: whole chunks per brick row, rows 16 bytes apart
        // in the level (so every row of a brick has the same alignment), and
        // both buffers 16-byte aligned
        GC_REQUIRE(p.nsmall < (1ull << 32), "too many bricks in one level");
        p.fast = (p.eb == 1 || p.eb == 2 || p.eb == 4) && (p.B & (p.B - 1)) == 0 && (p.B * p.eb) % 16 == 0 &&
                 (static_cast<uint64_t>(p.D[0]) * p.eb) % 16 == 0 &&
                 reinterpret_cast<uintptr_t>(level) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
        p.b_shift = p.cpr_shift = 0;
        while ((1u << p.b_shift) < p.B) ++p.b_shift;
        while (p.fast && (16u << p.cpr_shift) < p.B * p.eb) ++p.cpr_shift;
        if (launch_brick_slabs(static_cast<const uint8_t *>(level), static_cast<uint8_t *>(out), p, as_stream(stream)))
            return;
        // one warp per brick: 8 warps per block, enough blocks to fill every SM
        const uint64_t grid = std::max<uint64_t>(1, std::min<uint64_t>((p.nsmall + 7) / 8,
                                                                       static_cast<uint64_t>(sm_count()) * 8));
        brick_kernel<<<static_cast<unsigned>(grid), 256, 0, as_stream(stream)>>>(
            static_cast<const uint8_t *>(level), static_cast<uint8_t *>(out), p);
        GC_CUDA(cudaGetLastError());
        count_launch();
    });
}

int gc_bricks_empty(const void *bricks, uint64_t nb_big_bricks, const gc_volume_desc *vol,
                    float threshold, uint8_t *flags, void *stream) {
    return guard([&] {
        GC_REQUIRE(bricks && vol && flags, "null argument");
        validate_volume(*vol);
        const uint64_t B = vol->brick_size;
        const uint64_t values = B * B * B * vol->big_brick_size[0] * vol->big_brick_size[1] *
                                vol->big_brick_size[2] * vol->channels;
        if (nb_big_bricks == 0) return;
        const uint32_t cb = channel_bytes(*vol);
        const uint64_t bytes = values * cb;
        if (bytes % 16 == 0 && reinterpret_cast<uintptr_t>(bricks) % 16 == 0 && (cb == 1 || cb == 2 || cb == 4)) {
            const auto *in = static_cast<const uint4 *>(bricks);
            const uint64_t sms = static_cast<uint64_t>(sm_count());
            // a warp per big brick, above 32 KiB only where the bricks are warps enough
            if (bytes < (32u << 10) || (bytes <= (128u << 10) && nb_big_bricks >= sms * 48)) {
                const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((nb_big_bricks + 7) / 8, sms * 64));
                auto go = [&](auto kernel) {
                    kernel<<<blocks, 256, 0, as_stream(stream)>>>(in, nb_big_bricks, bytes / 16, threshold, flags);
                };
                cb == 1 ? go(empty_warp_kernel<1>) : cb == 2 ? go(empty_warp_kernel<2>) : go(empty_warp_kernel<4>);
            } else {
                const bool look = nb_big_bricks > sms * 4;
                const uint32_t per =
                    static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>(8, nb_big_bricks / (sms * 8))));
                const unsigned blocks = static_cast<unsigned>((nb_big_bricks + per - 1) / per);
                auto go = [&](auto kernel) {
                    kernel<<<blocks, 256, 0, as_stream(stream)>>>(in, nb_big_bricks, bytes / 16, per, threshold, flags);
                };
                if (cb == 1)
                    look ? go(empty_block_kernel<1, true>) : go(empty_block_kernel<1, false>);
                else if (cb == 2)
                    look ? go(empty_block_kernel<2, true>) : go(empty_block_kernel<2, false>);
                else
                    look ? go(empty_block_kernel<4, true>) : go(empty_block_kernel<4, false>);
            }
            GC_CUDA(cudaGetLastError());
            count_launch();
            return;
        }
        const uint64_t grid = std::min<uint64_t>(nb_big_bricks, static_cast<uint64_t>(sm_count()) * 16);
        empty_kernel<<<static_cast<unsigned>(grid), 256, 0, as_stream(stream)>>>(
            static_cast<const uint8_t *>(bricks), nb_big_bricks, values, channel_bytes(*vol), threshold,
            flags);
        GC_CUDA(cudaGetLastError());
        count_launch();
    });
}

}  // extern "C"
