// Per-frame cache kernels: LRU update, miss-list compaction, brick install,
// completude.
//
// LRU update.  The reference builds a bool mask (create_usage_mask,
// GcCore/src/cuda/libGPUCache/CacheManagerKernels.cu:8-29) and runs two
// thrust::copy_if over 28-byte LruContent records into a freshly allocated
// device_vector (CacheDevice.hpp:200-219): a stable partition, used slots
// first.  That is one stable 1-bit radix pass on the key "used this frame"
// (usage[slot] == timestamp).  Here the order is a list of 4-byte slot ids:
//   frame_scan     : total_used = #slots with usage == ts (one read of usage)
//   lru_partition  : per 4096-item tile, ballot/popc + block scan of the used
//                    flags, the tile's exclusive prefix P from the counts its
//                    predecessors published, then used id -> out[P + rank],
//                    unused id at global index i -> out[total_used + i -
//                    used_before(i)].
// Miss list.  The reference compacts indexes i in [0, size - 1) with
// req[i] == ts with thrust::copy_if over a counting iterator into a full-size
// size_t vector, keeps the first 50 and decodes them with coord_1D_to_3D
// (CacheManager.hpp:409-474, CacheManagerKernels.cu:32-72).  frame_scan does
// the scan, cap and decode in one pass of its own blocks.
// Every wait for a predecessor's count is bounded; on expiry the kernel sets
// ScanCtl::err.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "cache.cuh"
#include "gc_internal.h"
#include "value_range.cuh"

namespace gc {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr uint32_t kMaxSpins = 1u << 22;
// lru_partition: 16 slot ids a lane; frame_scan: eight 16-byte words a lane
constexpr uint32_t kLruItems = 16, kLruTile = kThreads * kLruItems;
constexpr uint32_t kScanWords = 8, kScanTile = kThreads * kScanWords * 4;

// A tile's status word: the published bit, then its count.  In a scan of more than
// a number of tiles (kScanGrouped, kLruGrouped) the words are followed by one per
// whole group of kGroup tiles, with the group's sum, which its last tile publishes.
// The words are all that is handed over, so relaxed accesses do (no other memory
// is ordered by them).
//
// With groups a tile reads at most 256 words and one per 256 tiles, without them
// one per tile before it, which grows with the square of the tiles; but a sum
// comes a hop later.  Request scan: 6.4 M entries (782 tiles), misses in most,
// 19.7 us without, 17.4 with groups; update of a 403 M entry directory (49,297
// tiles) with 10,000 misses / a miss in every tile 589 / 1,549 -> 447 / 688 us.
// LRU update, every tile of which waits: 8,192 tiles 220 us without, 247 with
// groups; 16,384 487 / 466; 32,768 1,254 / 910.
constexpr uint64_t kPublished = 1ull << 32;
constexpr uint32_t kGroup = 256, kScanGrouped = 256, kLruGrouped = 12288;
__host__ __device__ constexpr uint32_t whole_groups(uint32_t tiles, uint32_t grouped) {
    return tiles > grouped ? tiles / kGroup : 0u;
}
__device__ __forceinline__ void publish(uint64_t *status, uint32_t count) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(status), "l"(kPublished | count) : "memory");
}
__device__ __forceinline__ uint64_t status_of(const uint64_t *status) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(status) : "memory");
    return v;
}

// Sum of one value per thread over a block, for all threads.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *s_warp) {
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t += s_warp[w];
    return t;
}

// This thread's share of the sum of n published words, each waited for (bounded).
__device__ __forceinline__ uint32_t published(const uint64_t *words, uint32_t n, uint32_t *err) {
    uint32_t sum = 0, spins = 0;
#pragma unroll 4
    for (uint32_t j = threadIdx.x; j < n; j += kThreads) {
        uint64_t v = status_of(words + j);
        while (!(v & kPublished)) {
            if (++spins > kMaxSpins) {
                atomicOr(err, kErrLookback);
                break;
            }
            __nanosleep(32);
            v = status_of(words + j);
        }
        sum += static_cast<uint32_t>(v);
    }
    return sum;
}

// True for the tiles that publish their group's sum, and so call predecessors.
__device__ __forceinline__ bool ends_group(uint32_t tile, uint32_t groups) {
    return tile < groups * kGroup && tile % kGroup == kGroup - 1u;
}

// The number of flagged items in the tiles before `tile`, whose count `total` this
// tile's block has published: the threads wait for the tiles before it (in its
// group, and for the whole groups before that, where the scan has groups), so that
// no tile waits for a chain of others.  Tiles are handed out by a ticket, so every
// predecessor's block has started.
// only_group: the tile has nothing flagged and wants no sum.
__device__ uint32_t predecessors(uint64_t *status, uint32_t tile, uint32_t tiles, uint32_t groups, uint32_t total,
                                 bool only_group, uint32_t *err, uint32_t *s_warp) {
    const uint32_t group = groups ? tile / kGroup : 0u, first = group * kGroup;
    uint32_t sum = published(status + first, tile - first, err);
    if (ends_group(tile, groups)) {
        const uint32_t in_group = block_sum(sum, s_warp);
        if (threadIdx.x == 0) publish(status + tiles + group, in_group + total);
    }
    if (only_group) return 0;
    sum += published(status + tiles, group, err);
    return block_sum(sum, s_warp);
}

// True in the block that ends a launch last: it leaves the tickets and status
// words as the next launch expects them, with no memset between.
__device__ __forceinline__ bool ends_launch(ScanCtl *ctl) {
    __shared__ uint32_t s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&ctl->done, 1u) == gridDim.x - 1u;
        __threadfence();
    }
    __syncthreads();
    return s_last != 0;
}

__global__ void __launch_bounds__(kThreads) lru_partition_kernel(const uint32_t *__restrict__ order_in,
                                                                 uint32_t *__restrict__ order_out,
                                                                 const uint32_t *__restrict__ usage,
                                                                 uint32_t ts, uint32_t n,
                                                                 const uint32_t *__restrict__ count,
                                                                 uint64_t *status, ScanCtl *ctl) {
    __shared__ uint32_t s_tile, s_warp[kWarps], s_used[kWarps];
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // a warp's 512 consecutive items, 32 at a time
    const uint64_t base = static_cast<uint64_t>(tile) * kLruTile + warp * (32u * kLruItems) + lane;
    uint32_t ids[kLruItems], mine = 0, used = 0;
#pragma unroll
    for (uint32_t k = 0; k < kLruItems; ++k) ids[k] = base + 32u * k < n ? __ldg(order_in + base + 32u * k) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < kLruItems; ++k)
        mine |= (base + 32u * k < n && usage[ids[k]] == ts ? 1u : 0u) << k;
#pragma unroll
    for (uint32_t k = 0; k < kLruItems; ++k) used += __popc(__ballot_sync(0xffffffffu, (mine >> k) & 1u));
    if (lane == 0) s_used[warp] = used;
    __syncthreads();
    uint32_t total = 0, before = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) {
        before += w < warp ? s_used[w] : 0u;
        total += s_used[w];
    }
    if (threadIdx.x == 0) publish(status + tile, total);
    const uint32_t groups = whole_groups(gridDim.x, kLruGrouped);
    before += predecessors(status, tile, gridDim.x, groups, total, false, &ctl->err, s_warp);
    const uint32_t total_used = *count;
    bool bad = false;
#pragma unroll
    for (uint32_t k = 0; k < kLruItems; ++k) {
        const uint64_t i = base + 32u * k;
        const uint32_t flags = __ballot_sync(0xffffffffu, (mine >> k) & 1u);
        const uint32_t used_before = before + __popc(flags & ((1u << lane) - 1u));
        if (i < n) {
            const uint64_t dst = (mine >> k) & 1u ? used_before : total_used + i - used_before;
            if (dst < n)
                order_out[dst] = ids[k];
            else
                bad = true;  // only after an expired wait
        }
        before += __popc(flags);
    }
    if (bad) atomicOr(&ctl->err, kErrLookback);
    if (ends_launch(ctl)) {
        for (uint32_t j = threadIdx.x; j < gridDim.x + groups; j += kThreads) status[j] = 0;
        if (threadIdx.x == 0) ctl->ticket = ctl->done = 0;
    }
}

// The whole LRU update of a pool of up to kClusterSlots slots in one launch of one
// thread-block cluster: every block partitions 1024 kItems slots, and the blocks
// read one another's counts from distributed shared memory between the two
// halves, so neither a count kernel before nor waits through memory are needed.
// Bound by latency -- two dependent loads, a cluster barrier, a store -- so the
// slots are spread over as many of the eight blocks as there are.  Install frame
// of a 32,768-slot cache from render to installed bricks: 31 -> 21 us.
template <uint32_t kItems>
__global__ void __launch_bounds__(1024) lru_cluster_kernel(const uint32_t *__restrict__ order_in,
                                                           uint32_t *__restrict__ order_out,
                                                           const uint32_t *__restrict__ usage, uint32_t ts, uint32_t n,
                                                           uint32_t *__restrict__ count) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ uint32_t s_used[32], s_total;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, block = cluster.block_rank();
    // a warp's 512 consecutive items, 32 at a time
    const uint32_t base = block * (1024u * kItems) + warp * (32u * kItems) + lane;
    uint32_t ids[kItems], mine = 0, used = 0;
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) ids[k] = base + 32u * k < n ? __ldg(order_in + base + 32u * k) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k)
        mine |= (base + 32u * k < n && usage[ids[k]] == ts ? 1u : 0u) << k;
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) used += __popc(__ballot_sync(0xffffffffu, (mine >> k) & 1u));
    if (lane == 0) s_used[warp] = used;
    __syncthreads();
    const uint32_t of_warp = s_used[lane];
    if (threadIdx.x < 32u) {
        const uint32_t total = __reduce_add_sync(0xffffffffu, of_warp);
        if (lane == 0) s_total = total;
    }
    cluster.sync();
    const uint32_t blocks = cluster.num_blocks();
    const uint32_t of_block = lane < blocks ? *cluster.map_shared_rank(&s_total, lane) : 0u;
    uint32_t before = __reduce_add_sync(0xffffffffu, (lane < block ? of_block : 0u) + (lane < warp ? of_warp : 0u));
    const uint32_t total_used = __reduce_add_sync(0xffffffffu, of_block);
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) {
        const uint32_t i = base + 32u * k;
        const uint32_t flags = __ballot_sync(0xffffffffu, (mine >> k) & 1u);
        const uint32_t used_before = before + __popc(flags & ((1u << lane) - 1u));
        if (i < n) order_out[(mine >> k) & 1u ? used_before : total_used + i - used_before] = ids[k];
        before += __popc(flags);
    }
    if (block == 0 && threadIdx.x == 0) *count = total_used;
    cluster.sync();  // no block ends while another reads its count
}

// coord_1D_to_3D (CacheManagerKernels.cu:32-72) of an entry (the page directory
// has fewer than 2^32).
__device__ __forceinline__ uint4 decode_request(uint32_t i, uint32_t mx, uint32_t my, const LevelTables &lt) {
    const uint32_t row = i / mx, x = i - row * mx, z = row / my, y = row - z * my;
    uint32_t sum = 0, level = 0;
    for (level = 0; level < lt.nlevels; ++level) {
        sum += lt.nb[level][0];
        if (x < sum) break;
    }
    if (level >= lt.nlevels) level = lt.nlevels - 1;
    return make_uint4(x - (sum - lt.nb[level][0]), y, z, level);
}

// The scans of a frame, each by blocks of its own: the request scan (scan_tiles
// blocks) and the number of slots used (count_blocks[k] blocks for the brick
// pool and the table pool of a two-level directory).  One launch, bound by the
// read of the request buffer (from L2 when the frames follow one another).  A
// request tile holds 8192 entries, eight 16-byte loads in flight a lane; it only
// counts and publishes unless it has flagged entries, and then waits for its
// predecessors' counts alone, not for a chain of them.  The miss list goes to the
// device list and straight into the host's pinned copy: only the misses cross
// the link, and no copy follows the scan.  6.4 M entries with 5000 misses: 29 us
// (a chained look-back over 4096-entry tiles) -> 12 us.
template <bool kCounts>  // false: no slots to count
__global__ void __launch_bounds__(kThreads) frame_scan_kernel(const FrameScan a, const LevelTables lt) {
    __shared__ uint32_t s_tile, s_warp[kWarps], s_used[kWarps];
    __shared__ uint16_t s_entry[kScanTile];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t groups = whole_groups(a.scan_tiles, kScanGrouped);
    if (blockIdx.x < a.scan_tiles) {
        if (threadIdx.x == 0) s_tile = atomicAdd(&a.ctl->ticket, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        // a warp's 1024 consecutive entries, 128 at a time
        const uint64_t base = static_cast<uint64_t>(tile) * kScanTile + warp * (128u * kScanWords) + 4u * lane;
        uint4 v[kScanWords];
        uint32_t flags = 0;  // four bits a word
#pragma unroll
        for (uint32_t u = 0; u < kScanWords; ++u)
            if (base + 128u * u + 4u <= a.nscan) v[u] = __ldcg(reinterpret_cast<const uint4 *>(a.req + base + 128u * u));
#pragma unroll
        for (uint32_t u = 0; u < kScanWords; ++u) {
            const uint64_t i = base + 128u * u;
            if (i + 4u <= a.nscan) {
                flags |= ((v[u].x == a.ts ? 1u : 0u) | (v[u].y == a.ts ? 2u : 0u) | (v[u].z == a.ts ? 4u : 0u) |
                          (v[u].w == a.ts ? 8u : 0u))
                         << (4u * u);
            } else {
                for (uint32_t k = 0; k < 4u; ++k)
                    if (i + k < a.nscan) flags |= (__ldcg(a.req + i + k) == a.ts ? 1u : 0u) << (4u * u + k);
            }
        }
        const uint32_t used = __reduce_add_sync(0xffffffffu, __popc(flags));
        if (lane == 0) s_used[warp] = used;
        __syncthreads();
        uint32_t total = 0, rank = 0;
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w) {
            rank += w < warp ? s_used[w] : 0u;
            total += s_used[w];
        }
        if (tile != a.silent_tile && tile < a.scan_tiles) {  // (beyond: calls that share the scratch overlapped)
            if (threadIdx.x == 0) publish(a.status + tile, total);
            if (total) {
                // the tile's flagged entries in order, then decoded by all threads
                for (uint32_t u = 0; u < kScanWords; ++u) {
                    const uint32_t f = (flags >> (4u * u)) & 15u;
                    if (!__any_sync(0xffffffffu, f)) continue;
                    uint32_t r = rank;  // after the flagged entries of the lanes before
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k) {
                        const uint32_t bal = __ballot_sync(0xffffffffu, (f >> k) & 1u);
                        r += __popc(bal & ((1u << lane) - 1u));
                        rank += __popc(bal);
                    }
                    for (uint32_t k = 0; k < 4u; ++k)
                        if ((f >> k) & 1u)
                            s_entry[r++] = static_cast<uint16_t>(warp * (128u * kScanWords) + 128u * u + 4u * lane + k);
                }
                const uint32_t first =
                    predecessors(a.status, tile, a.scan_tiles, groups, total, false, &a.ctl->err, s_warp);  // also a barrier
                const uint32_t n = first < a.maxreq ? min(total, a.maxreq - first) : 0u;
                for (uint32_t r = threadIdx.x; r < n; r += kThreads) {
                    const uint4 b = decode_request(tile * kScanTile + s_entry[r], a.mx, a.my, lt);
                    a.list[first + r] = b;
                    if (a.host_list) a.host_list[first + r] = b;
                }
            } else if (ends_group(tile, groups)) {
                predecessors(a.status, tile, a.scan_tiles, groups, 0u, true, &a.ctl->err, s_warp);
            }
        }
    } else if constexpr (kCounts) {
        uint32_t blk = blockIdx.x - a.scan_tiles;
        const uint32_t k = blk < a.count_blocks[0] ? 0u : 1u;
        if (k) blk -= a.count_blocks[0];
        // four 16-byte loads in flight a thread: bound by HBM, not by the latency of one
        // word after the other (update of a 2 M slot pool 30 -> 26 us, 33 M 388 -> 221)
        const uint32_t *__restrict__ usage = a.usage[k];
        const uint4 *__restrict__ words = reinterpret_cast<const uint4 *>(usage);
        const uint32_t n = a.nslots[k], n4 = n / 4u, step = a.count_blocks[k] * kThreads;
        const uint32_t at = blk * kThreads + threadIdx.x;
        uint32_t c = 0;
        for (uint64_t i0 = at; i0 < n4; i0 += 4ull * step) {
            uint4 v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                if (i0 + u * step < n4) v[u] = __ldg(words + i0 + u * step);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                if (i0 + u * step < n4)
                    c += (v[u].x == a.ts ? 1u : 0u) + (v[u].y == a.ts ? 1u : 0u) + (v[u].z == a.ts ? 1u : 0u) +
                         (v[u].w == a.ts ? 1u : 0u);
        }
        if (at < n % 4u) c += usage[4u * n4 + at] == a.ts ? 1u : 0u;
        c = block_sum(c, s_warp);
        if (threadIdx.x == 0 && c) atomicAdd(&a.ctl->used[k], c);
    }
    if (!ends_launch(a.ctl)) return;
    // the last block: the totals, and everything as the next launch expects it
    uint32_t sum = 0;
    bool missing = false;
    const uint32_t in_groups = groups * kGroup;  // tiles summed by their groups
    for (uint32_t j = in_groups + threadIdx.x; j < a.scan_tiles + groups; j += kThreads) {
        const uint64_t v = status_of(a.status + j);
        missing = missing || !(v & kPublished);
        sum += static_cast<uint32_t>(v);
        a.status[j] = 0;
    }
    for (uint32_t j = threadIdx.x; j < in_groups; j += kThreads) a.status[j] = 0;
    missing = __syncthreads_or(missing);
    sum = block_sum(sum, s_warp);
    if (threadIdx.x == 0) {
        ScanCtl *ctl = a.ctl;
        if (missing) ctl->err |= kErrLookback;
        for (int k = 0; k < 2; ++k) {
            if (kCounts && a.count_blocks[k]) {
                *a.count[k] = *static_cast<volatile uint32_t *>(&ctl->used[k]);
                ctl->used[k] = 0;
            }
        }
        if (a.scan_tiles) {
            ctl->total = sum;
            if (a.host_total) *a.host_total = sum;
            if (a.out_total) {  // a caller's own list: the result word tells a failure, and the next call starts clean
                *a.out_total = *static_cast<volatile uint32_t *>(&ctl->err) ? GC_MISS_LIST_FAILED : sum;
                ctl->err = 0;
            }
        }
        ctl->ticket = ctl->done = 0;
    }
}

// ---------------------------------------------------------------------------
// Brick install (CacheManager::load_new_bricks, CacheManager.hpp:502-632).

// MRPD coordinate of a normalized brick origin (K_MultiResolutionPageDirectory::set,
// K_MultiResolutionPageDirectory.hpp:193-205).
__device__ __forceinline__ uint64_t mrpd_index(const LevelTables &lt, uint32_t level, float vx, float vy, float vz,
                                               uint32_t mx, uint32_t my) {
    const uint32_t x = lt.off[level] + static_cast<uint32_t>(__fmul_rn(vx, static_cast<float>(lt.nb[level][0])));
    const uint32_t y = static_cast<uint32_t>(__fmul_rn(vy, static_cast<float>(lt.nb[level][1])));
    const uint32_t z = static_cast<uint32_t>(__fmul_rn(vz, static_cast<float>(lt.nb[level][2])));
    return x + static_cast<uint64_t>(y) * mx + static_cast<uint64_t>(z) * mx * my;
}
// The same brick as (x inside the level, y, z): its place in a two-level directory.
__device__ __forceinline__ uint3 brick_at(const LevelTables &lt, uint32_t level, float vx, float vy, float vz) {
    return make_uint3(static_cast<uint32_t>(__fmul_rn(vx, static_cast<float>(lt.nb[level][0]))),
                      static_cast<uint32_t>(__fmul_rn(vy, static_cast<float>(lt.nb[level][1]))),
                      static_cast<uint32_t>(__fmul_rn(vz, static_cast<float>(lt.nb[level][2]))));
}
__device__ __forceinline__ bool brick_inside(const LevelTables &lt, uint32_t level, uint3 q) {
    return q.x < lt.nb[level][0] && q.y < lt.nb[level][1] && q.z < lt.nb[level][2];
}
// The brick entry of q in a two-level directory, or null when its block is
// not resident.
__device__ __forceinline__ uint4 *pt_entry_of(const PageTable &pt, const LevelTables &lt, uint32_t level, uint3 q) {
    const uint32_t t = pt.top[pt_word(pt, lt, level, q.x, q.y, q.z)];
    if (!(t & 1u)) return nullptr;
    return pt.table + pt_entry(pt, t >> 1, pt_local(pt, q.x, q.y, q.z));
}
// Page-directory entry (x, y, z, 1) of pool slot `slot`.
__device__ __forceinline__ uint4 slot_entry(uint32_t slot, uint32_t sx, uint32_t sy, uint32_t B) {
    return make_uint4((slot % sx) * B, ((slot / sx) % sy) * B, (slot / (sx * sy)) * B, 1u);
}

// compute_volume_position (CacheManagerKernels.cu:75-86):
// x / (V.x * (1 / (B - 2c))) + FLT_EPSILON.
__device__ __forceinline__ float4 brick_origin(const LevelTables &lt, uint4 b, float one_over_beff) {
    const float eps = 1.1920928955078125e-7f;
    float4 v;
    v.x = __fadd_rn(__fdiv_rn(static_cast<float>(b.x), __fmul_rn(static_cast<float>(lt.vvox[b.w][0]), one_over_beff)), eps);
    v.y = __fadd_rn(__fdiv_rn(static_cast<float>(b.y), __fmul_rn(static_cast<float>(lt.vvox[b.w][1]), one_over_beff)), eps);
    v.z = __fadd_rn(__fdiv_rn(static_cast<float>(b.z), __fmul_rn(static_cast<float>(lt.vvox[b.w][2]), one_over_beff)), eps);
    v.w = 0.f;
    return v;
}

// dereference_old_bricks (CacheManagerKernels.hpp:115-145) for one slot of the
// LRU tail, whose payload still names its old brick.
__device__ __forceinline__ void evict_slot(const InstallArgs &a, const LevelTables &lt, uint32_t slot) {
    const float4 vp = a.slot_vpos[slot];
    const uint32_t level = a.slot_level[slot];
    if (vp.x < 0.f) return;  // slot never held a brick
    const uint64_t e = mrpd_index(lt, level, vp.x, vp.y, vp.z, a.mx, a.my);
    if (e >= a.nentries) return;
    if (a.pt.shift) {
        // Two levels: the entry is cleared only where it still names this
        // slot -- after its block was evicted the brick may be unreachable,
        // or resident again in another slot.
        const uint3 q = brick_at(lt, level, vp.x, vp.y, vp.z);
        if (!brick_inside(lt, level, q)) return;
        uint4 *pe = pt_entry_of(a.pt, lt, level, q);
        if (!pe) return;
        const uint4 cur = *pe, mine = slot_entry(slot, a.sx, a.sy, a.B);
        if (cur.w != 1u || cur.x != mine.x || cur.y != mine.y || cur.z != mine.z) return;
        *pe = make_uint4(0, 0, 0, 0);
    } else {
        a.mrpd[e] = make_uint4(0, 0, 0, 0);
    }
    a.entry_bins[e] = a.user_bins ? a.user_bins[e] : ~0ull;
}

// Value range of a brick as value bins (empty-space skipping): min and max
// over its voxels (covering included), normalized like the samplers, widened
// by one bin on either side.  `at(v)` gives the address of voxel v; one
// block per brick (up to 288 threads); the result is valid in thread 0.
// The value bins of the range [lo, hi] (normalized like the samplers), widened
// by one bin on either side.
__device__ __forceinline__ unsigned long long bins_of_range(float lo, float hi) {
    auto bin = [](float x) {
        const float f = floorf(x * static_cast<float>(kValueBins));
        return f < 0.f ? 0 : (f > kValueBins - 1.f ? static_cast<int>(kValueBins) - 1 : static_cast<int>(f));
    };
    const int b0 = max(bin(lo) - 1, 0), b1 = min(bin(hi) + 1, static_cast<int>(kValueBins) - 1);
    const unsigned long long upto = b1 >= 63 ? ~0ull : ((1ull << (b1 + 1)) - 1ull);
    return upto & ~((1ull << b0) - 1ull);
}
// The block's value bins from each thread's min and max; the result is valid in
// thread 0.
__device__ unsigned long long block_bins_from(float lo, float hi) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __shared__ float s_lo[9], s_hi[9];
    const uint32_t warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31u) == 0) {
        s_lo[warp] = lo;
        s_hi[warp] = hi;
    }
    __syncthreads();
    if (threadIdx.x != 0) return 0;
    for (uint32_t w = 1; w < (blockDim.x + 31) / 32; ++w) {
        lo = fminf(lo, s_lo[w]);
        hi = fmaxf(hi, s_hi[w]);
    }
    return bins_of_range(lo, hi);
}
// Two 8-bit channels: 32 bins each, channel 0 in the low half.  mn and mx hold the
// thread's bounds, channel 0 in the low 16 bits; the result is valid in thread 0.
__device__ unsigned long long block_bins_of_two(uint32_t mn, uint32_t mx) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = min_u16x2(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = max_u16x2(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    __shared__ uint32_t s_mn[9], s_mx[9];
    const uint32_t warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31u) == 0) {
        s_mn[warp] = mn;
        s_mx[warp] = mx;
    }
    __syncthreads();
    if (threadIdx.x != 0) return 0;
    for (uint32_t w = 1; w < (blockDim.x + 31) / 32; ++w) {
        mn = min_u16x2(mn, s_mn[w]);
        mx = max_u16x2(mx, s_mx[w]);
    }
    auto bins = [](uint32_t lo, uint32_t hi) {  // bin of v: floor(32 v / 255), at most 31; one more on either side
        const uint32_t b0 = min(lo * 32u / 255u, 31u), b1 = min(min(hi * 32u / 255u, 31u) + 1u, 31u);
        const uint32_t upto = b1 == 31u ? ~0u : (2u << b1) - 1u;
        return upto & ~((1u << (b0 ? b0 - 1u : 0u)) - 1u);
    };
    return bins(mn & 0xffffu, mx & 0xffffu) | static_cast<unsigned long long>(bins(mn >> 16, mx >> 16)) << 32;
}
template <class At>
__device__ unsigned long long block_value_bins(uint32_t nvox, uint32_t eb, At at) {
    float lo = 3.4e38f, hi = -3.4e38f;
    for (uint32_t v = threadIdx.x; v < nvox; v += blockDim.x) {
        const uint8_t *p = at(v);
        float x;
        if (eb == 1)
            x = static_cast<float>(*p) * (1.0f / 255.0f);
        else if (eb == 2)
            x = static_cast<float>(*reinterpret_cast<const uint16_t *>(p)) * (1.0f / 65535.0f);
        else
            x = *reinterpret_cast<const float *>(p);
        lo = fminf(lo, x);
        hi = fmaxf(hi, x);
    }
    return block_bins_from(lo, hi);
}

// Min and max over the voxels of a 16-byte chunk, into (lo, hi) as the
// samplers normalize them (integer min / max first: the normalization is
// monotone, so the result is block_value_bins').
__device__ __forceinline__ void chunk_range(uint4 c, uint32_t eb, float &lo, float &hi) {
    if (eb == 1) {
        const uint32_t mn = __vminu4(__vminu4(c.x, c.y), __vminu4(c.z, c.w));
        const uint32_t mx = __vmaxu4(__vmaxu4(c.x, c.y), __vmaxu4(c.z, c.w));
        const uint32_t mn1 = min(min(mn & 0xffu, (mn >> 8) & 0xffu), min((mn >> 16) & 0xffu, mn >> 24));
        const uint32_t mx1 = max(max(mx & 0xffu, (mx >> 8) & 0xffu), max((mx >> 16) & 0xffu, mx >> 24));
        lo = fminf(lo, static_cast<float>(mn1) * (1.0f / 255.0f));
        hi = fmaxf(hi, static_cast<float>(mx1) * (1.0f / 255.0f));
    } else if (eb == 2) {
        const uint32_t mn = __vminu2(__vminu2(c.x, c.y), __vminu2(c.z, c.w));
        const uint32_t mx = __vmaxu2(__vmaxu2(c.x, c.y), __vmaxu2(c.z, c.w));
        lo = fminf(lo, static_cast<float>(min(mn & 0xffffu, mn >> 16)) * (1.0f / 65535.0f));
        hi = fmaxf(hi, static_cast<float>(max(mx & 0xffffu, mx >> 16)) * (1.0f / 65535.0f));
    } else {
        lo = fminf(fminf(lo, fminf(__uint_as_float(c.x), __uint_as_float(c.y))),
                   fminf(__uint_as_float(c.z), __uint_as_float(c.w)));
        hi = fmaxf(fmaxf(hi, fmaxf(__uint_as_float(c.x), __uint_as_float(c.y))),
                   fmaxf(__uint_as_float(c.z), __uint_as_float(c.w)));
    }
}

// Value bins of every brick of one level, read from the level's big bricks
// on the device: the mask the install computes for the same brick in a pool
// slot.  One block per brick of the level's brick grid (x fastest).
__global__ void __launch_bounds__(256) brick_bins_kernel(const uint8_t *__restrict__ level, uint32_t nbx, uint32_t nby,
                                                         uint32_t nbz, uint32_t gbx, uint32_t gby, uint32_t bb0,
                                                         uint32_t bb1, uint32_t bb2, uint32_t B, uint32_t eb,
                                                         unsigned long long *bins) {
    const uint64_t i = blockIdx.x;
    const uint32_t x = static_cast<uint32_t>(i % nbx), y = static_cast<uint32_t>((i / nbx) % nby),
                   z = static_cast<uint32_t>(i / (static_cast<uint64_t>(nbx) * nby));
    if (z >= nbz) return;
    const uint32_t gx = x / bb0, gy = y / bb1, gz = z / bb2;
    const uint32_t bvx = bb0 * B, bvy = bb1 * B, bvz = bb2 * B;
    const uint8_t *big =
        level + ((static_cast<uint64_t>(gz) * gby + gy) * gbx + gx) * (static_cast<uint64_t>(bvx) * bvy * bvz * eb);
    const uint32_t ox = (x - gx * bb0) * B, oy = (y - gy * bb1) * B, oz = (z - gz * bb2) * B;
    const unsigned long long m = block_value_bins(B * B * B, eb, [&](uint32_t v) {
        const uint32_t lx = v % B, ly = (v / B) % B, lz = v / (B * B);
        return big + ((static_cast<uint64_t>(oz + lz) * bvy + (oy + ly)) * bvx + (ox + lx)) * eb;
    });
    if (threadIdx.x == 0) bins[i] = m;
}

// The same for bricks of whole 16-byte row chunks in a 16-byte aligned level: G
// threads per brick read it 16 bytes a lane with four loads in flight.  Bound by
// the read of the store.  A warp per brick (G = 32) up to 16 KiB, so that no
// block barrier follows a brick's few loads; a block above, where one warp would
// take 64 KiB bricks in 32 dependent turns, and for few bricks of more than 2 KiB
// (warps / blocks: 16^3 floats in big bricks of 2^3, 64 bricks 10.5 / 4.8 us, 512 10.5 /
// 6.7; 16^3 u8 in big bricks 64 6.2 / 4.4, without 512 4.7 / 6.2).  The bricks of a 768^3 u16
// volume (16^3, 1.36 GB): 1970 -> 185 us, 7.4 TB/s.
template <int EB, int G>
__global__ void __launch_bounds__(256) brick_bins_vec_kernel(const uint8_t *__restrict__ level, uint32_t n,
                                                             uint32_t nbx, uint32_t nby, uint32_t gbx, uint32_t gby,
                                                             uint32_t bb0, uint32_t bb1, uint32_t bb2, uint32_t B,
                                                             uint32_t cpr, unsigned long long *bins) {
    const uint32_t i = G == 256 ? blockIdx.x : blockIdx.x * (256 / G) + threadIdx.x / G;
    const uint32_t lane = threadIdx.x % G;
    if (i >= n) return;  // the same for the G threads of the brick
    const uint32_t x = i % nbx, r = i / nbx, y = r % nby, z = r / nby;
    const uint32_t gx = x / bb0, gy = y / bb1, gz = z / bb2;
    const uint32_t chunks = B * B * cpr;  // per brick
    const uint64_t big = (static_cast<uint64_t>(gz) * gby + gy) * gbx + gx;
    const bool whole = bb0 == 1 && bb1 == 1;  // the brick's chunks lie one after the other
    const uint4 *p = reinterpret_cast<const uint4 *>(level) + big * (static_cast<uint64_t>(bb0) * bb1 * bb2 * chunks) +
                     ((static_cast<uint64_t>(z - gz * bb2) * B * (bb1 * B) + (y - gy * bb1) * B) * bb0 + (x - gx * bb0)) * cpr;
    ValueRange<EB> range;
    for (uint32_t c0 = lane; c0 < chunks; c0 += 4u * G) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t c = c0 + u * G;
            if (c < chunks) {
                uint64_t at = c;
                if (!whole) {
                    const uint32_t row = c / cpr, q = c - row * cpr, lz = row / B, ly = row - lz * B;
                    at = static_cast<uint64_t>(lz * (bb1 * B) + ly) * (bb0 * cpr) + q;
                }
                v[u] = __ldcs(p + at);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c0 + u * G < chunks) range.add(v[u]);
    }
    float lo = 3.4e38f, hi = -3.4e38f;
    if (lane < chunks) range.normalized(lo, hi);
    if constexpr (G == 256) {
        const unsigned long long m = block_bins_from(lo, hi);
        if (lane == 0) bins[i] = m;
    } else {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) bins[i] = bins_of_range(lo, hi);
    }
}

void launch_brick_bins(const uint8_t *level, const uint32_t nb[3], const uint32_t nbig[3], const uint32_t bb[3],
                       uint32_t B, uint32_t eb, unsigned long long *bins, cudaStream_t s) {
    const uint64_t n = static_cast<uint64_t>(nb[0]) * nb[1] * nb[2];
    if (n == 0) return;
    GC_REQUIRE(n < (1ull << 31), "too many bricks in one level");
    const uint32_t n32 = static_cast<uint32_t>(n);
    if ((B * eb) % 16 == 0 && B <= 512 && reinterpret_cast<uintptr_t>(level) % 16 == 0) {
        const uint32_t cpr = B * eb / 16;
        const uint32_t chunks = B * B * cpr, sms = static_cast<uint32_t>(sm_count());
        const bool warp = chunks <= 128 || (chunks <= 1024 && n32 >= sms * (chunks <= 512 ? 2u : 8u));
        auto go = [&](auto kernel) {
            kernel<<<warp ? div_up(n32, 8u) : n32, 256, 0, s>>>(level, n32, nb[0], nb[1], nbig[0], nbig[1], bb[0], bb[1],
                                                               bb[2], B, cpr, bins);
        };
        if (eb == 1)
            warp ? go(brick_bins_vec_kernel<1, 32>) : go(brick_bins_vec_kernel<1, 256>);
        else if (eb == 2)
            warp ? go(brick_bins_vec_kernel<2, 32>) : go(brick_bins_vec_kernel<2, 256>);
        else
            warp ? go(brick_bins_vec_kernel<4, 32>) : go(brick_bins_vec_kernel<4, 256>);
    } else {
        brick_bins_kernel<<<n32, 256, 0, s>>>(level, nb[0], nb[1], nb[2], nbig[0], nbig[1], bb[0], bb[1], bb[2], B, eb,
                                             bins);
    }
    GC_CUDA(cudaGetLastError());
    count_launch();
}

// One block per brick of the list, its first 256 threads copying and one more
// warp keeping the books meanwhile, so that an install is two launches.
//   books: dereference_old_bricks for the slot the brick takes, then the slot's
//   new payload (compute_lru_volume_position + copy_lru_position,
//   CacheManagerKernels.cu:90-114), and the owner word of the brick's entry (see
//   install_reference_kernel);
//   copy (write_brick, CacheManagerKernels.hpp:59-107): B^3 voxels from the staged
//   big brick into the LRU-tail slot, 16 bytes at a time when rows allow it.
// An evicted entry is read by nothing before install_reference_kernel.
constexpr uint32_t kCopyThreads = 256;
__global__ void __launch_bounds__(kCopyThreads + 32) install_place_kernel(InstallArgs a, const LevelTables lt,
                                                                          float one_over_beff) {
    const uint32_t i = blockIdx.x;
    const uint4 b = a.asked[i];
    if (threadIdx.x == kCopyThreads) {
        const float4 v = brick_origin(lt, b, one_over_beff);
        const uint64_t c = mrpd_index(lt, b.w, v.x, v.y, v.z, a.mx, a.my);
        a.coords[i] = c;
        if (c < a.nentries) atomicMin(a.owner + c, i);
        if (i < a.n_nonempty) {
            const uint32_t slot = a.order[a.nslots - a.n_nonempty + i];
            evict_slot(a, lt, slot);
            a.slot_level[slot] = b.w;
            a.slot_vpos[slot] = v;
        }
    }
    if (i >= a.n_nonempty) return;  // an empty brick: books only
    const uint32_t slot = a.order[a.nslots - a.n_nonempty + i];
    const uint32_t tid = threadIdx.x;  // the last warp copies nothing and only joins the block's barriers
    // the brick's volume: voxel width and big-brick shape of its level
    const uint32_t B = a.B, eb = lt.eb[b.w];
    const uint32_t *BB = lt.bb[b.w];
    const uint32_t bvx = BB[0] * B, bvy = BB[1] * B;
    uint32_t bi = i, ox = 0, oy = 0, oz = 0;
    if (a.big_index) {  // else every big brick is one brick, staged in list order
        bi = a.big_index[i];
        const uint4 bc = a.big_coord[bi];
        ox = (b.x - bc.x * BB[0]) * B, oy = (b.y - bc.y * BB[1]) * B, oz = (b.z - bc.z * BB[2]) * B;
    }
    const uint8_t *src = a.staging + bi * a.big_stride;
    uint8_t *dst = a.pool + static_cast<uint64_t>(slot) * a.slot_bytes;
    const uint32_t row_bytes = B * eb;
    const uint32_t rows = B * B;
    const uint32_t vec_per_row = row_bytes / 16;
    const bool pow2 = (B & (B - 1u)) == 0u && (vec_per_row & (vec_per_row - 1u)) == 0u;
    if (row_bytes % 16 == 0 && pow2 && (reinterpret_cast<uintptr_t>(src) % 16 == 0) && ((bvx * eb) % 16 == 0)) {
        // 16-byte chunks, four loads in flight per thread before their
        // stores; the brick's value range is taken from the loaded chunks
        // (one read of the brick for both)
        const uint32_t qs = __ffs(vec_per_row) - 1u, bs = __ffs(B) - 1u;
        const uint32_t nvec = rows * vec_per_row;
        const bool bins = a.slot_bins && a.nc == 1, two = a.slot_bins && a.nc == 2 && eb == 2;
        float lo = 3.4e38f, hi = -3.4e38f;
        ValueRange<1> range;  // two 8-bit channels: even and odd bytes
        for (uint32_t v0 = tid < kCopyThreads ? tid : nvec; v0 < nvec; v0 += 4u * kCopyThreads) {
            uint4 val[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t v = v0 + u * kCopyThreads;
                if (v < nvec) {
                    const uint32_t r = v >> qs, q = v & (vec_per_row - 1u);
                    const uint32_t ly = r & (B - 1u), lz = r >> bs;
                    const uint64_t soff =
                        ((static_cast<uint64_t>(oz + lz) * bvy + (oy + ly)) * bvx + ox) * eb + q * 16u;
                    val[u] = __ldcs(reinterpret_cast<const uint4 *>(src + soff));
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t v = v0 + u * kCopyThreads;
                if (v < nvec) {
                    reinterpret_cast<uint4 *>(dst)[v] = val[u];
                    if (bins) chunk_range(val[u], eb, lo, hi);
                    if (two) range.add(val[u]);
                }
            }
        }
        if (!a.slot_bins) return;
        if (two) {
            const unsigned long long b2 = block_bins_of_two(range.mn_channels(), range.mx_channels());
            if (threadIdx.x == 0) a.slot_bins[slot] = b2;
            return;
        }
        if (a.nc != 1) {
            if (threadIdx.x == 0) a.slot_bins[slot] = ~0ull;  // never skipped
            return;
        }
        const unsigned long long b2 = block_bins_from(lo, hi);
        if (threadIdx.x == 0) a.slot_bins[slot] = b2;
        return;
    } else {
        const uint32_t nbytes = rows * row_bytes;
        for (uint32_t v = tid < kCopyThreads ? tid : nbytes; v < nbytes; v += kCopyThreads) {
            const uint32_t r = v / row_bytes, q = v % row_bytes;
            const uint32_t ly = r % B, lz = r / B;
            const uint64_t soff = ((static_cast<uint64_t>(oz + lz) * bvy + (oy + ly)) * bvx + ox) * eb + q;
            dst[v] = src[soff];
        }
    }
    if (!a.slot_bins) return;
    __syncthreads();
    if (a.nc != 1) {
        if (threadIdx.x == 0) a.slot_bins[slot] = ~0ull;  // never skipped
        return;
    }
    const unsigned long long bins = block_value_bins(B * B * B, eb, [&](uint32_t v) { return dst + v * eb; });
    if (threadIdx.x == 0) a.slot_bins[slot] = bins;
}

// reference_new_bricks (CacheManagerKernels.hpp:308-357) for the MRPD-only
// hierarchy: in list order (non-empty first), an unmapped entry becomes
// {slot position, 1} or {0, 0, 0, 2} for an empty brick; an entry that is
// already mapped or empty is left alone.  The reference walks the list in one
// thread; here each brick is one thread, and a brick whose MRPD entry also
// belongs to an earlier list element yields to it, which is the serial order:
// install_place_kernel leaves the lowest list index naming each entry in `owner`,
// and only that element acts (and puts the owner word back).
__global__ void install_reference_kernel(InstallArgs a, const LevelTables lt, float one_over_beff) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const uint64_t c = a.coords[i];
    if (c >= a.nentries || a.owner[c] != i) return;  // an earlier element names the same entry
    a.owner[c] = 0xffffffffu;  // later readers see a value that is not their index either way
    uint4 *pe = a.mrpd + c;
    if (a.pt.shift) {
        // two levels: the entry lives in the block of its directory word (none
        // when the table pool had no slot left for it: the brick stays unmapped)
        const uint4 b = a.asked[i];
        const float4 v = brick_origin(lt, b, one_over_beff);
        const uint3 q = brick_at(lt, b.w, v.x, v.y, v.z);
        if (!brick_inside(lt, b.w, q)) return;
        pe = pt_entry_of(a.pt, lt, b.w, q);
        if (!pe) return;
    }
    const uint4 e = *pe;
    if (e.w == 1u || e.w == 2u) return;  // mapped or empty already (3 = in flight: install it)
    if (i < a.n_nonempty) {
        const uint32_t slot = a.order[a.nslots - a.n_nonempty + i];
        *pe = slot_entry(slot, a.sx, a.sy, a.B);
        a.entry_bins[c] = a.slot_bins[slot];
    } else {
        *pe = make_uint4(0, 0, 0, 2u);
    }
}

// Two-level directory: table blocks for the new bricks.  Each element that
// acts for its entry (the owner) and whose directory word has no block claims
// the word; the lowest element index wins.
__global__ void install_pt_claim_kernel(InstallArgs a, const LevelTables lt, float one_over_beff) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    uint32_t word = 0xffffffffu;
    const uint64_t c = a.coords[i];
    if (c < a.nentries && a.owner[c] == i) {
        const uint4 b = a.asked[i];
        const float4 v = brick_origin(lt, b, one_over_beff);
        const uint3 q = brick_at(lt, b.w, v.x, v.y, v.z);
        const uint32_t w = pt_word(a.pt, lt, b.w, q.x, q.y, q.z);
        if (brick_inside(lt, b.w, q) && !(a.pt.top[w] & 1u)) {
            word = w;
            atomicMin(a.pt_claim + w, i);
        }
    }
    a.pt_word_of[i] = word;
}

// The claimed words in list order (one block): the k-th winner gets the k-th
// of the table slots taken from the LRU tail.
__global__ void __launch_bounds__(1024) install_pt_rank_kernel(InstallArgs a) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_base;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (uint32_t i0 = 0; i0 < a.n; i0 += blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        const uint32_t w = i < a.n ? a.pt_word_of[i] : 0xffffffffu;
        const bool win = w != 0xffffffffu && a.pt_claim[w] == i;
        const uint32_t bal = __ballot_sync(0xffffffffu, win);
        if (lane == 0) s_warp[warp] = __popc(bal);
        __syncthreads();
        uint32_t before = s_base;
        for (uint32_t k = 0; k < warp; ++k) before += s_warp[k];
        if (win) a.pt_jobs[before + __popc(bal & ((1u << lane) - 1u))] = make_uint2(w, i);
        __syncthreads();
        if (threadIdx.x == 0)
            for (uint32_t k = 0; k < nwarps; ++k) s_base += s_warp[k];
        __syncthreads();
    }
    if (threadIdx.x == 0) *a.pt_njobs = s_base;
}

// One block per claimed word: the table slot at LRU-tail position k leaves
// the block it held (its directory word cleared, the value bins of its mapped
// entries reverted), is cleared and takes the claimed word.  Claims beyond
// the table pool's size get no slot.
__global__ void __launch_bounds__(256) install_pt_apply_kernel(InstallArgs a, const LevelTables lt,
                                                               float one_over_beff) {
    const uint32_t m = *a.pt_njobs, k = blockIdx.x;
    if (k >= m) return;
    const uint2 job = a.pt_jobs[k];
    const uint32_t npt = min(m, a.pt_slots);
    if (k >= npt) {
        if (threadIdx.x == 0) a.pt_claim[job.x] = 0xffffffffu;
        return;
    }
    const uint32_t slot = a.pt_order[a.pt_slots - npt + k];
    const uint32_t P = 1u << a.pt.shift, P3 = P * P * P;
    uint4 *blk = a.pt.table + pt_entry(a.pt, slot, 0);
    const uint4 old = a.pt_keys[slot];
    if (old.w != 0xffffffffu) {
        for (uint32_t j = threadIdx.x; j < P3; j += blockDim.x) {
            if (blk[j].w != 1u) continue;
            const uint32_t dx = j & (P - 1u), dy = (j >> a.pt.shift) & (P - 1u), dz = j >> (2u * a.pt.shift);
            const uint64_t e = static_cast<uint64_t>(lt.off[old.w] + old.x + dx) +
                               static_cast<uint64_t>(old.y + dy) * a.mx +
                               static_cast<uint64_t>(old.z + dz) * a.mx * a.my;
            a.entry_bins[e] = a.user_bins ? a.user_bins[e] : ~0ull;
        }
    }
    __syncthreads();  // the old entries are read before they are cleared
    for (uint32_t j = threadIdx.x; j < P3; j += blockDim.x) blk[j] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) {
        if (old.w != 0xffffffffu) a.pt.top[pt_word(a.pt, lt, old.w, old.x, old.y, old.z)] = 0u;
        const uint4 b = a.asked[job.y];
        const float4 v = brick_origin(lt, b, one_over_beff);
        const uint3 q = brick_at(lt, b.w, v.x, v.y, v.z);
        const uint32_t msk = ~(P - 1u);
        a.pt_keys[slot] = make_uint4(q.x & msk, q.y & msk, q.z & msk, b.w);
        a.pt.top[job.x] = slot << 1 | 1u;
        a.pt_claim[job.x] = 0xffffffffu;
    }
}

__global__ void __launch_bounds__(256) completude_kernel(const float4 *__restrict__ vpos, uint32_t n,
                                                         uint32_t *__restrict__ count) {
    uint32_t c = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        c += (vpos[i].x != -1.f) ? 1u : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

// ---------------------------------------------------------------------------
static uint32_t lru_tiles(uint64_t n) { return static_cast<uint32_t>((n + kLruTile - 1) / kLruTile); }
static uint32_t scan_tiles(uint64_t n) { return static_cast<uint32_t>((n + kScanTile - 1) / kScanTile); }
uint32_t lru_status_words(uint64_t n) { return lru_tiles(n) + whole_groups(lru_tiles(n), kLruGrouped); }
uint32_t scan_status_words(uint64_t n) { return scan_tiles(n) + whole_groups(scan_tiles(n), kScanGrouped); }

void launch_frame_scan(FrameScan a, const LevelTables &lt, cudaStream_t s) {
    a.scan_tiles = a.nscan ? scan_tiles(a.nscan) : 0u;
    uint32_t grid = a.scan_tiles;
    for (int k = 0; k < 2; ++k) {
        // a block per 4096 slots, at most two per SM
        a.count_blocks[k] = a.nslots[k] ? std::min(div_up(a.nslots[k], 4096u), static_cast<uint32_t>(sm_count()) * 2u) : 0u;
        grid += a.count_blocks[k];
    }
    if (grid > a.scan_tiles)
        frame_scan_kernel<true><<<grid, kThreads, 0, s>>>(a, lt);
    else
        frame_scan_kernel<false><<<grid, kThreads, 0, s>>>(a, lt);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

void launch_lru_partition(const uint32_t *order_in, uint32_t *order_out, const uint32_t *usage, uint32_t ts,
                          uint32_t nslots, const uint32_t *count, uint64_t *status, ScanCtl *ctl, cudaStream_t s) {
    lru_partition_kernel<<<lru_tiles(nslots), kThreads, 0, s>>>(order_in, order_out, usage, ts, nslots, count, status,
                                                                ctl);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

void launch_lru_cluster(const uint32_t *order_in, uint32_t *order_out, const uint32_t *usage, uint32_t ts,
                        uint32_t nslots, uint32_t *count, cudaStream_t s) {
    static_assert(kClusterSlots == 8u * 16u * 1024u, "a portable cluster has up to 8 blocks");
    uint32_t items = 1;
    while (items < 16u && items * 8192u < nslots) items *= 2u;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(div_up(nslots, 1024u * items));
    cfg.blockDim = dim3(1024);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cfg.gridDim.x;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto go = [&](auto kernel) { GC_CUDA(cudaLaunchKernelEx(&cfg, kernel, order_in, order_out, usage, ts, nslots, count)); };
    switch (items) {
        case 1: go(lru_cluster_kernel<1>); break;
        case 2: go(lru_cluster_kernel<2>); break;
        case 4: go(lru_cluster_kernel<4>); break;
        case 8: go(lru_cluster_kernel<8>); break;
        default: go(lru_cluster_kernel<16>); break;
    }
    count_launch();
}

__global__ void live_bins_kernel(const LevelTables lt, const float4 *__restrict__ slot_vpos,
                                 const uint32_t *__restrict__ slot_level,
                                 const unsigned long long *__restrict__ slot_bins, uint32_t nslots, uint32_t mx,
                                 uint32_t my, uint64_t nentries, unsigned long long *entry_bins, const PageTable pt,
                                 uint32_t sx, uint32_t sy, uint32_t B) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nslots; i += gridDim.x * blockDim.x) {
        const float4 vp = slot_vpos[i];
        if (vp.x < 0.f) continue;  // slot never held a brick
        const uint32_t level = slot_level[i];
        const uint64_t e = mrpd_index(lt, level, vp.x, vp.y, vp.z, mx, my);
        if (e >= nentries) continue;
        if (pt.shift) {  // two levels: only a slot its entry names is live
            const uint3 q = brick_at(lt, level, vp.x, vp.y, vp.z);
            if (!brick_inside(lt, level, q)) continue;
            const uint4 *pe = pt_entry_of(pt, lt, level, q);
            const uint4 mine = slot_entry(i, sx, sy, B);
            if (!pe || pe->w != 1u || pe->x != mine.x || pe->y != mine.y || pe->z != mine.z) continue;
        }
        entry_bins[e] = slot_bins[i];
    }
}

void launch_live_bins(const LevelTables &lt, const float4 *slot_vpos, const uint32_t *slot_level,
                      const unsigned long long *slot_bins, uint32_t nslots, uint32_t mx, uint32_t my,
                      uint64_t nentries, unsigned long long *entry_bins, const PageTable &pt, uint32_t sx,
                      uint32_t sy, uint32_t B, cudaStream_t s) {
    const uint32_t grid = std::max(1u, std::min<uint32_t>(div_up(nslots, 256), static_cast<uint32_t>(sm_count()) * 4));
    live_bins_kernel<<<grid, 256, 0, s>>>(lt, slot_vpos, slot_level, slot_bins, nslots, mx, my, nentries, entry_bins,
                                          pt, sx, sy, B);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

void launch_install(const InstallArgs &a, const LevelTables &lt, cudaStream_t s) {
    if (a.n == 0) return;
    const float one_over_beff = 1.0f / static_cast<float>(a.Beff);
    install_place_kernel<<<a.n, kCopyThreads + 32, 0, s>>>(a, lt, one_over_beff);
    GC_CUDA(cudaGetLastError());
    count_launch();
    if (a.pt.shift) {
        install_pt_claim_kernel<<<div_up(a.n, 256u), 256, 0, s>>>(a, lt, one_over_beff);
        GC_CUDA(cudaGetLastError());
        install_pt_rank_kernel<<<1, 1024, 0, s>>>(a);
        GC_CUDA(cudaGetLastError());
        install_pt_apply_kernel<<<a.n, 256, 0, s>>>(a, lt, one_over_beff);
        GC_CUDA(cudaGetLastError());
        count_launch(3);
    }
    install_reference_kernel<<<div_up(a.n, 256u), 256, 0, s>>>(a, lt, one_over_beff);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

__global__ void pt_flatten_kernel(const PageTable pt, const LevelTables lt, uint32_t mx, uint32_t my,
                                  uint64_t nentries, uint4 *out) {
    for (uint64_t e = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; e < nentries;
         e += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t X = static_cast<uint32_t>(e % mx), y = static_cast<uint32_t>((e / mx) % my);
        const uint32_t z = static_cast<uint32_t>(e / (static_cast<uint64_t>(mx) * my));
        uint4 v = make_uint4(0, 0, 0, 0);
        for (uint32_t l = 0; l < lt.nlevels; ++l) {
            if (X < lt.off[l] || X >= lt.off[l] + lt.nb[l][0]) continue;
            const uint3 q = make_uint3(X - lt.off[l], y, z);
            if (brick_inside(lt, l, q)) {
                const uint32_t t = pt.top[pt_word(pt, lt, l, q.x, q.y, q.z)];
                if (t & 1u) v = pt.table[pt_entry(pt, t >> 1, pt_local(pt, q.x, q.y, q.z))];
            }
            break;
        }
        out[e] = v;
    }
}

void launch_pt_flatten(const PageTable &pt, const LevelTables &lt, uint32_t mx, uint32_t my, uint64_t nentries,
                       uint4 *out, cudaStream_t s) {
    const uint32_t grid =
        static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>((nentries + 255) / 256, sm_count() * 8ull)));
    pt_flatten_kernel<<<grid, 256, 0, s>>>(pt, lt, mx, my, nentries, out);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

__global__ void pt_init_kernel(uint32_t *order, uint4 *keys, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        order[i] = i;
        keys[i] = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
    }
}

void launch_pt_init(uint32_t *order, uint4 *keys, uint32_t nslots, cudaStream_t s) {
    pt_init_kernel<<<std::max(1u, std::min<uint32_t>(div_up(nslots, 256), 4096)), 256, 0, s>>>(order, keys, nslots);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

// Brick gather from device-readable host memory (the direct upload route):
// block-strided over bricks, each brick copied by the whole block with
// 16-byte loads when aligned.  The reads travel over the host link; the
// writes land in the device staging buffer the install kernels read.
// kIlp independent loads per thread are in flight before their stores: the
// host link's latency (microseconds) needs many bytes in flight per SM.
// src(b): brick b as {address, bytes}.
struct ListedBricks {
    const ulonglong2 *__restrict__ src;
    __device__ __forceinline__ ulonglong2 operator()(uint32_t b) const { return src[b]; }
};
// Brick b of a miss list in the host stores of its volume (each big brick one
// brick); nothing to read where the volume's source is not a host store.
struct MissedBricks {
    const uint4 *__restrict__ list;
    const StoreMap &m;
    __device__ __forceinline__ ulonglong2 operator()(uint32_t b) const {
        const uint4 e = list[b];
        const StoreLevel &l = m.level[e.w];
        return make_ulonglong2(l.store + ((static_cast<uint64_t>(e.z) * l.nby + e.y) * l.nbx + e.x) * l.bytes,
                               l.store ? l.bytes : 0u);
    }
};
template <typename W, class Src>
__device__ __forceinline__ void gather_bricks(const Src src, uint32_t n, uint64_t stride, uint8_t *__restrict__ dst) {
    constexpr uint32_t kIlp = 2;
    for (uint32_t b = blockIdx.x; b < n; b += gridDim.x) {
        const ulonglong2 e = src(b);
        const W *sp = reinterpret_cast<const W *>(e.x);
        W *dp = reinterpret_cast<W *>(dst + static_cast<uint64_t>(b) * stride);
        const uint64_t words = e.y / sizeof(W);
        const uint64_t step = static_cast<uint64_t>(blockDim.x) * kIlp;
        for (uint64_t i0 = threadIdx.x; i0 < words; i0 += step) {
            W v[kIlp];
#pragma unroll
            for (uint32_t k = 0; k < kIlp; ++k) {
                const uint64_t i = i0 + static_cast<uint64_t>(k) * blockDim.x;
                if (i < words) v[k] = sp[i];
            }
#pragma unroll
            for (uint32_t k = 0; k < kIlp; ++k) {
                const uint64_t i = i0 + static_cast<uint64_t>(k) * blockDim.x;
                if (i < words) dp[i] = v[k];
            }
        }
    }
}
// At most 32 registers per thread (128 threads, 16 blocks): fits beside the ray caster.
template <typename W>
__global__ void __launch_bounds__(128, 16) gather_bricks_kernel(const ulonglong2 *__restrict__ src, uint32_t n,
                                                               uint64_t stride, uint8_t *__restrict__ dst) {
    gather_bricks<W>(ListedBricks{src}, n, stride, dst);
}
template <typename W>
__global__ void __launch_bounds__(128, 16) gather_missed_kernel(const uint4 *__restrict__ list, const StoreMap m,
                                                               uint32_t n, uint64_t stride, uint8_t *__restrict__ dst) {
    gather_bricks<W>(MissedBricks{list, m}, n, stride, dst);
}

void launch_gather_missed(const uint4 *list, const StoreMap &m, uint32_t n, uint64_t stride, uint8_t *dst, bool vec16,
                          cudaStream_t s) {
    if (n == 0) return;
    const uint32_t grid = std::min<uint32_t>(n, static_cast<uint32_t>(sm_count()));  // as beside a render (below)
    if (vec16)
        gather_missed_kernel<uint4><<<grid, 128, 0, s>>>(list, m, n, stride, dst);
    else
        gather_missed_kernel<uint8_t><<<grid, 128, 0, s>>>(list, m, n, stride, dst);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

void launch_gather_bricks(const ulonglong2 *src, uint32_t n, uint64_t stride, uint8_t *dst, bool vec16,
                          cudaStream_t s) {
    if (n == 0) return;
    // Next to a persistent ray-caster launch: at its occupancy each SM
    // sub-partition keeps 1024 registers free, room for one warp of 32
    // registers per thread -- 128-thread blocks (one warp per
    // sub-partition), one per SM, run during the render instead of after
    // it (two 16-byte loads in flight per thread).  A second block per
    // SM, resident before the render's blocks arrive, would hold
    // registers a ray-caster block needs.
    const uint32_t grid = std::min<uint32_t>(n, static_cast<uint32_t>(sm_count()));
    if (vec16)
        gather_bricks_kernel<uint4><<<grid, 128, 0, s>>>(src, n, stride, dst);
    else
        gather_bricks_kernel<uint8_t><<<grid, 128, 0, s>>>(src, n, stride, dst);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

// In-flight marks of the batched form's overlapped loads: the entries of a
// miss list (x, y, z, level) handed to the loader are flagged 3 so that rays
// stop there without requesting them again; after the install, the entries
// still flagged (bricks that did not load) go back to 0.
__device__ __forceinline__ uint64_t list_entry_index(const LevelTables &lt, uint4 b, uint32_t mx, uint32_t my) {
    return static_cast<uint64_t>(lt.off[b.w] + b.x) + static_cast<uint64_t>(b.y) * mx +
           static_cast<uint64_t>(b.z) * mx * my;
}

__global__ void mark_in_flight_kernel(const uint4 *__restrict__ list, const ScanCtl *ctl, uint32_t maxreq,
                                      const LevelTables lt, uint32_t mx, uint32_t my, uint64_t nentries, uint4 *mrpd) {
    const uint32_t n = min(ctl->total, maxreq);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint4 b = list[i];
        if (b.w >= lt.nlevels) continue;
        const uint64_t e = list_entry_index(lt, b, mx, my);
        if (e < nentries && mrpd[e].w == 0u) mrpd[e].w = 3u;
    }
}

__global__ void unmark_in_flight_kernel(const uint4 *__restrict__ list, uint32_t n, const LevelTables lt,
                                        uint32_t mx, uint32_t my, uint64_t nentries, uint4 *mrpd) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint4 b = list[i];
        if (b.w >= lt.nlevels) continue;
        const uint64_t e = list_entry_index(lt, b, mx, my);
        if (e < nentries && mrpd[e].w == 3u) mrpd[e] = make_uint4(0, 0, 0, 0);
    }
}

void launch_mark_in_flight(const uint4 *list, const ScanCtl *ctl, uint32_t maxreq, const LevelTables &lt,
                           uint32_t mx, uint32_t my, uint64_t nentries, uint4 *mrpd, cudaStream_t s) {
    const uint32_t grid = std::max(1u, std::min<uint32_t>(div_up(maxreq, 256), static_cast<uint32_t>(sm_count()) * 2));
    mark_in_flight_kernel<<<grid, 256, 0, s>>>(list, ctl, maxreq, lt, mx, my, nentries, mrpd);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

void launch_unmark_in_flight(const uint4 *list, uint32_t n, const LevelTables &lt, uint32_t mx, uint32_t my,
                             uint64_t nentries, uint4 *mrpd, cudaStream_t s) {
    if (n == 0) return;
    const uint32_t grid = std::max(1u, std::min<uint32_t>(div_up(n, 256), static_cast<uint32_t>(sm_count()) * 2));
    unmark_in_flight_kernel<<<grid, 256, 0, s>>>(list, n, lt, mx, my, nentries, mrpd);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

void launch_completude(const float4 *slot_vpos, uint32_t nslots, uint32_t *count, cudaStream_t s) {
    GC_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), s));
    const uint32_t grid = std::min<uint32_t>(div_up(nslots, 256), static_cast<uint32_t>(sm_count()) * 4);
    completude_kernel<<<std::max(1u, grid), 256, 0, s>>>(slot_vpos, nslots, count);
    GC_CUDA(cudaGetLastError());
    count_launch();
}

}  // namespace gc

// ---------------------------------------------------------------------------
// Miss list without allocation.
//
// Some callers cannot allocate device memory at the moment they need the miss
// list: a host that records its frame into a CUDA graph (memory allocation is
// not allowed while a stream is being captured), a render loop with a hard
// frame deadline that must not block in the allocator (cudaMalloc can wait for
// the device), or a plug-in whose host application owns every byte of device
// memory and hands it only input and output buffers.  For them the scan's
// scratch -- a status word per 8192-entry tile and per 256 tiles and the scan
// control block -- lives in this file-scope device array instead of memory
// obtained from cudaMalloc.  Every GPU that loads the library holds it until
// the process exits.
namespace gc {

constexpr uint32_t kNoAllocMaxTiles = 1024;  // request buffers of up to 1024 * 8192 entries
constexpr uint64_t kNoAllocMaxEntries = static_cast<uint64_t>(kNoAllocMaxTiles) * kScanTile;

// ScanCtl, then the status words
constexpr uint32_t kNoAllocWords =
    kNoAllocMaxTiles + whole_groups(kNoAllocMaxTiles, kScanGrouped) + sizeof(ScanCtl) / sizeof(uint64_t);
static_assert(sizeof(ScanCtl) % sizeof(uint64_t) == 0, "ScanCtl must fill whole scratch words");
static __device__ __align__(256) uint64_t g_noalloc_scratch[kNoAllocWords];  // 8 KiB + 64 B

// Host code cannot use g_noalloc_scratch as a device address (the name is a
// host-side stand-in); the device address is looked up once per device, with
// that device current.
constexpr int kNoAllocMaxDevices = 64;
static uint64_t *g_noalloc_ptr[kNoAllocMaxDevices] = {};
static std::mutex g_noalloc_mu;

// Test hook of the error path: GC_TEST_NOALLOC_SILENT_TILE=<k> makes scan tile
// k publish nothing, so that the bounded waits of the later tiles with flagged
// entries run out (or, with none, the end of the launch finds the word missing).
static uint32_t noalloc_silent_tile() {
    const char *v = std::getenv("GC_TEST_NOALLOC_SILENT_TILE");
    return (v && *v) ? static_cast<uint32_t>(std::strtoul(v, nullptr, 10)) : 0xffffffffu;
}

static uint64_t *noalloc_scratch() {
    int dev = 0;
    GC_CUDA(cudaGetDevice(&dev));
    GC_REQUIRE(dev >= 0 && dev < kNoAllocMaxDevices, "device index out of range");
    std::lock_guard<std::mutex> g(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        uint64_t *p = nullptr;
        GC_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_noalloc_scratch));
        g_noalloc_ptr[dev] = p;
    }
    return g_noalloc_ptr[dev];
}

}  // namespace gc

extern "C" int gc_miss_list_noalloc(const uint32_t *requests, uint64_t n_entries, uint32_t timestamp,
                                    const gc_layout *layout, uint32_t max_requests, uint32_t *out_list,
                                    uint32_t *out_total, void *stream) {
    using namespace gc;
    return guard([&] {
        GC_REQUIRE(requests && layout && out_list && out_total, "null argument");
        // the scan reads the request words and writes the list 16 bytes at a time
        GC_REQUIRE(reinterpret_cast<uintptr_t>(requests) % 16 == 0 && reinterpret_cast<uintptr_t>(out_list) % 16 == 0,
                   "requests and out_list must be 16-byte aligned");
        GC_REQUIRE(reinterpret_cast<uintptr_t>(out_total) % 4 == 0, "out_total must be 4-byte aligned");
        GC_REQUIRE(n_entries >= 2, "the request buffer needs at least 2 entries");
        GC_REQUIRE(n_entries - 1 <= kNoAllocMaxEntries,
                   "request buffer too large for the allocation-free scan: at most 8388609 entries "
                   "(1024 tiles of 8192) are supported");
        GC_REQUIRE(max_requests >= 1, "max_requests must be >= 1");
        GC_REQUIRE(layout->nb_levels >= 1 && layout->nb_levels <= GC_MAX_LEVELS, "bad layout");
        // level tables of the page directory (levels packed along x)
        LevelTables lt;
        std::memset(&lt, 0, sizeof(lt));
        lt.nlevels = layout->nb_levels;
        uint32_t mx = 0, my = 0, mz = 0;
        for (uint32_t l = 0; l < layout->nb_levels; ++l) {
            lt.off[l] = mx;
            for (int a = 0; a < 3; ++a) lt.nb[l][a] = layout->nb_bricks[l][a];
            mx += layout->nb_bricks[l][0];
            my = std::max(my, layout->nb_bricks[l][1]);
            mz = std::max(mz, layout->nb_bricks[l][2]);
        }
        GC_REQUIRE(static_cast<uint64_t>(mx) * my * mz == n_entries,
                   "n_entries does not match the page directory of the layout");
        cudaStream_t s = as_stream(stream);
        ScanCtl *ctl = reinterpret_cast<ScanCtl *>(noalloc_scratch());
        uint64_t *status = reinterpret_cast<uint64_t *>(ctl + 1);
        // The scan leaves the scratch as it found it, but calls that overlapped (see
        // the header) may not have: every call starts from zeros.
        GC_CUDA(cudaMemsetAsync(ctl, 0, sizeof(ScanCtl) + scan_status_words(n_entries - 1) * sizeof(uint64_t), s));
        FrameScan a{};
        a.req = requests;
        a.nscan = n_entries - 1;
        a.ts = timestamp;
        a.maxreq = max_requests;
        a.list = reinterpret_cast<uint4 *>(out_list);
        a.mx = mx;
        a.my = my;
        a.status = status;
        a.ctl = ctl;
        a.out_total = out_total;
        a.silent_tile = noalloc_silent_tile();
        launch_frame_scan(a, lt, s);
    });
}
