// sort.cu -- stable LSD radix sort of (Morton key, body id) pairs.
//
// Replaces the third-party webgpu-radix-sort@1.0.7 kernel that the reference
// dispatches at src/simulation.ts:400 (constructed at :132-140 with
// bit_count 32 over mortonCodes/bodyIndices).  The contract is the stable
// sort by key: equal keys keep ascending body id, which the index tie-break of
// the hierarchy build (lbvh.wgsl:78-80) then turns into a unique tree.
//
// Design (onesweep, one kernel per 8-bit digit):
//  - The digit histograms of every pass come from the encode kernel, so each
//    pass reads its keys exactly once.
//  - A CTA takes the next tile (512 threads x sort_items keys) from an atomic
//    counter (so lower tiles are always already running), ranks its keys warp
//    by warp (stable: item-major, lane-minor = memory order), publishes its
//    per-digit counts, stages the tile in shared memory in digit order, and
//    then resolves its global offsets by a decoupled look-back over the tiles
//    before it, several tiles per round trip.  The look-back spin is bounded;
//    on giving up it raises kErrLookbackSpin instead of hanging.
//  - Staged keys and ids are written out in runs, so global stores are
//    contiguous per digit.
//  - Pass 0 does not read ids: it writes the identity permutation of
//    lbvh.wgsl:68 directly.
//  - The passes alternate between two buffers and end in the public codes /
//    ids (an odd number of passes, ensembles only, starts in the others).
//
// What bounds it: shared-memory wavefronts and the chain of a tile's phases, not
// memory (16.8M 64-bit keys: 2.9 TB/s; wider look-backs, smaller tiles with
// more CTAs per SM and larger ones with fewer were all slower).  The ranking was
// half of 165 instructions a warp and 32 keys while it found a digit's lanes by
// eight ballots; now they meet in a mask in shared memory.  All passes before
// -> now: 800k 53 -> 43 us, ensembles' 5 passes of 1.2M keys 89 -> 74, 3M 127 ->
// 104, 64-bit keys 16.8M 1.20 -> 1.10 ms.
#include <cuda/atomic>

#include "bh_internal.cuh"

namespace bh {

constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kFlagMask = 3u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1;
#ifndef BH_SORT_LOOK_BATCH
#define BH_SORT_LOOK_BATCH 4
#endif
constexpr int kLookBatch = BH_SORT_LOOK_BATCH;  // predecessor tiles read per look-back round

// Exclusive scans of two values over the block's 256 digit threads (threads
// past them pass 0, so the digits' prefixes are unaffected by them).
__device__ __forceinline__ uint2 block_excl_scan2(uint32_t a, uint32_t b, uint2* s_tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = a, y = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, o), v = __shfl_up_sync(0xFFFFFFFFu, y, o);
        if (lane >= o) {
            x += u;
            y += v;
        }
    }
    if (lane == 31) s_tot[warp] = make_uint2(x, y);
    __syncthreads();
    uint32_t bx = 0, by = 0;
#pragma unroll
    for (int w = 0; w < kRadix / 32; ++w)
        if (w < warp) {
            const uint2 t = s_tot[w];
            bx += t.x;
            by += t.y;
        }
    return make_uint2(bx + x - a, by + y - b);
}

#ifndef BH_SORT_MIN_BLOCKS
#define BH_SORT_MIN_BLOCKS 2
#endif

template <typename K, int kSortItems, bool FIRST>
__global__ void __launch_bounds__(kSortThreads, BH_SORT_MIN_BLOCKS)
onesweep_kernel(const K* __restrict__ keys_in, const uint32_t* __restrict__ ids_in,
                K* __restrict__ keys_out, uint32_t* __restrict__ ids_out, uint32_t n, int pass,
                StepScratch* __restrict__ scratch, uint32_t* __restrict__ status, uint32_t tiles,
                uint32_t* __restrict__ err, uint32_t spin_cap, uint32_t debug_flags) {
    wait_previous_kernel();
    constexpr int W = kSortThreads / 32;
    constexpr int kSortTile = kSortThreads * kSortItems;
    __shared__ uint32_t s_whist[W][kRadix];  // a warp's counts, then its first places
    __shared__ uint32_t s_gbase[kRadix];
    __shared__ uint2 s_tot[W];
    __shared__ uint32_t s_tile;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    K* s_keys = reinterpret_cast<K*>(s_dyn);
    uint32_t* s_ids = reinterpret_cast<uint32_t*>(s_keys + kSortTile);
    // While ranking, the lanes that hold each digit.  (In memory of its own it
    // took L1 from the walks of other handles that start beside a sort: three
    // in rotation 8.71 against 8.16 ms a step at 16.8M bodies.)
    uint32_t(*s_mask)[kRadix] = reinterpret_cast<uint32_t(*)[kRadix]>(s_dyn);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(&scratch->tile_ctr[pass], 1u);
    for (int i = lane; i < kRadix; i += 32) {
        s_whist[warp][i] = 0;
        s_mask[warp][i] = 0;
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t seg = tile * kSortTile + (uint32_t)warp * 32u * kSortItems;
    const int shift = pass * kRadixBits;

    K key[kSortItems];
    uint32_t id[kSortItems];
    uint32_t rank[(kSortItems + 1) / 2];  // two 16-bit ranks each
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        uint32_t idx = seg + (uint32_t)k * 32u + (uint32_t)lane;
        // Places past the end get the largest key: they rank last in the last
        // tile, and nothing reads that tile's counts.
        key[k] = ~(K)0;
        if (idx < n) key[k] = keys_in[idx];
    }
    // Warp-local stable ranking: the lanes with a digit meet in its mask.  (Two
    // ranks a register, ids loaded afterwards: with 64-bit keys all three spill.)
    const unsigned me = 1u << lane;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t d = (uint32_t)(key[k] >> shift) & 0xFFu;
        atomicOr(&s_mask[warp][d], me);
        __syncwarp();
        const unsigned peers = s_mask[warp][d];
        const uint32_t base = s_whist[warp][d];
        __syncwarp();
        const uint32_t below = __popc(peers & (me - 1u));
        rank[k / 2] = k & 1 ? rank[k / 2] | (base + below) << 16 : base + below;
        if (below == 0) {  // the lowest of them
            s_mask[warp][d] = 0;
            s_whist[warp][d] = base + (uint32_t)__popc(peers);
        }
        __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t idx = seg + (uint32_t)k * 32u + (uint32_t)lane;
        id[k] = FIRST ? idx : idx < n ? ids_in[idx] : 0u;
    }
    __syncthreads();
    // Per digit (threads 0..255): exclusive prefix over warps, and the tile's count.
    static_assert(kSortThreads >= kRadix && kSortThreads % 32 == 0, "one thread per digit");
    const bool digit_thread = tid < kRadix;
    const uint32_t d = digit_thread ? (uint32_t)tid : 0u;
    uint32_t tile_cnt = 0;
    if (digit_thread) {
#pragma unroll
        for (int w = 0; w < W; ++w) tile_cnt += s_whist[w][d];
    }
    // Publish this tile's aggregate (or inclusive prefix for tile 0).
    uint32_t* my_status = status + ((size_t)pass * tiles + tile) * kRadix;
    if (digit_thread) {
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> a(my_status[d]);
        a.store((tile == 0 ? kFlagPrefix : kFlagAggregate) | tile_cnt, cuda::memory_order_relaxed);
    }
    const uint2 before = block_excl_scan2(tile_cnt, digit_thread ? scratch->hist[pass][d] : 0u, s_tot);
    const uint32_t tile_excl = before.x, glob_excl = before.y;
    if (digit_thread) {
        uint32_t run = tile_excl;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t c = s_whist[w][d];
            s_whist[w][d] = run;
            run += c;
        }
    }
    __syncthreads();
    // Stage in digit order before the look-back: the tile's own work is done
    // while the tiles before it finish theirs, so the walk back is shorter.
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t p = s_whist[warp][(uint32_t)(key[k] >> shift) & 0xFFu] + (k & 1 ? rank[k / 2] >> 16 : rank[k / 2] & 0xFFFFu);
        s_keys[p] = key[k];
        s_ids[p] = id[k];
    }
    // Decoupled look-back over earlier tiles, one digit per thread, reading
    // kLookBatch tiles per round trip (nearest first): the values are used up
    // to the first inclusive prefix, and re-read from the first tile that has
    // not published yet.
    uint32_t excl = 0;
    if (tile > 0 && digit_thread) {
        uint32_t* st = status + (size_t)pass * tiles * kRadix + d;
        int t = (int)tile - 1;
        uint32_t spins = 0;
        while (true) {
            uint32_t v[kLookBatch];
#pragma unroll
            for (int j = 0; j < kLookBatch; ++j) {
                v[j] = kFlagPrefix;  // below tile 0: never used
                if (t - j >= 0) {
                    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> a(st[(size_t)(t - j) * kRadix]);
                    v[j] = a.load(cuda::memory_order_relaxed);
                }
            }
            // Test hook: tile 1 of the first pass never sees its only
            // predecessor, tile 0 (entry j = 0), publish.
            if (FIRST && (debug_flags & kDebugLookbackUnpublished) && tile == 1u) v[0] = 0u;
            bool done = false;
            int used = 0;
#pragma unroll
            for (int j = 0; j < kLookBatch; ++j) {
                if (done || used < j || (v[j] & kFlagMask) == 0u) continue;
                excl += v[j] & kValueMask;
                used = j + 1;
                done = (v[j] & kFlagMask) == kFlagPrefix || t - j == 0;
            }
            if (done) break;
            t -= used;
            if (used == 0) {
                if (++spins > spin_cap) {
                    atomicOr(err, kErrLookbackSpin);
                    break;
                }
                if (spins > 64) __nanosleep(64);
            }
        }
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> a(my_status[d]);
        a.store(kFlagPrefix | (excl + tile_cnt), cuda::memory_order_relaxed);
    }
    // (place in the tile to place in the output: one wrapping addition)
    if (digit_thread) s_gbase[d] = glob_excl + excl - tile_excl;
    __syncthreads();
    const uint32_t tile_base = tile * kSortTile;
    const uint32_t tile_n = (n - tile_base) < (uint32_t)kSortTile ? (n - tile_base) : (uint32_t)kSortTile;
    for (uint32_t i = (uint32_t)tid; i < tile_n; i += kSortThreads) {
        K kk = s_keys[i];
        uint32_t dd = (uint32_t)(kk >> shift) & 0xFFu;
        uint32_t dst = s_gbase[dd] + i;
        // Offsets are in range unless a look-back gave up; never write outside.
        if (dst < n) {
            keys_out[dst] = kk;
            ids_out[dst] = s_ids[i];
        } else {
            atomicOr(err, kErrLookbackSpin);
        }
    }
}

// One pass per key byte, or fewer when the high bytes are
// known to be zero (ensemble keys: system id above a 32-bit Morton code).
int sort_passes(const DeviceBuffers& b) { return b.sort_passes > 0 ? b.sort_passes : b.key_bytes; }

// Keys per thread.  Many keys keep a large sort's tiles (and its look-back) few;
// a small one has fewer tiles than SMs, so it lasts as long as one tile: short
// tiles below 450k keys.  All passes, 12 / 6 / 3 / 2 keys (us): 2k bodies
// 31 / 21 / 18 / 16, 16k 33 / 25 / 23 / 20, 100k 35 / 29 / 27 / 27, 400k
// 41 / 36 / 39 / 49, 500k 41 / 40 / 44 / 57, 800k 45 / 46 / 62 / 77; 64-bit keys
// 100k 78 / 60 / 51 / 52, 300k 86 / 68 / 70 / 76, 600k 94 / 88 / 107 / 128.
constexpr int kSmallItems = 3, kLargeItems = 12;
constexpr uint32_t kSmallSort = 450000;
static int sort_items(uint32_t n) { return n < kSmallSort ? kSmallItems : kLargeItems; }
uint32_t sort_tiles(uint32_t n) {
    const uint32_t tile = (uint32_t)(kSortThreads * sort_items(n));
    return (uint32_t)(((uint64_t)n + tile - 1) / tile);
}

// Dynamic shared memory: the staged tile, and before it the digit masks.
template <typename K, int ITEMS>
constexpr size_t sort_smem() {
    const size_t tile = (size_t)kSortThreads * ITEMS * (sizeof(K) + sizeof(uint32_t));
    const size_t masks = (size_t)(kSortThreads / 32) * kRadix * sizeof(uint32_t);
    return tile > masks ? tile : masks;
}

template <typename K, int ITEMS>
static void sort_impl(const DeviceBuffers& b, cudaStream_t s) {
    const size_t smem = sort_smem<K, ITEMS>();
    const int passes = sort_passes(b);
    const bool odd = passes & 1;  // the last pass writes codes / ids
    K* kin = (K*)sort_input(b);
    K* kout = (K*)(odd ? b.codes : b.codes_alt);
    uint32_t* iin = odd ? b.ids_alt : b.ids;
    uint32_t* iout = odd ? b.ids : b.ids_alt;
    for (int p = 0; p < passes; ++p) {
        if (p == 0)
            launch_chained(onesweep_kernel<K, ITEMS, true>, b.tiles, kSortThreads, smem, s, (const K*)kin, (const uint32_t*)nullptr, kout, iout, b.n, p, b.scratch, b.status, b.tiles, b.err, b.spin_cap,
                b.debug_flags);
        else
            launch_chained(onesweep_kernel<K, ITEMS, false>, b.tiles, kSortThreads, smem, s, (const K*)kin, (const uint32_t*)iin, kout, iout, b.n, p, b.scratch, b.status, b.tiles, b.err, b.spin_cap,
                b.debug_flags);
        K* tk = kin; kin = kout; kout = tk;
        uint32_t* ti = iin; iin = iout; iout = ti;
    }
}

template <typename K, int ITEMS>
static cudaError_t set_sort_attributes() {
    const int smem = (int)sort_smem<K, ITEMS>();
    cudaError_t e = cudaFuncSetAttribute(onesweep_kernel<K, ITEMS, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(onesweep_kernel<K, ITEMS, false>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

// Opt the sort kernels into more than 48 KB of dynamic shared memory on the
// current device (called once per device before any launch or capture).
cudaError_t sort_init_attributes() {
    cudaError_t e;
    if ((e = set_sort_attributes<uint32_t, kLargeItems>()) != cudaSuccess) return e;
    if ((e = set_sort_attributes<uint64_t, kLargeItems>()) != cudaSuccess) return e;
    if ((e = set_sort_attributes<uint32_t, kSmallItems>()) != cudaSuccess) return e;
    return set_sort_attributes<uint64_t, kSmallItems>();
}

void launch_sort(const DeviceBuffers& b, cudaStream_t s) {
    if (b.n == 0) return;
    const bool small = sort_items(b.n) == kSmallItems;
    if (b.key_bytes == 8) {
        if (small) sort_impl<uint64_t, kSmallItems>(b, s);
        else sort_impl<uint64_t, kLargeItems>(b, s);
    } else {
        if (small) sort_impl<uint32_t, kSmallItems>(b, s);
        else sort_impl<uint32_t, kLargeItems>(b, s);
    }
}

}  // namespace bh
