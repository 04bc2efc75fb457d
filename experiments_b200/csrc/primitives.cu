// GPU primitives for sm_100a: fill, single-pass exclusive scan, one-launch LSD
// radix sort (8-bit digits) and bound search.
//
// Replaces the reference's OpenCL primitive objects:
//   btFillCL         BB/btFillCL.cpp:42-110,   PR/Fill/FillKernels.cl:47-96
//   btPrefixScanCL   BB/btPrefixScanCL.cpp:46-126, PR/Scan/PrefixScanKernels.cl:38-154
//   btRadixSort32CL  BB/btRadixSort32CL.cpp:161-535, PR/Sort/RadixSort32Kernels.cl:271,337,797
//   btBoundSearchCL  BB/btBoundSearchCL.cpp:78-136, PR/Search/BoundSearchKernels.cl:42-104
//
// Design: the reference sorts 4 bits per pass (8 passes x 3 kernels each,
// fixed 120 work-groups). Here a sort is one launch over 8 bits a pass: a
// resident grid of one block per SM, each block with a contiguous range of the
// keys. A pass counts the range's digits, meets the other blocks at a grid
// barrier, adds up the counts of the blocks before it, and then ranks its range
// tile by tile, staging each tile in shared memory in digit order so that the
// scatter writes contiguous runs. Sorts of up to 8,192 keys run in one block.
// Every wait is bounded; a wait that gives up sets *err_flag.
#include "b3_internal.h"

#include <algorithm>

namespace {

constexpr int kRadix = 256;
constexpr int kSortThreads = 1024;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortMaxBlocks = 256;
constexpr int kSortItems = 8;            // keys per thread of a tile at most
constexpr int kBlockSortMax = 8 * kSortThreads;  // the one-block sort

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

// An element count: on the device, or known at the launch (n_dev null).
__device__ __forceinline__ int dev_n(const int32_t* n_dev, int n) { return n_dev ? *n_dev : n; }

// Block-wide exclusive scan of one value per thread (blockDim = 256).
__device__ __forceinline__ uint32_t block_excl_scan_256(uint32_t v, uint32_t* warp_tot,
                                                         uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = (lane < 8) ? warp_tot[lane] : 0u;
        uint32_t s = t;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < 8) warp_tot[lane] = s - t;  // exclusive warp offsets
        if (lane == 7 && total) *total = s;
    }
    __syncthreads();
    uint32_t r = warp_tot[warp] + x - v;
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------------------
// Fill
// ---------------------------------------------------------------------------
__global__ void k_fill_u32(uint32_t* __restrict__ dst, uint32_t v, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = v;
}
__global__ void k_fill_int2(int2* __restrict__ dst, int2 v, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = v;
}

// ---------------------------------------------------------------------------
// Radix sort: keys and digits
// ---------------------------------------------------------------------------
// Key i of a sort input: split arrays hold the keys contiguously; the
// interleaved form (btSortData, BB/btRadixSort32CL.h:7-11) holds (key, value)
// pairs, key first.
template <bool kPairs>
__device__ __forceinline__ uint32_t sort_key(const uint32_t* __restrict__ keys, int64_t i) {
    if (kPairs) return reinterpret_cast<const uint2*>(keys)[i].x;
    return keys[i];
}

// Lanes of the warp with this lane's digit, of `bits` bits; a ballot per bit.
// (__match_any_sync in its place: 239 us instead of 195 for 4,194,304 pairs.)
__device__ __forceinline__ uint32_t same_digit(uint32_t d, int bits, uint32_t valid) {
    uint32_t peers = valid;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (b < bits) {
            const uint32_t m = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= (d >> b) & 1u ? m : ~m;
        }
    }
    return peers;
}

// Digit starts of a tile from its per-warp counts: cnt[w][d] becomes the keys of
// digit d in the warps before w, start[d] the keys of smaller digits; returns
// (to thread d) the tile's count of digit d.
__device__ __forceinline__ uint32_t tile_starts(uint16_t (*cnt)[kRadix], uint32_t* start, uint32_t* warp_tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t total = 0;
    if (threadIdx.x < kRadix) {
#pragma unroll 8
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = cnt[w][threadIdx.x];
            cnt[w][threadIdx.x] = (uint16_t)total;
            total += c;
        }
        uint32_t x = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[warp] = x;
        start[threadIdx.x] = x - total;
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
        uint32_t before = 0;
        for (int w = 0; w < warp; ++w) before += warp_tot[w];
        start[threadIdx.x] += before;
    }
    __syncthreads();
    return total;
}

// ---------------------------------------------------------------------------
// Radix sort over a resident grid
// ---------------------------------------------------------------------------
// One launch for all passes. What a pass costs beyond its 16 bytes a pair of
// traffic is the prefix over the blocks: with look-back over tiles (a kernel per
// pass) the walk through some 700 tiles in flight took 50 of 75 us at 4,194,304
// pairs; here it is one barrier and a sum over at most 148 rows of counts, for a
// second read of the keys, mostly from L2. Sorts of 32-bit pairs, before and now:
// 4,194,304 428 -> 195 us, 500,000 99 -> 54, 16,000,000 (24 bits) 1,063 -> 521,
// 20,000 (24 bits) 49 -> 28. What bounds it now is the ranking (some 190
// instructions a key and warp, schedulers 47 % busy between the tile's barriers);
// two blocks of 512 threads to an SM measured 202 us.
template <int kItems>
struct SortSmem {
    uint32_t stage[kSortThreads * kItems];  // a tile's keys in digit order, then its values
    uint16_t cnt[kSortWarps][kRadix];
    uint32_t start[kRadix];
    uint32_t next[kRadix];   // where the block's next key of each digit goes
    uint32_t base[kRadix];   // that, less the digit's start in the tile
    uint32_t part[kSortThreads];
    uint32_t warpTot[8];
};

struct SortArgs {
    const uint32_t *kin, *vin;
    uint32_t *kA, *vA, *kB, *vB;  // pass 0 writes A, pass 1 B, and so on
    const int32_t* n_dev;
    int n_host, key_bits;
    uint32_t* counts;             // [blocks][256]
    uint32_t* bar;
    int32_t* err;
};

// kPairs: the key pointers hold interleaved (key, value) pairs and the value
// pointers are unused.
template <bool kPairs, int kItems>
__global__ void __launch_bounds__(kSortThreads, 1) k_sort(SortArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortSmem<kItems>& S = *reinterpret_cast<SortSmem<kItems>*>(smem_raw);
    constexpr int kTile = kSortThreads * kItems;
    b3dev::GridBarrier barrier(A.bar, A.err, nullptr, b3dev::kSpinLimit, false);
    const int n = dev_n(A.n_dev, A.n_host);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool has_vals = kPairs || A.vin != nullptr;
    const uint32_t lt = b3dev::lanemask_lt();
    // the block's range: whole tiles while there are enough, else an even share
    const int blocks = (int)gridDim.x;
    int share = (n + blocks - 1) / blocks;
    share = (share + kSortThreads - 1) / kSortThreads * kSortThreads;
    const int r0 = (int)min((int64_t)n, (int64_t)share * blockIdx.x), r1 = (int)min((int64_t)n, (int64_t)r0 + share);
    const uint32_t *kin = A.kin, *vin = A.vin;
    for (int shift = 0, p = 0; shift < A.key_bits; shift += 8, ++p) {
        uint32_t* kout = (p & 1) ? A.kB : A.kA;
        uint32_t* vout = (p & 1) ? A.vB : A.vA;
        const int bits = min(8, A.key_bits - shift);
        const uint32_t mask = (1u << bits) - 1u;
        auto key_at = [&](int i) { return kPairs ? __ldcg(&reinterpret_cast<const uint2*>(kin)[i].x) : __ldcg(&kin[i]); };
        // the range's digit counts; a digit that the whole warp shares (the high
        // digits of cell keys) is counted once for it
        for (int d = t; d < kRadix; d += kSortThreads) S.next[d] = 0u;
        __syncthreads();
        for (int i0 = r0 + t; i0 - lane < r1; i0 += 4 * kSortThreads) {
            uint32_t k[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) k[u] = i0 + u * kSortThreads < r1 ? (key_at(i0 + u * kSortThreads) >> shift) & mask : kRadix;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t lead = __shfl_sync(0xffffffffu, k[u], 0);
                const bool same = __all_sync(0xffffffffu, k[u] == lead);
                if (k[u] < kRadix && (!same || lane == 0)) atomicAdd(&S.next[k[u]], same ? 32u : 1u);
            }
        }
        __syncthreads();
        if (t < kRadix) A.counts[(size_t)blockIdx.x * kRadix + t] = S.next[t];
        if (!barrier.wait()) return;
        // each digit's keys in all blocks and in those before this one: four rows
        // of threads, a quarter of the blocks each
        {
            const int d = t & (kRadix - 1), q = t / kRadix;
            uint32_t all = 0, mine = 0;
#pragma unroll 8
            for (int b = q; b < blocks; b += kSortThreads / kRadix) {
                const uint32_t c = __ldcg(&A.counts[(size_t)b * kRadix + d]);
                all += c;
                mine += b < (int)blockIdx.x ? c : 0u;
            }
            S.part[t] = mine;
            S.stage[t] = all;
            __syncthreads();
            uint32_t tot = 0, before = 0;
            if (t < kRadix) {
#pragma unroll
                for (int k = 0; k < kSortThreads / kRadix; ++k) {
                    tot += S.stage[k * kRadix + t];
                    before += S.part[k * kRadix + t];
                }
                uint32_t x = tot;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (lane == 31) S.warpTot[warp] = x;
                before += x - tot;
            }
            __syncthreads();
            if (t < kRadix) {
                for (int w = 0; w < warp; ++w) before += S.warpTot[w];
                S.next[t] = before;
            }
            __syncthreads();
        }
        for (int base = r0; base < r1; base += kTile) {
            const int m = min(kTile, r1 - base);
            // striped within each warp: lane l, item i -> w*32*I + i*32 + l
            const int first = warp * 32 * kItems + lane;
            uint32_t k[kItems], pos[kItems];
#pragma unroll
            for (int i = 0; i < kItems; ++i) k[i] = first + i * 32 < m ? key_at(base + first + i * 32) : 0xFFFFFFFFu;
            for (int d = lane; d < kRadix / 2; d += 32) reinterpret_cast<uint32_t*>(&S.cnt[warp][0])[d] = 0u;
            __syncwarp();
            // stable ranks within the warp
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                const bool valid = first + i * 32 < m;
                const uint32_t d = (k[i] >> shift) & mask;
                const uint32_t peers = same_digit(d, bits, __ballot_sync(0xffffffffu, valid));
                const uint32_t c = S.cnt[warp][d];
                pos[i] = c + __popc(peers & lt);
                __syncwarp();
                if (valid && (peers & lt) == 0u) S.cnt[warp][d] = (uint16_t)(c + __popc(peers));
                __syncwarp();
            }
            __syncthreads();
            const uint32_t tot = tile_starts(S.cnt, S.start, S.warpTot);
            if (t < kRadix) {
                S.base[t] = S.next[t] - S.start[t];
                S.next[t] += tot;
            }
            // the tile's keys in digit order; their values are fetched meanwhile
            uint32_t v[kItems];
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                const bool valid = first + i * 32 < m;
                const uint32_t d = (k[i] >> shift) & mask;
                pos[i] += S.start[d] + S.cnt[warp][d];
                if (valid) S.stage[pos[i]] = k[i];
                v[i] = 0u;
                if (has_vals && valid)
                    v[i] = kPairs ? __ldcg(&reinterpret_cast<const uint2*>(kin)[base + first + i * 32].y)
                                  : __ldcg(&vin[base + first + i * 32]);
            }
            __syncthreads();
            // scatter contiguous digit runs: the keys, then the values through the
            // same buffer
            uint32_t dst[kItems], key[kItems];
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                const int j = i * kSortThreads + t;
                if (j < m) {
                    key[i] = S.stage[j];
                    dst[i] = S.base[(key[i] >> shift) & mask] + j;
                    if (!kPairs) kout[dst[i]] = key[i];
                }
            }
            __syncthreads();
            if (has_vals) {
#pragma unroll
                for (int i = 0; i < kItems; ++i)
                    if (first + i * 32 < m) S.stage[pos[i]] = v[i];
                __syncthreads();
#pragma unroll
                for (int i = 0; i < kItems; ++i) {
                    const int j = i * kSortThreads + t;
                    if (j < m) {
                        if (kPairs) reinterpret_cast<uint2*>(kout)[dst[i]] = make_uint2(key[i], S.stage[j]);
                        else vout[dst[i]] = S.stage[j];
                    }
                }
                __syncthreads();
            }
        }
        kin = kout;
        vin = vout;
        if (shift + 8 < A.key_bits && !barrier.wait()) return;
    }
}

// ---------------------------------------------------------------------------
// Radix sort of up to kBlockSortMax keys: every pass in one block
// ---------------------------------------------------------------------------
// A pass over a few thousand keys is all latency; here it is a ranking and an
// exchange through shared memory, without barriers between blocks (4,000 pairs
// of 16 bits 33 -> 14 us, launches included).
template <int kItems>
struct BlockSortSmem {
    uint32_t keys[kSortThreads * kItems];
    uint32_t vals[kSortThreads * kItems];
    uint16_t cnt[kSortWarps][kRadix];
    uint32_t start[kRadix];
    uint32_t warpTot[8];
};
template <bool kPairs, int kItems>
__global__ void __launch_bounds__(kSortThreads)
k_block_sort(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
             const int32_t* n_dev, int n_host, int key_bits) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BlockSortSmem<kItems>& S = *reinterpret_cast<BlockSortSmem<kItems>*>(smem_raw);
    const int n = min(dev_n(n_dev, n_host), kSortThreads * kItems);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool has_vals = kPairs || vals_in != nullptr;
    const uint32_t lt = b3dev::lanemask_lt();
    const int first = warp * 32 * kItems + lane;
    uint32_t k[kItems], v[kItems], rank[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const int idx = first + i * 32;
        k[i] = 0xFFFFFFFFu;
        v[i] = 0u;
        if (idx < n) {
            if (kPairs) {
                const uint2 kv = reinterpret_cast<const uint2*>(keys_in)[idx];
                k[i] = kv.x;
                v[i] = kv.y;
            } else {
                k[i] = keys_in[idx];
                if (has_vals) v[i] = vals_in[idx];
            }
        }
    }
    for (int shift = 0; shift < key_bits; shift += 8) {
        const int bits = min(8, key_bits - shift);
        const uint32_t mask = (1u << bits) - 1u;
        for (int d = lane; d < kRadix / 2; d += 32) reinterpret_cast<uint32_t*>(&S.cnt[warp][0])[d] = 0u;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            const bool valid = first + i * 32 < n;
            const uint32_t d = (k[i] >> shift) & mask;
            const uint32_t peers = same_digit(d, bits, __ballot_sync(0xffffffffu, valid));
            const uint32_t base = S.cnt[warp][d];
            rank[i] = base + __popc(peers & lt);
            __syncwarp();
            if (valid && (peers & lt) == 0u) S.cnt[warp][d] = (uint16_t)(base + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        tile_starts(S.cnt, S.start, S.warpTot);
#pragma unroll
        for (int i = 0; i < kItems; ++i)
            if (first + i * 32 < n) {
                const uint32_t d = (k[i] >> shift) & mask;
                const uint32_t pos = S.start[d] + S.cnt[warp][d] + rank[i];
                S.keys[pos] = k[i];
                S.vals[pos] = v[i];
            }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kItems; ++i)
            if (first + i * 32 < n) {
                k[i] = S.keys[first + i * 32];
                v[i] = S.vals[first + i * 32];
            }
    }
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const int idx = first + i * 32;
        if (idx < n) {
            if (kPairs) {
                reinterpret_cast<uint2*>(keys_out)[idx] = make_uint2(k[i], v[i]);
            } else {
                keys_out[idx] = k[i];
                if (has_vals) vals_out[idx] = v[i];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Exclusive scan with decoupled look-back
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kScanThreads)
k_scan_u32(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, const int32_t* n_dev, int n_host,
           unsigned long long* __restrict__ status, int32_t* __restrict__ tile_counter,
           uint32_t* __restrict__ d_total, int32_t* __restrict__ err_flag) {
    __shared__ uint32_t sm[kScanTile + kScanTile / 32];
    __shared__ uint32_t warp_tot[8];
    __shared__ uint32_t tile_excl;
    __shared__ int tile_sh;
    const int n = dev_n(n_dev, n_host);
    const int num_tiles = (n + kScanTile - 1) / kScanTile;
    const unsigned long long FA = 1ull << 32, FP = 2ull << 32;
    if (n <= 0 && blockIdx.x == 0 && threadIdx.x == 0 && d_total) *d_total = 0;
    for (;;) {
        if (threadIdx.x == 0) tile_sh = atomicAdd(tile_counter, 1);
        __syncthreads();
        const int tile = tile_sh;
        if (tile >= num_tiles) break;
        const int64_t base = (int64_t)tile * kScanTile;
        const int tn = (int)min((int64_t)kScanTile, (int64_t)n - base);
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            const int j = i * kScanThreads + threadIdx.x;
            sm[j + j / 32] = (j < tn) ? src[base + j] : 0u;
        }
        __syncthreads();
        uint32_t loc[kScanItems];
        uint32_t run = 0;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            const int j = threadIdx.x * kScanItems + i;
            loc[i] = run;
            run += sm[j + j / 32];
        }
        const uint32_t texcl = block_excl_scan_256(run, warp_tot, nullptr);
        if (threadIdx.x == kScanThreads - 1) warp_tot[0] = texcl + run;  // tile aggregate
        __syncthreads();
        const uint32_t agg = warp_tot[0];
        // one warp looks back, 32 preceding tiles at a time
        if (threadIdx.x < 32) {
            unsigned long long* my = status + tile;
            const int lane = threadIdx.x;
            uint32_t excl = 0;
            if (lane == 0) b3dev::st_release_u64(my, (tile == 0 ? FP : FA) | agg);
            int t = tile - 1, spins = 0;
            while (t >= 0) {
                const unsigned long long s = t - lane >= 0 ? b3dev::ld_acquire_u64(status + t - lane) : FP;
                const unsigned missing = __ballot_sync(0xffffffffu, (s >> 32) == 0);
                const unsigned whole = __ballot_sync(0xffffffffu, (s >> 32) == 2);
                // tiles up to the nearest inclusive prefix, and before a missing one
                const int stop = whole ? __ffs(whole) - 1 : 31;
                const int gap = missing ? __ffs(missing) - 1 : 32;
                const int use = min(stop + 1, gap);
                excl += __reduce_add_sync(0xffffffffu, lane < use ? (uint32_t)s : 0u);
                if (use == stop + 1 && whole) break;
                t -= use;
                if (use == 0 && ++spins > b3dev::kSpinLimit) {
                    if (lane == 0) atomicExch(err_flag, 1);
                    break;
                }
            }
            if (lane == 0) {
                if (tile > 0) b3dev::st_release_u64(my, FP | (unsigned long long)(uint32_t)(excl + agg));
                tile_excl = excl;
                if (tile == num_tiles - 1 && d_total) *d_total = excl + agg;
            }
        }
        __syncthreads();
        const uint32_t off = tile_excl + texcl;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            const int j = threadIdx.x * kScanItems + i;
            sm[j + j / 32] = off + loc[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            const int j = i * kScanThreads + threadIdx.x;
            if (j < tn) dst[base + j] = sm[j + j / 32];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Bound search over sorted keys
// ---------------------------------------------------------------------------
// kPairs: the sorted input is interleaved (key, value) pairs (btSortData).
template <bool kPairs>
__global__ void k_bound_lower(const uint32_t* __restrict__ keys, const int32_t* n_dev, int n_host,
                              uint32_t* __restrict__ dst, int64_t n_dst) {
    const int n = dev_n(n_dev, n_host);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t k = sort_key<kPairs>(keys, i);
        if ((i == 0 || sort_key<kPairs>(keys, i - 1) != k) && k < (uint64_t)n_dst) dst[k] = (uint32_t)i;
    }
}
// kPairs also follows SearchSortDataUpperKernel (PR/Search/BoundSearchKernels.cl:66-86)
// where no key 0 is present: its first work item compares the first key
// with 0 and writes dst[0] = 0.
template <bool kPairs>
__global__ void k_bound_upper(const uint32_t* __restrict__ keys, const int32_t* n_dev, int n_host,
                              uint32_t* __restrict__ dst, int64_t n_dst) {
    const int n = dev_n(n_dev, n_host);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t k = sort_key<kPairs>(keys, i);
        if ((i == n - 1 || sort_key<kPairs>(keys, i + 1) != k) && k < (uint64_t)n_dst) dst[k] = (uint32_t)(i + 1);
        if (kPairs && i == 0 && k != 0u && n_dst > 0) dst[0] = 0u;
    }
}
template <bool kPairs>
__global__ void k_bound_count(const uint32_t* __restrict__ keys, const int32_t* n_dev, int n_host,
                              uint32_t* __restrict__ dst, int64_t n_dst) {
    const int n = dev_n(n_dev, n_host);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t k = sort_key<kPairs>(keys, i);
        if ((i == 0 || sort_key<kPairs>(keys, i - 1) != k) && k < (uint64_t)n_dst) {
            int64_t j = i;
            // run length by binary search for the first index with a larger key
            int64_t lo = i + 1, hi = n;
            while (lo < hi) {
                int64_t mid = (lo + hi) >> 1;
                if (sort_key<kPairs>(keys, mid) == k) lo = mid + 1; else hi = mid;
            }
            dst[k] = (uint32_t)(lo - j);
        }
    }
}

int grid_for(int64_t n, int threads, int numSMs, int perSM = 8) {
    int64_t g = (n + threads - 1) / threads;
    g = std::max<int64_t>(1, std::min<int64_t>(g, (int64_t)numSMs * perSM));
    return (int)g;
}

}  // namespace

namespace b3 {

static inline int sort_passes(int key_bits) { return (key_bits + 7) / 8; }

size_t radix_scratch_bytes(int64_t n_max, int key_bits) {
    (void)n_max;
    (void)key_bits;
    // [grid barrier, 256 B][digit counts per block]
    return 256 + (size_t)kSortMaxBlocks * kRadix * 4;
}

// Large dynamic shared memory of a kernel, opted in once per device.
static int allow_smem(const void* kern, size_t smem) {
    if (smem > 48 * 1024) B3_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return B3_OK;
}

template <bool kPairs, int kItems>
static int block_sort(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, const int32_t* n_dev,
                      int n, int key_bits, cudaStream_t st) {
    const size_t smem = sizeof(BlockSortSmem<kItems>);
    B3_TRY(allow_smem((const void*)k_block_sort<kPairs, kItems>, smem));
    k_block_sort<kPairs, kItems><<<1, kSortThreads, smem, st>>>(kin, vin, kout, vout, n_dev, n, key_bits);
    B3_CHECK_LAUNCH();
    return B3_OK;
}

// Sorts that fit one block; the result goes straight to kout / vout, which may
// be the input.
static bool fits_block(int64_t n_max) { return n_max <= kBlockSortMax; }
template <bool kPairs>
static int block_sort_any(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout,
                          const int32_t* n_dev, int64_t n_max, int key_bits, cudaStream_t st) {
    if (key_bits < 1 || key_bits > 32) return B3_ERR_INVALID_ARG;
    if (n_max <= 0) return B3_OK;
    const int n = (int)n_max;
    if (n <= 1 * kSortThreads) return block_sort<kPairs, 1>(kin, vin, kout, vout, n_dev, n, key_bits, st);
    if (n <= 2 * kSortThreads) return block_sort<kPairs, 2>(kin, vin, kout, vout, n_dev, n, key_bits, st);
    if (n <= 4 * kSortThreads) return block_sort<kPairs, 4>(kin, vin, kout, vout, n_dev, n, key_bits, st);
    return block_sort<kPairs, 8>(kin, vin, kout, vout, n_dev, n, key_bits, st);
}

template <bool kPairs, int kItems>
static int sort_grid(SortArgs& A, int64_t n_expect, cudaStream_t st, int numSMs) {
    const size_t smem = sizeof(SortSmem<kItems>);
    const void* kern = (const void*)k_sort<kPairs, kItems>;
    B3_TRY(allow_smem(kern, smem));
    const int64_t want = std::max<int64_t>(1, (n_expect + kSortThreads - 1) / kSortThreads);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min<int64_t>(want, std::min(numSMs, kSortMaxBlocks)));
    cfg.blockDim = dim3(kSortThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {&A};
    B3_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
    return B3_OK;
}

// Passes of one sort: pass 0 reads (kin, vin) and writes buffer A, pass 1
// reads A and writes B, and so on; the result is in A when the pass count
// is odd, else in B. The input may be A or B itself (in-place sorts). A block's
// threads take as many keys each as an even share of the likely count gives
// them, up to 8: more would leave warps of a short range idle.
template <bool kPairs>
static int radix_sort_core(const uint32_t* kin, const uint32_t* vin, uint32_t* kA, uint32_t* vA, uint32_t* kB,
                           uint32_t* vB, const int32_t* n_dev, int64_t n_max, int64_t n_expect, int key_bits,
                           void* scratch, size_t scratch_bytes, int32_t* err_flag, cudaStream_t st, int numSMs,
                           bool cleared = false) {
    if (key_bits < 1 || key_bits > 32) return B3_ERR_INVALID_ARG;
    if (scratch_bytes < radix_scratch_bytes(n_max, key_bits)) return B3_ERR_CAPACITY;
    if (n_max <= 0) return B3_OK;
    if (!cleared) B3_CUDA(cudaMemsetAsync(scratch, 0, 16, st));
    SortArgs A = {kin, vin, kA, vA, kB, vB, n_dev, (int)n_max, key_bits,
                  reinterpret_cast<uint32_t*>((unsigned char*)scratch + 256), (uint32_t*)scratch, err_flag};
    const int64_t each = n_expect / ((int64_t)numSMs * kSortThreads);
    if (each < 1) return sort_grid<kPairs, 1>(A, n_expect, st, numSMs);
    if (each < 2) return sort_grid<kPairs, 2>(A, n_expect, st, numSMs);
    if (each < 4) return sort_grid<kPairs, 4>(A, n_expect, st, numSMs);
    return sort_grid<kPairs, kSortItems>(A, n_expect, st, numSMs);
}

bool radix_result_in_alt(int64_t n_max, int key_bits) { return !fits_block(n_max) && (sort_passes(key_bits) & 1) != 0; }

int radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt,
                     const int32_t* n_dev, int64_t n_max, int key_bits, void* scratch,
                     size_t scratch_bytes, int32_t* err_flag, cudaStream_t st, bool* result_in_alt,
                     int numSMs, int64_t n_expect, bool cleared) {
    *result_in_alt = radix_result_in_alt(n_max, key_bits);
    if (fits_block(n_max)) return block_sort_any<false>(keys, vals, keys, vals, n_dev, n_max, key_bits, st);
    return radix_sort_core<false>(keys, vals, keys_alt, vals ? vals_alt : nullptr, keys, vals, n_dev, n_max,
                                  n_expect > 0 ? n_expect : n_max, key_bits, scratch, scratch_bytes, err_flag, st,
                                  numSMs, cleared);
}

int radix_sort_kv_out(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                      uint32_t* keys_tmp, uint32_t* vals_tmp, const int32_t* n_dev, int64_t n_max, int key_bits,
                      void* scratch, size_t scratch_bytes, int32_t* err_flag, cudaStream_t st, int numSMs,
                      bool cleared) {
    if (fits_block(n_max))
        return block_sort_any<false>(keys_in, vals_in, keys_out, vals_out, n_dev, n_max, key_bits, st);
    // the first pass writes the buffer that makes the last pass land in out
    const bool odd = (sort_passes(key_bits) & 1) != 0;
    uint32_t* kA = odd ? keys_out : keys_tmp;
    uint32_t* vA = odd ? vals_out : vals_tmp;
    uint32_t* kB = odd ? keys_tmp : keys_out;
    uint32_t* vB = odd ? vals_tmp : vals_out;
    return radix_sort_core<false>(keys_in, vals_in, kA, vals_in ? vA : nullptr, kB, vals_in ? vB : nullptr,
                                  n_dev, n_max, n_max, key_bits, scratch, scratch_bytes, err_flag, st, numSMs,
                                  cleared);
}

int radix_sort_interleaved(uint2* kv, uint2* kv_alt, const int32_t* n_dev, int64_t n_max, int key_bits,
                           void* scratch, size_t scratch_bytes, int32_t* err_flag, cudaStream_t st,
                           bool* result_in_alt, int numSMs, bool cleared) {
    uint32_t* a = reinterpret_cast<uint32_t*>(kv_alt);
    uint32_t* b = reinterpret_cast<uint32_t*>(kv);
    *result_in_alt = radix_result_in_alt(n_max, key_bits);
    if (fits_block(n_max)) return block_sort_any<true>(b, nullptr, b, nullptr, n_dev, n_max, key_bits, st);
    return radix_sort_core<true>(b, nullptr, a, nullptr, b, nullptr, n_dev, n_max, n_max, key_bits, scratch,
                                 scratch_bytes, err_flag, st, numSMs, cleared);
}

size_t scan_scratch_bytes(int64_t n_max) {
    const int64_t tiles = std::max<int64_t>(1, (n_max + kScanTile - 1) / kScanTile);
    return 256 + (size_t)tiles * 8;
}

int exclusive_scan_u32(const uint32_t* src, uint32_t* dst, const int32_t* n_dev, int64_t n_max,
                       uint32_t* d_total, void* scratch, size_t scratch_bytes, int32_t* err_flag,
                       cudaStream_t st, int numSMs, bool cleared) {
    const size_t need = scan_scratch_bytes(n_max);
    if (scratch_bytes < need) return B3_ERR_CAPACITY;
    if (!cleared) B3_CUDA(cudaMemsetAsync(scratch, 0, need, st));
    int32_t* counter = (int32_t*)scratch;
    unsigned long long* status = (unsigned long long*)((unsigned char*)scratch + 256);
    if (n_max <= 0) {
        if (d_total) B3_CUDA(cudaMemsetAsync(d_total, 0, sizeof(uint32_t), st));
        return B3_OK;
    }
    const int64_t tiles = std::max<int64_t>(1, (n_max + kScanTile - 1) / kScanTile);
    int occ = 1;
    B3_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_scan_u32, kScanThreads, 0));
    occ = std::max(1, occ);
    const int grid = (int)std::min<int64_t>(tiles, (int64_t)numSMs * occ);
    k_scan_u32<<<grid, kScanThreads, 0, st>>>(src, dst, n_dev, (int)n_max, status, counter, d_total, err_flag);
    B3_CHECK_LAUNCH();
    return B3_OK;
}

int fill_u32(uint32_t* dst, uint32_t v, int64_t n, cudaStream_t st) {
    if (n <= 0) return B3_OK;
    k_fill_u32<<<grid_for(n, 256, 148, 16), 256, 0, st>>>(dst, v, n);
    B3_CHECK_LAUNCH();
    return B3_OK;
}

template <bool kPairs>
static int bound_search_t(const uint32_t* keys, const int32_t* n_dev, int64_t n_max, uint32_t* dst,
                          int64_t n_dst, int mode, cudaStream_t st) {
    if (n_max <= 0) return B3_OK;
    const int g = grid_for(n_max, 256, 148, 16);
    if (mode == 0) k_bound_lower<kPairs><<<g, 256, 0, st>>>(keys, n_dev, (int)n_max, dst, n_dst);
    else if (mode == 1) k_bound_upper<kPairs><<<g, 256, 0, st>>>(keys, n_dev, (int)n_max, dst, n_dst);
    else k_bound_count<kPairs><<<g, 256, 0, st>>>(keys, n_dev, (int)n_max, dst, n_dst);
    B3_CHECK_LAUNCH();
    return B3_OK;
}

int bound_search(const uint32_t* keys, const int32_t* n_dev, int64_t n_max, uint32_t* dst,
                 int64_t n_dst, int mode, cudaStream_t st) {
    return bound_search_t<false>(keys, n_dev, n_max, dst, n_dst, mode, st);
}

int bound_search_interleaved(const uint2* kv, const int32_t* n_dev, int64_t n_max, uint32_t* dst, int64_t n_dst,
                             int mode, cudaStream_t st) {
    return bound_search_t<true>(reinterpret_cast<const uint32_t*>(kv), n_dev, n_max, dst, n_dst, mode, st);
}

int fill_int2(int2* dst, int2 v, int64_t n, cudaStream_t st) {
    if (n <= 0) return B3_OK;
    k_fill_int2<<<grid_for(n, 256, 148, 16), 256, 0, st>>>(dst, v, n);
    B3_CHECK_LAUNCH();
    return B3_OK;
}

}  // namespace b3
