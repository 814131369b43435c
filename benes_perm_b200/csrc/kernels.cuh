// SPDX-License-Identifier: Apache-2.0
//
// sm_100a kernels of the compact encoder.
//
// Level kernels (global memory) run one routing level over every node of
// the level at once; they are used while nodes are larger than a tile.
// The tile kernel (tile.cuh) takes one node per CTA into shared memory and
// finishes its whole subtree there, down to the middle-group ranks.
//
// Per internal node and level (src/benes.cpp:226-315):
//   inverse      inv[p[i]] = i (node-local)
//   union        one parity union per output pair (inv[2k], inv[2k+1]) on
//                pair-nodes: colour(u) != colour(w) becomes
//                x(u/2) ^ x(w/2) = 1 ^ (u&1) ^ (w&1), x(k) = colour(2k)
//   orient       odd nodes: flip the tail's component so the tail is colour 0
//   roots        x(k) = parity to the component minimum (the canonical
//                colouring: each component's smallest vertex gets colour
//                0); the input switch of pair k is x(k).  Nodes that fit L2
//                are coloured by walks instead (walk.cuh)
//   settle       a level whose union-find chains get long (settle.cuh)
//   outputs      output switch of output pair k is colour(inv[2k]); the
//                children's inverses follow from the same two reads (the
//                values p are read at level 0 only)
//   emit         switch bits into the clustered blob layout: word copies of
//                long packet runs, word blocks of short ones, bits for the
//                rest
//
// The kernels are bound by memory latency and random-access throughput, not
// by instruction issue: their loops keep several independent loads per
// thread in flight.
#pragma once

#include "device.cuh"
#include "plan.hpp"

#include <cstdint>

namespace bpb200 {

constexpr uint32_t kTileThreads = 512;
// 4 slots per thread: more threads keep more of the scattered inverse stores
// in flight (measured on B200 when every level of 2^30 uniform entries had
// its own inverse: 207 ms per compress, 8 slots 227, 16 slots 243; it now
// runs on level 0 of inputs of up to 2^23 entries only).
#ifndef BPB200_INVERSE_ITEMS
#define BPB200_INVERSE_ITEMS 4
#endif
constexpr int kInverseItems = BPB200_INVERSE_ITEMS; // slots per thread in level_inverse
// level_union shape: 2 output pairs per thread at 6 blocks of 256 per SM
// measured fastest on B200 at 2^30 uniform entries (169 ms per compress with
// loads on every level; 1 at 8 blocks: 169, 2 at 4: 172, 4 at 4: 181).
#ifndef BPB200_UNION_ITEMS
#define BPB200_UNION_ITEMS 2
#endif
#ifndef BPB200_UNION_MIN_BLOCKS
#define BPB200_UNION_MIN_BLOCKS 6
#endif
// Nodes of up to this many entries (64 MB of union-find words) are united by
// compare-and-swaps alone, larger ones by loads first: at 2^30 entries the
// levels of 2^24, 2^25 and 2^26-entry nodes took 10.6, 11.6 and 23.2 ms with
// swaps, 14.0, 14.4 and 16.8 ms with loads.
constexpr uint64_t kSwapMaxNode = 1ull << 25;
constexpr int kUnionItems = BPB200_UNION_ITEMS; // output pairs per thread in level_union
// level_roots shape: pair-nodes per thread (1, 2, 4 or 8; 32 / items lanes
// assemble one colour word) and the minimum resident blocks of 256 per SM.
// The finds are latency-bound, so more resident warps beat more finds per
// thread (2^30 uniform entries, first seven levels, before the claims below:
// 1 pair-node at 8 blocks 55 ms, 2 at 8 57 ms, 4 at 4 61 ms).
#ifndef BPB200_RESOLVE_ITEMS
#define BPB200_RESOLVE_ITEMS 2
#endif
#ifndef BPB200_FINAL_MIN_BLOCKS
#define BPB200_FINAL_MIN_BLOCKS 8
#endif
constexpr int kResolveItems = BPB200_RESOLVE_ITEMS;
static_assert(kResolveItems == 1 || kResolveItems == 2 || kResolveItems == 4 ||
    kResolveItems == 8, "level_roots assembles colour words from 1, 2, 4 or 8 bits per lane");
// Control words of a level: work counters of its claiming kernels, zeroed
// for every level at once before the first launch.
enum : int {
    kCtlClaimInverse = 0, // level_inverse
    kCtlClaimPlace = 1,   // level_place
    kCtlChains = 2,       // kErrGaveUp: a union-find walk met a long chain (give_up)
    kCtlClaimUnion = 3,   // level_union
    kCtlClaimRoots = 4,   // level_roots
    kCtlArrived = 5,      // level_settle: blocks at its barriers
    kCtlChanged = 6,      // level_settle: two words, last pass with work left
    kCtlDeferred = 8,     // unions put off
    kCtlWords = 12
};

// What a union-find level's kernels share about its long chains: the level's
// control words, the word that says it is given up (kErrGaveUp in its
// kCtlChains word or, in a batched launch, in the permutation's status word)
// and the list of unions put off (in the memory of the output switch bits,
// which are written later; no list in a batched launch).
struct Chains {
    uint32_t* ctl;
    uint32_t* flag;
    uint2* list;
    uint32_t room;
};
constexpr uint32_t kStopClaims = 0x80000000u;
__host__ __device__ __forceinline__ Chains level_chains(uint32_t* ctl, uint32_t* ybits,
    uint32_t room) {
    return Chains{ctl, ctl + kCtlChains, reinterpret_cast<uint2*>(ybits), room};
}

// Gives a union-find level up: its roots are left to level_settle.
__device__ __forceinline__ void give_up(const Chains& c) {
    atomicOr(c.flag, kErrGaveUp);
    atomicOr(c.ctl + kCtlClaimRoots, kStopClaims);
}
__device__ __forceinline__ bool given_up(const Chains& c) {
    return (*(volatile uint32_t*)c.flag & kErrGaveUp) != 0;
}

// Gives the level up and puts a union off.  Once the list is full the others
// stop too: level_settle then does all of them again.
__device__ __forceinline__ void defer(const Chains& c, uint2 rec) {
    give_up(c);
    const uint32_t at = c.list != nullptr ? atomicAdd(c.ctl + kCtlDeferred, 1u) : 0u;
    if (at < c.room) {
        c.list[at] = rec;
    } else {
        atomicOr(c.ctl + kCtlClaimUnion, kStopClaims);
    }
}

struct TileShape {
    uint32_t slots;   // padded entry slots needed at the deepest level
    uint32_t smem;    // dynamic shared memory bytes
};

// 32-bit node-size test: every level here has fewer than 2^32 nodes.
__device__ __forceinline__ uint32_t size_at(const LevelInfo& lv, uint32_t level, uint32_t node) {
    const uint32_t rev = level == 0 ? 0u : (__brev(node) >> (32 - level));
    return (uint32_t)lv.q + ((uint64_t)rev < lv.r ? 1u : 0u);
}

// ------------------------------------------------------------ level kernels

// Inverse of level 0: inv[p[i]] = i.  With `uf`, every pair-node also starts
// as its own root, whatever its values: a stale word could point outside.
template <typename T>
__device__ __forceinline__ void level_inverse_run(Grid grid, const Plan* __restrict__ plan,
    const T* __restrict__ src, uint32_t* __restrict__ inv, uint32_t* __restrict__ uf,
    uint32_t* claims, uint32_t* status) {
    const uint32_t s = (uint32_t)plan->levels[0].q;
    const bool aligned = ((uintptr_t)src & 15u) == 0;
    uint64_t first;
    while (claim_chunk(claims, (uint64_t)blockDim.x * kInverseItems, s, &first)) {
        const uint64_t e0 = first + (uint64_t)threadIdx.x * kInverseItems;
        if (e0 >= s) {
            continue;
        }
        T v[kInverseItems];
        if (aligned && e0 + kInverseItems <= s) {
            constexpr int kVec = 16 / sizeof(T);
#pragma unroll
            for (int q = 0; q < kInverseItems / kVec; ++q) {
                const uint4 chunk = __ldcs(reinterpret_cast<const uint4*>(src + e0) + q);
                const T* parts = reinterpret_cast<const T*>(&chunk);
#pragma unroll
                for (int r = 0; r < kVec; ++r) v[q * kVec + r] = parts[r];
            }
        } else {
#pragma unroll
            for (int q = 0; q < kInverseItems; ++q) {
                v[q] = e0 + q < s ? src[e0 + q] : (T)0;
            }
        }
        const uint32_t i0 = (uint32_t)e0;
#pragma unroll
        for (int q = 0; q < kInverseItems; ++q) {
            if (e0 + q < s) {
                const uint32_t i = i0 + q;
                if (uf != nullptr && (i & 1u) == 0) {
                    uf[i >> 1] = i & ~1u;
                }
                const uint64_t val = (uint64_t)v[q];
                if (val >= s) {
                    atomicOr(status, kErrNotPermutation);
                } else {
                    inv[val] = i;
                }
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) level_inverse(const Plan* __restrict__ plan,
    const T* __restrict__ src, uint32_t* __restrict__ inv, uint32_t* __restrict__ uf,
    uint32_t* claims, uint32_t* status) {
    wait_for_previous();
    level_inverse_run<T>(launch_grid(), plan, src, inv, uf, claims, status);
}

// ---------------------------------------------------------------------------
// Partitioned inverse for levels whose nodes do not fit in L2.  A plain
// scatter inv[p[i]] = i there costs one HBM read-modify-write of a 32-byte
// sector per entry (about 21 G entries/s on B200).  Instead:
//   level_bucket  streams the values once and appends (destination, i)
//                 records to the 2^kPlaceLog2-slot destination window they
//                 land in.  A block sorts its 4096 records by window in
//                 shared memory (counts, a scan, one global reservation per
//                 window) and writes them out in that order, so a window's
//                 records leave as runs of whole sectors;
//   level_place   replays each window's records; the writes of one window
//                 stay inside an L2-resident 32 MB range.
// Bound by HBM for the bucket pass (8 + 8 + 2 bytes per uint64 entry) and by
// L2's random writes for the replay (2^30 at 220 G/s: 4.9 ms).  2^30 uniform
// uint64 entries, both kernels: 13.5 ms; 28.5 ms with every thread writing
// its records where they fell, 8 bytes to a sector.  Windows of 2^24 slots
// (64 MB, half of L2): 14.8 ms; 2^25: 29.5 ms, the window no longer fits.
// 2^24 entries: 0.236 ms against 0.273 before and 0.275 with 2^24 slots.
// A window receives at most as many records as it has slots when the input
// is a permutation; an overfull window means a repeated value.
// ---------------------------------------------------------------------------
#ifndef BPB200_PLACE_LOG2
#define BPB200_PLACE_LOG2 23
#endif
constexpr uint32_t kPlaceLog2 = BPB200_PLACE_LOG2; // slots per destination window (log2)
constexpr uint32_t kMaxWindows = 256;
static_assert((1ull << 31) >> kPlaceLog2 <= kMaxWindows, "windows must cover 2^31 slots");
constexpr int kBucketItems = 16;
constexpr int kBucketThreads = 256; // block size of level_bucket: a thread per window
static_assert(kMaxWindows <= kBucketThreads, "one window per thread in the scan");

// Slots [e_lo, e_hi) of level 0 (all of it, or one part of an input still
// being uploaded; e_lo a multiple of 4 so vector loads stay aligned).
template <typename T>
__global__ void __launch_bounds__(kBucketThreads, 4) level_bucket(const Plan* __restrict__ plan,
    const T* __restrict__ src, uint2* __restrict__ records, uint32_t* __restrict__ cursor,
    uint32_t* __restrict__ uf, uint32_t* status, uint64_t e_lo, uint64_t e_hi) {
    __shared__ uint2 sorted[kBucketThreads * kBucketItems];
    __shared__ uint32_t count[kMaxWindows];
    __shared__ uint32_t local[kMaxWindows]; // the window's first record in `sorted`
    __shared__ uint32_t start[kMaxWindows]; // and in its region of `records`
    __shared__ uint32_t sums[kBucketThreads / 32];
    constexpr int kVec = 16 / sizeof(T);
    constexpr uint32_t kChunk = kBucketThreads * kBucketItems;
    wait_for_previous();
    const uint64_t n = plan->levels[0].cap;
    const uint64_t total = e_hi < n ? e_hi : n;
    const bool aligned = ((uintptr_t)src & 15u) == 0 && (e_lo & 3u) == 0;
    const uint32_t t = threadIdx.x;
    for (uint64_t c0 = e_lo + (uint64_t)blockIdx.x * kChunk; c0 < total;
         c0 += (uint64_t)gridDim.x * kChunk) {
        const bool whole = aligned && c0 + kChunk <= total;
        if (t < kMaxWindows) count[t] = 0;
        __syncthreads();
        auto item = [&](int q) -> uint32_t { // offset in the chunk of this thread's value q
            return whole ? (t + kBucketThreads * (q / kVec)) * kVec + q % kVec
                         : t + kBucketThreads * q;
        };
        T v[kBucketItems];
        if (whole) {
#pragma unroll
            for (int q = 0; q < kBucketItems / kVec; ++q) {
                const uint4 part = __ldcs(reinterpret_cast<const uint4*>(src + c0) + t +
                    kBucketThreads * q);
                const T* parts = reinterpret_cast<const T*>(&part);
#pragma unroll
                for (int r = 0; r < kVec; ++r) v[q * kVec + r] = parts[r];
            }
        } else {
#pragma unroll
            for (int q = 0; q < kBucketItems; ++q) {
                v[q] = c0 + item(q) < total ? src[c0 + item(q)] : (T)0;
            }
        }
        uint32_t dest[kBucketItems], rank[kBucketItems];
#pragma unroll
        for (int q = 0; q < kBucketItems; ++q) {
            dest[q] = ~0u;
            if (c0 + item(q) < total) {
                if ((uint64_t)v[q] >= n) {
                    atomicOr(status, kErrNotPermutation);
                } else {
                    dest[q] = (uint32_t)v[q];
                    rank[q] = atomicAdd(&count[dest[q] >> kPlaceLog2], 1u);
                }
            }
        }
        // union-find roots of the chunk's pair-nodes (unconditional: see
        // level_inverse)
        const uint64_t pairs = ((c0 + kChunk < total ? c0 + kChunk : total) + 1) / 2;
#pragma unroll
        for (int q = 0; q < kBucketItems / 2; ++q) {
            const uint64_t id = c0 / 2 + t + kBucketThreads * q;
            if (id < pairs) uf[id] = (uint32_t)id << 1;
        }
        __syncthreads();
        const uint32_t mine = t < kMaxWindows ? count[t] : 0;
        uint32_t upto = mine;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, upto, d);
            if ((t & 31u) >= (uint32_t)d) upto += o;
        }
        if ((t & 31u) == 31u) sums[t / 32] = upto;
        if (mine != 0) start[t] = atomicAdd(cursor + t, mine);
        __syncthreads();
        uint32_t all = 0;
#pragma unroll
        for (uint32_t k = 0; k < kBucketThreads / 32; ++k) {
            if (k < t / 32) upto += sums[k];
            all += sums[k];
        }
        if (t < kMaxWindows) local[t] = upto - mine;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kBucketItems; ++q) {
            if (dest[q] == ~0u) continue;
            sorted[local[dest[q] >> kPlaceLog2] + rank[q]] =
                make_uint2(dest[q], (uint32_t)c0 + item(q));
        }
        __syncthreads();
        for (uint32_t k = t; k < all; k += kBucketThreads) {
            const uint2 r = sorted[k];
            const uint32_t b = r.x >> kPlaceLog2;
            const uint64_t at = ((uint64_t)b << kPlaceLog2) + start[b] + (k - local[b]);
            if (at < n && at < ((uint64_t)(b + 1) << kPlaceLog2)) {
                records[at] = r;
            } else {
                atomicOr(status, kErrNotPermutation); // more values than slots: a repeat
            }
        }
        __syncthreads();
    }
}

constexpr int kPlaceItems = 16;

__device__ __forceinline__ void level_place_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, const uint2* __restrict__ records, const uint32_t* __restrict__ cursor,
    uint32_t* __restrict__ inv, uint32_t* claims) {
    const LevelInfo& lv = plan->levels[level];
    const uint64_t total = lv.cap << level;
    const uint64_t chunk = (uint64_t)blockDim.x * kPlaceItems;
    uint64_t first;
    while (claim_chunk(claims, chunk, total, &first)) {
#pragma unroll
        for (int q = 0; q < kPlaceItems; ++q) {
            const uint64_t at = first + (uint64_t)q * blockDim.x + threadIdx.x;
            if (at >= total) break;
            const uint32_t b = (uint32_t)(at >> kPlaceLog2);
            if ((at & ((1ull << kPlaceLog2) - 1)) < cursor[b]) {
                const uint2 r = __ldcs(records + at);
                inv[r.x] = r.y;
            }
        }
    }
}

__global__ void __launch_bounds__(256) level_place(const Plan* __restrict__ plan,
    uint32_t level, const uint2* __restrict__ records, const uint32_t* __restrict__ cursor,
    uint32_t* __restrict__ inv, uint32_t* claims) {
    wait_for_previous();
    level_place_run(launch_grid(), plan, level, records, cursor, inv, claims);
}

// Unions of output pairs [p0, p0 + kUnionItems) below `end`; returns whether
// one met a long chain and puts those off (with `chains`).  `swap`: see
// uf_unite_many.
__device__ __forceinline__ bool unite_outputs(const LevelInfo& lv, uint32_t level,
    const uint32_t* __restrict__ inv, uint32_t* uf, uint64_t p0, uint64_t end, bool swap,
    const Chains* chains, uint32_t* status) {
    const uint32_t pcap = (uint32_t)lv.pcap;
    uint32_t j = (uint32_t)(p0 / pcap);
    uint32_t k = (uint32_t)(p0 - (uint64_t)j * pcap);
    uint32_t s = size_at(lv, level, j);
    uint32_t a[kUnionItems], b[kUnionItems], rel[kUnionItems];
    uint32_t u[kUnionItems], w[kUnionItems], base[kUnionItems];
    uint32_t pending = 0;
#pragma unroll
    for (int q = 0; q < kUnionItems; ++q) {
        if (p0 + q < end && k < s / 2) {
            pending |= 1u << q;
            const uint2 both = *reinterpret_cast<const uint2*>(inv + 2 * ((uint64_t)j * pcap + k));
            u[q] = both.x;
            w[q] = both.y;
            base[q] = j * pcap;
            rel[q] = s; // stash the node size for the range check below
        }
        if (++k == pcap) {
            k = 0;
            ++j;
            s = size_at(lv, level, j);
        }
    }
#pragma unroll
    for (int q = 0; q < kUnionItems; ++q) {
        if (pending & (1u << q)) {
            if (u[q] >= rel[q] || w[q] >= rel[q]) {
                atomicOr(status, not_permutation(level));
                pending &= ~(1u << q);
                continue;
            }
            a[q] = base[q] + (u[q] >> 1);
            b[q] = base[q] + (w[q] >> 1);
            rel[q] = 1u ^ (u[q] & 1u) ^ (w[q] & 1u);
        }
    }
    pending = swap ? uf_unite_many<kUnionItems, true>(uf, a, b, rel, pending, status)
                   : uf_unite_many<kUnionItems, false>(uf, a, b, rel, pending, status);
    if (chains != nullptr) {
#pragma unroll
        for (int q = 0; q < kUnionItems; ++q) {
            if (pending & (1u << q)) defer(*chains, make_uint2(a[q], (b[q] << 1) | rel[q]));
        }
    }
    return pending != 0;
}

// Blocks claim chunks of output pairs in address order (claim_chunk), so the
// union-find words being linked at any time belong to the few nodes those
// chunks cover: once a node's words fit in L2 the random finds hit there.
__device__ __forceinline__ void level_union_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ inv, uint32_t* uf, const Chains& chains,
    uint32_t* status) {
    const LevelInfo& lv = plan->levels[level];
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t begin = nr.lo * lv.pcap;
    const uint64_t total = lv.pcap << nr.shift;
    uint64_t first;
    while (claim_chunk(chains.ctl + kCtlClaimUnion, (uint64_t)blockDim.x * kUnionItems, total,
        &first)) {
        const uint64_t p0 = begin + first + (uint64_t)threadIdx.x * kUnionItems;
        if (p0 >= begin + total) {
            continue;
        }
        unite_outputs(lv, level, inv, uf, p0, begin + total, lv.cap <= kSwapMaxNode, &chains,
            status);
    }
}

__global__ void __launch_bounds__(256, BPB200_UNION_MIN_BLOCKS) level_union(const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ inv, uint32_t* uf, const __grid_constant__ Chains chains,
    uint32_t* status) {
    wait_for_previous();
    level_union_run(launch_grid(), plan, level, inv, uf, chains, status);
}

// ---------------------------------------------------------------------------
// Unions by windows, for nodes whose union-find words do not fit L2.  There a
// union is a few dependent random accesses to HBM.  Since a walk only ever
// looks at the larger of its two ends, the unions can be kept in buckets by
// that end's window of 2^kUnionWindowLog2 pair-nodes and worked off from the
// highest window down:
//   union_bucket  appends every output pair's union (larger end, smaller end
//                 and relation) to its window's bucket;
//   union_window  works off one bucket: each union is walked while its larger
//                 end lies in the window, whose words stay in L2, and is
//                 appended to a lower window's bucket when it leaves.
// A window's region holds two records per pair-node, as many unions as can
// start in it; a union that finds its region full is finished on the spot.
// 2^30 uniform entries, levels of 2^30 to 2^26-entry nodes: 19.1, 16.4, 15.9,
// 15.6 and 15.5 ms against 36.1, 33.7, 29.6, 23.1 and 16.6 ms with the same
// unions in the order of the output pairs; nodes of 2^25 entries (11.8 ms in
// that order, level_union) already fit.
// ---------------------------------------------------------------------------
constexpr uint32_t kUnionWindowLog2 = 24;
constexpr uint32_t kUnionWindows = 128; // up to 2^31 pair-nodes
constexpr int kUnionBucketItems = 4;    // unions per thread and round

// Appends this thread's pending records to their windows' buckets; all
// threads of the block call.  Returns the records that found no room.
template <int K>
__device__ __forceinline__ uint32_t union_append(uint2* __restrict__ records,
    uint32_t* __restrict__ cursor, uint64_t capacity, const uint2 (&rec)[K], uint32_t pending,
    uint32_t* count, uint32_t* start) {
    for (uint32_t v = threadIdx.x; v < kUnionWindows; v += blockDim.x) count[v] = 0;
    __syncthreads();
    uint32_t at[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
        if (pending & (1u << i)) at[i] = atomicAdd(&count[rec[i].x >> kUnionWindowLog2], 1u);
    }
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < kUnionWindows; v += blockDim.x) {
        if (count[v] != 0) start[v] = atomicAdd(cursor + v, count[v]);
    }
    __syncthreads();
    uint32_t left = 0;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        if (!(pending & (1u << i))) continue;
        const uint32_t v = rec[i].x >> kUnionWindowLog2;
        const uint64_t slot = (uint64_t)start[v] + at[i];
        const uint64_t pos = ((uint64_t)v << (kUnionWindowLog2 + 1)) + slot;
        if (slot < (2ull << kUnionWindowLog2) && pos < capacity) {
            records[pos] = rec[i];
        } else {
            left |= 1u << i;
        }
    }
    __syncthreads(); // count and start are free again
    return left;
}

// Finishes the unions that found no room.
template <int K>
__device__ __forceinline__ void union_finish(uint32_t* uf, const uint2 (&rec)[K], uint32_t left,
    const Chains& chains, uint32_t* status) {
    uint32_t a[K], b[K], rel[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
        a[i] = rec[i].x;
        b[i] = rec[i].y >> 1;
        rel[i] = rec[i].y & 1u;
    }
    left = uf_unite_many<K, false>(uf, a, b, rel, left, status);
#pragma unroll
    for (int i = 0; i < K; ++i) {
        if (left & (1u << i)) defer(chains, make_uint2(a[i], (b[i] << 1) | rel[i]));
    }
}

__global__ void __launch_bounds__(256) union_bucket(const Plan* __restrict__ plan, uint32_t level,
    const uint32_t* __restrict__ inv, uint32_t* uf, uint2* __restrict__ records,
    uint32_t* __restrict__ cursor, uint64_t capacity, const __grid_constant__ Chains chains, uint32_t* status) {
    wait_for_previous();
    __shared__ uint32_t count[kUnionWindows];
    __shared__ uint32_t start[kUnionWindows];
    const LevelInfo& lv = plan->levels[level];
    const uint32_t ps = (uint32_t)lv.pcap;
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t first = nr.lo * ps;
    const uint64_t end = first + ((uint64_t)ps << nr.shift);
    const uint64_t chunk = (uint64_t)blockDim.x * kUnionBucketItems;
    for (uint64_t c = first + (uint64_t)blockIdx.x * chunk; c < end; c += (uint64_t)gridDim.x * chunk) {
        uint2 both[kUnionBucketItems], rec[kUnionBucketItems];
        uint32_t pending = 0;
#pragma unroll
        for (int i = 0; i < kUnionBucketItems; ++i) {
            const uint64_t p = c + (uint64_t)i * blockDim.x + threadIdx.x;
            both[i] = p < end ? __ldcs(reinterpret_cast<const uint2*>(inv) + p) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < kUnionBucketItems; ++i) {
            const uint64_t p = c + (uint64_t)i * blockDim.x + threadIdx.x;
            if (p >= end) continue;
            const uint32_t j = (uint32_t)p / ps;
            const uint32_t k = (uint32_t)p - j * ps;
            const uint32_t s = size_at(lv, level, j);
            if (k >= s / 2) continue;
            const uint32_t u = both[i].x, w = both[i].y;
            if (u >= s || w >= s) {
                atomicOr(status, not_permutation(level));
                continue;
            }
            const uint32_t a = j * ps + (u >> 1), b = j * ps + (w >> 1);
            const uint32_t rel = 1u ^ (u & 1u) ^ (w & 1u);
            if (a == b) {
                if (rel != 0) atomicOr(status, kErrInconsistent);
                continue;
            }
            rec[i] = make_uint2(max(a, b), (min(a, b) << 1) | rel);
            pending |= 1u << i;
        }
        const uint32_t left = union_append<kUnionBucketItems>(records, cursor, capacity, rec,
            pending, count, start);
        if (left != 0) union_finish<kUnionBucketItems>(uf, rec, left, chains, status);
    }
}

// A union that has come half of kLongChain halves the rest of its path: x,
// whose word is w, goes to its grandparent; both are true facts, so the racy
// store can only write a true one.  Returns the word that leads from x to
// where the walk goes on.  Uniform inputs never get here, but the compiler
// makes a slower loop of union_window without the branch: 3.07 ms for the
// windows of 100,000,007 entries' top two levels, 2.84 with it (and 3.08
// where `chains` is a __grid_constant__).
__device__ __forceinline__ uint32_t uf_halve(uint32_t* uf, uint32_t x, uint32_t w) {
    const uint32_t up = *(volatile uint32_t*)(uf + (w >> 1));
    if ((up >> 1) == (w >> 1)) {
        return w; // the parent is a root
    }
    const uint32_t over = (up & ~1u) | ((w ^ up) & 1u);
    uf[x] = over;
    return over;
}

__global__ void __launch_bounds__(256, 6) union_window(uint32_t window, uint32_t* uf,
    uint2* __restrict__ records, uint32_t* __restrict__ cursor, uint64_t capacity,
    const Chains chains, uint32_t* status) {
    wait_for_previous();
    const volatile uint32_t* stop = chains.ctl + kCtlClaimUnion;
    if (__syncthreads_or((*stop & kStopClaims) != 0)) return; // too many unions put off
    __shared__ uint32_t count[kUnionWindows];
    __shared__ uint32_t start[kUnionWindows];
    const uint64_t base = (uint64_t)window << (kUnionWindowLog2 + 1);
    uint64_t total = cursor[window]; // complete: only higher windows add to it
    const uint64_t room = capacity - base;
    if (total > (2ull << kUnionWindowLog2)) total = 2ull << kUnionWindowLog2;
    if (total > room) total = room;
    constexpr int K = 2;
    const uint64_t chunk = (uint64_t)blockDim.x * K;
    for (uint64_t c = (uint64_t)blockIdx.x * chunk; c < total; c += (uint64_t)gridDim.x * chunk) {
        uint2 rec[K];
        uint32_t live = 0, pending = 0;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            const uint64_t at = c + (uint64_t)i * blockDim.x + threadIdx.x;
            if (at < total) {
                rec[i] = __ldcs(records + base + at);
                live |= 1u << i;
            }
        }
        for (uint32_t it = 0; live != 0; ++it) {
            uint32_t w[K];
#pragma unroll
            for (int i = 0; i < K; ++i) {
                if (live & (1u << i)) w[i] = atomicCAS(uf + rec[i].x, rec[i].x << 1, rec[i].y);
            }
#pragma unroll
            for (int i = 0; i < K; ++i) {
                if (!(live & (1u << i))) continue;
                if (w[i] == rec[i].x << 1) { // a root: linked
                    live &= ~(1u << i);
                    continue;
                }
                const uint32_t over = it < kLongChain / 2 ? w[i] : uf_halve(uf, rec[i].x, w[i]);
                const uint32_t up = over >> 1, b = rec[i].y >> 1;
                const uint32_t rel = (rec[i].y ^ over) & 1u;
                rec[i] = make_uint2(max(up, b), (min(up, b) << 1) | rel);
                if (up == b) {
                    if (rel != 0) atomicOr(status, kErrInconsistent);
                    live &= ~(1u << i);
                } else if (rec[i].x >> kUnionWindowLog2 != window) {
                    live &= ~(1u << i); // on to a lower window
                    pending |= 1u << i;
                } else if (it == kLongChain) {
                    defer(chains, rec[i]);
                    live &= ~(1u << i);
                }
            }
        }
        const uint32_t left = union_append<K>(records, cursor, capacity, rec, pending, count, start);
        if (left != 0) union_finish<K>(uf, rec, left, chains, status);
    }
}

__device__ __forceinline__ void level_orient_run(Grid grid, const Plan* __restrict__ plan, uint32_t level,
    const uint32_t* __restrict__ inv, uint32_t* uf, const Chains& chains,
    uint32_t* status) {
    if (given_up(chains)) return;
    const LevelInfo& lv = plan->levels[level];
    const uint32_t pcap = (uint32_t)lv.pcap;
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t nodes_end = nr.lo + (1ull << nr.shift);
    for (uint64_t j = nr.lo + (uint64_t)grid.bid * blockDim.x + threadIdx.x; j < nodes_end;
         j += (uint64_t)grid.nblk * blockDim.x) {
        const uint32_t s = size_at(lv, level, (uint32_t)j);
        if ((s & 1u) == 0) {
            continue;
        }
        if (inv[2 * j * pcap + s - 1] >= s) {
            atomicOr(status, not_permutation(level));
            continue;
        }
        const uint32_t x[1] = {(uint32_t)j * pcap + (s >> 1)};
        Found f[1];
        if (uf_find_many<1>(uf, x, f, 1u) != 0) {
            give_up(chains);
        } else if (f[0].bit) {
            atomicOr(uf + f[0].root, 1u);
        }
    }
}

__global__ void level_orient(const Plan* __restrict__ plan, uint32_t level,
    const uint32_t* __restrict__ inv, uint32_t* uf, const __grid_constant__ Chains chains, uint32_t* status) {
    wait_for_previous();
    level_orient_run(launch_grid(), plan, level, inv, uf, chains, status);
}

// Switch addresses of every node of the levels above the tile's: level l's
// nodes start at element 2^l of in_addr / out_addr.
__device__ __forceinline__ void level_descriptors_run(Grid grid, const Plan* __restrict__ plan,
    NodeAddress* __restrict__ in_addr, NodeAddress* __restrict__ out_addr) {
    const uint64_t end = 1ull << plan->tile_level;
    for (uint64_t i = 1 + (uint64_t)grid.bid * blockDim.x + threadIdx.x; i < end;
         i += (uint64_t)grid.nblk * blockDim.x) {
        const uint32_t level = high_bit(i);
        const uint64_t j = i - (1ull << level);
        const NodeRange nr = level_nodes(*plan, level);
        if (j >= nr.lo && j < nr.lo + (1ull << nr.shift)) {
            in_addr[i] = node_address(*plan, 0, level, j);
            out_addr[i] = node_address(*plan, 1, level, j);
        }
    }
}

// Input switch bits of a union-find level: bit k = colour of input 2k = the
// pair-node's parity to its root, flipped by the root's orientation flag;
// kResolveItems pair-nodes per thread.  Finds that shortened paths as they
// went, in grid-stride order on nodes up to 2^26 entries, took 58 ms per
// compress at 2^30 entries, these 44 ms.
__device__ __forceinline__ void level_roots_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, uint32_t* uf, uint32_t* __restrict__ xbits,
    const Chains& chains) {
    const LevelInfo& lv = plan->levels[level];
    const uint32_t pcap = (uint32_t)lv.pcap;
    // this call's pair-nodes [lo_pair, end); chunks start at a 32-pair
    // boundary at or below lo_pair so colour words are written whole
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t lo_pair = nr.lo * pcap;
    const uint64_t end = lo_pair + ((uint64_t)pcap << nr.shift);
    const uint64_t begin = lo_pair & ~31ull;
    const uint64_t total = end - begin;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t chunk = (uint64_t)blockDim.x * kResolveItems;
    // Chunks are claimed in address order and every pair-node's root goes
    // back into its word: parents are smaller than their children, so most
    // finds end at a parent that was resolved before them.
    uint64_t first;
    while (claim_chunk(chains.ctl + kCtlClaimRoots, chunk, total, &first)) {
        const uint64_t p0 = begin + first + (uint64_t)threadIdx.x * kResolveItems;
        uint32_t j = (uint32_t)(p0 / pcap);
        uint32_t k = (uint32_t)(p0 - (uint64_t)j * pcap);
        uint32_t s = size_at(lv, level, j);
        uint32_t live = 0;
        uint32_t x[kResolveItems];
#pragma unroll
        for (int q = 0; q < kResolveItems; ++q) {
            x[q] = (uint32_t)(p0 + q);
            if (p0 + q >= lo_pair && p0 + q < end && k < s - s / 2) live |= 1u << q;
            if (++k == pcap) {
                k = 0;
                ++j;
                s = size_at(lv, level, j);
            }
        }
        Found f[kResolveItems];
        if (uf_find_many<kResolveItems>(uf, x, f, live) != 0) {
            give_up(chains);
            live = 0;
        }
        uint32_t mine = 0; // this lane's kResolveItems colour bits
#pragma unroll
        for (int q = 0; q < kResolveItems; ++q) {
            if (!(live & (1u << q))) continue;
            mine |= (f[q].bit ^ (uf[f[q].root] & 1u)) << q;
            if (f[q].root != x[q]) {
                uf[x[q]] = (f[q].root << 1) | f[q].bit;
            }
        }
        // 32 / kResolveItems lanes hold one 32-pair colour word
        constexpr uint32_t kWordLanes = 32 / kResolveItems;
        uint32_t v = mine << ((lane & (kWordLanes - 1)) * kResolveItems);
#pragma unroll
        for (uint32_t d = 1; d < kWordLanes; d <<= 1) {
            v |= __shfl_xor_sync(0xffffffffu, v, d);
        }
        if ((lane & (kWordLanes - 1)) == 0 && p0 < end) {
            xbits[p0 >> 5] = v;
        }
    }
}

__global__ void __launch_bounds__(256, BPB200_FINAL_MIN_BLOCKS) level_roots(
    const Plan* __restrict__ plan, uint32_t level, uint32_t* uf, uint32_t* __restrict__ xbits,
    const __grid_constant__ Chains chains) {
    wait_for_previous();
    level_roots_run(launch_grid(), plan, level, uf, xbits, chains);
}

// Output side of a level, in natural (node, output pair) order: the output
// switch bits and the children, so no level below the first scatters an
// inverse.  Output pair k of node j joins outputs 2k and 2k+1, fed by inputs
// u0 = inv[2k] and u1 = inv[2k+1], whose colours differ.  Its switch bit is
// y = colour(u0) (src/benes.cpp:306-310: the output bit of input i is
// colour(i) ^ (p[i] & 1), and p[u0] = 2k).  Of the two, the colour-0 input
// inv[2k + y] is routed to the left child, where it sits at input pair
// inv[2k + y] >> 1 and carries value k (src/benes.cpp:313-314); the other
// goes right with the same value.  So
//     left_inv[k] = inv[2k + y] >> 1,  right_inv[k] = inv[2k + 1 - y] >> 1,
// and an odd node's tail output s - 1, whose input is coloured 0, gives
// left_inv[s / 2] = inv[s - 1] >> 1.  A thread takes two output pairs, which
// make one output pair of each child: one 16-byte load of inv, one 8-byte
// store per child inverse, and, for a child level coloured by walks
// (`child_edge`), that pair's edges and a cleared stamp (`child_stamp`); for one coloured by union-find
// (`child_uf`), its pair-node's root.  An odd child's tail is stored with
// its virtual partner.  The edges are the only random writes (their node
// fits L2); xbits gathers one bit per output pair.  A value out of range
// (only possible when the input was not a permutation, which level 0
// reports, or after a walk gave up) leaves 0xffffffff, which every user
// range-checks.
__device__ __forceinline__ void level_outputs_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ inv, const uint32_t* __restrict__ xbits,
    uint32_t* __restrict__ ybits, uint32_t* __restrict__ child_inv,
    uint32_t* __restrict__ child_edge, uint32_t* __restrict__ child_stamp,
    uint32_t* __restrict__ child_uf) {
    const LevelInfo& lv = plan->levels[level];
    const LevelInfo& cl = plan->levels[level + 1];
    const uint32_t ps = (uint32_t)lv.pcap;
    const uint32_t hs = ps / 2; // quads of outputs per node
    const uint32_t cps = (uint32_t)cl.pcap;
    // this call's quads; the loop starts at a 32-quad boundary so each warp
    // assembles whole bit words (bits before `first` stay zero)
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t first = nr.lo * hs;
    const uint64_t end = first + ((uint64_t)hs << nr.shift);
    const uint64_t begin = first & ~31ull;
    const uint32_t lane = threadIdx.x & 31;
    // one quad a thread, blocks starting in address order, so the child nodes
    // being scattered to at any time fit L2 (in grid-stride order the output
    // pass took 407 ms per compress at 2^30 entries)
    const uint64_t stride = (uint64_t)grid.nblk * blockDim.x;
    for (uint64_t g = begin + (uint64_t)grid.bid * blockDim.x + threadIdx.x; g - lane < end;
         g += stride) {
        uint32_t ys = 0;
        if (g >= first && g < end) {
            const uint32_t j = (uint32_t)g / hs;
            const uint32_t k0 = 2 * ((uint32_t)g - j * hs);
            const uint32_t s = size_at(lv, level, j);
            const uint32_t half = s / 2;
            if (k0 < s - half) {
                const uint4 four = __ldcs(reinterpret_cast<const uint4*>(inv) + g);
                uint32_t left[2], right[2];
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    const uint32_t u = i == 0 ? four.x : four.z;
                    const uint32_t w = i == 0 ? four.y : four.w;
                    bool y = false;
                    left[i] = right[i] = ~0u;
                    if (k0 + i < half) {
                        if (u < s && w < s) {
                            const uint32_t q = j * ps + (u >> 1);
                            y = (((xbits[q >> 5] >> (q & 31)) ^ u) & 1u) != 0;
                            left[i] = (y ? w : u) >> 1;
                            right[i] = (y ? u : w) >> 1;
                        }
                    } else if (k0 + i == half && u < s) { // the odd tail
                        left[i] = u >> 1;
                    }
                    ys |= (y ? 1u : 0u) << i;
                }
                auto child = [&](uint32_t node, uint32_t cs, const uint32_t (&v)[2]) {
                    if (k0 >= cs) return;
                    const uint64_t at = 2ull * node * cps;
                    const uint32_t w = k0 + 1 < cs ? v[1] : cs; // virtual partner
                    __stcs(reinterpret_cast<uint2*>(child_inv + at + k0), make_uint2(v[0], w));
                    const uint32_t id = node * cps + (k0 >> 1);
                    if (child_edge != nullptr) {
                        child_stamp[id] = 0;
                        if (v[0] < cs && w < cs + (cs & 1u)) {
                            child_edge[at + v[0]] = w;
                            child_edge[at + w] = v[0];
                        }
                    } else if (child_uf != nullptr) {
                        child_uf[id] = id << 1;
                    }
                };
                child(2 * j, s - half, left);
                child(2 * j + 1, half, right);
            }
        }
        // lane i holds bits 2i and 2i + 1 of the 64 from quad g - lane
        const uint32_t two = ys << (2 * (lane & 15));
        const uint32_t low = __reduce_or_sync(0xffffffffu, lane < 16 ? two : 0u);
        const uint32_t high = __reduce_or_sync(0xffffffffu, lane < 16 ? 0u : two);
        if (lane < 2) {
            ybits[((g - lane) >> 4) + lane] = lane == 0 ? low : high;
        }
    }
}

__global__ void __launch_bounds__(256) level_outputs(const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ inv, const uint32_t* __restrict__ xbits,
    uint32_t* __restrict__ ybits, uint32_t* __restrict__ child_inv,
    uint32_t* __restrict__ child_edge, uint32_t* __restrict__ child_stamp,
    uint32_t* __restrict__ child_uf) {
    wait_for_previous();
    level_outputs_run(launch_grid(), plan, level, inv, xbits, ybits, child_inv, child_edge,
        child_stamp, child_uf);
}

// Switch bits of one section at one level, packet-major: thread t maps to
// (packet, node, pair-in-span) with the pair fastest, then the node, so for
// full packets consecutive threads land on consecutive blob bits and a
// warp issues one or two atomics instead of one per bit.
__device__ __forceinline__ void level_emit_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, int side, const uint32_t* __restrict__ bits,
    const NodeAddress* __restrict__ addr, uint32_t* __restrict__ blob, uint64_t first_packet) {
    const LevelInfo& lv = plan->levels[level];
    const LevelSide& ls = lv.side[side];
    const GroupInfo& gi = plan->groups[side][ls.group];
    const uint32_t span_log2 = gi.depth - ls.rel - 1;
    const uint32_t pcap = (uint32_t)lv.pcap;
    const uint64_t max_pairs = lv.cap / 2;
    const uint64_t packets = (max_pairs + (1ull << span_log2) - 1) >> span_log2;
    const NodeRange nr = level_nodes(*plan, level);
    const uint32_t shift = nr.shift + span_log2; // log2(nodes * span)
    const uint64_t total = packets > first_packet ? (packets - first_packet) << shift : 0;
    const uint64_t section_bit = plan->section_offset[side] * 8;
    const uint64_t stride = (uint64_t)grid.nblk * blockDim.x;
    for (uint64_t t = (uint64_t)grid.bid * blockDim.x + threadIdx.x;
         t - (threadIdx.x & 31) < total; t += stride) {
        bool set = false;
        uint64_t dest = 0;
        if (t < total) {
            const uint64_t packet = first_packet + (t >> shift);
            const uint64_t rem = t & ((1ull << shift) - 1);
            const uint32_t node = (uint32_t)(nr.lo + (rem >> span_log2));
            const uint64_t pair = (packet << span_log2) + (rem & ((1ull << span_log2) - 1));
            const uint32_t s = size_at(lv, level, node);
            if (pair < s / 2) {
                const uint64_t q = (uint64_t)node * pcap + pair;
                set = ((bits[q >> 5] >> (q & 31)) & 1u) != 0;
                if (set) {
                    dest = section_bit + switch_bit(addr[node], pair);
                }
            }
        }
        emit_bit(blob, dest, set, 0xffffffffu);
    }
}

// Block form of level_emit for short runs (span_log2 < 5), on the packets
// every node of the level fills (packet < full_packets: below the smallest
// node's tail packet, so every node contributes `span` switches and every
// path's run starts at path * span inside the packet, SectionAddress using
// packet 0's prefix for all non-tail packets).  Inside such a packet the
// level's switches of one cluster root are then one contiguous block,
// path-major: thread per 32-bit word of a block, gathering the `span`-bit
// fields of 32 / span consecutive nodes, one or two atomics per word.
__device__ __forceinline__ void level_emit_blocks_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, int side, const uint32_t* __restrict__ bits,
    const NodeAddress* __restrict__ addr, uint32_t* __restrict__ blob, uint64_t full_packets) {
    const LevelInfo& lv = plan->levels[level];
    const LevelSide& ls = lv.side[side];
    const GroupInfo& gi = plan->groups[side][ls.group];
    const uint32_t rel = ls.rel;
    const uint32_t span_log2 = gi.depth - rel - 1;
    const uint32_t span_mask = (1u << (1u << span_log2)) - 1u; // span <= 16 bits
    const uint32_t pcap = (uint32_t)lv.pcap;
    // nodes per word: 32 / span, or all 2^rel nodes of a root when fewer
    const uint32_t per_word_log2 = min(5u - span_log2, rel);
    const uint32_t words_log2 = rel - per_word_log2; // words per block (log2)
    const uint64_t per_root = full_packets << words_log2;
    // this call's nodes hold whole cluster roots (the host uses this form
    // only then)
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t root_lo = nr.lo >> rel;
    const uint64_t total = (per_root << (nr.shift - rel));
    const uint64_t section_bit = plan->section_offset[side] * 8;
    const uint64_t stride = (uint64_t)grid.nblk * blockDim.x;
    for (uint64_t t = (uint64_t)grid.bid * blockDim.x + threadIdx.x; t < total; t += stride) {
        const uint64_t root = root_lo + t / per_root;
        const uint64_t rem = t - (root - root_lo) * per_root;
        const uint64_t packet = rem >> words_log2;
        const uint32_t word = (uint32_t)(rem & ((1ull << words_log2) - 1));
        const uint32_t node0 = (uint32_t)(root << rel) + (word << per_word_log2);
        uint32_t v = 0;
        for (uint32_t i = 0; i < (1u << per_word_log2); ++i) {
            const uint64_t q = (uint64_t)(node0 + i) * pcap + (packet << span_log2);
            const uint64_t wq = q >> 5;
            const uint32_t field =
                __funnelshift_r(bits[wq], bits[wq + 1], (uint32_t)(q & 31)) & span_mask;
            v |= field << (i << span_log2);
        }
        if (v == 0) {
            continue;
        }
        const uint64_t dest = section_bit +
            switch_bit(addr[(uint32_t)(root << rel)], packet << span_log2) + ((uint64_t)word << 5);
        const uint32_t off = (uint32_t)(dest & 31);
        atomicOr(blob + (dest >> 5), v << off);
        if (off != 0 && (v >> (32 - off)) != 0) {
            atomicOr(blob + (dest >> 5) + 1, v >> (32 - off));
        }
    }
}

// Transposed form of level_emit_blocks for cluster roots of at least 32
// nodes (rel >= 5): a warp takes 32 consecutive nodes of one root and a
// window of 32 / span full packets.  Each lane loads one 32-bit window of
// its node's switches (span bits per packet, consecutive packets adjacent),
// and lane L then assembles output word L with 32 / span shuffles: packet
// L / span of the window, nodes (L % span) * 32 / span onwards.  Two loads
// per lane replace the 2 * 32 / span loads per word of the block form.
__device__ __forceinline__ void level_emit_transpose_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, int side, const uint32_t* __restrict__ bits,
    const NodeAddress* __restrict__ addr, uint32_t* __restrict__ blob, uint64_t full_packets) {
    const LevelInfo& lv = plan->levels[level];
    const LevelSide& ls = lv.side[side];
    const GroupInfo& gi = plan->groups[side][ls.group];
    const uint32_t rel = ls.rel;                 // >= 5
    const uint32_t span_log2 = gi.depth - rel - 1; // < 5
    const uint32_t span_mask = (1u << (1u << span_log2)) - 1u;
    const uint32_t per_window_log2 = 5 - span_log2; // packets per lane window
    const uint32_t pcap = (uint32_t)lv.pcap;
    const uint64_t windows = (full_packets + (1ull << per_window_log2) - 1) >> per_window_log2;
    // 32-node groups of this call's nodes (at least 32 of them, aligned)
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t groups = 1ull << (nr.shift - 5);
    const uint64_t total_warps = groups * windows;
    const uint64_t section_bit = plan->section_offset[side] * 8;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)grid.nblk * blockDim.x) >> 5;
    for (uint64_t wi = ((uint64_t)grid.bid * blockDim.x + threadIdx.x) >> 5; wi < total_warps;
         wi += warps) {
        const uint64_t group = wi / windows;
        const uint64_t k0 = (wi - group * windows) << per_window_log2;
        const uint32_t node = (uint32_t)(nr.lo + (group << 5)) + lane;
        const uint64_t q = (uint64_t)node * pcap + (k0 << span_log2);
        const uint64_t wq = q >> 5;
        uint32_t window = __funnelshift_r(bits[wq], bits[wq + 1], (uint32_t)(q & 31));
        // packets at or past full_packets belong to level_emit
        const uint64_t valid = full_packets - k0; // > 0
        if (valid < (1ull << per_window_log2)) {
            window &= (1u << (uint32_t)(valid << span_log2)) - 1u;
        }
        const uint32_t p_local = lane >> span_log2;
        const uint32_t g_out = lane & ((1u << span_log2) - 1u);
        uint32_t v = 0;
        for (uint32_t n = 0; n < (1u << per_window_log2); ++n) {
            const uint32_t w = __shfl_sync(0xffffffffu, window,
                (int)((g_out << per_window_log2) + n));
            v |= ((w >> (p_local << span_log2)) & span_mask) << (n << span_log2);
        }
        const uint64_t packet = k0 + p_local;
        if (v == 0 || packet >= full_packets) {
            continue;
        }
        const uint32_t root_node = node & ~((1u << rel) - 1u);
        const uint32_t n0 = (node & ((1u << rel) - 1u)) & ~31u; // first node of the group
        const uint64_t dest = section_bit + switch_bit(addr[root_node], packet << span_log2) +
            ((uint64_t)n0 << span_log2) + ((uint64_t)g_out << 5);
        const uint32_t off = (uint32_t)(dest & 31);
        atomicOr(blob + (dest >> 5), v << off);
        if (off != 0 && (v >> (32 - off)) != 0) {
            atomicOr(blob + (dest >> 5) + 1, v >> (32 - off));
        }
    }
}

// Word-wise form of level_emit for levels whose packets carry at least 32
// switches of each node (span_log2 >= 5).  The switches of one node inside
// one packet are a contiguous run of the node's bits and land on a
// contiguous run of blob bits (SwitchBitAddress::bit moves by one per pair
// inside a packet), so the level is a set of bit-range copies: thread per
// 32-switch chunk, one funnel shift to align the source and one or two
// atomics for the destination words (neighbouring runs share edge words).
// Chunks start at multiples of 32 pairs, so a chunk never crosses a packet.
__device__ __forceinline__ void level_emit_words_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, int side, const uint32_t* __restrict__ bits,
    const NodeAddress* __restrict__ addr, uint32_t* __restrict__ blob) {
    const LevelInfo& lv = plan->levels[level];
    const LevelSide& ls = lv.side[side];
    const GroupInfo& gi = plan->groups[side][ls.group];
    const uint32_t span_log2 = gi.depth - ls.rel - 1;
    const uint32_t pcap = (uint32_t)lv.pcap;
    const uint64_t max_pairs = lv.cap / 2;
    const uint64_t packets = (max_pairs + (1ull << span_log2) - 1) >> span_log2;
    const uint32_t cshift = span_log2 - 5;  // log2(chunks per run)
    const NodeRange nr = level_nodes(*plan, level);
    const uint32_t shift = nr.shift + cshift; // log2(nodes * chunks per run)
    const uint64_t total = packets << shift;
    const uint64_t section_bit = plan->section_offset[side] * 8;
    const uint64_t stride = (uint64_t)grid.nblk * blockDim.x;
    for (uint64_t t = (uint64_t)grid.bid * blockDim.x + threadIdx.x; t < total; t += stride) {
        const uint64_t packet = t >> shift;
        const uint64_t rem = t & ((1ull << shift) - 1);
        const uint32_t node = (uint32_t)(nr.lo + (rem >> cshift));
        const uint64_t pair0 = (packet << span_log2) + ((rem & ((1ull << cshift) - 1)) << 5);
        const uint64_t half = size_at(lv, level, node) / 2;
        if (pair0 >= half) {
            continue;
        }
        const uint64_t q = (uint64_t)node * pcap + pair0;
        // the bit arrays keep one spare word, so bits[w + 1] is always there
        const uint64_t w = q >> 5;
        uint32_t v = __funnelshift_r(bits[w], bits[w + 1], (uint32_t)(q & 31));
        if (half - pair0 < 32) {
            v &= (1u << (uint32_t)(half - pair0)) - 1u;
        }
        if (v == 0) {
            continue;
        }
        const uint64_t dest = section_bit + switch_bit(addr[node], pair0);
        const uint32_t off = (uint32_t)(dest & 31);
        atomicOr(blob + (dest >> 5), v << off);
        if (off != 0 && (v >> (32 - off)) != 0) {
            atomicOr(blob + (dest >> 5) + 1, v >> (32 - off));
        }
    }
}

// Emission forms: the launches of one section at one level (see
// emission_launches, encode.cu).
enum EmitForm : int { kEmitWords = 0, kEmitTranspose, kEmitBlocks, kEmitBits, kEmitForms };

// Both sections' switch bits of one level in one launch: part k owns blocks
// [first, first + blocks).
struct EmitPart {
    int32_t form;
    int32_t side;
    uint32_t first;
    uint32_t blocks;
    uint64_t full; // full packets (block forms) or first packet (per-bit form)
};
struct EmitParts {
    uint32_t count;
    uint32_t blocks;
    EmitPart part[4];
};

__device__ __forceinline__ void level_emit_form(Grid g, int form, const Plan* __restrict__ plan,
    uint32_t level, int side, const uint32_t* __restrict__ bits,
    const NodeAddress* __restrict__ addr, uint32_t* __restrict__ blob, uint64_t full) {
    switch (form) {
    case kEmitWords:
        level_emit_words_run(g, plan, level, side, bits, addr, blob);
        break;
    case kEmitTranspose:
        level_emit_transpose_run(g, plan, level, side, bits, addr, blob, full);
        break;
    case kEmitBlocks:
        level_emit_blocks_run(g, plan, level, side, bits, addr, blob, full);
        break;
    default:
        level_emit_run(g, plan, level, side, bits, addr, blob, full);
        break;
    }
}

__global__ void __launch_bounds__(256) level_emit(const Plan* __restrict__ plan, uint32_t level,
    const __grid_constant__ EmitParts parts, const uint32_t* __restrict__ xbits,
    const uint32_t* __restrict__ ybits, const NodeAddress* __restrict__ in_addr,
    const NodeAddress* __restrict__ out_addr, uint32_t* __restrict__ blob) {
    wait_for_previous();
    uint32_t k = 0;
    while (k + 1 < parts.count && parts.part[k + 1].first <= blockIdx.x) ++k;
    const EmitPart& p = parts.part[k];
    level_emit_form(Grid{blockIdx.x - p.first, p.blocks}, p.form, plan, level, p.side,
        p.side == 0 ? xbits : ybits, p.side == 0 ? in_addr : out_addr, blob, p.full);
}

} // namespace bpb200
