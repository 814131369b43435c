// SPDX-License-Identifier: Apache-2.0
//
// Canonical colouring of the global levels by two-way walks over contracted
// lists.
//
// A node's constraint graph (src/benes.cpp:238-252) is held as its output
// edges: edge[u] is the input that shares input u's output pair, two words
// per pair-node k = inputs {2k, 2k+1}.  The graph is a set of cycles over
// pair-nodes: a path that enters pair-node k at input w leaves it at w^1 and
// goes on to edge[w^1].  All inputs at which a directed path enters have one
// colour; the path walked backwards enters at their partners, which have the
// other.  An odd node's unpaired input t = s-1 gets a virtual partner s, and
// its unpaired output a virtual partner output fed by s, so the tail's path
// closes into a cycle too.  With key(w) = w, or (w - t) mod 2^32 in an odd
// node (which puts t and s first), the canonical rule (odd tail colour 0,
// else the component's smallest input, src/benes.cpp:253-297) says: the
// colour of input w is the low bit of the smallest key on the directed cycle
// through w, because that cycle passes the component's smallest pair-node at
// exactly one of its two inputs.
//
// List 0 is the pair-nodes.  One element of a list in 8, at a hashed place
// (ruler_slot), is an element of the next list.  Two walks leave it, one per
// direction, each up to the next such element or to an element stamped by a
// walk that came the other way, so every element is passed about once, half
// the steps of one-way walks.  A stamp names the walk that passed: kStamp |
// ruler << 1 | (direction ^ side of entry); a walk that enters a stamped
// element at side b goes on as directed ruler (stamp ^ b).  One atomic
// exchange leaves the stamp and fetches what was there: the stamps are then
// only ever touched by atomics and the edges only read.  (Plain loads and
// stores to the same words, whether stamps in the place of edges or in an
// array of their own, cost 13 and 18 ms per level at 2^30 entries against
// 5.6 ms: every sector moved between the two L2 halves at each change.)  A
// walk that meets another replaces the stamp it finds by one that says the
// same.  Each directed ruler keeps its successor and the smallest key its
// own walk saw; a ruler's two walks together cover the stretches around it,
// so folding min(m0, m1 ^ 1) over the rulers of a cycle (^ 1 mirrors a key
// to the other direction) covers the whole cycle.  Lists are contracted
// (list_contract) until a node's elements fit one CTA, which colours them in
// shared memory (list_rank); the colours then go back down the lists
// (list_expand) and to the pair-nodes (level_colours).
//
// Cycles without any ruler are short for all but contrived inputs: each of
// their elements walks them whole.  A walk longer than its cap sets
// kErrGaveUp and the host encodes the permutation again with union-find on
// every level.  Indexes read from memory are range-checked throughout: an
// input that is not a permutation, or a level after a walk that gave up,
// leaves arbitrary words behind.
//
// What bounds the walks: random L2 accesses (a node's edges fit L2 up to
// kWalkMaxNode entries); larger nodes are coloured by union-find.
#pragma once

#include "device.cuh"
#include "kernels.cuh"
#include "plan.hpp"

#include <cstdint>

namespace bpb200 {

#ifndef BPB200_WALK_MAX_LOG2
#define BPB200_WALK_MAX_LOG2 23
#endif
constexpr uint64_t kWalkMaxNode = 1ull << BPB200_WALK_MAX_LOG2; // larger: union-find
static_assert(BPB200_WALK_MAX_LOG2 >= 13 && BPB200_WALK_MAX_LOG2 <= 28, "walk limit out of range");
constexpr uint32_t kRulerLog2 = 3;          // elements per element of the next list (log2)
constexpr uint32_t kRankRulerLog2 = 3;      // the same inside list_rank
constexpr uint32_t kWalkCap = 1u << 16;     // longest walk between rulers
constexpr uint32_t kShortCap = 1u << 10;    // longest cycle without rulers
constexpr uint32_t kStamp = 0x80000000u;    // an element's stamp starts as 0
constexpr uint32_t kNone = 0xffffffffu;     // successor of an absent element
constexpr uint32_t kMaxLists = 5;           // lists of rulers: 1..kMaxLists
constexpr uint32_t kRankMaxLog2 = 14;       // most elements of a node list_rank takes (log2)
constexpr uint32_t kRankMinLog2 = 10;

// Element of list e that element i of list e + 1 stands for.
__host__ __device__ __forceinline__ uint32_t ruler_slot(uint32_t i) {
    return (i << kRulerLog2) + ((i * 0x9E3779B1u) >> (32 - kRulerLog2));
}
__host__ __device__ __forceinline__ bool is_ruler(uint32_t element) {
    return element == ruler_slot(element >> kRulerLog2);
}

// This call's elements of list e (0: pair-nodes): those that stand for the
// pair-nodes [pair_lo, pair_end) lie in [lo, hi); the first and the last may
// stand for a pair-node outside and are absent then.
struct ListRange {
    uint32_t lo, hi;
};

BP_HD ListRange list_range(uint64_t pair_lo, uint64_t pair_end, uint32_t e) {
    return ListRange{(uint32_t)(pair_lo >> (kRulerLog2 * e)),
        (uint32_t)((pair_end - 1) >> (kRulerLog2 * e)) + 1};
}

// Pair-node that element i of list e stands for.
__device__ __forceinline__ uint32_t pair_of(uint32_t i, uint32_t e) {
    for (; e > 0; --e) {
        i = ruler_slot(i);
    }
    return i;
}

// Smallest key of the stretches around a ruler, for paths that enter it in
// direction 0 (direction 1: ^ 1).
__device__ __forceinline__ uint32_t around(uint4 state) { return min(state.y, state.w ^ 1u); }

// The edges of level 0, from its inverse: one thread per output pair.  Every
// later level's edges are written by its parent's output pass, which clears
// the stamps as well.  A slot no value was routed to means a repeated value.
__device__ __forceinline__ void level_edges_run(Grid grid, const Plan* __restrict__ plan,
    const uint32_t* __restrict__ inv, uint32_t* __restrict__ edge, uint32_t* __restrict__ stamp,
    uint32_t* status) {
    const uint32_t s = (uint32_t)plan->levels[0].q;
    const uint32_t np = s - s / 2;
    bool bad = false;
    for (uint32_t k = grid.bid * blockDim.x + threadIdx.x; k < np; k += grid.nblk * blockDim.x) {
        const uint2 both = reinterpret_cast<const uint2*>(inv)[k];
        stamp[k] = 0;
        const uint32_t u = both.x;
        const uint32_t w = 2 * k + 1 < s ? both.y : s;
        if (u >= s || (2 * k + 1 < s && w >= s)) {
            bad = true;
            continue;
        }
        edge[u] = w;
        edge[w] = u;
    }
    if (bad) atomicOr(status, kErrNotPermutation);
}

__global__ void __launch_bounds__(256) level_edges(const Plan* __restrict__ plan,
    const uint32_t* __restrict__ inv, uint32_t* __restrict__ edge, uint32_t* __restrict__ stamp,
    uint32_t* status) {
    wait_for_previous();
    level_edges_run(launch_grid(), plan, inv, edge, stamp, status);
}

// One direction of a walk, advanced one element at a time.  `enter` is the
// side and element it enters next, `best` its smallest key so far.
struct Walk {
    uint32_t enter, best, next;
    bool live;
};

// Walks over the pair-nodes: state[r] = {successor, smallest key} of ruler
// r's two directions.  One thread per ruler, both directions in lockstep, so
// two loads are in flight; blocks start in address order, so the walks in
// flight at any moment touch few nodes.  (Persistent warps that hand every
// lane its next walk as soon as one ends took 11.8 ms per level at 2^30
// entries: the hand-over cost more than the lanes idle behind the longest
// walk of their warp.)  mark[r] = 0 resets the stamps of list_contract.
__device__ __forceinline__ void level_walk_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ edge, uint32_t* stamp,
    uint4* __restrict__ state, uint32_t* __restrict__ mark, uint32_t* status) {
    const LevelInfo& lv = plan->levels[level];
    const uint32_t ps = (uint32_t)lv.pcap;
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t pair_lo = nr.lo * ps;
    const uint64_t pair_end = pair_lo + ((uint64_t)ps << nr.shift);
    const ListRange rr = list_range(pair_lo, pair_end, 1);
    bool bad = false;
    for (uint32_t r = rr.lo + grid.bid * blockDim.x + threadIdx.x; r < rr.hi;
         r += grid.nblk * blockDim.x) {
        mark[r] = 0;
        const uint32_t q = ruler_slot(r);
        const bool in_range = q >= pair_lo && q < pair_end;
        const uint32_t j = in_range ? q / ps : 0u;
        const uint32_t base = j * ps;
        const uint32_t s = in_range ? size_at(lv, level, j) : 0u;
        const uint32_t limit = 2 * (s - s / 2);
        const uint32_t own = 2 * (q - base);
        if (own >= limit) {
            state[r] = make_uint4(kNone, kNone, kNone, kNone);
            continue;
        }
        const uint2* __restrict__ node = reinterpret_cast<const uint2*>(edge) + base;
        const uint32_t bias = (s & 1u) != 0 ? 0u - (s - 1) : 0u;
        const uint2 mine = node[own >> 1];
        Walk w[2] = {{mine.y, own + bias, 2 * r, mine.y < limit},
            {mine.x, own + 1 + bias, 2 * r + 1, mine.x < limit}};
        bad |= !w[0].live || !w[1].live;
        for (uint32_t step = 0; (w[0].live || w[1].live) && step < kWalkCap; ++step) {
            bool ruler[2];
            uint2 v[2];
            uint32_t found[2];
#pragma unroll
            for (uint32_t d = 0; d < 2; ++d) {
                const uint32_t at = base + (w[d].enter >> 1);
                ruler[d] = is_ruler(at);
                v[d] = make_uint2(0u, 0u);
                found[d] = kStamp;
                if (w[d].live && !ruler[d]) {
                    v[d] = node[w[d].enter >> 1];
                    found[d] = atomicExch(stamp + at, kStamp | (r << 1) | (d ^ (w[d].enter & 1u)));
                }
            }
#pragma unroll
            for (uint32_t d = 0; d < 2; ++d) {
                if (!w[d].live) continue;
                const uint32_t side = w[d].enter & 1u;
                if ((found[d] & kStamp) != 0) {
                    w[d].next = side ^ (ruler[d]
                        ? ((base + (w[d].enter >> 1)) >> kRulerLog2) << 1 : found[d] & ~kStamp);
                    w[d].live = false;
                } else {
                    w[d].best = min(w[d].best, w[d].enter + bias);
                    w[d].enter = side != 0 ? v[d].x : v[d].y;
                    if (w[d].enter >= limit) {
                        bad = true;
                        w[d].live = false;
                    }
                }
            }
        }
        bad |= w[0].live || w[1].live;
        state[r] = make_uint4(w[0].next, w[0].best, w[1].next, w[1].best);
    }
    if (bad) atomicOr(status, kErrGaveUp);
}

__global__ void __launch_bounds__(256, 8) level_walk(const Plan* __restrict__ plan, uint32_t level,
    const uint32_t* __restrict__ edge, uint32_t* stamp, uint4* __restrict__ state,
    uint32_t* __restrict__ mark, uint32_t* status) {
    wait_for_previous();
    level_walk_run(launch_grid(), plan, level, edge, stamp, state, mark, status);
}

// Walks over list e (state, mark), giving list e + 1 (up_state, up_mark).
// Same walks as level_walk with a list element's two successors in the place
// of a pair-node's edges and its stamp in mark[]; one walk per thread, in
// address order.
__device__ __forceinline__ void list_contract_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, uint32_t e, const uint4* __restrict__ state, uint32_t* mark,
    uint4* __restrict__ up_state, uint32_t* __restrict__ up_mark, uint32_t* status) {
    const uint32_t ps = (uint32_t)plan->levels[level].pcap;
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t pair_lo = nr.lo * ps;
    const uint64_t pair_end = pair_lo + ((uint64_t)ps << nr.shift);
    const ListRange from = list_range(pair_lo, pair_end, e);
    const ListRange to = list_range(pair_lo, pair_end, e + 1);
    uint2* half = reinterpret_cast<uint2*>(up_state);
    bool bad = false;
    for (uint64_t unit = 2ull * to.lo + (uint64_t)grid.bid * blockDim.x + threadIdx.x;
         unit < 2ull * to.hi; unit += (uint64_t)grid.nblk * blockDim.x) {
        const uint32_t up = (uint32_t)(unit >> 1);
        const uint32_t r = ruler_slot(up);
        if ((unit & 1) == 0) up_mark[up] = 0;
        uint4 st = make_uint4(kNone, kNone, kNone, kNone);
        if (r >= from.lo && r < from.hi) st = state[r];
        if (st.x == kNone) {
            half[unit] = make_uint2(kNone, kNone);
            continue;
        }
        uint32_t cur = (r << 1) | (uint32_t)(unit & 1);
        uint32_t m = ~0u, next = kNone;
        for (uint32_t step = 0; next == kNone; ++step) {
            m = min(m, around(st) ^ (cur & 1u));
            cur = (cur & 1u) != 0 ? st.z : st.x;
            const uint32_t at = cur >> 1;
            if (at < from.lo || at >= from.hi || step == kWalkCap) {
                bad = true;
                next = (uint32_t)unit;
            } else if (is_ruler(at)) {
                next = ((at >> kRulerLog2) << 1) | (cur & 1u);
            } else {
                st = state[at];
                const uint32_t found = atomicExch(mark + at, kStamp | ((uint32_t)unit ^ (cur & 1u)));
                if ((found & kStamp) != 0) {
                    next = (found & ~kStamp) ^ (cur & 1u);
                }
            }
        }
        half[unit] = make_uint2(next, m);
    }
    if (bad) atomicOr(status, kErrGaveUp);
}

__global__ void __launch_bounds__(256) list_contract(const Plan* __restrict__ plan,
    uint32_t level, uint32_t e, const uint4* __restrict__ state, uint32_t* mark,
    uint4* __restrict__ up_state, uint32_t* __restrict__ up_mark, uint32_t* status) {
    wait_for_previous();
    list_contract_run(launch_grid(), plan, level, e, state, mark, up_state, up_mark, status);
}

// Colours of list e's elements (colour[i]: the colour of paths that enter
// element i in direction 0) from those of list e + 1.
__device__ __forceinline__ void list_expand_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, uint32_t e, const uint4* __restrict__ state,
    const uint32_t* __restrict__ mark, const uint8_t* __restrict__ up_colour,
    uint8_t* __restrict__ colour, uint32_t* status) {
    const uint32_t ps = (uint32_t)plan->levels[level].pcap;
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t pair_lo = nr.lo * ps;
    const uint64_t pair_end = pair_lo + ((uint64_t)ps << nr.shift);
    const ListRange from = list_range(pair_lo, pair_end, e);
    const ListRange to = list_range(pair_lo, pair_end, e + 1);
    bool bad = false;
    for (uint32_t i = from.lo + grid.bid * blockDim.x + threadIdx.x; i < from.hi;
         i += grid.nblk * blockDim.x) {
        const uint32_t stamp = mark[i];
        uint32_t c;
        if (is_ruler(i)) {
            c = up_colour[i >> kRulerLog2];
        } else if ((stamp & kStamp) != 0) {
            const uint32_t up = (stamp & ~kStamp) >> 1;
            const bool in_range = up >= to.lo && up < to.hi;
            bad |= !in_range;
            c = in_range ? up_colour[up] ^ (stamp & 1u) : 0u;
        } else {
            uint4 st = state[i];
            if (st.x == kNone) continue;
            uint32_t cur = i << 1, m = ~0u, step = 0;
            do {
                m = min(m, around(st) ^ (cur & 1u));
                cur = (cur & 1u) != 0 ? st.z : st.x;
                const uint32_t at = cur >> 1;
                if (at < from.lo || at >= from.hi || ++step == kShortCap) {
                    bad = true;
                    break;
                }
                st = state[at];
            } while (cur != i << 1);
            c = m & 1u;
        }
        colour[i] = (uint8_t)(c & 1u);
    }
    if (bad) atomicOr(status, kErrGaveUp);
}

__global__ void __launch_bounds__(256) list_expand(const Plan* __restrict__ plan, uint32_t level,
    uint32_t e, const uint4* __restrict__ state, const uint32_t* __restrict__ mark,
    const uint8_t* __restrict__ up_colour, uint8_t* __restrict__ colour, uint32_t* status) {
    wait_for_previous();
    list_expand_run(launch_grid(), plan, level, e, state, mark, up_colour, colour, status);
}

// Most elements of one node in list e (one more at either end when nodes
// start inside an element's bucket).
BP_HD uint32_t list_node_max(uint64_t ps, uint32_t e) {
    const uint32_t sh = kRulerLog2 * e;
    return (ps & ((1ull << sh) - 1)) == 0 ? (uint32_t)(ps >> sh) : (uint32_t)((ps - 1) >> sh) + 2;
}

// Element of a node's list that ruler i of list_rank stands for.
__device__ __forceinline__ uint32_t rank_slot(uint32_t i) {
    return (i << kRankRulerLog2) + ((i * 0x9E3779B1u) >> (32 - kRankRulerLog2));
}

// Dynamic shared memory of list_rank for nodes of `count` elements.
BP_HD uint32_t rank_smem(uint32_t count) {
    const uint32_t rulers = ((count - 1) >> kRankRulerLog2) + 1;
    return count * 8 + rulers * 16;
}
constexpr uint32_t kRankThreads = 1024;
constexpr uint32_t kRankBatch = 5; // directed states per thread, at least 2 * rulers / threads

// Threads of a list_rank launch: one per 4 elements, so a thread's loads of
// list states are few; at most kRankBatch directed states each.
BP_HD uint32_t rank_threads(uint32_t count) {
    uint32_t t = 128;
    while (t < kRankThreads && t * 4 < count) t *= 2;
    return t;
}

// Colours of every element of list e, one CTA per node: the node's list is
// contracted once more in shared memory by the tile's ruler walk and
// finished by pointer tripling over the rulers.  Element i's word holds the
// local directed successors: low half that of direction 1, high half that of
// direction 0 (so a path entering at side b leaves through half b ^ 1, as
// with a pair-node's edges), or a stamp.
__device__ __forceinline__ void list_rank_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, uint32_t e, const uint4* __restrict__ state, uint8_t* __restrict__ colour,
    uint32_t* status, uint32_t* smem) {
    const uint32_t ps = (uint32_t)plan->levels[level].pcap;
    const NodeRange nr = level_nodes(*plan, level);
    const uint32_t tid = threadIdx.x;
    bool bad = false;
    for (uint64_t j = nr.lo + grid.bid; j < nr.lo + (1ull << nr.shift); j += grid.nblk) {
        const uint64_t pair_lo = j * ps;
        const ListRange range = list_range(pair_lo, pair_lo + ps, e);
        const uint32_t count = range.hi - range.lo;
        const uint32_t rulers = ((count - 1) >> kRankRulerLog2) + 1;
        volatile uint32_t* link = smem;
        volatile uint16_t* link16 = reinterpret_cast<volatile uint16_t*>(smem);
        uint32_t* key = smem + count;
        uint32_t* smin = key + count;      // 2 * rulers
        uint32_t* snext = smin + 2 * rulers;
        __syncthreads(); // the previous node's arrays are free
        constexpr uint32_t kBatch = 8; // states in flight per thread
        for (uint32_t i0 = tid; i0 < count; i0 += kBatch * blockDim.x) {
            uint4 st[kBatch];
#pragma unroll
            for (uint32_t b = 0; b < kBatch; ++b) {
                const uint32_t i = i0 + b * blockDim.x;
                st[b] = make_uint4(kNone, 0u, 0u, 0u);
                if (i < count) {
                    const uint32_t q = pair_of(range.lo + i, e);
                    if (q >= pair_lo && q < pair_lo + ps) st[b] = state[range.lo + i];
                }
            }
#pragma unroll
            for (uint32_t b = 0; b < kBatch; ++b) {
                const uint32_t i = i0 + b * blockDim.x;
                if (i >= count) break;
                uint32_t word = 0x8000u; // not here: nothing leads to it
                uint32_t k = ~0u;
                if (st[b].x != kNone) {
                    uint32_t x = st[b].x - 2 * range.lo, z = st[b].z - 2 * range.lo;
                    if (x >= 2 * count || z >= 2 * count) {
                        bad = true;
                        x = 2 * i;
                        z = 2 * i + 1;
                    }
                    word = z | (x << 16);
                    k = around(st[b]);
                }
                key[i] = k;
                link[i] = word;
            }
        }
        __syncthreads();
        // rulers first: their word moves to the state, a stamp takes its place
        for (uint32_t r = tid; r < rulers; r += blockDim.x) {
            const uint32_t i = rank_slot(r);
            const uint32_t word = i < count ? link[i] : 0x8000u;
            snext[2 * r] = word;
            if ((word & 0x8000u) == 0) link16[2 * i] = (uint16_t)(0x8000u | (r << 1));
        }
        __syncthreads();
        for (uint32_t r = tid; r < rulers; r += blockDim.x) {
            const uint32_t word = snext[2 * r];
            if ((word & 0x8000u) != 0) {
                snext[2 * r] = 2 * r;
                snext[2 * r + 1] = 2 * r + 1;
                smin[2 * r] = smin[2 * r + 1] = ~0u;
                continue;
            }
            const uint32_t own = key[rank_slot(r)];
            uint32_t wa = word >> 16, wb = word & 0xffffu;
            uint32_t ma = own, mb = own ^ 1u;
            uint32_t va, vb;
            bool ga = true, gb = true;
            for (uint32_t step = 0; step <= count; ++step) {
                // both walks and their keys in flight together; a walk that
                // has ended reads its last word again
                va = link[wa >> 1];
                vb = link[wb >> 1];
                const uint32_t ka = key[wa >> 1] ^ (wa & 1u);
                const uint32_t kb = key[wb >> 1] ^ (wb & 1u);
                ga = (va & 0x8000u) == 0;
                gb = (vb & 0x8000u) == 0;
                if (ga) link16[wa & ~1u] = (uint16_t)(0x8000u | (r << 1) | (wa & 1u));
                if (gb) link16[wb & ~1u] = (uint16_t)(0x8000u | (r << 1) | (~wb & 1u));
                if (!ga && !gb) break;
                ma = ga ? min(ma, ka) : ma;
                mb = gb ? min(mb, kb) : mb;
                wa = ga ? (va >> ((~wa & 1u) << 4)) & 0xffffu : wa;
                wb = gb ? (vb >> ((~wb & 1u) << 4)) & 0xffffu : wb;
            }
            const uint32_t na = ga ? 2 * r : (va & 0x7fffu) ^ (wa & 1u);
            const uint32_t nb = gb ? 2 * r + 1 : (vb & 0x7fffu) ^ (wb & 1u);
            bad |= ga || gb || na >= 2 * rulers || nb >= 2 * rulers;
            const uint32_t m = min(ma, mb ^ 1u);
            smin[2 * r] = m;
            smin[2 * r + 1] = m ^ 1u;
            snext[2 * r] = na < 2 * rulers ? na : 2 * r;
            snext[2 * r + 1] = nb < 2 * rulers ? nb : 2 * r + 1;
        }
        __syncthreads();
        for (uint32_t reach = 1; reach < rulers + 1; reach *= 3) {
            uint32_t om[kRankBatch], on[kRankBatch];
#pragma unroll
            for (uint32_t b = 0; b < kRankBatch; ++b) {
                const uint32_t i = tid + b * blockDim.x;
                if (i >= 2 * rulers) continue;
                const uint32_t n1 = snext[i];
                const uint32_t n2 = snext[n1];
                om[b] = min(smin[i], min(smin[n1], smin[n2]));
                on[b] = snext[n2];
            }
            __syncthreads();
#pragma unroll
            for (uint32_t b = 0; b < kRankBatch; ++b) {
                const uint32_t i = tid + b * blockDim.x;
                if (i >= 2 * rulers) continue;
                smin[i] = om[b];
                snext[i] = on[b];
            }
            __syncthreads();
        }
        for (uint32_t i = tid; i < count; i += blockDim.x) {
            const uint32_t word = link[i];
            uint32_t c;
            if ((word & 0x8000u) != 0) {
                if (key[i] == ~0u) continue; // another node's, or absent
                const uint32_t r2 = word & 0x7ffeu;
                c = r2 < 2 * rulers ? smin[r2] ^ word : 0u;
            } else { // a cycle without rulers
                uint32_t cur = 2 * i, v = word, m = ~0u, step = 0;
                do {
                    m = min(m, key[cur >> 1] ^ (cur & 1u));
                    cur = (cur & 1u) != 0 ? v & 0xffffu : v >> 16;
                    if (cur >= 2 * count || ++step == kShortCap) {
                        bad = true;
                        break;
                    }
                    v = link[cur >> 1];
                } while (cur != 2 * i);
                c = m;
            }
            colour[range.lo + i] = (uint8_t)(c & 1u);
        }
    }
    if (bad) atomicOr(status, kErrGaveUp);
}

__global__ void __launch_bounds__(kRankThreads, 1) list_rank(const Plan* __restrict__ plan,
    uint32_t level, uint32_t e, const uint4* __restrict__ state, uint8_t* __restrict__ colour,
    uint32_t* status) {
    extern __shared__ __align__(16) uint32_t rank_shared[];
    wait_for_previous();
    list_rank_run(launch_grid(), plan, level, e, state, colour, status, rank_shared);
}

// Input switch bits of a walk level: the colour of input 2k of every
// pair-node k, from the stamp of the walk that passed it and that ruler's
// colour.  One thread per pair-node, in address order.
__device__ __forceinline__ void level_colours_run(Grid grid, const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ edge, const uint32_t* __restrict__ stamp,
    const uint8_t* __restrict__ colour, uint32_t* __restrict__ xbits, uint32_t* status) {
    const LevelInfo& lv = plan->levels[level];
    const uint32_t ps = (uint32_t)lv.pcap;
    // this call's pair-nodes; the loop starts at a 32-pair boundary so each
    // warp assembles whole bit words (bits before `first` stay zero)
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t first = nr.lo * ps;
    const uint64_t end = first + ((uint64_t)ps << nr.shift);
    const ListRange rr = list_range(first, end, 1);
    const uint2* pairs = reinterpret_cast<const uint2*>(edge);
    bool bad = false;
    for (uint64_t p = (first & ~31ull) + (uint64_t)grid.bid * blockDim.x + threadIdx.x;
         p - (threadIdx.x & 31) < end; p += (uint64_t)grid.nblk * blockDim.x) {
        uint32_t x = 0;
        if (p >= first && p < end) {
            const uint32_t q = (uint32_t)p;
            const uint32_t v = __ldcs(stamp + q);
            if (is_ruler(q)) {
                x = colour[q >> kRulerLog2];
            } else if ((v & kStamp) != 0) {
                const uint32_t r = (v & ~kStamp) >> 1;
                // padding pair-nodes hold anything; their bits are not used
                if (r >= rr.lo && r < rr.hi) x = colour[r] ^ v;
            } else {
                const uint32_t j = q / ps;
                const uint32_t k = q - j * ps;
                const uint32_t s = size_at(lv, level, j);
                const uint32_t limit = 2 * (s - s / 2);
                if (2 * k < limit) { // a cycle without rulers: walk it whole
                    const uint2* node = pairs + (uint64_t)j * ps;
                    const uint32_t bias = (s & 1u) != 0 ? 0u - (s - 1) : 0u;
                    uint32_t cur = 2 * k, step = 0;
                    uint2 word = node[k];
                    x = ~0u;
                    do {
                        x = min(x, cur + bias);
                        cur = (cur & 1u) != 0 ? word.x : word.y;
                        if (cur >= limit || ++step == kShortCap) {
                            bad = true;
                            break;
                        }
                        word = node[cur >> 1];
                    } while (cur != 2 * k);
                }
            }
        }
        const unsigned word = __ballot_sync(0xffffffffu, (x & 1u) != 0);
        if ((threadIdx.x & 31) == 0) {
            xbits[p >> 5] = word;
        }
    }
    if (bad) atomicOr(status, kErrGaveUp);
}

__global__ void __launch_bounds__(256) level_colours(const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ edge, const uint32_t* __restrict__ stamp,
    const uint8_t* __restrict__ colour, uint32_t* __restrict__ xbits, uint32_t* status) {
    wait_for_previous();
    level_colours_run(launch_grid(), plan, level, edge, stamp, colour, xbits, status);
}

} // namespace bpb200
