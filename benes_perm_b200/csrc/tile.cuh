// SPDX-License-Identifier: Apache-2.0
//
// Tile kernel: one CTA per node of the tile level; the node's whole subtree
// (every remaining routing level plus the middle-group ranks) is encoded in
// shared memory, on 16-bit node-local indexes.
//
// A node is held as its inverse (inv[o] = the input routed to output o) and
// as its output edges: edge[u] is the input that shares input u's output
// pair, edge[inv[2k]] = inv[2k+1] and back.  With pair-node k = inputs
// {2k, 2k+1}, one 32-bit word per pair-node holds both edges, and the
// constraint graph (src/benes.cpp:238-252) is a set of cycles over
// pair-nodes: a path that enters pair-node k at input w leaves it at w^1 and
// goes on to edge[w^1].  The inputs at which a path enters all have one
// colour, and walked backwards the path enters at their partners, which have
// the other.  An odd node's unpaired input t = s-1 gets a virtual partner s,
// and its unpaired output a virtual partner output fed by s, which closes
// the tail's path into a cycle as well.  The canonical rule (the odd tail
// has colour 0, else the component's smallest input has) is then: with
// key(v) = v, or (v - t) mod 2^16 in an odd node (which puts t and s first),
// the colour of input v is the low bit of the smallest key on the directed
// cycle through v, because that cycle passes the component's smallest
// pair-node at exactly one of its two inputs.
//
// What bounds it: shared-memory latency and instruction issue; nothing
// leaves the SM between the input load and the switch bits.
#pragma once

#include "device.cuh"
#include "kernels.cuh"
#include "plan.hpp"

#include <cstdint>

namespace bpb200 {

__host__ __device__ inline uint32_t align_up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

// Division by a per-level constant: floor(n / d) = umulhi(n, ceil(2^32 / d))
// exactly whenever n * d < 2^32 (the rounding error n * (m - 2^32/d) / 2^32
// stays below 1/d), which holds for tile indices: n and d are below 2^16.
struct FastDiv {
    uint32_t d, m;
    __device__ explicit FastDiv(uint32_t div)
        : d(div), m(div > 1 ? 0xffffffffu / div + 1u : 0u) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const {
        return d > 1 ? __umulhi(n, m) : n;
    }
};

// Pair-nodes per node in the tile's arrays: the level's pair-nodes rounded
// up to an even number, so that a node's inverse starts on an 8-byte
// boundary and four outputs (two output pairs) are one 64-bit load.
__host__ __device__ inline uint32_t tile_pair_stride(uint64_t pcap) {
    return ((uint32_t)pcap + 1u) & ~1u;
}

// One pair-node in 2^tile_ruler_log2 is a ruler (see the walk below), and
// nodes of at most tile_serial_pairs pair-nodes are coloured by one thread
// each.  Large tiles are bound by instruction issue: few rulers, and serial
// nodes of up to 64 pair-nodes (8192 entries: 2^26 entries' tiles 3.47 ms
// against 3.67 with a ruler per 4).  Tiles of up to 4096 slots leave most of
// their SM idle and wait for their longest walk: a ruler per 4 and fewer
// serial nodes (1000 entries: 68.4 -> 63.2 us a call, 4096: 85.3 -> 81.5; a
// ruler per 2: 67.3 and 88.6).
constexpr uint32_t kSmallTileSlots = 4096;
__host__ __device__ inline uint32_t tile_ruler_log2(uint32_t slots) {
    return slots <= kSmallTileSlots ? 2u : 3u;
}
__host__ __device__ inline uint32_t tile_serial_pairs(uint32_t slots) {
    return slots <= kSmallTileSlots ? 32u : 64u;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory accesses of the walks, by 32-bit address: words that other
// threads of the block rewrite meanwhile, and a store without a branch.
__device__ __forceinline__ uint32_t shared_load(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ void shared_store16_if(bool yes, uint32_t addr, uint32_t v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t"
                 "@p st.volatile.shared.u16 [%1], %2;\n\t}"
                 :: "r"((uint32_t)yes), "r"(addr), "h"((uint16_t)v) : "memory");
}

// Slots per node in the tile's arrays: two per pair-node of the stride, or,
// at the leaf level, a leaf's entries if those are fewer.
__host__ __device__ inline uint32_t tile_node_slots(uint64_t pcap, bool leaf_level, uint32_t leaf) {
    const uint32_t slots = 2 * tile_pair_stride(pcap);
    return leaf_level && leaf < slots ? leaf : slots;
}

// Words of one section's switch bits at one level, with a spare word.
__host__ __device__ inline uint32_t tile_bit_words(uint32_t slots) { return slots / 64 + 2; }

// Byte offsets of the smem arrays; identical on host (sizing) and device.
// `slots`: nodes * tile_node_slots at the level that needs most; `levels`:
// routing levels in the tile.
__host__ __device__ inline uint32_t tile_smem_layout(uint32_t slots, uint32_t levels,
    uint32_t* off) {
    const uint32_t rulers = (slots >> (tile_ruler_log2(slots) + 1)) + 1;
    uint32_t o = 0;
    off[0] = o; o = align_up(o + slots * 2, 16);           // inverse, even levels
    off[1] = o; o = align_up(o + slots * 2, 16);           // inverse, odd levels
    off[2] = o; o = align_up(o + slots * 2, 16);           // edges, one word per pair-node
    off[3] = o; o = align_up(o + rulers * 8, 16);          // directed ruler states
    off[4] = o; // switch bits of every level, input and output section
    o = align_up(o + 2 * levels * tile_bit_words(slots) * 4, 16);
    return o;
}

// Colours one node of at most 64 pair-nodes (Mask: 32 or 64 bits) with one
// thread: cycle after cycle from the smallest unvisited pair-node, the odd
// tail's first, exactly the canonical order, so every cycle's first input
// has colour 0 and no minimum is needed.  One dependent shared-memory load
// per pair-node.  Returns bit k = colour of input 2k.
template <typename Mask>
__device__ __forceinline__ Mask tile_colour_node(const uint32_t* edge, uint32_t s) {
    const uint32_t np = s - s / 2;
    Mask todo = np >= sizeof(Mask) * 8 ? ~(Mask)0 : (((Mask)1 << np) - 1);
    Mask x = 0;
    uint32_t w = (s & 1u) != 0 ? s - 1 : 0u;
    for (uint32_t i = 0; i < np; ++i) {
        const uint32_t k = w >> 1;
        const uint32_t v = edge[k];
        todo &= ~((Mask)1 << k);
        x |= (Mask)(w & 1u) << k;
        w = (w & 1u) != 0 ? v & 0xffffu : v >> 16;
        if (((todo >> (w >> 1)) & 1u) == 0) { // cycle closed
            w = 2u * (uint32_t)(sizeof(Mask) == 8 ? __ffsll((long long)todo) : __ffs((int)todo)) - 2u;
        }
    }
    return x;
}

// Levels [T0, stop) of one node of level T0.  stop = the routing depth: the
// whole subtree, down to the ranks.  An earlier stop leaves the inverses of
// the nodes of level `stop` (all of them internal) in next_inv, laid out as
// level_outputs does: a stage of the subtree, after which more CTAs go on.
// kPlanNear: the plan is already in shared memory.
template <typename T, bool kPlanNear = false>
__device__ __forceinline__ void tile_body(const Plan* __restrict__ plan_ptr,
    const T* __restrict__ src, uint32_t* __restrict__ blob, uint32_t* status, uint32_t slots,
    uint32_t tile, unsigned char* smem, uint32_t T0, uint32_t stop,
    uint32_t* __restrict__ next_inv) {
    uint32_t off[5];
    tile_smem_layout(slots, stop - T0, off);
    uint16_t* invs[2] = {(uint16_t*)(smem + off[0]), (uint16_t*)(smem + off[1])};
    uint32_t* edge = (uint32_t*)(smem + off[2]);
    uint16_t* edge16 = (uint16_t*)edge;
    uint32_t* state = (uint32_t*)(smem + off[3]);
    volatile uint32_t* vstate = state;
    uint32_t* level_bits = (uint32_t*)(smem + off[4]);
    const uint32_t bit_words = tile_bit_words(slots);
    const uint32_t ruler_log2 = tile_ruler_log2(slots);
    const uint32_t serial_pairs = tile_serial_pairs(slots);

    const Plan& plan = *plan_ptr;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31;
    const uint32_t warp = tid >> 5;
    const uint32_t nwarps = blockDim.x >> 5;
    const uint32_t D = plan.depth;
    const uint32_t leaf = plan.leaf;
    const uint32_t J = tile;

    if (T0 > 0 && size_at(plan.levels[T0 - 1], T0 - 1, J >> 1) <= leaf) {
        return; // child of a leaf: not part of the tree
    }
    // The levels and groups the tile works on, into L1: their first uses would
    // otherwise be chains of dependent L2 reads at every level.
    if (!kPlanNear) {
        uint32_t sum = 0;
        const char* lo = reinterpret_cast<const char*>(&plan);
        auto touch = [&](const void* from, const void* to) {
            const uint32_t a = (uint32_t)((const char*)from - lo) & ~127u;
            const uint32_t b = (uint32_t)((const char*)to - lo);
            for (uint32_t at = a + 128 * tid; at < b; at += 128 * blockDim.x) {
                sum += *reinterpret_cast<const uint32_t*>(lo + at);
            }
        };
        touch(&plan, &plan.groups[0][plan.group_count[0]]);
        touch(&plan.groups[1][0], &plan.groups[1][plan.group_count[1]]);
        touch(&plan.levels[0], &plan.levels[D + 1]);
        asm volatile("" :: "r"(sum));
    }
    // The tile's own node: its inverse and edges, or, when it is a leaf, its
    // values.  A whole permutation (tile level 0) is given by its values, a
    // node of a later level by its inverse.  A tile that is not a permutation
    // ends here, so everything below runs on valid indexes.
    {
        const LevelInfo& l0 = plan.levels[T0];
        const uint32_t s0 = size_at(l0, T0, J);
        const uint32_t np = s0 - s0 / 2;
        const uint32_t ps0 = tile_pair_stride(l0.pcap);
        uint16_t* inv = invs[0];
        uint32_t* inv32 = reinterpret_cast<uint32_t*>(inv);
        const bool is_leaf = s0 <= leaf;
        bool bad = false;
        // every load of a batch is issued before any is used
        constexpr int kBatch = 8;
        if (T0 == 0) {
            // never-written inverse slots mean a repeated value
            for (uint32_t e = tid; e < ps0; e += blockDim.x) inv32[e] = ~0u;
            __syncthreads();
            for (uint32_t i0 = tid; i0 < s0; i0 += kBatch * blockDim.x) {
                uint64_t v[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const uint32_t i = i0 + q * blockDim.x;
                    v[q] = i < s0 ? (uint64_t)__ldcs(src + i) : 0;
                }
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const uint32_t i = i0 + q * blockDim.x;
                    if (i >= s0) {
                        break;
                    }
                    if (v[q] >= s0) {
                        bad = true;
                    } else {
                        inv[is_leaf ? i : (uint32_t)v[q]] = (uint16_t)(is_leaf ? v[q] : i);
                    }
                }
            }
            __syncthreads();
            for (uint32_t k = tid; k < np && !is_leaf; k += blockDim.x) {
                const uint32_t both = inv32[k];
                const uint32_t u = both & 0xffffu;
                const uint32_t w = 2 * k + 1 < s0 ? both >> 16 : s0; // virtual partner
                if (u >= s0 || (2 * k + 1 < s0 && w >= s0)) {
                    bad = true;
                } else {
                    edge16[u] = (uint16_t)w;
                    edge16[w] = (uint16_t)u;
                }
            }
        } else {
            // never-written edges mean a repeated value
            for (uint32_t k = tid; k < np; k += blockDim.x) edge[k] = ~0u;
            __syncthreads();
            const uint2* in = reinterpret_cast<const uint2*>(src) + (uint64_t)J * l0.pcap;
            for (uint32_t k0 = tid; k0 < np; k0 += kBatch * blockDim.x) {
                uint2 v[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const uint32_t k = k0 + q * blockDim.x;
                    v[q] = k < np ? __ldcs(in + k) : make_uint2(0u, 0u);
                }
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const uint32_t k = k0 + q * blockDim.x;
                    if (k >= np) {
                        break;
                    }
                    const uint32_t u = v[q].x;
                    const uint32_t w = 2 * k + 1 < s0 ? v[q].y : s0; // virtual partner
                    if (u >= s0 || (2 * k + 1 < s0 && w >= s0)) {
                        bad = true;
                    } else {
                        inv32[k] = u | (w << 16);
                        edge16[u] = (uint16_t)w;
                        edge16[w] = (uint16_t)u;
                    }
                }
            }
            __syncthreads();
            for (uint32_t k = tid; k < np; k += blockDim.x) {
                const uint32_t both = edge[k];
                bad |= (both & 0xffffu) == 0xffffu || (both >> 16) == 0xffffu;
            }
        }
        if (__syncthreads_or(bad)) {
            if (tid == 0) atomicOr(status, not_permutation(T0));
            return;
        }
    }

    for (uint32_t t = 0; T0 + t < stop; ++t) {
        const uint32_t level = T0 + t;
        const LevelInfo& lv = plan.levels[level];
        const uint32_t nodes = 1u << t;
        const uint32_t first = J << t;
        const uint32_t q32 = (uint32_t)lv.q;
        const uint32_t r32 = (uint32_t)lv.r;
        const uint32_t ps = tile_pair_stride(lv.pcap);
        const uint32_t stride = 2 * ps;
        const FastDiv by_ps(ps);
        const uint16_t* cur = invs[t & 1]; // this level's inverse
        uint16_t* nxt = invs[(t + 1) & 1]; // the children's (values, for leaves)
        uint32_t* xbits = level_bits + 2 * t * bit_words;
        uint32_t* ybits = xbits + bit_words;
        // uniform per level: whether every node here exists / is internal
        const bool all_exist = level == 0 || plan.levels[level - 1].q > leaf;
        const bool all_internal = q32 > leaf && all_exist;
        auto node_size = [&](uint32_t path) {
            // levels without large nodes (all of a power-of-two count): q
            if (r32 == 0) return q32;
            return q32 + ((__brev(first + path) >> (32 - level)) < r32 ? 1u : 0u);
        };
        auto exists = [&](uint32_t path) {
            return all_exist ||
                size_at(plan.levels[level - 1], level - 1, (first + path) >> 1) > leaf;
        };
        auto internal_node = [&](uint32_t path, uint32_t s) {
            return all_internal || (s > leaf && exists(path));
        };

        // key(w) = (w + bias) mod 2^16 (see the top of this file)
        auto key_bias = [](uint32_t s) { return (s & 1u) != 0 ? 0u - (s - 1u) : 0u; };

        {
            // ---- input switch bits: the colour of input 2k of every pair-node
            if (ps <= serial_pairs) {
                for (uint32_t e = tid; e < (nodes * ps + 31) / 32 + 1; e += blockDim.x) xbits[e] = 0;
                __syncthreads();
                for (uint32_t path = tid; path < nodes; path += blockDim.x) {
                    const uint32_t s = node_size(path);
                    if (!internal_node(path, s)) {
                        continue;
                    }
                    const uint32_t at = path * ps;
                    uint64_t x;
                    if (ps <= 32) {
                        x = tile_colour_node<uint32_t>(edge + at, s);
                    } else {
                        x = tile_colour_node<uint64_t>(edge + at, s);
                    }
                    const uint32_t sh = at & 31;
                    const uint64_t lo = x << sh;
                    uint32_t* word = xbits + (at >> 5);
                    if ((uint32_t)lo != 0) atomicOr(word, (uint32_t)lo);
                    if ((lo >> 32) != 0) atomicOr(word + 1, (uint32_t)(lo >> 32));
                    if (sh != 0 && (x >> (64 - sh)) != 0) {
                        atomicOr(word + 2, (uint32_t)(x >> (64 - sh)));
                    }
                }
            } else {
                // Ruler walks.  One pair-node in 2^ruler_log2 (hashed) is
                // a ruler; a thread walks both directions away from it until
                // each meets a ruler or a pair-node stamped by a walk coming
                // the other way, so every pair-node is passed about once.  A
                // passed pair-node's edge word becomes the stamp 0x8000 |
                // ruler << 1 | (direction ^ side of entry): each pair-node
                // needs its edges once only.  Rulers are stamped first, as
                // passed by their own direction 0.  A walk that enters a
                // stamped pair-node at input w goes on as directed ruler
                // stamp ^ (w & 1); two walks crossing may both stamp the
                // pair-nodes where they cross, with stamps that say the same.
                const uint32_t rulers = (nodes * ps + (1u << ruler_log2) - 1) >> ruler_log2;
                const uint32_t edge_addr = smem_addr(edge);
                for (uint32_t r = tid; r < rulers; r += blockDim.x) {
                    const uint32_t at = (r << ruler_log2) +
                        ((r * 0x9E3779B1u) >> (32 - ruler_log2));
                    const uint32_t path = by_ps(at);
                    const uint32_t s = path < nodes ? node_size(path) : 0;
                    const bool real = at - path * ps < s - s / 2 && internal_node(path, s);
                    state[2 * r] = real ? edge[at] : 0x80000000u; // no input index: padding
                    if (real) edge16[2 * at] = (uint16_t)(0x8000u | (r << 1));
                }
                __syncthreads();
                for (uint32_t r = tid; r < rulers; r += blockDim.x) {
                    const uint32_t mine = state[2 * r];
                    if (mine == 0x80000000u) {
                        state[2 * r] = 0xffff0000u | (2 * r);
                        state[2 * r + 1] = 0xffff0000u | (2 * r + 1);
                        continue;
                    }
                    const uint32_t at = (r << ruler_log2) +
                        ((r * 0x9E3779B1u) >> (32 - ruler_log2));
                    const uint32_t path = by_ps(at);
                    const uint32_t base = path * ps;
                    const uint32_t bias = key_bias(node_size(path));
                    const uint32_t v0 = 2 * (at - base);
                    // both walks advance together, two loads in flight
                    uint32_t wa = mine >> 16, wb = mine & 0xffffu;
                    uint32_t ma = (v0 + bias) & 0xffffu, mb = (v0 + 1 + bias) & 0xffffu;
                    const uint32_t mark = 0x8000u | (r << 1);
                    const uint32_t at0 = edge_addr + 4 * base;
                    uint32_t pa, pb; // 0 while the walk goes on
                    uint32_t qa, qb;
                    do {
                        qa = at0 + ((wa << 1) & ~3u);
                        qb = at0 + ((wb << 1) & ~3u);
                        const uint32_t va = shared_load(qa), vb = shared_load(qb);
                        pa = va & 0x8000u;
                        pb = vb & 0x8000u;
                        shared_store16_if(pa == 0, qa, mark | (wa & 1u));
                        shared_store16_if(pb == 0, qb, mark | (~wb & 1u));
                        ma = pa == 0 ? min(ma, (wa + bias) & 0xffffu) : ma;
                        mb = pb == 0 ? min(mb, (wb + bias) & 0xffffu) : mb;
                        wa = pa == 0 ? (va >> ((~wa & 1u) << 4)) & 0xffffu : wa;
                        wb = pb == 0 ? (vb >> ((~wb & 1u) << 4)) & 0xffffu : wb;
                    } while ((pa & pb) == 0);
                    // the stamps the walks ended at are still there: stamps
                    // are only ever replaced by ones that say the same
                    const uint32_t na = (shared_load(qa) & 0x7fffu) ^ (wa & 1u);
                    const uint32_t nb = (shared_load(qb) & 0x7fffu) ^ (wb & 1u);
                    const uint32_t m = min(ma, mb ^ 1u);
                    state[2 * r] = (m << 16) | na;
                    state[2 * r + 1] = ((m ^ 1u) << 16) | nb;
                }
                __syncthreads();
                // Each directed ruler state holds the smallest key of the
                // stretch up to `next` (both half-walks of every ruler in
                // it): three hops a round at least quadruple the stretch.
                // States change in place: a state read early or late is a
                // shorter or a longer stretch, both true.
                for (uint32_t reach = 1; reach < (ps >> ruler_log2) + 2; reach *= 4) {
                    for (uint32_t i = tid; i < 2 * rulers; i += blockDim.x) {
                        uint32_t me = vstate[i];
#pragma unroll
                        for (uint32_t hop = 0; hop < 3; ++hop) {
                            const uint32_t far = vstate[me & 0xffffu];
                            me = (min(me, far) & 0xffff0000u) | (far & 0xffffu);
                        }
                        vstate[i] = me;
                    }
                    __syncthreads();
                }
                const uint32_t total = nodes * ps;
                for (uint32_t base = warp * 32; base < total; base += nwarps * 32) {
                    const uint32_t q = base + lane;
                    const uint32_t v = q < total ? edge[q] : 0x8000u;
                    // padding pair-nodes hold anything: their bits are
                    // never used, but the ruler must stay in range
                    uint32_t x = (state[min(v & 0x7ffeu, 2 * rulers - 2)] >> 16) ^ v;
                    if ((v & 0x8000u) == 0) { // a cycle without rulers, or padding
                        const uint32_t path = by_ps(q);
                        const uint32_t k = q - path * ps;
                        const uint32_t s = node_size(path);
                        if (k < s - s / 2 && internal_node(path, s)) {
                            const uint32_t bias = key_bias(s);
                            uint32_t w = 2 * k, word = v;
                            x = ~0u; // the smallest key: walk the cycle whole
                            for (uint32_t step = 0; step < ps; ++step) {
                                x = min(x, (w + bias) & 0xffffu);
                                w = (w & 1u) != 0 ? word & 0xffffu : word >> 16;
                                if (w == 2 * k) break;
                                word = edge[path * ps + (w >> 1)];
                            }
                        }
                    }
                    const unsigned word = __ballot_sync(0xffffffffu, (x & 1u) != 0);
                    if (lane == 0) {
                        xbits[base >> 5] = word;
                    }
                }
            }
            __syncthreads();
            // ---- output switch bits, and the children: output pair k's
            // colour-0 input inv[2k + y] goes left with value k, the other
            // right (as level_outputs does for the global levels).  A thread
            // takes two output pairs, which make one output pair of each
            // child: it writes that pair of the children's inverses and both
            // of its edges, or a leaf child's values.
            {
                const LevelInfo& cl = plan.levels[level + 1];
                const uint32_t cstride = tile_node_slots(cl.pcap, level + 1 == D, leaf);
                const bool hand_over = level + 1 == stop && stop < D;
                const uint32_t hs = ps / 2;
                const FastDiv by_hs(hs);
                const uint32_t total = nodes * hs;
                for (uint32_t base = warp * 32; base < total; base += nwarps * 32) {
                    const uint32_t idx = base + lane;
                    bool y[2] = {false, false};
                    if (idx < total) {
                        const uint32_t path = by_hs(idx);
                        const uint32_t k0 = 2 * (idx - path * hs);
                        const uint32_t s = node_size(path);
                        const uint32_t half = s / 2;
                        const uint32_t sl = s - half;
                        if (k0 < sl && internal_node(path, s)) {
                            const uint2 four = *reinterpret_cast<const uint2*>(cur + path * stride + 2 * k0);
                            uint32_t left[2], right[2];
#pragma unroll
                            for (uint32_t i = 0; i < 2; ++i) {
                                const uint32_t both = i == 0 ? four.x : four.y;
                                const uint32_t u = both & 0xffffu;
                                if (k0 + i < half) {
                                    const uint32_t q = path * ps + (u >> 1);
                                    y[i] = (((xbits[q >> 5] >> (q & 31)) ^ u) & 1u) != 0;
                                }
                                // the odd tail output (k = half) goes left: y stays 0
                                left[i] = (y[i] ? both >> 16 : u) >> 1;
                                right[i] = (y[i] ? u : both >> 16) >> 1;
                            }
                            auto child = [&](uint32_t cpath, uint32_t cs, const uint32_t (&v)[2]) {
                                if (k0 >= cs) return;
                                uint16_t* to = nxt + cpath * cstride;
                                const bool two = k0 + 1 < cs;
                                const uint32_t w = two ? v[1] : cs; // virtual partner
                                if (hand_over) {
                                    reinterpret_cast<uint2*>(next_inv)[
                                        (uint64_t)(2 * first + cpath) * cl.pcap + (k0 >> 1)] =
                                        make_uint2(v[0], w);
                                } else if (cs > leaf) {
                                    *reinterpret_cast<uint32_t*>(to + k0) = v[0] | (w << 16);
                                    edge16[cpath * cstride + v[0]] = (uint16_t)w;
                                    edge16[cpath * cstride + w] = (uint16_t)v[0];
                                } else {
                                    to[v[0]] = (uint16_t)k0;
                                    if (two) to[v[1]] = (uint16_t)(k0 + 1);
                                }
                            };
                            child(2 * path, sl, left);
                            child(2 * path + 1, half, right);
                        }
                    }
                    // lane i holds bits 2i and 2i + 1 of the 64 from 2 * base
                    const uint32_t two = ((y[0] ? 1u : 0u) | (y[1] ? 2u : 0u)) << (2 * (lane & 15));
                    const uint32_t low = __reduce_or_sync(0xffffffffu, lane < 16 ? two : 0u);
                    const uint32_t high = __reduce_or_sync(0xffffffffu, lane < 16 ? 0u : two);
                    if (lane < 2) {
                        ybits[(base >> 4) + lane] = lane == 0 ? low : high;
                    }
                }
            }
        }
        __syncthreads();
    }

    // ---- switch bits and middle-group ranks out, all levels at once: a warp
    // task is one section of up to 32 nodes of a level (in large tiles one of
    // several parts of that), or the ranks of up to 32 leaves.  Keeping every level's bits until here costs 1/32 of the
    // tile's memory per level; going out level by level, with two barriers
    // and a wave of node addresses each time, took a third of a small tile's
    // time.
    const uint32_t levels = stop - T0;
    const bool leaves = stop == D;
    uint32_t tasks = 0;
    auto parts_of = [&](uint32_t t) { // 128 words of bits a part
        const uint32_t parts = (slots >> 13) >> (t < 5 ? 0 : t - 5);
        return parts > 1 ? parts : 1u;
    };
    auto tasks_of = [&](uint32_t t) { return (t < 5 ? 2u : 2u << (t - 5)) * parts_of(t); };
    for (uint32_t t = 0; t < levels; ++t) tasks += tasks_of(t);
    const uint32_t leaf_tasks = levels < 5 ? 1u : 1u << (levels - 5);
    const bool mixed = levels > 0 && plan.levels[D - 1].q <= leaf; // leaves at level D - 1 too
    if (leaves) {
        tasks += leaf_tasks + (mixed ? (levels < 6 ? 1u : 1u << (levels - 6)) : 0u);
    }
    for (uint32_t task = warp; task < tasks; task += nwarps) {
        uint32_t t = 0, at = task;
        for (; t < levels; ++t) {
            const uint32_t here = tasks_of(t);
            if (at < here) break;
            at -= here;
        }
        const bool is_leaf = t == levels;
        if (is_leaf && at >= leaf_tasks) { // level D - 1's leaves
            at -= leaf_tasks;
            --t;
        }
        const uint32_t level = T0 + t;
        const LevelInfo& lv = plan.levels[level];
        const uint32_t first = J << t;
        const uint32_t q32 = (uint32_t)lv.q;
        const uint32_t r32 = (uint32_t)lv.r;
        const bool all_exist = level == 0 || plan.levels[level - 1].q > leaf;
        auto node_size = [&](uint32_t path) {
            if (r32 == 0) return q32;
            return q32 + ((__brev(first + path) >> (32 - level)) < r32 ? 1u : 0u);
        };
        auto exists = [&](uint32_t path) {
            return all_exist ||
                size_at(plan.levels[level - 1], level - 1, (first + path) >> 1) > leaf;
        };
        const uint32_t wave_log2 = t < 5 ? t : 5; // log2 of the task's nodes
        const uint32_t slot_mask = (1u << wave_log2) - 1;
        if (is_leaf) {
            const uint32_t path = (at << 5) + lane;
            const uint32_t s = lane <= slot_mask ? node_size(path) : leaf + 1;
            if (s <= leaf && exists(path)) {
                int section = 0;
                const uint64_t bit = leaf_rank_bit(plan, level, first + path, &section);
                bool valid = true;
                const U128 rank = thread_factoradic_rank(
                    invs[t & 1] + path * tile_node_slots(lv.pcap, level == D, leaf), s, &valid);
                if (valid) {
                    thread_emit_rank(blob, plan.section_offset[section] * 8 + bit,
                        plan.fact_bits[s], rank);
                } else {
                    atomicOr(status, not_permutation(T0));
                }
            }
            continue;
        }
        const uint32_t parts = parts_of(t);
        const uint32_t part = at % parts;
        at /= parts;
        const int side = (int)(at & 1);
        const uint32_t w0 = (at >> 1) << 5;
        const uint32_t ps = tile_pair_stride(lv.pcap);
        const uint32_t* bits = level_bits + (2 * t + side) * bit_words;
        const LevelSide& ls = lv.side[side];
        const GroupInfo& gi = plan.groups[side][ls.group];
        const uint32_t span_log2 = gi.depth - ls.rel - 1;
        const uint64_t packet_bits[2] = {gi.packet_bits[0], gi.packet_bits[1]};
        // this lane's node: its switches (0: not an internal node) and the
        // blob bits of its run in packet 0 and in its tail packet
        uint32_t my_half = 0, my_large = 0;
        uint64_t my_full = 0, my_tail = 0;
        {
            const uint32_t path = w0 + (lane & slot_mask);
            const uint32_t s = node_size(path);
            if (s > leaf && exists(path)) {
                const NodeAddress a = node_address(plan, side, level, first + path);
                const uint64_t start = plan.section_offset[side] * 8 + a.base;
                my_half = s / 2;
                my_large = a.packet_bits != packet_bits[0] ? 1u : 0u;
                my_full = start + a.full_prefix;
                my_tail = start + a.tail_prefix;
            }
        }
        // blob bit of switch `pair` of node `slot`; all lanes call
        auto bit_of = [&](uint32_t slot, uint32_t pair, uint32_t half) {
            const uint32_t packet = pair >> span_log2;
            const uint64_t full = __shfl_sync(0xffffffffu, my_full, slot);
            const uint64_t tail = __shfl_sync(0xffffffffu, my_tail, slot);
            const uint32_t large = __shfl_sync(0xffffffffu, my_large, slot);
            return (packet == (half - 1) >> span_log2 ? tail : full) +
                packet * (large != 0 ? packet_bits[1] : packet_bits[0]) +
                (pair & ((1u << span_log2) - 1));
        };
        auto put = [&](uint64_t dest, uint32_t v) {
            if (v == 0) return;
            const uint32_t sh = (uint32_t)(dest & 31);
            atomicOr(blob + (dest >> 5), v << sh);
            if (sh != 0 && (v >> (32 - sh)) != 0) {
                atomicOr(blob + (dest >> 5) + 1, v >> (32 - sh));
            }
        };
        const uint32_t packets = ((uint32_t)lv.cap / 2 + (1u << span_log2) - 1) >> span_log2;
        if (span_log2 >= 5) {
            // runs of at least 32 switches: word-wise copies as in
            // level_emit_words
            const uint32_t cshift = span_log2 - 5;
            const uint32_t cs = wave_log2 + cshift;
            const uint32_t chunks = packets << cs;
            for (uint32_t base = part * 32; base < chunks; base += parts * 32) {
                const uint32_t c = base + lane;
                const uint32_t packet = c >> cs;
                const uint32_t rem = c & ((1u << cs) - 1);
                const uint32_t slot = rem >> cshift;
                const uint32_t pair0 =
                    (packet << span_log2) + ((rem & ((1u << cshift) - 1)) << 5);
                const uint32_t half = __shfl_sync(0xffffffffu, my_half, slot);
                const uint64_t dest = bit_of(slot, pair0, half);
                if (c < chunks && pair0 < half) {
                    const uint32_t q = (w0 + slot) * ps + pair0;
                    uint32_t v = __funnelshift_r(bits[q >> 5], bits[(q >> 5) + 1], q & 31);
                    if (half - pair0 < 32) {
                        v &= (1u << (half - pair0)) - 1u;
                    }
                    put(dest, v);
                }
            }
            continue;
        }
        // short runs: the packets every node fills go out as word blocks
        // (see level_emit_blocks_run), the rest bit by bit
        uint32_t full = 0;
        if (q32 > leaf && all_exist && q32 / 2 >= 1) {
            full = ((q32 / 2) - 1) >> span_log2;
        }
        if (full > packets) {
            full = packets;
        }
        if (full > 0) {
            // nodes per word: within a word, a cluster root and the task
            uint32_t g_log2 = 5 - span_log2;
            g_log2 = g_log2 < ls.rel ? g_log2 : ls.rel;
            g_log2 = g_log2 < wave_log2 ? g_log2 : wave_log2;
            const uint32_t span_mask = (1u << (1u << span_log2)) - 1u;
            const uint32_t groups_log2 = wave_log2 - g_log2;
            const uint32_t work = full << groups_log2;
            for (uint32_t base = part * 32; base < work; base += parts * 32) {
                const uint32_t c = base + lane;
                const uint32_t packet = c >> groups_log2;
                const uint32_t slot0 = (c & ((1u << groups_log2) - 1)) << g_log2;
                // below every node's tail packet: any half past it will do
                const uint64_t dest = bit_of(slot0, packet << span_log2, 0u);
                if (c < work) {
                    uint32_t v = 0;
                    for (uint32_t i = 0; i < (1u << g_log2); ++i) {
                        const uint32_t q = (w0 + slot0 + i) * ps + (packet << span_log2);
                        const uint32_t field =
                            __funnelshift_r(bits[q >> 5], bits[(q >> 5) + 1], q & 31) & span_mask;
                        v |= field << (i << span_log2);
                    }
                    put(dest, v);
                }
            }
        }
        const uint32_t shift = wave_log2 + span_log2;
        const uint32_t rest = (packets - full) << shift;
        for (uint32_t base = part * 32; base < rest; base += parts * 32) {
            const uint32_t c = base + lane;
            const uint32_t packet = full + (c >> shift);
            const uint32_t rem = c & ((1u << shift) - 1);
            const uint32_t slot = rem >> span_log2;
            const uint32_t pair = (packet << span_log2) + (rem & ((1u << span_log2) - 1));
            const uint32_t half = __shfl_sync(0xffffffffu, my_half, slot);
            const uint64_t dest = bit_of(slot, pair, half);
            bool set = false;
            if (c < rest && pair < half) {
                const uint32_t q = (w0 + slot) * ps + pair;
                set = ((bits[q >> 5] >> (q & 31)) & 1u) != 0;
            }
            emit_bit(blob, dest, set, 0xffffffffu);
        }
    }
}

// One permutation: one CTA per node of the tile level.
template <typename T>
__global__ void __launch_bounds__(kTileThreads, 2) tile_encode(const Plan* __restrict__ plan,
    const T* __restrict__ src, uint32_t* __restrict__ blob, uint32_t* status, uint32_t slots,
    uint32_t part_first, uint32_t level, uint32_t stop, uint32_t* __restrict__ next_inv) {
    extern __shared__ __align__(16) unsigned char smem[];
    wait_for_previous();
    // a sharded call encodes only its own nodes (level_nodes); a launch may
    // cover a part of them, from part_first on
    const uint32_t first = (uint32_t)level_nodes(*plan, level).lo + part_first;
    tile_body<T>(plan, src, blob, status, slots, first + blockIdx.x, smem, level, stop, next_inv);
}

// Tiles too large for two CTAs per SM (nodes of 16384 entries, up to about
// 200 KB of shared memory): one CTA of twice the threads per SM keeps the
// same number of resident warps.
template <typename T>
__global__ void __launch_bounds__(2 * kTileThreads, 1) tile_encode_wide(
    const Plan* __restrict__ plan, const T* __restrict__ src, uint32_t* __restrict__ blob,
    uint32_t* status, uint32_t slots, uint32_t part_first, uint32_t level, uint32_t stop,
    uint32_t* __restrict__ next_inv) {
    extern __shared__ __align__(16) unsigned char smem[];
    wait_for_previous();
    const uint32_t first = (uint32_t)level_nodes(*plan, level).lo + part_first;
    tile_body<T>(plan, src, blob, status, slots, first + blockIdx.x, smem, level, stop, next_inv);
}

struct Header {
    uint32_t bytes;
    uint8_t data[84];
};

// Word i of a blob that holds its header and nothing else.  The header ends
// before the first section bit.
__device__ __forceinline__ uint32_t header_word(const Header& h, uint64_t i) {
    uint32_t v = 0;
    for (uint32_t k = 0; k < 4; ++k) {
        if (4 * i + k < h.bytes) v |= (uint32_t)h.data[4 * i + k] << (8 * k);
    }
    return v;
}

// A permutation that is one tile, as a single launch: the plan and the
// header come as kernel parameters, the block keeps the plan in shared
// memory at byte `plan_at` (0: no room, it stays a parameter), clears the blob and leaves the status word at `status_out`
// (device or pinned host memory).  A plan upload, a memset, a header kernel
// and a status download around the tile took 40 of the 90 us of a 1000-entry
// call.
struct TileSingle {
    Plan plan;
    Header header;
};

template <typename T>
__global__ void __launch_bounds__(2 * kTileThreads, 1) tile_encode_single(
    const __grid_constant__ TileSingle one, const T* __restrict__ src,
    uint32_t* __restrict__ blob, uint32_t blob_words, uint32_t* status_out, uint32_t slots,
    uint32_t plan_at) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t status;
    const Plan* plan = &one.plan;
    if (plan_at != 0) {
        uint32_t* near = reinterpret_cast<uint32_t*>(smem + plan_at);
        const uint32_t* from = reinterpret_cast<const uint32_t*>(&one.plan);
        for (uint32_t i = threadIdx.x; i < sizeof(Plan) / 4; i += blockDim.x) near[i] = from[i];
        plan = reinterpret_cast<const Plan*>(near);
    }
    for (uint32_t i = threadIdx.x; i < blob_words; i += blockDim.x) {
        blob[i] = header_word(one.header, i);
    }
    if (threadIdx.x == 0) status = 0;
    __syncthreads();
    tile_body<T, true>(plan, src, blob, &status, slots, 0, smem, 0, plan->depth, nullptr);
    __syncthreads();
    if (threadIdx.x == 0) *(volatile uint32_t*)status_out = status;
}

// Tiles of many permutations in one launch (the batched and serving forms):
// job k owns blocks [first_block, first_block + tiles); the launch's dynamic
// shared memory covers the largest job.
// A job whose permutation is a single tile (tile level 0) also clears its
// blob, writes the header and resets its status word first: its CTA is the
// only writer of that blob.
struct TileJob {
    const Plan* plan;
    const void* src;
    uint32_t* blob;
    uint32_t* status;
    uint32_t* next_inv;    // a stage's output (tile_body), null for whole subtrees
    uint32_t slots;
    uint32_t level;
    uint32_t stop;
    uint32_t first_block;
    uint32_t tiles;
    uint32_t blob_words;   // words to clear (single-tile jobs)
    uint32_t header_bytes;
    uint8_t header[84];
};

template <typename T>
__device__ __forceinline__ void tile_batch_body(const TileJob* __restrict__ jobs, uint32_t njobs,
    unsigned char* smem) {
    uint32_t lo = 0, hi = njobs;
    while (hi - lo > 1) { // last job whose first block is <= blockIdx.x
        const uint32_t mid = (lo + hi) / 2;
        if (jobs[mid].first_block <= blockIdx.x) lo = mid; else hi = mid;
    }
    const TileJob& job = jobs[lo];
    if (job.tiles == 1 && job.blob_words != 0) {
        for (uint32_t i = threadIdx.x; i < job.blob_words; i += blockDim.x) job.blob[i] = 0;
        __syncthreads();
        uint8_t* b = reinterpret_cast<uint8_t*>(job.blob);
        for (uint32_t i = threadIdx.x; i < job.header_bytes; i += blockDim.x) b[i] = job.header[i];
        if (threadIdx.x == 0) *job.status = 0;
        __syncthreads();
    }
    tile_body<T>(job.plan, (const T*)job.src, job.blob, job.status, job.slots,
        blockIdx.x - job.first_block, smem, job.level, job.stop, job.next_inv);
}

template <typename T>
__global__ void __launch_bounds__(kTileThreads, 2) tile_encode_batch(
    const TileJob* __restrict__ jobs, uint32_t njobs) {
    extern __shared__ __align__(16) unsigned char smem[];
    wait_for_previous();
    tile_batch_body<T>(jobs, njobs, smem);
}

// Stages of many permutations: one large node per SM.
template <typename T>
__global__ void __launch_bounds__(2 * kTileThreads, 1) tile_encode_batch_wide(
    const TileJob* __restrict__ jobs, uint32_t njobs) {
    extern __shared__ __align__(16) unsigned char smem[];
    wait_for_previous();
    tile_batch_body<T>(jobs, njobs, smem);
}

} // namespace bpb200
