// SPDX-License-Identifier: Apache-2.0
//
// Forward and inverse lookup of one index in a compact blob, shared by the
// device verifier kernel (lookup.inc) and a host test probe.
//
// Restates the reference's read path, lookup() in src/internal.hpp:1035-1124:
// descend from the root reading one switch per level (input section for a
// forward lookup, output section for an inverse one), decode the leaf's
// factoradic rank, then climb back reading the switches of the other
// section.  On the closed-form plan the node reached at level l is the
// string of left/right turns taken so far (children of node j are 2j and
// 2j + 1), so the climb recomputes each ancestor and its turn from the leaf
// node's index instead of keeping the reference's frame stack.
#pragma once

#include "plan.hpp"

#include <cstdint>

namespace bpb200 {

// Status bits of one lookup (ORed over a batch).
enum LookupStatus : uint32_t {
    kLookupOk = 0,
    kLookupOutOfRange = 1u, // index >= size (std::out_of_range in the reference)
    kLookupTruncated = 2u,  // a bit address fell outside the blob
    kLookupBadPlan = 4u,    // descent ran past the routing depth
};

struct BlobBits {
    const uint8_t* data;
    uint64_t len; // bytes
};

// Bit `bit` (LSB-first) of the section starting at byte `offset`
// (read_bit, src/internal.hpp:1005-1013).
BP_HD uint32_t blob_bit(const BlobBits& b, uint64_t offset, uint64_t bit, uint32_t* status) {
    const uint64_t byte = offset + (bit >> 3);
    if (byte >= b.len) {
        *status |= kLookupTruncated;
        return 0;
    }
    return (uint32_t)(b.data[byte] >> (bit & 7)) & 1u;
}

// Bits [first, first + bits) (bits <= 128) of the section at byte `offset`,
// LSB-first (read_rank, src/internal.hpp:1015-1033): 32-bit words from the
// aligned word that holds the first bit; words that reach over either end of
// the blob are put together from its bytes.
BP_HD void blob_rank(const BlobBits& b, uint64_t offset, uint64_t first, uint32_t bits,
    uint32_t (&rank)[4], uint32_t* status) {
    rank[0] = rank[1] = rank[2] = rank[3] = 0;
    if (bits == 0) {
        return;
    }
    if (offset + ((first + bits - 1) >> 3) >= b.len) {
        *status |= kLookupTruncated;
        return;
    }
    const uintptr_t base = (uintptr_t)b.data;
    const uint64_t at = (uint64_t)(base & 3) * 8 + offset * 8 + first; // bit from the aligned base
    const uint32_t shift = (uint32_t)(at & 31);
    const uint64_t word0 = at >> 5;
    const uint32_t words = (shift + bits + 31) >> 5; // 1..5
    uint32_t below = 0;
    for (uint32_t i = 0; i < 5; ++i) {
        uint32_t w = 0;
        if (i < words) {
            // byte range of the word inside the blob
            const int64_t lo = (int64_t)((word0 + i) * 4) - (int64_t)(base & 3);
            if (lo >= 0 && (uint64_t)lo + 4 <= b.len) {
                w = *reinterpret_cast<const uint32_t*>(b.data + lo);
            } else {
                for (int k = 0; k < 4; ++k) {
                    if (lo + k >= 0 && (uint64_t)(lo + k) < b.len) {
                        w |= (uint32_t)b.data[lo + k] << (8 * k);
                    }
                }
            }
        }
        if (i > 0) {
            rank[i - 1] = shift == 0 ? below : (below >> shift) | (w << (32 - shift));
        }
        below = w;
    }
    for (uint32_t i = 0; i < 4; ++i) { // drop the bits of the next rank
        const uint32_t keep = bits > 32 * i ? bits - 32 * i : 0;
        if (keep < 32) rank[i] &= (1u << keep) - 1u;
    }
}

BP_HD uint32_t mul_high(uint32_t a, uint32_t b) {
    return (uint32_t)(((uint64_t)a * b) >> 32);
}
BP_HD uint64_t mul_high(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// Leaf step of the lookup: the local permutation of `size` (<= 32) entries
// encoded by the factoradic rank, applied forward to `index` (p[index]) or
// inverted (the i with p[i] == index).
//
// The rank is the mixed-radix number with digits d[i] = #{k < i : p[k] <
// p[i]}, radix i + 1 (encode_factoradic, src/internal.hpp:148-167), so the
// lowest digit is d[size-1].  Digits come off from the top entry down: one
// long division of the rank by the product of the next radices (below 2^27)
// leaves a remainder whose digits are 32-bit divisions by a reciprocal,
// floor(n / r) = mul_high(n, ceil(2^32 / r)), exact while n * r < 2^32.  The
// long division's limbs are divided by a 64-bit reciprocal rounded down,
// whose quotient is at most one too small.
// Inverse: entry k has the d[k]-th smallest value of the entries up to k, so
// the wanted value's rank t among them either is d[k], or loses one when
// d[k] < t.  Forward: the same steps backwards, from entry `index` up:
// p[index] starts as d[index] and gains one for every later entry whose
// digit is not above it.
BP_HD uint32_t leaf_apply(const Plan& p, uint32_t (&rank)[4], uint32_t size,
    uint32_t index, bool inverse) {
    uint8_t digits[32];
    uint32_t t = index;
    uint32_t i = size;
    while (i > 0) {
        const DigitGroup group = p.digit_groups[i];
        uint64_t rem = 0;
        for (int k = 3; k >= 0; --k) {
            if (rem == 0 && rank[k] == 0) {
                continue; // leading zero limbs
            }
            const uint64_t cur = (rem << 32) | rank[k];
            uint64_t quot = mul_high(cur, group.reciprocal);
            rem = cur - quot * group.product;
            if (rem >= group.product) {
                rem -= group.product;
                ++quot;
            }
            rank[k] = (uint32_t)quot;
        }
        uint32_t rest = (uint32_t)rem;
        for (uint32_t g = 0; g < group.digits; ++g) {
            const uint32_t radix = i--; // entry i's digit, after the decrement
            uint32_t digit = 0;
            if (radix > 1) {
                const uint32_t q = mul_high(rest, p.digit_reciprocal[radix]);
                digit = rest - q * radix;
                rest = q;
            }
            if (inverse) {
                if (digit == t) {
                    return i;
                }
                t -= digit < t ? 1u : 0u;
            } else if (i == index) {
                uint32_t value = digit;
                for (uint32_t k = index + 1; k < size; ++k) {
                    value += digits[k] <= value ? 1u : 0u;
                }
                return value;
            } else {
                digits[i] = (uint8_t)digit;
            }
        }
    }
    return 0; // unreachable for index < size
}

// What a path needs of one level and section, gathered from the plan: the
// device kernel keeps the table of its call in shared memory.
struct PathLevel {
    uint64_t prefix0[2];        // by cluster root size
    uint64_t prefix_tail[2][2]; // by root and node size
    uint64_t packet_bits[2];
    uint32_t q, r;              // node sizes of the level (low words; see path_node_size)
    uint32_t group;
    uint32_t start;             // first level of the group
    uint32_t rel;
    uint32_t span_log2;
};

BP_HD PathLevel path_level(const Plan& p, int side, uint32_t level) {
    const LevelInfo& lv = p.levels[level];
    const LevelSide& ls = lv.side[side];
    const GroupInfo& gi = p.groups[side][ls.group];
    PathLevel t;
    for (int rs = 0; rs < 2; ++rs) {
        t.prefix0[rs] = ls.prefix0[rs];
        t.prefix_tail[rs][0] = ls.prefix_tail[rs][0];
        t.prefix_tail[rs][1] = ls.prefix_tail[rs][1];
        t.packet_bits[rs] = gi.packet_bits[rs];
    }
    t.q = (uint32_t)lv.q;
    t.r = (uint32_t)lv.r;
    t.group = ls.group;
    t.start = gi.start;
    t.rel = ls.rel;
    t.span_log2 = gi.depth - ls.rel - 1; // unused past the last routing level
    return t;
}

// The plan itself as the source of path levels (host probe).
struct PlanLevels {
    const Plan* plan;
    BP_HD PathLevel at(int side, uint32_t level) const { return path_level(*plan, side, level); }
};

// Switch addresses along one query's path through one section.  All nodes of
// the path inside one cluster group share the cluster root, so its base is
// worked out once per group; below it only the packet that holds the wanted
// pair is looked at (node_address works out both kinds).
struct PathAddress {
    uint64_t base = 0;  // blob bit of the cluster's packets
    uint64_t root_count = 0;
    uint32_t group = ~0u;
    uint32_t rs = 0;    // 1: the cluster root is a large node

    template <typename Int>
    BP_HD uint64_t bit(const Plan& p, const PathLevel& t, int side, uint32_t level, Int node,
        Int size, Int pair) {
        if (t.group != group) {
            group = t.group;
            base = p.section_offset[side] * 8 + cluster_base(p, side, group, level, node);
            rs = node_is_large(p.levels[t.start], t.start, node >> t.rel) ? 1u : 0u;
            root_count = p.levels[t.start].q + rs;
        }
        const Int path = node & (((Int)1 << t.rel) - 1);
        const Int span = (Int)1 << t.span_log2;
        const Int packet = pair >> t.span_log2;
        const uint64_t at = base + (uint64_t)packet * t.packet_bits[rs] + (pair & (span - 1));
        const bool tail = packet == (size / 2 - 1) >> t.span_log2;
        // packet_path_bits in Int arithmetic: switches of the nodes left of
        // this one in the packet, by the two node sizes of the level
        const Int small = (Int)(root_count >> t.rel);
        const Int large = (Int)root_count & (((Int)1 << t.rel) - 1);
        const Int first = tail ? packet << t.span_log2 : 0;
        auto share = [&](Int count) -> Int {
            const Int half = count / 2;
            return count <= p.leaf || first >= half ? 0 : (half - first < span ? half - first : span);
        };
        const Int each = share(small);
        uint64_t before = (uint64_t)path * each;
        if (large != 0 && path != 0) {
            const Int more = share(small + 1) - each;
            if (more != 0) before += count_large(path, t.rel, large) * more;
        }
        return at + before +
            (tail ? t.prefix_tail[rs][size != (Int)p.levels[level].q ? 1 : 0] : t.prefix0[rs]);
    }
};

// node_size, in 32 bits where those hold every index.
BP_HD uint64_t path_node_size(const Plan& p, const PathLevel&, uint32_t level, uint64_t node) {
    return node_size(p.levels[level], level, node);
}
BP_HD uint32_t path_node_size(const Plan&, const PathLevel& t, uint32_t level, uint32_t node) {
#if defined(__CUDA_ARCH__)
    const uint32_t reversed = level == 0 ? 0u : __brev(node) >> (32 - level);
#else
    const uint32_t reversed = (uint32_t)reverse_bits(node, level);
#endif
    return t.q + (reversed < t.r ? 1u : 0u);
}

// Forward (p[value]) or inverse (p^-1[value]) lookup.  Returns a
// LookupStatus; *out is valid when it is kLookupOk.  Int holds every index
// and node of the permutation: 32 bits up to 2^31 entries, else 64.
// `levels` gives the path levels of a section (PlanLevels, or a table).
template <typename Int, typename Levels>
BP_HD uint32_t lookup_path(const Plan& p, const Levels& levels, const BlobBits& blob,
    uint64_t value, bool inverse, uint64_t* out) {
    if (value >= p.n) {
        return kLookupOutOfRange;
    }
    uint32_t status = 0;
    const int down = inverse ? 1 : 0; // section read on the way down
    const int up = 1 - down;
    Int index = (Int)value;
    Int node = 0;
    Int size = (Int)p.n;
    uint32_t level = 0;
    PathAddress way_down;
    while (size > p.leaf) {
        if (level >= p.depth) {
            return kLookupBadPlan;
        }
        bool right = false;
        if ((size & 1) == 0 || index != size - 1) { // the odd tail passes straight left
            const uint64_t bit =
                way_down.bit(p, levels.at(down, level), down, level, node, size, (Int)(index >> 1));
            right = blob_bit(blob, 0, bit, &status) != (uint32_t)(index & 1);
        }
        index >>= 1;
        node = 2 * node + (right ? 1 : 0);
        ++level;
        size = path_node_size(p, levels.at(down, level), level, node);
    }
    int section = 0;
    const uint64_t rank_bit = leaf_rank_bit(p, level, node, &section);
    uint32_t rank[4];
    blob_rank(blob, p.section_offset[section], rank_bit, p.fact_bits[size], rank, &status);
    index = leaf_apply(p, rank, (uint32_t)size, (uint32_t)index, inverse);
    PathAddress way_up;
    for (uint32_t l = level; l-- > 0;) {
        const Int at = node >> (level - l);
        const uint32_t right = (uint32_t)(node >> (level - 1 - l)) & 1u;
        const auto& here = levels.at(up, l);
        const Int count = path_node_size(p, here, l, at);
        if (right == 0 && (count & 1) != 0 && index == count / 2) {
            index = count - 1; // back out through the odd tail
            continue;
        }
        const uint64_t bit = way_up.bit(p, here, up, l, at, count, index);
        index = 2 * index + (right ^ blob_bit(blob, 0, bit, &status));
    }
    *out = index;
    return status;
}

BP_HD uint32_t lookup_one(const Plan& p, const BlobBits& blob, uint64_t value, bool inverse,
    uint64_t* out) {
    const PlanLevels levels{&p};
    return p.n <= (1ull << 31) ? lookup_path<uint32_t>(p, levels, blob, value, inverse, out)
                               : lookup_path<uint64_t>(p, levels, blob, value, inverse, out);
}

} // namespace bpb200
