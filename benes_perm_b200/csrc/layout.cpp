// SPDX-License-Identifier: Apache-2.0
#include "layout.hpp"

#include <algorithm>
#include <cstring>

namespace bpb200 {
namespace {

struct Fail {
    int code;
    const char* message;
};

uint64_t add(uint64_t a, uint64_t b) {
    if (b > UINT64_MAX - a) {
        throw Fail{kOverflow, "compressed permutation is too large"};
    }
    return a + b;
}

// ceil(log2(c!)) exactly: bit width of c! - 1 (src/internal.hpp:173-183).
uint32_t factoradic_bits(uint32_t c) {
    unsigned __int128 f = 1;
    for (uint32_t i = 2; i <= c; ++i) {
        f *= i;
    }
    f -= 1;
    uint32_t bits = 0;
    while (f != 0) {
        ++bits;
        f >>= 1;
    }
    return bits;
}

const uint32_t* factoradic_table() {
    static const struct Table {
        uint32_t bits[33];
        Table() {
            for (uint32_t c = 0; c <= 32; ++c) bits[c] = factoradic_bits(c);
        }
    } table;
    return table.bits;
}

struct DigitTables {
    uint32_t reciprocal[33] = {};
    DigitGroup groups[33] = {};
};

const DigitTables& digit_tables() {
    static const DigitTables tables = [] {
        DigitTables t;
        for (uint32_t i = 1; i <= 32; ++i) {
            t.reciprocal[i] = i > 1 ? 0xffffffffu / i + 1u : 0u;
            uint32_t product = i, digits = 1;
            while (digits < i && (uint64_t)product * (i - digits) < (1u << 27)) {
                product *= i - digits;
                ++digits;
            }
            t.groups[i] = {~0ull / product, product, digits};
        }
        return t;
    }();
    return tables;
}

// Switches and middle bits of the subtrees of every level's two node sizes,
// q_l = floor(n / 2^l) and q_l + 1 (FormatSizeCache, src/internal.hpp:225-313,
// memoises the same recursion).  Both halves of either size are one of the
// next level's two, so the tables fill from the leaves up in a few steps per
// level.  Level 0's second size belongs to no node and may wrap around.
class Sizes {
public:
    Sizes(uint64_t n, uint32_t leaf, uint32_t depth) : n_(n), leaf_(leaf) {
        for (uint32_t l = depth + 2; l-- > 0;) {
            for (uint32_t big = 0; big < 2; ++big) {
                const uint64_t c = small(l) + big;
                if (c <= leaf_) {
                    switches_[l][big] = 0;
                    middle_[l][big] = factoradic_table()[c];
                    continue;
                }
                const uint32_t lo = (uint32_t)(c / 2 - small(l + 1));
                const uint32_t hi = (uint32_t)(c - c / 2 - small(l + 1));
                if (l == 0 && big == 1) {
                    switches_[l][big] = c / 2 + switches_[l + 1][hi] + switches_[l + 1][lo];
                    middle_[l][big] = middle_[l + 1][hi] + middle_[l + 1][lo];
                } else {
                    switches_[l][big] = add(c / 2, add(switches_[l + 1][hi], switches_[l + 1][lo]));
                    middle_[l][big] = add(middle_[l + 1][hi], middle_[l + 1][lo]);
                }
            }
        }
    }

    uint64_t switches(uint32_t level, uint32_t big) const { return switches_[level][big]; }
    uint64_t middle(uint32_t level, uint32_t big) const { return middle_[level][big]; }

    // Switches of the first `depth` levels of the subtrees of the two sizes
    // of level `start`.
    void top_switches(uint32_t start, uint32_t depth, uint64_t (&out)[2]) const {
        uint64_t below[2] = {0, 0};
        for (uint32_t l = start + depth; l-- > start;) {
            uint64_t here[2];
            for (uint32_t big = 0; big < 2; ++big) {
                const uint64_t c = small(l) + big;
                here[big] = c <= leaf_ ? 0
                    : c / 2 + below[c - c / 2 - small(l + 1)] + below[c / 2 - small(l + 1)];
            }
            below[0] = here[0];
            below[1] = here[1];
        }
        out[0] = below[0];
        out[1] = below[1];
    }

private:
    uint64_t small(uint32_t l) const { return l < 64 ? n_ >> l : 0; }

    uint64_t n_;
    uint32_t leaf_;
    uint64_t switches_[66][2];
    uint64_t middle_[66][2];
};

// packet_path_bits over all 2^rel nodes of a level of a cluster: of those
// exactly root mod 2^rel are large.
uint64_t packet_level_bits(uint64_t root, uint32_t depth, uint32_t rel, uint64_t packet,
    uint32_t leaf) {
    const uint64_t small = root >> rel;
    const uint64_t nodes = 1ull << rel;
    const uint64_t large = root & (nodes - 1);
    const uint64_t span = 1ull << (depth - rel - 1);
    const uint64_t first = packet * span;
    auto share = [&](uint64_t count) {
        return count <= leaf || first >= count / 2 ? 0 : std::min(count / 2 - first, span);
    };
    return large * share(small + 1) + (nodes - large) * share(small);
}

uint32_t routing_depth(uint64_t count, uint32_t leaf) {
    uint32_t d = 0;
    while (count > leaf) {
        count = count - count / 2;
        ++d;
    }
    return d;
}

uint8_t balanced_clusters(uint32_t depth, uint8_t* out) {
    if (depth == 0) {
        return 0;
    }
    if (depth == 1) {
        out[0] = 1;
        return 1;
    }
    out[0] = (uint8_t)((depth + 1) / 2);
    out[1] = (uint8_t)(depth / 2);
    return 2;
}

void check_clusters(const uint8_t* c, uint32_t n, uint32_t depth) {
    uint32_t sum = 0;
    for (uint32_t i = 0; i < n; ++i) {
        if (c[i] == 0) {
            throw Fail{kInvalidArgument, "cluster depths must be positive"};
        }
        sum += c[i];
    }
    if (sum != depth) {
        throw Fail{kInvalidArgument, "cluster depths do not span every routing level"};
    }
}

uint64_t bytes_of(uint64_t bits) { return bits / 8 + (bits % 8 != 0 ? 1 : 0); }

void layout_or_throw(uint64_t count, const Format& in, Layout* out) {
    Format f = in;
    if (f.middle_group_log2 == 0 || f.middle_group_log2 > 5) {
        throw Fail{kInvalidArgument, "middle_group_log2 must be between 1 and 5"};
    }
    if (f.middle_placement > 2) {
        throw Fail{kInvalidArgument, "invalid middle placement"};
    }
    if (f.input_cluster_count > 64 || f.output_cluster_count > 64) {
        throw Fail{kInvalidArgument, "cluster depths do not span every routing level"};
    }
    const uint32_t leaf = 1u << f.middle_group_log2;
    const uint32_t depth = routing_depth(count, leaf);
    if (f.input_cluster_count == 0) {
        f.input_cluster_count = balanced_clusters(depth, f.input_clusters);
    }
    if (f.output_cluster_count == 0) {
        f.output_cluster_count = balanced_clusters(depth, f.output_clusters);
    }
    check_clusters(f.input_clusters, f.input_cluster_count, depth);
    check_clusters(f.output_clusters, f.output_cluster_count, depth);
    if (depth == 0) {
        f.middle_placement = 0;
    }
    const Sizes sizes(count, leaf, depth);
    Layout L;
    L.format = f;
    L.size = count;
    L.depth = depth;
    L.switch_bits = sizes.switches(0, 0);
    L.middle_bits = sizes.middle(0, 0);
    L.header_bytes = add(20, (uint64_t)f.input_cluster_count + f.output_cluster_count);
    const uint64_t in_bytes = add(bytes_of(L.switch_bits),
        f.middle_placement == 1 ? bytes_of(L.middle_bits) : 0);
    const uint64_t out_bytes = add(bytes_of(L.switch_bits),
        f.middle_placement == 2 ? bytes_of(L.middle_bits) : 0);
    const uint64_t mid_bytes = f.middle_placement == 0 ? bytes_of(L.middle_bits) : 0;
    if (count > (1ull << 63)) {
        throw Fail{kOverflow, "logical network size is too large"};
    }
    uint64_t width = leaf;
    while (width < count) {
        width <<= 1;
    }
    L.network_size = width;
    L.input_offset = L.header_bytes;
    L.output_offset = add(L.header_bytes, in_bytes);
    L.middle_offset = add(L.output_offset, out_bytes);
    L.end_offset = add(L.middle_offset, mid_bytes);
    *out = L;
}

} // namespace

Error make_layout(uint64_t count, const Format& format, Layout* out) {
    try {
        layout_or_throw(count, format, out);
        return {};
    } catch (const Fail& f) {
        return {f.code, f.message};
    }
}

void write_header(const Layout& L, uint8_t* out) {
    static const uint8_t magic[8] = {'B', 'E', 'N', 'E', 'S', '0', '1', 0};
    std::memcpy(out, magic, 8);
    for (int i = 0; i < 8; ++i) {
        out[8 + i] = (uint8_t)(L.size >> (8 * i));
    }
    out[16] = L.format.middle_placement;
    out[17] = L.format.middle_group_log2;
    out[18] = L.format.input_cluster_count;
    out[19] = L.format.output_cluster_count;
    std::memcpy(out + 20, L.format.input_clusters, L.format.input_cluster_count);
    std::memcpy(out + 20 + L.format.input_cluster_count, L.format.output_clusters,
        L.format.output_cluster_count);
}

Error make_plan(const Layout& L, uint64_t tile_max, Plan* out) {
    try {
        Plan& p = *out;
        std::memset(&p, 0, sizeof p);
        const uint64_t n = L.size;
        const uint32_t leaf = 1u << L.format.middle_group_log2;
        if (L.depth > kMaxLevels - 1) {
            throw Fail{kLength, "permutation is too large for the B200 backend"};
        }
        const Sizes sizes(n, leaf, L.depth);
        p.n = n;
        p.leaf = leaf;
        p.depth = L.depth;
        p.placement = L.format.middle_placement;
        p.section_offset[0] = L.input_offset;
        p.section_offset[1] = L.output_offset;
        p.section_offset[2] = L.middle_offset;
        p.end_offset = L.end_offset;
        p.switch_bits = L.switch_bits;
        p.middle_bits = L.middle_bits;

        for (uint32_t l = 0; l <= L.depth; ++l) {
            LevelInfo& lv = p.levels[l];
            lv.q = n >> l;
            lv.r = n & ((1ull << l) - 1);
            lv.cap = lv.q + (lv.r != 0 ? 1 : 0);
            lv.pcap = ((lv.cap + 1) / 2 + 1) & ~1ull;
            for (int big = 0; big < 2; ++big) {
                lv.middle[big] = sizes.middle(l, big);
                for (int side = 0; side < 2; ++side) {
                    const bool embeds = L.format.middle_placement == (uint8_t)(side + 1);
                    lv.section[side][big] =
                        sizes.switches(l, big) + (embeds ? lv.middle[big] : 0);
                }
            }
        }

        for (int side = 0; side < 2; ++side) {
            const uint8_t* cl = side == 0 ? L.format.input_clusters : L.format.output_clusters;
            const uint32_t gc = side == 0 ? L.format.input_cluster_count : L.format.output_cluster_count;
            p.group_count[side] = gc;
            uint32_t start = 0;
            for (uint32_t g = 0; g < gc; ++g) {
                GroupInfo& gi = p.groups[side][g];
                gi.start = start;
                gi.depth = cl[g];
                sizes.top_switches(start, gi.depth, gi.group_bits);
                for (int big = 0; big < 2; ++big) {
                    const uint64_t root = p.levels[start].q + (uint64_t)big;
                    uint64_t bits = 0;
                    for (uint32_t l = 0; l < gi.depth; ++l) {
                        bits += packet_level_bits(root, gi.depth, l, 0, leaf);
                    }
                    gi.packet_bits[big] = bits;
                }
                start += gi.depth;
            }
            for (uint32_t l = 0; l <= L.depth && gc > 0; ++l) {
                uint32_t g = 0;
                while (g + 1 < gc && p.groups[side][g + 1].start <= l) {
                    ++g;
                }
                const GroupInfo& gi = p.groups[side][g];
                LevelSide& ls = p.levels[l].side[side];
                ls.group = g;
                ls.rel = l - gi.start;
                if (ls.rel >= gi.depth) {
                    continue; // leaf level past the last group: no switches
                }
                for (int rb = 0; rb < 2; ++rb) {
                    const uint64_t root = p.levels[gi.start].q + (uint64_t)rb;
                    uint64_t f0 = 0;
                    for (uint32_t up = 0; up < ls.rel; ++up) {
                        f0 += packet_level_bits(root, gi.depth, up, 0, leaf);
                    }
                    ls.prefix0[rb] = f0;
                    for (int nb = 0; nb < 2; ++nb) {
                        const uint64_t pairs = (p.levels[l].q + (uint64_t)nb) / 2;
                        const uint64_t tail = pairs == 0 ? 0 : (pairs - 1) >> (gi.depth - ls.rel - 1);
                        uint64_t ft = 0;
                        for (uint32_t up = 0; up < ls.rel; ++up) {
                            ft += packet_level_bits(root, gi.depth, up, tail, leaf);
                        }
                        ls.prefix_tail[rb][nb] = ft;
                    }
                }
            }
        }

        uint32_t tile = 0;
        while (tile < L.depth && p.levels[tile].cap > tile_max) {
            ++tile;
        }
        p.tile_level = tile;
        uint64_t slots = 0, pairs = 0;
        for (uint32_t l = 0; l <= tile; ++l) {
            const uint64_t s = (1ull << l) * 2 * p.levels[l].pcap;
            const uint64_t q = (1ull << l) * p.levels[l].pcap;
            slots = s > slots ? s : slots;
            pairs = q > pairs ? q : pairs;
        }
        p.max_slots = slots;
        p.max_pairs = pairs;
        for (uint32_t c = 0; c <= 32; ++c) {
            p.fact_bits[c] = factoradic_table()[c];
        }
        std::memcpy(p.digit_reciprocal, digit_tables().reciprocal, sizeof p.digit_reciprocal);
        std::memcpy(p.digit_groups, digit_tables().groups, sizeof p.digit_groups);
        return {};
    } catch (const Fail& f) {
        return {f.code, f.message};
    }
}

} // namespace bpb200
