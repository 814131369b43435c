// SPDX-License-Identifier: Apache-2.0
//
// Device building blocks shared by the level kernels and the tile kernel:
// parity union-find, warp-aggregated bit emission and the factoradic rank of
// a middle group.
#pragma once

#include "plan.hpp"

#include <cstdint>

namespace bpb200 {

// The block's place in the grid it works in: the launch's own grid for a
// one-permutation launch, or this permutation's share of the blocks of a
// batched launch over many permutations (serve.inc).  Kernel bodies index
// their work by it instead of blockIdx / gridDim.
struct Grid {
    uint32_t bid;
    uint32_t nblk;
};

__device__ __forceinline__ Grid launch_grid() { return Grid{blockIdx.x, gridDim.x}; }

// Start of every kernel of an encode's launch sequence, which is launched
// with programmatic stream serialisation (launch_next, encode.cu): its
// blocks may be resident before the kernel ahead of it has ended, and wait
// here until it has, with its writes visible.  The next kernel may be made
// resident as soon as this one's blocks all have started.  A kernel launched
// without the attribute passes through.
__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Device status word bits (read by the host after each call).
constexpr uint32_t kErrNotPermutation = 1u;  // value out of range or duplicated
constexpr uint32_t kErrIterationCap = 2u;    // a bounded loop ran out (no input reaches it)
constexpr uint32_t kErrInconsistent = 4u;    // colouring constraint violated
constexpr uint32_t kErrGaveUp = 8u;          // a walk ran too long: encode again with union-find
constexpr uint32_t kErrBelow = 16u;          // a node below level 0 is not a permutation

// What a node of `level` that is not a permutation says.  Level 0 checks
// every value of the input, so its finding is final; below it, the cause may
// also be a walk that gave up.
__device__ __forceinline__ uint32_t not_permutation(uint32_t level) {
    return level == 0 ? kErrNotPermutation : kErrBelow;
}

// Longest walk along a union-find chain.  Uniform inputs and single cycles
// stay below 45 steps (2^26 entries), but inputs that keep neighbours
// together can hang every pair-node under its predecessor, a chain as long
// as the node.  A walk that gets this far stops and gives its level up
// (give_up, defer; kernels.cuh): level_settle (settle.cuh) then shortens
// every chain and finishes the unions.
constexpr uint32_t kLongChain = 256;

// ------------------------------------------------------------------------
// Parity union-find over pair-nodes.
//
// Word layout: (parent << 1) | bit.  For a non-root the bit is the colour
// difference between the node and its parent; a root points to itself and
// its bit is the orientation flag set after all unions (it flips the colour
// of the whole component so that the odd tail ends up colour 0).  A link
// hangs a root under a smaller node, so a root is the smallest pair-node of
// its component and parents strictly decrease along any chain.  The unions
// write nothing but links and the resolving pass nothing but each node's own
// root: compressing paths on the way costs more than the shorter paths save,
// because the words near the roots then move between the two L2 halves all
// the time.  Chains that are long all the same are compressed afterwards
// (settle.cuh).
// ------------------------------------------------------------------------

struct Found {
    uint32_t root;
    uint32_t bit;
};

// K finds advanced in lockstep, K loads in flight; bits of `pending` name
// the finds to run.  Returns the finds that met a long chain: their `out` is
// an ancestor, not the root.
template <int K>
__device__ __forceinline__ uint32_t uf_find_many(const uint32_t* uf, const uint32_t (&x)[K],
    Found (&out)[K], uint32_t pending) {
#pragma unroll
    for (int i = 0; i < K; ++i) out[i] = {x[i], 0u};
    for (uint32_t it = 0; pending != 0 && it < kLongChain; ++it) {
        uint32_t w[K];
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (pending & (1u << i)) w[i] = uf[out[i].root];
        }
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (!(pending & (1u << i))) continue;
            if ((w[i] >> 1) == out[i].root) {
                pending &= ~(1u << i);
            } else {
                out[i].bit ^= w[i] & 1u;
                out[i].root = w[i] >> 1;
            }
        }
    }
    return pending;
}

// K unions x(a[i]) ^ x(b[i]) == rel[i] in lockstep.  Only the larger of the
// two nodes is looked at: while it has a parent it is replaced by that; once
// it is a root it is hung under the smaller node, which need not be a root
// (it lies in another component: a root is the smallest node of its own).
// Two thirds of a random graph's unions find their larger end still alone
// and touch one word (finding both roots, with path halving, took 251 ms per
// compress at 2^30 entries, this 162 ms).  Returns the unions that met a long
// chain and are not done: a, b and rel are as far as they came.
//
// A plain load may return an older word, which still names a true ancestor
// with its true parity; the link is a compare-and-swap on a root, and a
// failed one returns the word as it is.  `kSwap`: every look is a
// compare-and-swap that expects a root, so that words are only touched by
// atomics, faster while a node's words fit L2 (see level_union).
template <int K, bool kSwap>
__device__ __forceinline__ uint32_t uf_unite_many(uint32_t* uf, uint32_t (&a)[K],
    uint32_t (&b)[K], uint32_t (&rel)[K], uint32_t pending, uint32_t* err) {
    uint32_t w[K];
    auto look = [&](int i) {
        if (kSwap) {
            w[i] = atomicCAS(uf + a[i], a[i] << 1, (b[i] << 1) | rel[i]);
            if (w[i] == a[i] << 1) pending &= ~(1u << i); // linked
        } else {
            w[i] = uf[a[i]];
        }
    };
    auto settle = [&](int i) { // a above b; both the same: nothing left to do
        const uint32_t hi = max(a[i], b[i]);
        b[i] = min(a[i], b[i]);
        a[i] = hi;
        if (a[i] == b[i]) {
            if (rel[i] != 0) atomicOr(err, kErrInconsistent);
            pending &= ~(1u << i);
        }
    };
#pragma unroll
    for (int i = 0; i < K; ++i) {
        if (pending & (1u << i)) settle(i);
        if (pending & (1u << i)) look(i);
    }
    for (uint32_t it = 0; pending != 0 && it < kLongChain; ++it) {
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (!(pending & (1u << i))) continue;
            const uint32_t up = w[i] >> 1;
            if (!kSwap && up == a[i]) {
                w[i] = atomicCAS(uf + up, up << 1, (b[i] << 1) | rel[i]);
                if (w[i] == up << 1) pending &= ~(1u << i);
            } else {
                rel[i] ^= w[i] & 1u;
                a[i] = up;
                settle(i);
                if (pending & (1u << i)) look(i);
            }
        }
    }
    return pending;
}

// Blocks take chunks of `chunk` consecutive items in increasing order from
// *counter, so the items in flight across the whole GPU stay within a few
// chunks of each other.  (A grid-stride loop lets blocks drift apart and
// spreads node-local random accesses over far more memory than L2 holds.)
// Every thread of the block must call it.
__device__ __forceinline__ bool claim_chunk(uint32_t* counter, uint64_t chunk, uint64_t total,
    uint64_t* first) {
    __shared__ uint64_t s_first;
    __syncthreads();
    if (threadIdx.x == 0) {
        s_first = (uint64_t)atomicAdd(counter, 1u) * chunk;
    }
    __syncthreads();
    *first = s_first;
    return s_first < total;
}

// ------------------------------------------------------------------------
// Warp-aggregated emission of single bits into the blob.  Lanes of the
// warp named in `active` call it together; each lane with `set` ORs bit
// `abs_bit` (absolute bit position in the blob).  Lanes that hit the same
// 32-bit word combine first, so one atomic is issued per distinct word.
// ------------------------------------------------------------------------
__device__ __forceinline__ void emit_bit(uint32_t* blob, uint64_t abs_bit, bool set,
    unsigned active) {
    const unsigned writers = __ballot_sync(active, set);
    if (!set) {
        return;
    }
    const unsigned long long word = abs_bit >> 5;
    const unsigned group = __match_any_sync(writers, word);
    const unsigned v = __reduce_or_sync(group, 1u << (abs_bit & 31));
    if ((threadIdx.x & 31) == (unsigned)(__ffs(group) - 1)) {
        atomicOr(blob + word, v);
    }
}

// ------------------------------------------------------------------------
// Factoradic ranks of the middle groups.
// ------------------------------------------------------------------------
struct U128 {
    unsigned long long lo, hi;
};

// Factoradic rank of one middle group of `count` <= 32 entries v[0..count)
// (encode_factoradic, src/internal.hpp:148-167), by one thread: digit j =
// #{k < j : v[k] < v[j]} is a popc on the mask of values seen so far, and
// Horner's rule rank = rank * (j + 1) + digit_j sums digit_j * count!/(j+1)!.
// The rank stays below 20! < 2^62 through the first 20 entries, so those
// steps are 64-bit.  A thread per group costs about 10 instructions per
// entry; the earlier warp-per-group form (ballots, prefix-OR and a 128-bit
// shuffle tree) cost about 7 warp instructions per entry, 20 times more per
// group.  *valid is false when a value is out of range or repeated.
__device__ __forceinline__ U128 thread_factoradic_rank(const uint16_t* v, uint32_t count,
    bool* valid) {
    uint32_t seen = 0;
    bool ok = true;
    auto digit = [&](uint32_t j) {
        const uint32_t value = v[j];
        ok = ok && value < count;
        const uint32_t bit = 1u << (value & 31u);
        const uint32_t d = (uint32_t)__popc(seen & (bit - 1u));
        seen |= bit;
        return d;
    };
    U128 r = {0ull, 0ull};
    const uint32_t narrow = count < 20 ? count : 20;
    for (uint32_t j = 0; j < narrow; ++j) {
        r.lo = r.lo * (j + 1) + digit(j);
    }
    for (uint32_t j = 20; j < count; ++j) {
        const unsigned long long f = j + 1;
        const unsigned long long lo = r.lo * f;
        r.hi = __umul64hi(r.lo, f) + r.hi * f;
        r.lo = lo + digit(j);
        r.hi += r.lo < lo ? 1ull : 0ull;
    }
    *valid = ok && (uint32_t)__popc(seen) == count;
    return r;
}

// ORs the `nbits` (<= 118) bits of `rank` into the blob at absolute bit
// `abs`; rank < count! <= 2^nbits, so no bit at or above nbits is set.
__device__ __forceinline__ void thread_emit_rank(uint32_t* blob, uint64_t abs, uint32_t nbits,
    U128 rank) {
    if (nbits == 0) {
        return;
    }
    uint32_t* word = blob + (abs >> 5);
    const uint32_t shift = (uint32_t)(abs & 31);
    const uint32_t last = (shift + nbits - 1) >> 5; // destination words 0..last
    uint32_t w[5] = {(uint32_t)rank.lo, (uint32_t)(rank.lo >> 32), (uint32_t)rank.hi,
        (uint32_t)(rank.hi >> 32), 0u};
    uint32_t below = 0;
#pragma unroll
    for (uint32_t i = 0; i < 5; ++i) {
        const uint32_t v = __funnelshift_l(below, w[i], shift);
        below = w[i];
        if (i <= last && v != 0) {
            atomicOr(word + i, v);
        }
    }
}

} // namespace bpb200
