// SPDX-License-Identifier: Apache-2.0
//
// Union-find levels with long chains.
//
// The unions and finds of kernels.cuh follow parents one by one and compress
// nothing, which suits inputs whose chains stay short: uniform ones and
// single cycles.  Inputs that keep neighbours together build chains as long
// as a node: when each union joins pair-nodes k and k + 1, every pair-node
// ends up under its predecessor, in whatever order the unions run.  A walk
// over more than kLongChain words gives its level up (give_up), and
// level_settle then colours it from the words as they stand, each of which
// is a true fact:
//   flatten  every pair-node takes its ancestor's word over until it points
//            at its root; a pass multiplies the stretch a word covers by at
//            least kSettleHops + 1, so a chain of 2^29 takes ten passes;
//   unite    the unions put off or, when there were more than their list
//            holds, all output pairs' again.  Of two roots that a union still
//            joins one is linked each time, so the roots left to join at
//            least halve from round to round;
// and, once a round leaves nothing undone, orients the odd tails'
// components and writes the colours.  No input makes it fail.
//
// Its blocks wait on one another between the passes, so it is launched
// cooperatively, one block per SM, and returns at once where no walk gave
// up.  What bounds it: the words' dependent reads, at one block's warps per
// SM.  Device time of the whole call, ms, for uniform inputs, neighbours kept
// in pairs and blocks of 100,001 entries (in brackets: walks without a limit,
// which ran into a cap on the pairs):
//   2^24 + 2 entries     5.1, 5.9 (failed), 4.5 (320)
//   2^25 + 2 entries     9.9, 11.4 (failed), 10.0 (700)
//   100,000,007 entries  30.4, 33.7 (failed), 36.8 (2470)
// Doing all unions again in place of the listed ones took 6.0 and 4.7, 11.6
// and 10.3, 36.2 and 46 ms.  A limit of 1024 steps for the unions suits some
// inputs (p = 1,048,583 i mod 2^28: 77 ms, 122 with 256, uniform 86), and
// costs others more (2^28 in blocks: 184 ms, 119 with 256).  3, 5 or 16 hops a
// pass: within 5 % of 8.
#pragma once

#include "device.cuh"
#include "kernels.cuh"
#include "plan.hpp"

#include <cstdint>

namespace bpb200 {

constexpr uint32_t kSettleThreads = 1024;
constexpr uint32_t kSettleHops = 8;   // words read on per pass and pair-node
constexpr uint32_t kSettleItems = 4;  // pair-nodes in flight per thread
constexpr uint32_t kSettleRounds = 64; // more than log2 of any number of roots
constexpr uint32_t kBarrierPolls = 1u << 25; // several seconds, far above any pass

// Barrier of all blocks of a cooperative launch, with a flag: *any is whether
// some thread passed `mine`.  Returns false when the wait ran out; the status
// word then says so and every block returns.
struct SettleBarrier {
    uint32_t* ctl;
    uint32_t* status;
    uint32_t target = 0;
    uint32_t pass = 0;

    __device__ bool wait(bool mine, bool* any) {
        __shared__ uint32_t s_ok;
        ++pass;
        target += gridDim.x;
        // passes alternate between two words: one is written again only after
        // the next barrier, when every block has read it
        volatile uint32_t* changed = ctl + kCtlChanged + (pass & 1u);
        __threadfence();
        const bool here = __syncthreads_or(mine) != 0;
        if (threadIdx.x == 0) {
            if (here) *changed = pass;
            __threadfence();
            atomicAdd(ctl + kCtlArrived, 1u);
            const volatile uint32_t* arrived = ctl + kCtlArrived;
            uint32_t polls = 0;
            while (*arrived < target && polls < kBarrierPolls) {
                __nanosleep(200);
                ++polls;
            }
            s_ok = *arrived >= target ? 1u : 0u;
            if (s_ok == 0) atomicOr(status, kErrIterationCap);
            __threadfence();
        }
        __syncthreads();
        *any = *changed == pass;
        return s_ok != 0;
    }
};

// Points every pair-node in [lo, end) at its root and clears the roots'
// orientation flags.
__device__ __forceinline__ bool settle_flatten(SettleBarrier& barrier, const LevelInfo& lv,
    uint32_t level, uint32_t* uf, uint64_t lo, uint64_t end) {
    const uint32_t ps = (uint32_t)lv.pcap;
    const uint64_t chunk = (uint64_t)blockDim.x * kSettleItems;
    for (bool more = true; more;) {
        bool on = false; // some word does not point at its root yet
        for (uint64_t c = lo + blockIdx.x * chunk; c < end; c += gridDim.x * chunk) {
            uint32_t up[kSettleItems], bit[kSettleItems];
            uint32_t live = 0, moved = 0;
#pragma unroll
            for (uint32_t i = 0; i < kSettleItems; ++i) {
                const uint64_t p = c + i * blockDim.x + threadIdx.x;
                if (p >= end) continue;
                const uint32_t x = (uint32_t)p;
                const uint32_t j = x / ps;
                const uint32_t s = size_at(lv, level, j);
                if (x - j * ps >= s - s / 2) continue; // padding
                const uint32_t w = __ldcg(uf + x);
                up[i] = w >> 1;
                bit[i] = w & 1u;
                if (up[i] != x) {
                    live |= 1u << i;
                } else if (bit[i] != 0) {
                    uf[x] = x << 1;
                }
            }
            for (uint32_t hop = 0; hop < kSettleHops && live != 0; ++hop) {
                uint32_t w[kSettleItems];
#pragma unroll
                for (uint32_t i = 0; i < kSettleItems; ++i) {
                    if (live & (1u << i)) w[i] = __ldcg(uf + up[i]);
                }
#pragma unroll
                for (uint32_t i = 0; i < kSettleItems; ++i) {
                    if (!(live & (1u << i))) continue;
                    if ((w[i] >> 1) == up[i]) {
                        live &= ~(1u << i); // a root
                    } else {
                        up[i] = w[i] >> 1;
                        bit[i] ^= w[i] & 1u;
                        moved |= 1u << i;
                    }
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < kSettleItems; ++i) {
                if (moved & (1u << i)) {
                    uf[c + i * blockDim.x + threadIdx.x] = (up[i] << 1) | bit[i];
                }
            }
            on |= live != 0;
        }
        if (!barrier.wait(on, &more)) return false;
    }
    return true;
}

__global__ void __launch_bounds__(kSettleThreads, 1) level_settle(const Plan* __restrict__ plan,
    uint32_t level, const uint32_t* __restrict__ inv, uint32_t* uf, uint32_t* __restrict__ xbits,
    const __grid_constant__ Chains chains, uint32_t* status) {
    wait_for_previous();
    if (!given_up(chains)) return; // the same for all blocks: nothing here sets it
    const uint32_t deferred = chains.ctl[kCtlDeferred];
    const LevelInfo& lv = plan->levels[level];
    const uint32_t ps = (uint32_t)lv.pcap;
    const NodeRange nr = level_nodes(*plan, level);
    const uint64_t lo = nr.lo * ps;
    const uint64_t end = lo + ((uint64_t)ps << nr.shift);
    const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    SettleBarrier barrier{chains.ctl, status};
    bool again = deferred != 0;
    for (uint32_t round = 0; again; ++round) {
        if (!settle_flatten(barrier, lv, level, uf, lo, end)) return;
        if (round == kSettleRounds) {
            atomicOr(status, kErrIterationCap);
            return;
        }
        bool undone = false;
        if (deferred > chains.room) {
            for (uint64_t p0 = lo + id * kUnionItems; p0 < end; p0 += stride * kUnionItems) {
                undone |= unite_outputs(lv, level, inv, uf, p0, end, true, nullptr, status);
            }
        } else {
            for (uint64_t i = id; i < deferred; i += stride) {
                const uint2 r = chains.list[i];
                uint32_t a[1] = {r.x}, b[1] = {r.y >> 1}, rel[1] = {r.y & 1u};
                undone |= uf_unite_many<1, true>(uf, a, b, rel, 1u, status) != 0;
            }
        }
        if (!barrier.wait(undone, &again)) return;
    }
    if (!settle_flatten(barrier, lv, level, uf, lo, end)) return;
    // as level_orient
    for (uint64_t j = nr.lo + id; j < nr.lo + (1ull << nr.shift); j += stride) {
        const uint32_t s = size_at(lv, level, (uint32_t)j);
        if ((s & 1u) == 0) continue;
        if (inv[2 * j * ps + s - 1] >= s) atomicOr(status, not_permutation(level));
        const uint32_t x = (uint32_t)j * ps + (s >> 1);
        const uint32_t w = __ldcg(uf + x);
        if ((w >> 1) != x && (w & 1u) != 0) atomicOr(uf + (w >> 1), 1u);
    }
    if (!barrier.wait(false, &again)) return;
    // as level_roots
    for (uint64_t p = (lo & ~31ull) + id; p - (threadIdx.x & 31) < end; p += stride) {
        bool colour = false;
        if (p >= lo && p < end) {
            const uint32_t x = (uint32_t)p;
            const uint32_t j = x / ps;
            const uint32_t s = size_at(lv, level, j);
            if (x - j * ps < s - s / 2) {
                const uint32_t w = __ldcg(uf + x);
                colour = (w & 1u) != 0;
                if ((w >> 1) != x) colour ^= (__ldcg(uf + (w >> 1)) & 1u) != 0;
            }
        }
        const unsigned word = __ballot_sync(0xffffffffu, colour);
        if ((threadIdx.x & 31) == 0) xbits[p >> 5] = word;
    }
}

} // namespace bpb200
