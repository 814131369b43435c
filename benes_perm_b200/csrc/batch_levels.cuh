// SPDX-License-Identifier: Apache-2.0
//
// Batched level kernels: one launch runs one kernel step of one routing
// level for a whole group of permutations.
//
// The host builds, per routing level, a device work list of LevelJob
// entries, one per permutation whose level is still above its tile level:
// the permutation's plan and scratch, and for every kernel step the range
// of the launch's blocks that work on it (first[kind], blocks[kind]).  A
// block finds its job by binary search on `first`, then runs the same body
// as the one-permutation kernel over the job's share of the blocks (a Grid
// in place of blockIdx / gridDim).  Kernels that claim work from
// per-level counters keep claiming from the job's own control words, so
// the work in flight at any moment still covers a few nodes of one or two
// permutations.  A group of R permutations therefore needs one launch per
// kernel step per level instead of R, and the steps of short, latency-bound
// levels of different permutations (list contraction and ranking, small
// walks) run side by side on different SMs.
#pragma once

#include "kernels.cuh"
#include "tile.cuh"
#include "walk.cuh"

#include <cstdint>

namespace bpb200 {

enum BatchKind : int {
    kBInit = 0,
    kBInverse,
    kBEdges,
    kBWalk,
    kBRank,
    kBColours,
    kBUnion,
    kBOrient,
    kBRoots,
    kBOutputs,
    kBContract,                         // list e -> e + 1: kBContract + e - 1
    kBExpand = kBContract + kMaxLists,  // list e + 1 -> e: kBExpand + e - 1
    kBatchKinds = kBExpand + kMaxLists
};

// One permutation at one routing level of a batched launch sequence.
struct LevelJob {
    const Plan* plan;
    const void* src;         // level 0: the caller's input
    uint32_t* inv;           // this level's inverse
    uint32_t* child_inv;     // children's inverse
    uint32_t* edge;          // edges, or union-find words, of this level and then the next
    uint32_t* stamp;
    uint32_t* xbits;
    uint32_t* ybits;
    uint4* state[kMaxLists + 1];
    uint32_t* mark[kMaxLists + 1];
    uint8_t* colour[kMaxLists + 1];
    uint32_t* control;       // the level's control words
    uint32_t* status;
    NodeAddress* addr[2];
    uint32_t* blob;          // level 0: the blob whose header is written
    uint32_t level;
    uint32_t src_bytes;
    uint32_t top;            // list that list_rank colours
    uint32_t walks;          // 1: coloured by walks, 0: by union-find
    uint32_t child_walks;    // the next global level: 1 walks, 0 union-find, 2 none
    uint32_t header_bytes;   // level 0 only
    uint8_t header[84];
    uint32_t first[kBatchKinds];
    uint32_t blocks[kBatchKinds];
};

// One section's switch emission of one permutation at one level.
struct EmitJob {
    const Plan* plan;
    const uint32_t* bits;
    const NodeAddress* addr;
    uint32_t* blob;
    uint64_t full;           // full packets (block forms) or first packet (per-bit form)
    uint32_t level;
    int32_t side;
    int32_t form;
    uint32_t first;
    uint32_t blocks;
    uint32_t pad_;
};

// Word fills (blob clearing, validation sentinels).
struct FillJob {
    uint32_t* ptr;
    uint64_t words;
    uint32_t value;
    uint32_t first;
    uint32_t blocks;
    uint32_t pad_;
};

// The job whose block range holds this block: the last job with
// first <= blockIdx.x (jobs that own no blocks share the next job's first
// and are skipped by taking the last).
template <typename Job, typename First>
__device__ __forceinline__ const Job* batch_job(const Job* jobs, uint32_t n, First first_of,
    Grid* g) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (first_of(jobs[mid]) <= blockIdx.x) lo = mid; else hi = mid;
    }
    return jobs + lo;
}

__device__ __forceinline__ const LevelJob* level_job(const LevelJob* jobs, uint32_t n, int kind,
    Grid* g) {
    const LevelJob* j = batch_job(jobs, n, [kind](const LevelJob& x) { return x.first[kind]; }, g);
    g->bid = blockIdx.x - j->first[kind];
    g->nblk = j->blocks[kind];
    return j;
}

// A member that meets a long chain gives up as a whole: the host encodes it
// again by itself.
__device__ __forceinline__ Chains batch_chains(const LevelJob* j) {
    return Chains{j->control, j->status, nullptr, 0};
}

__global__ void __launch_bounds__(256) batch_fill(const FillJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const FillJob* j = batch_job(jobs, n, [](const FillJob& x) { return x.first; }, &g);
    g.bid = blockIdx.x - j->first;
    g.nblk = j->blocks;
    if (g.bid >= g.nblk) return;
    for (uint64_t i = (uint64_t)g.bid * blockDim.x + threadIdx.x; i < j->words;
         i += (uint64_t)g.nblk * blockDim.x) {
        j->ptr[i] = j->value;
    }
}

// Status word, blob header (after the blob was cleared by batch_fill) and
// switch addresses of every level.
__global__ void __launch_bounds__(256) batch_init(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBInit, &g);
    if (g.bid >= g.nblk) return;
    if (g.bid == 0) {
        if (threadIdx.x == 0) *j->status = 0;
        uint8_t* b = reinterpret_cast<uint8_t*>(j->blob);
        for (uint32_t i = threadIdx.x; i < j->header_bytes; i += blockDim.x) b[i] = j->header[i];
    }
    level_descriptors_run(g, j->plan, j->addr[0], j->addr[1]);
}

__global__ void __launch_bounds__(256) batch_inverse(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBInverse, &g);
    if (g.bid >= g.nblk) return;
    uint32_t* uf = j->walks ? nullptr : j->edge;
    uint32_t* claims = j->control + kCtlClaimInverse;
    if (j->src_bytes == 8) {
        level_inverse_run<uint64_t>(g, j->plan, (const uint64_t*)j->src, j->inv, uf, claims, j->status);
    } else {
        level_inverse_run<uint32_t>(g, j->plan, (const uint32_t*)j->src, j->inv, uf, claims, j->status);
    }
}

__global__ void __launch_bounds__(256) batch_edges(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBEdges, &g);
    if (g.bid >= g.nblk) return;
    level_edges_run(g, j->plan, j->inv, j->edge, j->stamp, j->status);
}

__global__ void __launch_bounds__(256) batch_walk(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBWalk, &g);
    if (g.bid >= g.nblk) return;
    level_walk_run(g, j->plan, j->level, j->edge, j->stamp, j->state[1], j->mark[1], j->status);
}

__global__ void __launch_bounds__(256) batch_contract(const LevelJob* jobs, uint32_t n, uint32_t e) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBContract + (int)e - 1, &g);
    if (g.bid >= g.nblk) return;
    list_contract_run(g, j->plan, j->level, e, j->state[e], j->mark[e], j->state[e + 1],
        j->mark[e + 1], j->status);
}

__global__ void __launch_bounds__(kRankThreads, 1) batch_rank(const LevelJob* jobs, uint32_t n) {
    extern __shared__ __align__(16) uint32_t rank_shared[];
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBRank, &g);
    if (g.bid >= g.nblk) return;
    list_rank_run(g, j->plan, j->level, j->top, j->state[j->top], j->colour[j->top], j->status,
        rank_shared);
}

__global__ void __launch_bounds__(256) batch_expand(const LevelJob* jobs, uint32_t n, uint32_t e) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBExpand + (int)e - 1, &g);
    if (g.bid >= g.nblk) return;
    list_expand_run(g, j->plan, j->level, e, j->state[e], j->mark[e], j->colour[e + 1],
        j->colour[e], j->status);
}

__global__ void __launch_bounds__(256) batch_colours(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBColours, &g);
    if (g.bid >= g.nblk) return;
    level_colours_run(g, j->plan, j->level, j->edge, j->stamp, j->colour[1], j->xbits, j->status);
}

__global__ void __launch_bounds__(256, BPB200_UNION_MIN_BLOCKS) batch_union(const LevelJob* jobs,
    uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBUnion, &g);
    if (g.bid >= g.nblk) return;
    level_union_run(g, j->plan, j->level, j->inv, j->edge, batch_chains(j), j->status);
}

__global__ void __launch_bounds__(256) batch_orient(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBOrient, &g);
    if (g.bid >= g.nblk) return;
    level_orient_run(g, j->plan, j->level, j->inv, j->edge, batch_chains(j), j->status);
}

__global__ void __launch_bounds__(256, 4) batch_roots(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBRoots, &g);
    if (g.bid >= g.nblk) return;
    level_roots_run(g, j->plan, j->level, j->edge, j->xbits, batch_chains(j));
}

__global__ void __launch_bounds__(256) batch_outputs(const LevelJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const LevelJob* j = level_job(jobs, n, kBOutputs, &g);
    if (g.bid >= g.nblk) return;
    level_outputs_run(g, j->plan, j->level, j->inv, j->xbits, j->ybits, j->child_inv,
        j->child_walks == 1 ? j->edge : nullptr, j->stamp, j->child_walks == 0 ? j->edge : nullptr);
}

// Switch emission: every (permutation, section, form) of the level in one
// launch.
__global__ void __launch_bounds__(256) batch_emit(const EmitJob* jobs, uint32_t n) {
    wait_for_previous();
    Grid g;
    const EmitJob* j = batch_job(jobs, n, [](const EmitJob& x) { return x.first; }, &g);
    g.bid = blockIdx.x - j->first;
    g.nblk = j->blocks;
    if (g.bid >= g.nblk) return;
    level_emit_form(g, j->form, j->plan, j->level, j->side, j->bits, j->addr, j->blob, j->full);
}

} // namespace bpb200
