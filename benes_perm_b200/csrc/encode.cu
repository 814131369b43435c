// SPDX-License-Identifier: Apache-2.0
//
// Host orchestration and C ABI of the B200 compact encoder.
//
// One call: plan on the host (closed-form layout, a few KB) -> prologue
// kernel (places the plan, clears blob and status, header bytes) -> level
// kernels for the levels whose nodes exceed a tile -> tile kernels (a stage
// of two levels where nodes or launches are small, then the rest of every
// subtree) in shared memory.  A permutation of one tile is one launch.
// Everything runs on one stream; scratch lives in a pooled per-device
// workspace so repeated calls allocate nothing.
#include "../../include/benes_b200.h"
#include "batch_levels.cuh"
#include "kernels.cuh"
#include "layout.hpp"
#include "plan.hpp"
#include "settle.cuh"
#include "tile.cuh"
#include "walk.cuh"

#include <cuda_runtime.h>
#include <dlfcn.h>
#include <immintrin.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

namespace bpb200 {
namespace {

constexpr uint64_t kTileMaxEntries = 8192;
constexpr uint32_t kTileSmemBudget = 224 * 1024;
// Above this a tile runs as one 1024-thread CTA per SM (tile_encode_wide).
constexpr uint32_t kTileSmemTwoPerSm = 112 * 1024;
constexpr int kLevelThreads = 256;

// Kernel kinds reported by bpb200_last_profile.
enum KernelKind : int {
    kKindPrologue = 0,
    kKindInverse,
    kKindDescriptors, // part of the prologue: never recorded, kept in the numbering
    kKindUnion,
    kKindOrient,
    kKindResolve,
    kKindOutputBits,
    kKindTile,
    kKindEmit,
    kKindWalk,
    kKindJump,
    kKindPlace, // partitioned inverse (level_bucket + level_place)
    kKernelKinds
};

struct CudaFail {
    cudaError_t err;
    const char* what;
};

void check(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        throw CudaFail{e, what};
    }
}

// ------------------------------------------------------------ workspace

// Device arrays of the ruler lists 1..kMaxLists (walk.cuh); index 0 unused.
struct WalkLists {
    uint4* state[kMaxLists + 1] = {};
    uint32_t* mark[kMaxLists + 1] = {};
    uint8_t* colour[kMaxLists + 1] = {};
};

constexpr uint64_t up256(uint64_t x) { return (x + 255) & ~255ull; }

// Elements of list e over `pairs` pair-nodes.
constexpr uint64_t list_elements(uint64_t pairs, uint32_t e) {
    return (pairs >> (kRulerLog2 * e)) + 2;
}

// Bytes of the lists over `pairs` pair-nodes; with `base`, places them there.
constexpr uint64_t place_lists(uint64_t pairs, unsigned char* base, WalkLists* out) {
    uint64_t at = 0;
    for (uint32_t e = 1; e <= kMaxLists; ++e) {
        const uint64_t n = list_elements(pairs, e);
        if (out != nullptr) {
            out->state[e] = reinterpret_cast<uint4*>(base + at);
            out->mark[e] = reinterpret_cast<uint32_t*>(base + at + up256(n * 16));
            out->colour[e] = reinterpret_cast<uint8_t*>(base + at + up256(n * 16) + up256(n * 4));
        }
        at += up256(n * 16) + up256(n * 4) + up256(n);
    }
    return at;
}

struct Workspace {
    int device = -1;
    cudaStream_t stream = nullptr;
    cudaStream_t copy_stream = nullptr; // early blob download of the host path
    cudaEvent_t start = nullptr, stop = nullptr;
    cudaEvent_t early = nullptr;        // the blob's first cluster groups are final
    cudaEvent_t parts[8] = {};          // tile parts done (progressive blob download)
    cudaEvent_t inparts[8] = {};        // input parts on the device (host path upload)
    Plan* d_plan = nullptr;
    Plan* h_plan = nullptr;       // pinned staging for the plan upload
    uint32_t* d_status = nullptr;
    uint32_t* h_status = nullptr; // pinned
    uint32_t* inv[2] = {nullptr, nullptr}; // levels alternate the two
    uint32_t* edge = nullptr;              // output edges of a walk level, or a
                                           // union-find level's words (one per pair-node)
    uint32_t* stamp = nullptr;             // walk stamps, one per pair-node
    uint32_t* xbits = nullptr;
    uint32_t* ybits = nullptr;
    WalkLists lists;                       // ruler lists of the walk levels
    void* lists_mem = nullptr;
    uint32_t* control = nullptr;           // per-level control words
    uint2* records = nullptr;              // partitioned-inverse records (kernels.cuh)
    uint32_t* cursor = nullptr;            // fill level of each destination window
    NodeAddress* addr[2] = {nullptr, nullptr};
    uint64_t slot_cap = 0, pair_cap = 0, node_cap = 0;
    void* input = nullptr;        // staging for host-path inputs
    uint64_t input_cap = 0;
    uint32_t* blob = nullptr;     // staging for host-path blobs
    uint64_t blob_cap = 0;
    std::vector<cudaEvent_t> events; // profiling events, reused across calls
    bool busy = false;

    void release_scratch() {
        for (void* p : {(void*)inv[0], (void*)inv[1], (void*)edge, (void*)stamp, (void*)xbits, (void*)ybits,
                 lists_mem, (void*)control, (void*)records, (void*)cursor, (void*)addr[0],
                 (void*)addr[1]}) {
            if (p) cudaFree(p);
        }
        inv[0] = inv[1] = edge = stamp = xbits = ybits = control = cursor = nullptr;
        lists = WalkLists();
        lists_mem = nullptr;
        records = nullptr;
        addr[0] = addr[1] = nullptr;
        slot_cap = pair_cap = node_cap = 0;
    }
    void destroy() {
        release_scratch();
        if (input) cudaFree(input);
        if (blob) cudaFree(blob);
        if (d_plan) cudaFree(d_plan);
        if (d_status) cudaFree(d_status);
        if (h_plan) cudaFreeHost(h_plan);
        if (h_status) cudaFreeHost(h_status);
        if (start) cudaEventDestroy(start);
        if (stop) cudaEventDestroy(stop);
        if (early) cudaEventDestroy(early);
        for (cudaEvent_t e : parts) {
            if (e) cudaEventDestroy(e);
        }
        for (cudaEvent_t e : inparts) {
            if (e) cudaEventDestroy(e);
        }
        if (stream) cudaStreamDestroy(stream);
        if (copy_stream) cudaStreamDestroy(copy_stream);
        for (cudaEvent_t e : events) cudaEventDestroy(e);
        *this = Workspace();
    }
};

std::mutex g_pool_mutex;
std::vector<std::unique_ptr<Workspace>> g_pool;

Workspace* acquire(int device) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    for (auto& w : g_pool) {
        if (!w->busy && w->device == device) {
            w->busy = true;
            return w.get();
        }
    }
    auto w = std::make_unique<Workspace>();
    w->device = device;
    check(cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    check(cudaEventCreate(&w->start), "cudaEventCreate");
    check(cudaEventCreate(&w->stop), "cudaEventCreate");
    check(cudaStreamCreateWithFlags(&w->copy_stream, cudaStreamNonBlocking), "cudaStreamCreate");
    check(cudaEventCreateWithFlags(&w->early, cudaEventDisableTiming), "cudaEventCreate");
    for (cudaEvent_t& e : w->parts) {
        check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    }
    for (cudaEvent_t& e : w->inparts) {
        check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    }
    check(cudaMalloc(&w->d_plan, sizeof(Plan)), "cudaMalloc(plan)");
    check(cudaMallocHost(&w->h_plan, sizeof(Plan)), "cudaMallocHost(plan)");
    check(cudaMalloc(&w->d_status, sizeof(uint32_t)), "cudaMalloc(status)");
    check(cudaMallocHost(&w->h_status, sizeof(uint32_t)), "cudaMallocHost(status)");
    w->busy = true;
    g_pool.push_back(std::move(w));
    return g_pool.back().get();
}

void release(Workspace* w) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    w->busy = false;
}

struct Lease {
    Workspace* w;
    explicit Lease(int device) : w(acquire(device)) {}
    ~Lease() { release(w); }
};

bool single_launch(const Plan& p);

// Grows the level scratch to fit `p`.  Growth at least doubles the previous
// capacities: freeing device memory synchronises the whole device, so a
// workspace that serves requests of varying sizes (the batched and serving
// forms) must reach its final size after a few calls, not one per call.
void ensure_scratch(Workspace& w, const Plan& p) {
    const bool levels = !single_launch(p);
    uint64_t slots = levels ? p.max_slots : 0;
    uint64_t pairs = levels ? p.max_pairs : 0;
    uint64_t nodes = levels ? (1ull << p.tile_level) : 0;
    const bool need_records = p.levels[0].cap > kWalkMaxNode;
    if (slots <= w.slot_cap && pairs <= w.pair_cap && nodes <= w.node_cap &&
        (w.records != nullptr || !need_records)) {
        return;
    }
    if (slots == 0) {
        return;
    }
    slots = std::max(slots, 2 * w.slot_cap);
    pairs = std::max(pairs, 2 * w.pair_cap);
    nodes = std::max(nodes, 2 * w.node_cap);
    w.release_scratch();
    check(cudaMalloc(&w.inv[0], slots * 4), "cudaMalloc(inverse)");
    check(cudaMalloc(&w.inv[1], slots * 4), "cudaMalloc(inverse)");
    check(cudaMalloc(&w.edge, slots * 4), "cudaMalloc(edges)");
    check(cudaMalloc(&w.stamp, pairs * 4), "cudaMalloc(stamps)");
    check(cudaMalloc(&w.xbits, (pairs / 32 + 4) * 4), "cudaMalloc(colour bits)");
    check(cudaMalloc(&w.ybits, (pairs / 32 + 4) * 4), "cudaMalloc(output bits)");
    check(cudaMalloc(&w.lists_mem, place_lists(pairs, nullptr, nullptr)), "cudaMalloc(ruler lists)");
    place_lists(pairs, (unsigned char*)w.lists_mem, &w.lists);
    check(cudaMalloc(&w.control, kMaxLevels * kCtlWords * 4), "cudaMalloc(control)");
    if (p.levels[0].cap > kWalkMaxNode) {
        // only levels with nodes above L2 size use the partitioned inverse
        check(cudaMalloc(&w.records, slots * sizeof(uint2)), "cudaMalloc(records)");
        check(cudaMalloc(&w.cursor, kMaxWindows * 4), "cudaMalloc(cursors)");
    }
    check(cudaMalloc(&w.addr[0], nodes * sizeof(NodeAddress)), "cudaMalloc(descriptors)");
    check(cudaMalloc(&w.addr[1], nodes * sizeof(NodeAddress)), "cudaMalloc(descriptors)");
    w.slot_cap = slots;
    w.pair_cap = pairs;
    w.node_cap = nodes;
}

// ------------------------------------------------------------ prologue

struct Prologue {
    Plan plan;
    Header header;
};

// First launch of an encode with global levels: places the plan, clears the
// blob but for its header, the status word and the level counters, fills
// level 0's inverse with 0xffffffff (a repeated value leaves such a slot
// behind) and works out the switch addresses of every global level.  One
// launch in the place of an upload, three memsets and two kernels.
__global__ void __launch_bounds__(256) prologue(const __grid_constant__ Prologue p, Plan* plan,
    uint32_t* status, uint32_t* __restrict__ blob, uint64_t blob_words,
    uint32_t* __restrict__ control, uint32_t control_words, uint32_t* __restrict__ inv,
    uint64_t inv_words, NodeAddress* __restrict__ in_addr, NodeAddress* __restrict__ out_addr) {
    const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t* from = reinterpret_cast<const uint32_t*>(&p.plan);
    for (uint64_t i = id; i < sizeof(Plan) / 4; i += stride) {
        reinterpret_cast<uint32_t*>(plan)[i] = from[i];
    }
    if (id == 0) *status = 0;
    for (uint64_t i = id; i < control_words; i += stride) control[i] = 0;
    for (uint64_t i = id; i < blob_words; i += stride) {
        blob[i] = i < sizeof(Header) / 4 ? header_word(p.header, i) : 0u;
    }
    for (uint64_t i = id; i < inv_words; i += stride) inv[i] = ~0u;
    level_descriptors_run(launch_grid(), &p.plan, in_addr, out_addr);
}

// Launches a kernel with one launch attribute set.  A cooperative launch of
// more blocks than the stream's context can hold at once (one that owns only
// a part of the SMs) is tried again with half of them.
template <typename... Params, typename... Args>
void launch_with(cudaLaunchAttributeID id, void (*kernel)(Params...), uint64_t blocks,
    uint32_t threads, uint32_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3((unsigned)blocks);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = st;
    cudaLaunchAttribute attribute{};
    attribute.id = id;
    if (id == cudaLaunchAttributeCooperative) {
        attribute.val.cooperative = 1;
    } else {
        attribute.val.programmaticStreamSerializationAllowed = 1;
    }
    config.attrs = &attribute;
    config.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&config, kernel, Params(args)...);
    while (e == cudaErrorCooperativeLaunchTooLarge && config.gridDim.x > 1) {
        cudaGetLastError(); // the error is not sticky
        config.gridDim.x /= 2;
        e = cudaLaunchKernelEx(&config, kernel, Params(args)...);
    }
    check(e, "kernel launch");
}

// Launches the next kernel of an encode's sequence: with programmatic stream
// serialisation, so its launch and the start of its blocks overlap the end
// of the kernel ahead, on which it waits itself (wait_for_previous).
template <typename... Params, typename... Args>
void launch_next(void (*kernel)(Params...), uint64_t blocks, uint32_t threads, uint32_t smem,
    cudaStream_t st, Args&&... args) {
    launch_with(cudaLaunchAttributeProgrammaticStreamSerialization, kernel, blocks, threads, smem,
        st, args...);
}

// ------------------------------------------------------------ tile sizing

// Shared memory of levels [t0, stop) of one node of level t0.
TileShape tile_shape(const Plan& p, uint32_t t0, uint32_t stop) {
    uint64_t slots = 0;
    const uint32_t end = stop == p.depth ? stop + 1 : stop; // the leaves, too
    for (uint32_t l = t0; l < end; ++l) {
        slots = std::max<uint64_t>(slots,
            (uint64_t)tile_node_slots(p.levels[l].pcap, l == p.depth, p.leaf) << (l - t0));
    }
    TileShape s;
    s.slots = (uint32_t)std::min<uint64_t>((slots + 3) & ~3ull, 1u << 30);
    uint32_t off[5];
    s.smem = tile_smem_layout(s.slots, stop - t0, off);
    if (slots >= 65536) {
        s.smem = UINT32_MAX;
    }
    return s;
}

TileShape tile_shape(const Plan& p, uint32_t t0) { return tile_shape(p, t0, p.depth); }

// Stages.  Nodes of up to 2^15 entries fit an SM for a level or two even
// when they are above the tile size: the levels from there to the tile level
// run as one launch of tile_encode_wide over [l, stop) instead of level
// kernels, which for so small nodes are all launches and latency (2^20
// entries: 672 -> 648 us) or random L2 accesses (2^30 entries, levels 15 and
// 16: 27 ms as level kernels, 15 ms as a stage).
// A launch of few tiles hands the subtree over after two levels to four
// times as many CTAs: a lone CTA takes 12 us for a level of 16384 entries,
// four take 6 (16384 entries: 187 -> 141 us, 2^16: 285 -> 230 us; tiles of
// 4096 entries lose more by the hand-over than they gain, 93 -> 103 us).
constexpr uint64_t kStageMaxNode = 1ull << 15;
constexpr uint32_t kStageLevels = 2;
constexpr uint64_t kFewTiles = 4 * 148;          // CTAs after the hand-over, at most
constexpr uint64_t kFewTilesMinNode = 4096;      // larger tiles only

// Level at which a stage from level l on stops, at or before `last`; 0: no
// stage.
uint32_t stage_stop(const Plan& p, uint32_t l, uint32_t last) {
    if (l >= last || p.levels[l].cap > kStageMaxNode || (p.shards > 1 && l < p.shard_level)) {
        return 0;
    }
    for (uint32_t stop = std::min(last, l + kStageLevels); stop > l; --stop) {
        // every node handed over has to be internal
        if (stop < p.depth && p.levels[stop].q > p.leaf &&
            tile_shape(p, l, stop).smem <= kTileSmemBudget) {
            return stop;
        }
    }
    return 0;
}

// Level at which a launch of the tiles of level l hands over, or 0: whole
// subtrees.
uint32_t few_tiles_stop(const Plan& p, uint32_t l) {
    const uint64_t tiles = 1ull << level_nodes(p, l).shift;
    if (tiles * 4 > kFewTiles || p.levels[l].cap <= kFewTilesMinNode) {
        return 0;
    }
    return stage_stop(p, l, p.depth);
}

// Threads per tile.  With more tiles than two per SM, 256: the tile is bound
// by instruction issue and by its barriers, and three small CTAs per SM wait
// less at theirs (tiles of 100,000,007 entries: 6.1 ms against 7.7 ms with
// 512).  Fewer tiles than that leave SMs idle, and one tile ends sooner with
// 512 (8192 entries: 107 us against 140 us).  Wide tiles fill an SM each.
unsigned tile_threads(uint64_t tiles, bool wide, uint64_t entries) {
    if (tiles > 2 * 148 && !wide) return kTileThreads / 2;
    unsigned t = 128;
    while (t < (wide ? 2 : 1) * kTileThreads && (uint64_t)t * 8 < entries) t *= 2;
    return t;
}

// Threads of a stage: 8 entries each, up to 1024.
unsigned stage_threads(uint64_t entries) { return tile_threads(1, true, entries); }

// Whether the whole permutation is one launch of one CTA.
bool single_launch(const Plan& p) { return p.tile_level == 0 && few_tiles_stop(p, 0) == 0; }

// Slots and pair-nodes of the largest level the launches keep in device
// memory: those down to the tile level and those that launches of few tiles
// hand over at, which a shard, having fewer tiles, does further down.
void size_levels(Plan& p) {
    p.max_slots = p.max_pairs = 0;
    auto hold = [&](uint32_t l) {
        p.max_slots = std::max<uint64_t>(p.max_slots, (2 * p.levels[l].pcap) << l);
        p.max_pairs = std::max<uint64_t>(p.max_pairs, p.levels[l].pcap << l);
    };
    for (uint32_t l = 0; l <= p.tile_level; ++l) hold(l);
    for (uint32_t l = p.tile_level; (l = few_tiles_stop(p, l)) != 0;) hold(l);
}

// Picks the tile level: the first level whose nodes fit `tile_max` entries
// and whose deepest padded tile level also fits the shared-memory budget.
void choose_tile(Plan& p, TileShape* shape, uint64_t tile_max = kTileMaxEntries) {
    uint32_t t0 = 0;
    while (t0 < p.depth && p.levels[t0].cap > tile_max) {
        ++t0;
    }
    TileShape s = tile_shape(p, t0);
    while (s.smem > kTileSmemBudget && t0 < p.depth) {
        ++t0;
        s = tile_shape(p, t0);
    }
    p.tile_level = t0;
    size_levels(p);
    *shape = s;
}

bool valid_shard(uint32_t shard, uint32_t shards) {
    return shards != 0 && (shards & (shards - 1)) == 0 && shard < shards;
}

// Restricts a plan whose tile level is chosen to one shard; false when the
// permutation is too small for that many.
bool set_shard(Plan& p, uint32_t shard, uint32_t shards) {
    uint32_t k = 0;
    while ((1u << k) < shards) ++k;
    if (!valid_shard(shard, shards) || k > p.tile_level) return false;
    p.shards = shards;
    p.shard = shard;
    p.shard_level = k;
    size_levels(p);
    return true;
}

std::atomic<int> g_force_union_find{0};

// ------------------------------------------------------------ tuning
//
// Launch choices that change speed but never bytes, per size class (the
// class of a permutation of n entries is ceil(log2 n)):
//   walk_blocks_per_sm  kept in the setting's layout; no kernel reads it
//                       (the walks take one ruler per thread)
//   walk_max_log2       largest node coloured by ruler walks (larger nodes
//                       by union-find); at most the compiled walk limit
//   jump_block_log2     largest list of a node's rulers ranked inside one
//                       CTA (2^10 to 2^14), longer ones are contracted first
//   tile_max_log2       largest node handed to the shared-memory tile
// The table comes from tuning.json beside this library (written by
// benes_perm_b200/tune.py; BPB200_TUNING_FILE names another file, "none"
// disables it), loaded once; classes it lacks take the nearest class it
// has, and without a table the compiled defaults apply.
struct Tuning {
    uint32_t walk_blocks_per_sm;
    uint32_t walk_max_log2;
    uint32_t jump_block_log2;
    uint32_t tile_max_log2;
};

Tuning default_tuning() {
    return Tuning{4, BPB200_WALK_MAX_LOG2, kRankMaxLog2, 13};
}

Tuning clamp_tuning(Tuning t) {
    auto clamp = [](uint32_t v, uint32_t lo, uint32_t hi) { return v < lo ? lo : (v > hi ? hi : v); };
    t.walk_blocks_per_sm = clamp(t.walk_blocks_per_sm, 1, 8);
    t.walk_max_log2 = clamp(t.walk_max_log2, 10, BPB200_WALK_MAX_LOG2);
    t.jump_block_log2 = clamp(t.jump_block_log2, 4, 18);
    t.tile_max_log2 = clamp(t.tile_max_log2, 9, 14);
    return t;
}

struct TuningTable {
    bool has[64] = {};
    Tuning at[64];
};

// Reads {"classes": {"<class>": {"<knob>": <int>, ...}, ...}}; anything
// else in the file is ignored.  A missing or malformed file gives an empty
// table.
TuningTable load_tuning_table() {
    TuningTable t;
    std::string path;
    if (const char* env = std::getenv("BPB200_TUNING_FILE")) {
        path = env;
    } else {
        Dl_info info{};
        if (dladdr((void*)&default_tuning, &info) != 0 && info.dli_fname != nullptr) {
            path = info.dli_fname;
            const size_t slash = path.find_last_of('/');
            path = (slash == std::string::npos ? std::string(".") : path.substr(0, slash)) +
                "/tuning.json";
        }
    }
    if (path.empty() || path == "none") return t;
    FILE* f = std::fopen(path.c_str(), "rb");
    if (f == nullptr) return t;
    std::string text;
    char buf[4096];
    size_t got;
    while ((got = std::fread(buf, 1, sizeof buf, f)) > 0) text.append(buf, got);
    std::fclose(f);
    size_t at = text.find("\"classes\"");
    if (at == std::string::npos) return t;
    at = text.find('{', at);
    while (at != std::string::npos) {
        const size_t q0 = text.find('"', at + 1);
        const size_t close = text.find('}', at + 1);
        if (q0 == std::string::npos || (close != std::string::npos && close < q0)) break;
        const size_t q1 = text.find('"', q0 + 1);
        const size_t open = text.find('{', q1);
        const size_t end = text.find('}', open);
        if (q1 == std::string::npos || open == std::string::npos || end == std::string::npos) break;
        const int cls = std::atoi(text.substr(q0 + 1, q1 - q0 - 1).c_str());
        Tuning v = default_tuning();
        const std::string body = text.substr(open + 1, end - open - 1);
        auto knob = [&](const char* name, uint32_t* field) {
            const size_t k = body.find(std::string("\"") + name + "\"");
            if (k == std::string::npos) return;
            const size_t colon = body.find(':', k);
            if (colon != std::string::npos) *field = (uint32_t)std::atoi(body.c_str() + colon + 1);
        };
        knob("walk_blocks_per_sm", &v.walk_blocks_per_sm);
        knob("walk_max_log2", &v.walk_max_log2);
        knob("jump_block_log2", &v.jump_block_log2);
        knob("tile_max_log2", &v.tile_max_log2);
        if (cls >= 0 && cls < 64) {
            t.has[cls] = true;
            t.at[cls] = clamp_tuning(v);
        }
        at = end;
    }
    return t;
}

std::mutex g_tuning_mutex;
bool g_tuning_forced = false;
Tuning g_tuning_force{};

uint32_t size_class(uint64_t n) {
    uint32_t c = 0;
    while (c < 63 && (1ull << c) < n) ++c;
    return c;
}

Tuning tuning_for(uint64_t count) {
    static const TuningTable table = load_tuning_table();
    {
        std::lock_guard<std::mutex> lock(g_tuning_mutex);
        if (g_tuning_forced) return g_tuning_force;
    }
    const int c = (int)size_class(count);
    for (int d = 0; d < 64; ++d) {
        if (c - d >= 0 && table.has[c - d]) return table.at[c - d];
        if (c + d < 64 && table.has[c + d]) return table.at[c + d];
    }
    return default_tuning();
}

int grid_for(uint64_t work, int threads) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t want = (work + threads - 1) / threads;
    const uint64_t cap = (uint64_t)sms * 16;
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(want, cap));
}

// Optional per-kernel timing: when enabled, every launch is bracketed by a
// pair of events and the per-kind totals are reported after the call.
struct Recorder {
    bool enabled = false;
    std::vector<cudaEvent_t>* pool = nullptr;
    struct Mark {
        int kind;
        int level;
        size_t first; // index of the opening event
    };
    std::vector<Mark> marks;
    uint32_t launches = 0;
    int level = -1; // routing level of the launches being recorded
    cudaStream_t st = nullptr;
    size_t used = 0;

    cudaEvent_t next() {
        if (used == pool->size()) {
            cudaEvent_t e;
            check(cudaEventCreate(&e), "cudaEventCreate");
            pool->push_back(e);
        }
        return (*pool)[used++];
    }
    // `kernels`: kernel launches f makes (counted in `launches`)
    template <typename F>
    void launch(int kind, F&& f, uint32_t kernels = 1) {
        launches += kernels;
        if (!enabled) {
            f();
            return;
        }
        const size_t i = used;
        check(cudaEventRecord(next(), st), "cudaEventRecord");
        f();
        check(cudaEventRecord(next(), st), "cudaEventRecord");
        marks.push_back({kind, level, i});
    }
    void collect(double* seconds, uint32_t* counts, std::vector<Mark>* per_launch,
        std::vector<double>* per_launch_seconds) {
        per_launch->clear();
        per_launch_seconds->clear();
        for (auto& m : marks) {
            float ms = 0;
            check(cudaEventElapsedTime(&ms, (*pool)[m.first], (*pool)[m.first + 1]),
                "cudaEventElapsedTime");
            seconds[m.kind] += ms * 1e-3;
            counts[m.kind] += 1;
            per_launch->push_back(m);
            per_launch_seconds->push_back(ms * 1e-3);
        }
    }
};

// The emission launches of one section at one level, in launch order:
// f(form, full, blocks) per launch.  Packet runs of at least 32 switches
// are copied word-wise; shorter runs go out as whole words where every node
// fills the packet (transposed across 32 nodes when a cluster root holds at
// least 32 nodes, else gathered per word), and the tail packets bit by bit
// (`full` is the number of full packets, the first packet of the per-bit
// form).
// The block forms assemble words across the nodes of a cluster root, so a
// sharded level uses them only when its nodes hold whole roots.
template <typename F>
void emission_launches(const Plan& p, uint32_t l, int side, F&& f) {
    const LevelInfo& lv = p.levels[l];
    const LevelSide& ls = lv.side[side];
    const NodeRange nr = level_nodes(p, l);
    const uint32_t span_log2 = p.groups[side][ls.group].depth - ls.rel - 1;
    const uint64_t packets = (lv.cap / 2 + (1ull << span_log2) - 1) >> span_log2;
    if (span_log2 >= 5) {
        f((int)kEmitWords, 0ull, grid_for(packets << (nr.shift + span_log2 - 5), kLevelThreads));
        return;
    }
    const uint64_t half_min = lv.q / 2;
    const uint32_t rel = ls.rel;
    const uint64_t full = half_min >= 1 && nr.shift >= rel ? (half_min - 1) >> span_log2 : 0;
    const uint32_t per_word_log2 = std::min<uint32_t>(5 - span_log2, rel);
    if (full > 0 && rel >= 5) {
        const uint64_t windows = (full + (32 >> span_log2) - 1) >> (5 - span_log2);
        const uint64_t threads = (windows << (nr.shift - 5)) * 32;
        f((int)kEmitTranspose, full, grid_for(threads, kLevelThreads));
    } else if (full > 0) {
        const uint64_t words = (full << (rel - per_word_log2)) << (nr.shift - rel);
        f((int)kEmitBlocks, full, grid_for(words, kLevelThreads));
    }
    f((int)kEmitBits, full,
        grid_for((packets - std::min(packets, full)) << (nr.shift + span_log2), kLevelThreads));
}

// Level 0's input still arriving from the host in parts: after wait(k) the
// stream has waited for part k, and entries [0, ends[k]) are on the device.
struct InputParts {
    std::vector<uint64_t> ends;
    std::function<void(uint32_t part)> wait;
};

// How the elements of one walk level's nodes are ranked: lists 1..top are
// built, list `top` by list_rank with `threads` and `smem`.
struct RankShape {
    uint32_t top;
    uint32_t threads;
    uint32_t smem;
};

RankShape rank_shape(const LevelInfo& lv, const Tuning& tune) {
    const uint32_t limit = 1u << std::min(kRankMaxLog2, std::max(kRankMinLog2, tune.jump_block_log2));
    RankShape r{1, 0, 0};
    while (r.top < kMaxLists && list_node_max(lv.pcap, r.top) > limit) ++r.top;
    const uint32_t count = list_node_max(lv.pcap, r.top);
    r.threads = rank_threads(count);
    r.smem = rank_smem(count);
    return r;
}

// Whether a level is coloured by walks (else by union-find).
bool walk_level(const LevelInfo& lv, const Tuning& tune, bool union_find_only) {
    return lv.cap <= (1ull << tune.walk_max_log2) && !union_find_only;
}

int device_sms() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

void allow_smem(const void* kernel);

// One global routing level: level 0 builds its inverse; then the colouring
// (walks, or union-find for nodes above L2 size), and the output pass, which
// writes the children; then both sections' switch bits.  `inv` holds this
// level's inverse; `child_inv` receives the next level's.
template <typename T>
void run_level(Workspace& w, Recorder& rec, cudaStream_t st, const Plan& p, const Tuning& tune,
    uint32_t l, const T* src, uint32_t* d_blob, uint32_t* inv, uint32_t* child_inv,
    bool union_find_only, const InputParts* input = nullptr) {
    const Plan* dp = w.d_plan;
    const LevelInfo& lv = p.levels[l];
    const NodeRange nr = level_nodes(p, l);
    const uint64_t prs = lv.pcap << nr.shift; // this call's pair-nodes
    const uint64_t pair_lo = nr.lo * lv.pcap;
    const uint64_t nodes = 1ull << nr.shift;
    const int gp = grid_for(prs, kLevelThreads);
    uint32_t* ctl = w.control + l * kCtlWords;
    const Chains chains = level_chains(ctl, w.ybits, (uint32_t)(prs / 64));
    const bool walks = walk_level(lv, tune, union_find_only);
    if (l == 0 && lv.cap > kWalkMaxNode && w.records != nullptr) {
        const uint64_t slots = lv.cap;
        const uint32_t windows = (uint32_t)((slots + (1ull << kPlaceLog2) - 1) >> kPlaceLog2);
        check(cudaMemsetAsync(w.cursor, 0, windows * 4, st), "cudaMemsetAsync(cursors)");
        auto bucket = [&](uint64_t lo, uint64_t hi) {
            const int gb = grid_for((hi - lo + kBucketItems - 1) / kBucketItems, kBucketThreads);
            level_bucket<T><<<gb, kBucketThreads, 0, st>>>(dp, src, w.records, w.cursor, w.edge,
                w.d_status, lo, hi);
        };
        const uint32_t parts = input != nullptr ? (uint32_t)input->ends.size() : 0;
        rec.launch(kKindPlace, [&] {
            if (parts == 0) {
                bucket(0, slots);
            } else {
                // each part is bucketed as soon as it is on the device, while
                // the later parts are still being uploaded
                uint64_t lo = 0;
                for (uint32_t k = 0; k < parts; ++k) {
                    input->wait(k);
                    const uint64_t hi = std::min<uint64_t>(input->ends[k], slots);
                    if (hi > lo) bucket(lo, hi);
                    lo = std::max(lo, hi);
                }
            }
            level_place<<<grid_for(slots, kLevelThreads), kLevelThreads, 0, st>>>(dp, l,
                w.records, w.cursor, inv, ctl + kCtlClaimPlace);
        }, parts == 0 ? 2 : parts + 1);
    } else if (l == 0) {
        rec.launch(kKindInverse, [&] {
            launch_next(level_inverse<T>,
                grid_for((lv.cap + kInverseItems - 1) / kInverseItems, kLevelThreads), kLevelThreads,
                0, st, dp, src, inv, walks ? nullptr : w.edge, ctl + kCtlClaimInverse, w.d_status);
        });
    }
    if (walks) {
        const RankShape shape = rank_shape(lv, tune);
        const ListRange rr = list_range(pair_lo, pair_lo + prs, 1);
        if (l == 0) {
            rec.launch(kKindInverse, [&] {
                launch_next(level_edges, gp, kLevelThreads, 0, st, dp, inv, w.edge, w.stamp,
                    w.d_status);
            });
        }
        rec.launch(kKindWalk, [&] {
            launch_next(level_walk, (rr.hi - rr.lo + kLevelThreads - 1) / kLevelThreads,
                kLevelThreads, 0, st, dp, l, w.edge, w.stamp, w.lists.state[1], w.lists.mark[1],
                w.d_status);
        });
        rec.launch(kKindJump, [&] {
            for (uint32_t e = 1; e < shape.top; ++e) {
                const ListRange to = list_range(pair_lo, pair_lo + prs, e + 1);
                launch_next(list_contract, grid_for(2ull * (to.hi - to.lo), kLevelThreads),
                    kLevelThreads, 0, st, dp, l, e, w.lists.state[e], w.lists.mark[e],
                    w.lists.state[e + 1], w.lists.mark[e + 1], w.d_status);
            }
            allow_smem((const void*)list_rank);
            launch_next(list_rank, std::min<uint64_t>(nodes, 1u << 20), shape.threads, shape.smem, st,
                dp, l, shape.top, w.lists.state[shape.top], w.lists.colour[shape.top], w.d_status);
            for (uint32_t e = shape.top; e-- > 1;) {
                const ListRange to = list_range(pair_lo, pair_lo + prs, e);
                launch_next(list_expand, grid_for(to.hi - to.lo, kLevelThreads), kLevelThreads, 0, st,
                    dp, l, e, w.lists.state[e], w.lists.mark[e], w.lists.colour[e + 1],
                    w.lists.colour[e], w.d_status);
            }
        }, 2 * shape.top - 1);
        rec.launch(kKindResolve, [&] {
            launch_next(level_colours, gp, kLevelThreads, 0, st, dp, l, w.edge, w.stamp,
                w.lists.colour[1], w.xbits, w.d_status);
        });
    } else {
        const bool by_windows = lv.cap > kSwapMaxNode && w.records != nullptr;
        if (by_windows) {
            const uint32_t low = (uint32_t)(pair_lo >> kUnionWindowLog2);
            const uint32_t high = (uint32_t)((pair_lo + prs - 1) >> kUnionWindowLog2);
            check(cudaMemsetAsync(w.cursor, 0, kUnionWindows * 4, st), "cudaMemsetAsync(cursors)");
            rec.launch(kKindUnion, [&] {
                launch_next(union_bucket, grid_for(prs / kUnionBucketItems, kLevelThreads),
                    kLevelThreads, 0, st, dp, l, inv, w.edge, w.records, w.cursor, w.slot_cap, chains,
                    w.d_status);
                for (uint32_t v = high + 1; v-- > low;) {
                    launch_next(union_window, device_sms() * 6, kLevelThreads, 0, st, v, w.edge,
                        w.records, w.cursor, w.slot_cap, chains, w.d_status);
                }
            }, 2 + high - low);
        }
        if (!by_windows) rec.launch(kKindUnion, [&] {
            launch_next(level_union, grid_for((prs + kUnionItems - 1) / kUnionItems, kLevelThreads),
                kLevelThreads, 0, st, dp, l, inv, w.edge, chains, w.d_status);
        });
        rec.launch(kKindOrient, [&] {
            launch_next(level_orient, grid_for(nodes, kLevelThreads), kLevelThreads, 0, st, dp, l, inv,
                w.edge, chains, w.d_status);
        });
        rec.launch(kKindResolve, [&] {
            launch_next(level_roots, grid_for((prs + kResolveItems - 1) / kResolveItems, kLevelThreads),
                kLevelThreads, 0, st, dp, l, w.edge, w.xbits, chains);
            launch_with(cudaLaunchAttributeCooperative, level_settle, device_sms(), kSettleThreads,
                0, st, dp, l, inv, w.edge, w.xbits, chains, w.d_status);
        }, 2);
    }
    rec.launch(kKindOutputBits, [&] {
        // the colours are all in xbits: the child level's edges or union-find
        // words take the place of this level's; tiles and stages build their own
        const bool global_child = l + 1 < p.tile_level &&
            (union_find_only || stage_stop(p, l + 1, p.tile_level) == 0);
        const bool child_walks = global_child && walk_level(p.levels[l + 1], tune, union_find_only);
        launch_next(level_outputs, (prs / 2 + 32 + kLevelThreads - 1) / kLevelThreads, kLevelThreads, 0, st, dp, l, inv,
            w.xbits, w.ybits, child_inv, child_walks ? w.edge : nullptr, w.stamp,
            global_child && !child_walks ? w.edge : nullptr);
    });
    // above the shard level every shard computes the level, shard 0 alone
    // writes its switches
    const bool emit = p.shards <= 1 || l >= p.shard_level || p.shard == 0;
    if (emit) {
        EmitParts parts{};
        for (int side = 0; side < 2; ++side) {
            emission_launches(p, l, side, [&](int form, uint64_t full, int blocks) {
                parts.part[parts.count++] = EmitPart{form, side, parts.blocks, (uint32_t)blocks, full};
                parts.blocks += (uint32_t)blocks;
            });
        }
        rec.launch(kKindEmit, [&] {
            launch_next(level_emit, parts.blocks, kLevelThreads, 0, st, dp, l, parts, w.xbits,
                w.ybits, w.addr[0] + (1ull << l), w.addr[1] + (1ull << l), d_blob);
        });
    }
    check(cudaGetLastError(), "level kernel launch");
}

// Raises a kernel's dynamic shared memory limit to the whole shared-memory
// budget, once per kernel and device.  Setting it per call to the call's own
// size raced between concurrent callers: the limit is per function, and a
// caller that lowered it between another caller's set and launch made that
// launch fail ("too many resources requested").  The limit only bounds what
// a launch may ask for; occupancy follows each launch's actual request.
void allow_smem(const void* kernel) {
    static std::mutex m;
    static std::vector<std::pair<const void*, int>> done;
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    std::lock_guard<std::mutex> lock(m);
    for (const auto& d : done) {
        if (d.first == kernel && d.second == dev) return;
    }
    check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
              (int)kTileSmemBudget),
        "cudaFuncSetAttribute");
    done.emplace_back(kernel, dev);
}

// Called after the launches of each global level are enqueued.
using LevelHook = std::function<void(uint32_t level)>;

// The tile launch split into parts at ascending tile indices (`cuts`, the
// last one the tile count), with a hook after each part's launch.
struct TileParts {
    std::vector<uint64_t> cuts;
    std::function<void(uint32_t part)> after_part;
};

template <typename T>
void launch_levels(Workspace& w, Recorder& rec, cudaStream_t st, const Plan& p,
    const TileShape& shape, const Tuning& tune, const Header& header, const T* d_in,
    uint32_t* d_blob, uint32_t* status_out, bool union_find_only, const LevelHook* after_level = nullptr,
    const TileParts* parts = nullptr, const InputParts* input = nullptr) {
    const Plan* dp = w.d_plan;
    const uint32_t t0 = p.tile_level;
    const uint64_t blob_words = (p.end_offset + 3) / 4;
    // level 0 reads the input at once unless it is bucketed part by part
    const bool by_parts = t0 > 0 && p.levels[0].cap > kWalkMaxNode && w.records != nullptr;
    for (uint32_t k = 0; input != nullptr && !by_parts && k < (uint32_t)input->ends.size(); ++k) {
        input->wait(k);
    }
    if (single_launch(p)) {
        rec.level = 0;
        rec.launch(kKindTile, [&] {
            const std::unique_ptr<TileSingle> one(new TileSingle); // not cleared: set at once
            one->plan = p;
            one->header = header;
            allow_smem((const void*)tile_encode_single<T>);
            const uint32_t plan_at = (shape.smem + 15) / 16 * 16;
            const bool near = plan_at + sizeof(Plan) <= kTileSmemBudget;
            tile_encode_single<T><<<1, stage_threads(p.n),
                near ? plan_at + sizeof(Plan) : shape.smem, st>>>(*one, d_in, d_blob,
                (uint32_t)blob_words, status_out, shape.slots, near ? plan_at : 0u);
        });
        check(cudaGetLastError(), "tile kernel launch");
        return;
    }
    rec.launch(kKindPrologue, [&] {
        const std::unique_ptr<Prologue> first(new Prologue); // not cleared: set at once
        first->plan = p;
        first->header = header;
        // (a stage from level 0 checks its input itself)
        const bool scatter = t0 > 0 && (union_find_only || stage_stop(p, 0, t0) == 0);
        const uint64_t inv_words = scatter ? p.levels[0].cap : 0;
        prologue<<<grid_for((blob_words + inv_words) / 8, 256), 256, 0, st>>>(*first, w.d_plan,
            w.d_status, d_blob, blob_words, w.control, t0 * kCtlWords, w.inv[0], inv_words,
            w.addr[0], w.addr[1]);
    });
    // inv[cur] holds the inverse of the level reached, from level 1 on
    uint32_t cur = 0;
    auto stage = [&](uint32_t l, uint32_t stop) {
        rec.level = (int)l;
        const TileShape part = tile_shape(p, l, stop);
        const uint64_t nodes = 1ull << level_nodes(p, l).shift;
        if ((2 * p.levels[stop].pcap) << stop > p.max_slots) { // see size_levels
            throw CudaFail{cudaErrorInvalidValue, "level scratch"};
        }
        const unsigned threads = stage_threads(p.levels[l].cap);
        rec.launch(kKindTile, [&] {
            if (l == 0) {
                allow_smem((const void*)tile_encode_wide<T>);
                launch_next(tile_encode_wide<T>, nodes, threads, part.smem, st, dp, d_in, d_blob,
                    w.d_status, part.slots, 0u, l, stop, w.inv[cur ^ 1]);
            } else {
                allow_smem((const void*)tile_encode_wide<uint32_t>);
                launch_next(tile_encode_wide<uint32_t>, nodes, threads, part.smem, st, dp,
                    w.inv[cur], d_blob, w.d_status, part.slots, 0u, l, stop, w.inv[cur ^ 1]);
            }
        });
        cur ^= 1;
    };
    for (uint32_t l = 0; l < t0;) {
        const uint32_t stop = union_find_only ? 0 : stage_stop(p, l, t0);
        if (stop != 0) {
            stage(l, stop);
        } else {
            rec.level = (int)l;
            run_level<T>(w, rec, st, p, tune, l, d_in, d_blob, w.inv[cur], w.inv[cur ^ 1],
                union_find_only, by_parts ? input : nullptr);
            cur ^= 1;
        }
        const uint32_t next = stop != 0 ? stop : l + 1;
        for (; l < next; ++l) {
            if (after_level != nullptr) {
                (*after_level)(l);
            }
        }
    }
    uint32_t last = t0;
    TileShape last_shape = shape;
    while (const uint32_t stop = few_tiles_stop(p, last)) {
        stage(last, stop);
        last = stop;
        last_shape = tile_shape(p, last);
    }
    rec.level = (int)last;
    const uint64_t tiles = 1ull << level_nodes(p, last).shift;
    if (tiles > 0x7fffffffull) {
        throw CudaFail{cudaErrorInvalidValue, "too many tiles"};
    }
    const bool wide = last_shape.smem > kTileSmemTwoPerSm;
    const unsigned threads = tile_threads(tiles, wide, p.levels[last].cap);
    auto kernel = wide ? tile_encode_wide<uint32_t> : tile_encode<uint32_t>;
    allow_smem((const void*)kernel);
    uint64_t lo = 0;
    const size_t count = parts != nullptr ? parts->cuts.size() : 1;
    for (size_t k = 0; k < count; ++k) {
        const uint64_t hi = parts != nullptr ? parts->cuts[k] : tiles;
        if (hi > lo) {
            rec.launch(kKindTile, [&] {
                launch_next(kernel, hi - lo, threads, last_shape.smem, st, dp, w.inv[cur], d_blob,
                    w.d_status, last_shape.slots, (uint32_t)lo, last, p.depth, nullptr);
            });
        }
        if (parts != nullptr && parts->after_part) {
            parts->after_part((uint32_t)k);
        }
        lo = hi;
    }
    check(cudaMemcpyAsync(status_out, w.d_status, 4, cudaMemcpyDefault, st), "status");
    check(cudaGetLastError(), "tile kernel launch");
}

struct Call {
    Layout layout;
    Plan* plan = nullptr;
    TileShape shape{};
    Tuning tune{};
};

void set_error(char* err, size_t len, const std::string& msg) {
    if (err != nullptr && len > 0) {
        std::snprintf(err, len, "%s", msg.c_str());
    }
}

Format to_format(const bpb200_format* f) {
    Format out;
    if (f == nullptr) {
        return out;
    }
    out.middle_group_log2 = f->middle_group_log2;
    out.middle_placement = f->middle_placement;
    out.input_cluster_count = f->input_cluster_count;
    out.output_cluster_count = f->output_cluster_count;
    std::memcpy(out.input_clusters, f->input_clusters, 64);
    std::memcpy(out.output_clusters, f->output_clusters, 64);
    return out;
}

// Device buffers must be aligned to the width the kernels access them with
// (4-byte blob words, entry-width input values); a misaligned pointer would
// fault on the device, so it is rejected here.
int check_device_buffers(const void* d_entries, uint32_t entry_bytes, const void* d_blob,
    char* err, size_t err_len) {
    if (((uintptr_t)d_blob & 3u) != 0) {
        set_error(err, err_len, "device blob must be 4-byte aligned");
        return kInvalidArgument;
    }
    if ((entry_bytes == 4 || entry_bytes == 8) &&
        ((uintptr_t)d_entries & (uintptr_t)(entry_bytes - 1)) != 0) {
        set_error(err, err_len, "device input must be aligned to its entry width");
        return kInvalidArgument;
    }
    return kOk;
}

// Validation shared by both entry points; fills the layout and plan.
// `tune` (null: the table's setting for `count`) fixes the tile size.
int prepare(uint64_t count, uint32_t entry_bytes, const bpb200_format* format,
    uint64_t blob_len, Workspace& w, Call* call, char* err, size_t err_len,
    const Tuning* tune = nullptr) {
    if (entry_bytes != 4 && entry_bytes != 8) {
        set_error(err, err_len, "entry width must be 4 or 8 bytes");
        return kInvalidArgument;
    }
    if (count == 0) {
        set_error(err, err_len, "permutation size is out of range");
        return kInvalidArgument;
    }
    if (entry_bytes == 4 && count > 0xffffffffull) {
        set_error(err, err_len, "permutation size requires 64-bit source values");
        return kInvalidArgument;
    }
    Error e = make_layout(count, to_format(format), &call->layout);
    if (!e.ok()) {
        set_error(err, err_len, e.message);
        return e.code;
    }
    if (count > (1ull << 31)) {
        set_error(err, err_len, "the b200 backend handles at most 2^31 entries");
        return kLength;
    }
    if (blob_len != call->layout.end_offset) {
        set_error(err, err_len, "blob length does not match the encoded size");
        return kLength;
    }
    call->plan = w.h_plan;
    call->tune = tune != nullptr ? *tune : tuning_for(count);
    const uint64_t tile_max = 1ull << call->tune.tile_max_log2;
    e = make_plan(call->layout, tile_max, call->plan);
    if (!e.ok()) {
        set_error(err, err_len, e.message);
        return e.code;
    }
    choose_tile(*call->plan, &call->shape, tile_max);
    if (call->shape.smem > kTileSmemBudget) {
        set_error(err, err_len, "tile does not fit in shared memory");
        return kLength;
    }
    return kOk;
}

// Per-thread record of the last call (the reference keeps device seconds
// thread_local too, src/benes.cpp:24).
thread_local double t_kernel_seconds[kKernelKinds];
thread_local uint32_t t_kernel_counts[kKernelKinds];
thread_local uint32_t t_launches = 0;
thread_local std::vector<Recorder::Mark> t_marks;
thread_local std::vector<double> t_mark_seconds;
std::atomic<int> g_profiling{0};

// Whether a permutation has to be encoded again with union-find: a walk gave
// up, and not because the input is no permutation.
bool gave_up(uint32_t status) {
    return (status & kErrGaveUp) != 0 && (status & kErrNotPermutation) == 0;
}

// Return code of a finished encode's status word.
int status_code(uint32_t status, char* err, size_t err_len) {
    if (status & (kErrNotPermutation | kErrBelow)) {
        set_error(err, err_len, "input must contain every value from zero through size minus one");
        return kInvalidArgument;
    }
    if (status & (kErrIterationCap | kErrInconsistent | kErrGaveUp)) {
        set_error(err, err_len, "b200 device status reported a failed colouring");
        return kRuntime;
    }
    return kOk;
}

// Queues the whole encode on `st` and waits for it.  When a walk gave up
// (contrived inputs only), or the test hook asks for it, the permutation is
// encoded a second time with union-find on every level; `again` (may be
// null) then says so: what the hooks handed out earlier is stale.
int run(Workspace& w, Call& call, cudaStream_t st, const void* d_in, uint32_t entry_bytes,
    uint32_t* d_blob, double* device_seconds, char* err, size_t err_len,
    const LevelHook* after_level = nullptr, const TileParts* parts = nullptr,
    const InputParts* input = nullptr, bool* again = nullptr) {
    const Plan& p = *call.plan;
    ensure_scratch(w, p);
    Recorder rec;
    rec.enabled = g_profiling.load() != 0;
    rec.pool = &w.events;
    rec.st = st;
    Header h{};
    // of the shards of one permutation only shard 0 writes the header
    h.bytes = p.shards > 1 && p.shard != 0 ? 0u : (uint32_t)call.layout.header_bytes;
    write_header(call.layout, h.data);
    check(cudaEventRecord(w.start, st), "cudaEventRecord");
    const int colouring = g_force_union_find.load();
    bool union_find_only = colouring == 1;
    uint32_t status = 0;
    for (int pass = 0; pass < 2; ++pass) {
        if (entry_bytes == 4) {
            launch_levels<uint32_t>(w, rec, st, p, call.shape, call.tune, h, (const uint32_t*)d_in,
                d_blob, w.h_status, union_find_only, after_level, parts, input);
        } else {
            launch_levels<uint64_t>(w, rec, st, p, call.shape, call.tune, h, (const uint64_t*)d_in,
                d_blob, w.h_status, union_find_only, after_level, parts, input);
        }
        check(cudaEventRecord(w.stop, st), "cudaEventRecord");
        check(cudaStreamSynchronize(st), "cudaStreamSynchronize");
        status = *w.h_status;
        if (union_find_only || p.tile_level == 0 || (!gave_up(status) && colouring != 2)) {
            break;
        }
        union_find_only = true;
        after_level = nullptr;
        parts = nullptr;
        input = nullptr; // all of it is on the device by now
        if (again != nullptr) *again = true;
    }
    float ms = 0;
    check(cudaEventElapsedTime(&ms, w.start, w.stop), "cudaEventElapsedTime");
    if (device_seconds) {
        *device_seconds = ms * 1e-3;
    }
    for (int k = 0; k < kKernelKinds; ++k) {
        t_kernel_seconds[k] = 0;
        t_kernel_counts[k] = 0;
    }
    rec.collect(t_kernel_seconds, t_kernel_counts, &t_marks, &t_mark_seconds);
    t_launches = rec.launches;
    return status_code(status, err, err_len);
}

// Whether the current device is an sm_100 part, cached per device: the
// check runs on every call, and a full cudaGetDeviceProperties costs
// milliseconds.
int current_device_ok(int* device) {
    static std::atomic<int> known[64]; // 0 unknown, 1 usable, 2 not usable
    if (cudaGetDevice(device) != cudaSuccess || *device < 0) {
        return 0;
    }
    if (*device < 64) {
        const int k = known[*device].load();
        if (k != 0) return k == 1 ? 1 : 0;
    }
    int major = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, *device) != cudaSuccess) {
        return 0;
    }
    const int ok = major == 10 ? 1 : 0;
    if (*device < 64) known[*device].store(ok ? 1 : 2);
    return ok;
}

template <typename Fn>
int guarded(char* err, size_t err_len, Fn&& fn) {
    try {
        return fn();
    } catch (const CudaFail& f) {
        set_error(err, err_len, std::string(f.what) + ": " + cudaGetErrorString(f.err));
        return kRuntime;
    } catch (const std::bad_alloc&) {
        set_error(err, err_len, "host allocation failed");
        return kRuntime;
    }
}

// Device staging of the host-path input and blob (grow-only).
void ensure_staging(Workspace& w, uint64_t in_bytes, uint64_t blob_len) {
    // grows at least twofold, like ensure_scratch
    if (in_bytes > w.input_cap) {
        const uint64_t cap = std::max(in_bytes, 2 * w.input_cap);
        if (w.input) cudaFree(w.input);
        w.input = nullptr;
        w.input_cap = 0;
        check(cudaMalloc(&w.input, cap), "cudaMalloc(input)");
        w.input_cap = cap;
    }
    const uint64_t blob_bytes = ((blob_len + 3) / 4 + 1) * 4;
    if (blob_bytes > w.blob_cap) {
        const uint64_t cap = std::max(blob_bytes, 2 * w.blob_cap);
        if (w.blob) cudaFree(w.blob);
        w.blob = nullptr;
        w.blob_cap = 0;
        check(cudaMalloc(&w.blob, cap), "cudaMalloc(blob)");
        w.blob_cap = cap;
    }
}

} // namespace
} // namespace bpb200

// Pinned staging rings for host copies and files.
#include "staging.inc"

namespace bpb200 {
namespace {

// Pieces of the blob that are final before the last launch, so the host
// path downloads them while the remaining work runs.  A section lists, per
// cluster group in order, each cluster's packets followed by the sections of
// its child clusters (cluster_base), so:
//  - after the last level of the first groups (the header and, per section,
//    the level-0 cluster's packets: `level`, `first[]`), when both sections
//    have more groups and those levels are all global;
//  - when the last group of both sections starts at or above the tile level,
//    after each of kTileParts tile launches: every byte before the first
//    last-group cluster whose tiles have not run yet (`cuts`, `upto[k][]`).
// The byte holding a piece's last bit may be shared with the next piece, so
// pieces end at the byte below it.
constexpr uint32_t kTileParts = 8;

struct EarlyPlan {
    bool levels = false;
    uint32_t level = 0;
    uint64_t first[2] = {0, 0};          // end of the first-group piece, per section
    std::vector<uint64_t> cuts;          // tile part ends (empty: one launch)
    std::vector<std::array<uint64_t, 2>> upto; // per part, per section: bytes final after it
};

EarlyPlan early_plan(const Plan& p) {
    EarlyPlan e;
    if (p.shards > 1 || p.tile_level == 0) {
        return e;
    }
    uint32_t last = 0;
    bool multi = true;
    for (int side = 0; side < 2; ++side) {
        if (p.group_count[side] < 2) {
            multi = false;
            break;
        }
        const GroupInfo& g = p.groups[side][0];
        last = std::max(last, g.start + g.depth - 1);
    }
    if (multi && last + 1 < p.tile_level) {
        // the single node of level 0 is small (r_0 = 0): its packets take
        // group_bits[0]
        e.levels = true;
        e.level = last;
        e.first[0] = p.section_offset[0] + p.groups[0][0].group_bits[0] / 8;
        e.first[1] = p.section_offset[1] + p.groups[1][0].group_bits[0] / 8;
    }
    uint32_t s_min = p.tile_level;
    uint32_t glast[2], slast[2];
    for (int side = 0; side < 2; ++side) {
        glast[side] = p.group_count[side] - 1;
        slast[side] = p.groups[side][glast[side]].start;
        s_min = std::min(s_min, slast[side]);
    }
    if (slast[0] > p.tile_level || slast[1] > p.tile_level || s_min == 0) {
        return e;
    }
    const uint64_t tiles = 1ull << p.tile_level;
    const uint64_t span = 1ull << (p.tile_level - s_min); // tiles per coarsest root
    if (tiles < (uint64_t)kTileParts * span || tiles < (uint64_t)kTileParts * 2048) {
        return e;
    }
    const uint64_t step = tiles / kTileParts / span * span;
    for (uint32_t k = 0; k + 1 < kTileParts; ++k) {
        const uint64_t cut = step * (k + 1);
        std::array<uint64_t, 2> at{};
        for (int side = 0; side < 2; ++side) {
            const uint64_t root = cut >> (p.tile_level - slast[side]);
            at[side] = p.section_offset[side] +
                cluster_base(p, side, glast[side], slast[side], root) / 8;
        }
        e.cuts.push_back(cut);
        e.upto.push_back(at);
    }
    e.cuts.push_back(tiles);
    return e;
}

// out[i] = (uint32_t)in[i] for i < n; true when some value needs more than
// 32 bits.  With AVX2 the stores bypass the cache (the pinned chunk is read
// next by the copy engine, not by this thread), which saves the read for
// ownership of every destination line.
__attribute__((target("avx2"))) bool narrow_values_avx2(const uint64_t* in, uint32_t* out,
    uint64_t n) {
    uint64_t i = 0;
    __m256i high = _mm256_setzero_si256();
    const __m256i pick = _mm256_setr_epi32(0, 2, 4, 6, 1, 3, 5, 7);
    if (((uintptr_t)out & 31) == 0) {
        for (; i + 8 <= n; i += 8) {
            const __m256i a = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(in + i));
            const __m256i b = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(in + i + 4));
            high = _mm256_or_si256(high, _mm256_or_si256(a, b));
            // low halves of a's four values, then of b's
            const __m256i la = _mm256_permutevar8x32_epi32(a, pick);
            const __m256i lb = _mm256_permutevar8x32_epi32(b, pick);
            _mm256_stream_si256(reinterpret_cast<__m256i*>(out + i),
                _mm256_permute2x128_si256(la, lb, 0x20));
        }
        _mm_sfence();
    }
    alignas(32) uint64_t lanes[4];
    _mm256_store_si256(reinterpret_cast<__m256i*>(lanes), high);
    uint64_t wide = lanes[0] | lanes[1] | lanes[2] | lanes[3];
    for (; i < n; ++i) {
        wide |= in[i];
        out[i] = (uint32_t)in[i];
    }
    return (wide >> 32) != 0;
}

bool narrow_values(const uint64_t* in, uint32_t* out, uint64_t n) {
    static const bool avx2 = __builtin_cpu_supports("avx2") != 0;
    if (avx2) {
        return narrow_values_avx2(in, out, n);
    }
    uint64_t wide = 0;
    for (uint64_t i = 0; i < n; ++i) {
        wide |= in[i];
        out[i] = (uint32_t)in[i];
    }
    return (wide >> 32) != 0;
}

constexpr uint32_t kInputParts = 8; // host-path upload parts (see compress_host)

// Narrowing of 64-bit host inputs before the upload (on unless the
// environment sets BPB200_NARROW_UPLOAD=0), with up to 16 host threads.
bool narrow_upload_enabled() {
    static const bool on = [] {
        const char* v = std::getenv("BPB200_NARROW_UPLOAD");
        return v == nullptr || std::strcmp(v, "0") != 0;
    }();
    return on;
}

int narrow_threads() {
    const unsigned hw = std::thread::hardware_concurrency();
    return (int)std::max(1u, std::min(16u, hw));
}

// Host-memory compress (bpb200_compress): upload, encode, download.
int compress_host(const void* entries, uint64_t count, uint32_t entry_bytes,
    const bpb200_format* format, uint8_t* blob, uint64_t blob_len, double* device_seconds,
    char* err, size_t err_len) {
    int device = 0;
    if (!current_device_ok(&device)) {
        set_error(err, err_len, "b200 backend is unavailable");
        return kUnavailable;
    }
    Lease lease(device);
    Workspace& w = *lease.w;
    Call call;
    int rc = prepare(count, entry_bytes, format, blob_len, w, &call, err, err_len);
    if (rc != kOk) {
        return rc;
    }
    const uint64_t in_bytes = count * entry_bytes;
    ensure_staging(w, in_bytes, blob_len);
    // 64-bit inputs of up to 2^32 entries cross PCIe as 32-bit values: the
    // ring's threads narrow them while the copy engine moves the chunks
    // already done, halving the bytes on the link.  Every valid value is
    // below count <= 2^32; a wider one means the input is not a permutation.
    const bool narrow = entry_bytes == 8 && count <= (1ull << 32) && in_bytes >= kStageMin &&
        narrow_upload_enabled();
    // Other pageable buffers of a few MB and more go through the pinned ring
    // (parallel host copies overlapping the transfer); pinned ones and small
    // ones are copied directly.
    const bool stage_in = !narrow && in_bytes >= kStageMin && !host_is_pinned(entries);
    const bool stage_out = blob_len >= kStageMin && !host_is_pinned(blob);
    std::unique_ptr<RingLease> ring;
    if (narrow || stage_in || stage_out) {
        ring = std::make_unique<RingLease>(device);
    }
    const uint32_t device_width = narrow ? 4u : entry_bytes;
    const uint64_t dev_bytes = count * device_width;
    // Narrowing fill: true when some value needs more than 32 bits.
    std::atomic<uint64_t> wide{0};
    const uint64_t* src64 = static_cast<const uint64_t*>(entries);
    const unsigned char* src8 = static_cast<const unsigned char*>(entries);
    auto fill = [&](unsigned char* dst, uint64_t len, uint64_t off) {
        if (narrow) {
            if (narrow_values(src64 + off / 4, reinterpret_cast<uint32_t*>(dst), len / 4)) {
                wide.fetch_or(1);
            }
        } else {
            std::memcpy(dst, src8 + off, len);
        }
        return true;
    };
    // When level 0 takes the partitioned inverse, the upload runs on the copy
    // stream in kInputParts parts and level 0 buckets each part as soon as it
    // is on the device (the bucket pass streams the input in order), so the
    // transfer overlaps that pass.  Part ends fall on staging-chunk bounds.
    const Plan& plan = *call.plan;
    const bool overlap = plan.shards <= 1 && plan.tile_level > 0 &&
        plan.levels[0].cap > kWalkMaxNode && dev_bytes >= kInputParts * kStageChunk;
    InputParts input;
    std::vector<uint64_t> part_bytes;
    std::mutex um;
    std::condition_variable ucv;
    uint32_t recorded = 0;
    bool upload_failed = false;
    std::thread uploader;
    struct JoinUpload {
        std::thread& t;
        ~JoinUpload() {
            if (t.joinable()) t.join();
        }
    } join_upload{uploader};
    if (overlap) {
        for (uint32_t k = 0; k < kInputParts; ++k) {
            const uint64_t want = dev_bytes / kInputParts * (k + 1);
            const uint64_t at = k + 1 == kInputParts ? dev_bytes
                : std::min(dev_bytes, (want + kStageChunk - 1) / kStageChunk * kStageChunk);
            part_bytes.push_back(at);
            input.ends.push_back(at / device_width);
        }
        if (narrow || stage_in) {
            uploader = std::thread([&] {
                uint32_t next = 0;
                const std::function<void(uint64_t)> on_issue = [&](uint64_t bytes) {
                    while (next < kInputParts && bytes >= part_bytes[next]) {
                        check(cudaEventRecord(w.inparts[next], w.copy_stream), "cudaEventRecord");
                        {
                            std::lock_guard<std::mutex> lock(um);
                            recorded = ++next;
                        }
                        ucv.notify_all();
                    }
                };
                bool ok = false;
                try {
                    ok = upload_staged(fill, dev_bytes, (unsigned char*)w.input, *ring->r,
                        w.copy_stream, narrow ? narrow_threads() : 0, &on_issue);
                } catch (const CudaFail&) {
                    ok = false;
                }
                if (!ok || next < kInputParts) {
                    std::lock_guard<std::mutex> lock(um);
                    upload_failed = true;
                }
                ucv.notify_all();
            });
            input.wait = [&](uint32_t k) {
                {
                    std::unique_lock<std::mutex> lock(um);
                    ucv.wait(lock, [&] { return upload_failed || recorded > k; });
                    if (recorded <= k) {
                        throw CudaFail{cudaErrorUnknown, "input upload"};
                    }
                }
                check(cudaStreamWaitEvent(w.stream, w.inparts[k], 0), "cudaStreamWaitEvent");
                if (k + 1 == kInputParts && uploader.joinable()) {
                    uploader.join(); // every chunk is queued; the ring is free for downloads
                }
            };
        } else {
            uint64_t lo = 0;
            for (uint32_t k = 0; k < kInputParts; ++k) {
                check(cudaMemcpyAsync((unsigned char*)w.input + lo, src8 + lo, part_bytes[k] - lo,
                          cudaMemcpyHostToDevice, w.copy_stream),
                    "input upload");
                check(cudaEventRecord(w.inparts[k], w.copy_stream), "cudaEventRecord");
                lo = part_bytes[k];
            }
            input.wait = [&](uint32_t k) {
                check(cudaStreamWaitEvent(w.stream, w.inparts[k], 0), "cudaStreamWaitEvent");
            };
        }
    } else if (narrow || stage_in) {
        upload_staged(fill, dev_bytes, (unsigned char*)w.input, *ring->r, w.stream,
            narrow ? narrow_threads() : 0);
    } else {
        check(cudaMemcpyAsync(w.input, entries, in_bytes, cudaMemcpyHostToDevice, w.stream),
            "input upload");
    }
    if (!overlap && wide.load() != 0) {
        check(cudaStreamSynchronize(w.stream), "cudaStreamSynchronize");
        set_error(err, err_len, "input must contain every value from zero through size minus one");
        return kInvalidArgument;
    }
    // Bytes [0, end) of the blob are the encoding; the first cluster groups
    // go down on the copy stream (through the ring on a helper thread for a
    // pageable blob) as soon as their last level is done.
    const uint64_t end = std::min<uint64_t>(blob_len, call.plan->end_offset);
    const unsigned char* d_bytes = (const unsigned char*)w.blob;
    auto download = [&](uint64_t off, uint64_t len, cudaStream_t st) {
        if (len == 0) {
            return;
        }
        if (stage_out) {
            if (!download_staged(
                    [blob, off](const unsigned char* src, uint64_t n, uint64_t o) {
                        std::memcpy(blob + off + o, src, n);
                        return true;
                    },
                    len, d_bytes + off, *ring->r, st)) {
                throw CudaFail{cudaErrorUnknown, "staged blob download"};
            }
        } else {
            check(cudaMemcpyAsync(blob + off, d_bytes + off, len, cudaMemcpyDeviceToHost, st),
                "blob download");
        }
    };
    // Early pieces go down on the copy stream after the event that makes
    // them final; a pageable blob goes through the ring on a helper thread,
    // which takes the pieces in order from a queue.
    EarlyPlan early;
    if (end == call.plan->end_offset) {
        early = early_plan(*call.plan);
    }
    uint64_t done[2] = {0, call.plan->section_offset[1]}; // bytes handed out, per section
    struct Piece {
        cudaEvent_t ev;
        uint64_t off, len;
    };
    std::mutex qm;
    std::condition_variable qcv;
    std::vector<Piece> queue;
    bool closed = false;
    std::atomic<int> helper_failed{0};
    std::thread helper;
    struct Join {
        std::thread& t;
        std::mutex& m;
        std::condition_variable& cv;
        bool& closed;
        ~Join() {
            {
                std::lock_guard<std::mutex> lock(m);
                closed = true;
            }
            cv.notify_all();
            if (t.joinable()) t.join();
        }
    } join{helper, qm, qcv, closed};
    if (stage_out && (early.levels || !early.cuts.empty())) {
        helper = std::thread([&] {
            size_t next = 0;
            for (;;) {
                Piece piece{};
                {
                    std::unique_lock<std::mutex> lock(qm);
                    qcv.wait(lock, [&] { return closed || next < queue.size(); });
                    if (next >= queue.size()) return;
                    piece = queue[next++];
                }
                try {
                    check(cudaStreamWaitEvent(w.copy_stream, piece.ev, 0), "cudaStreamWaitEvent");
                    download(piece.off, piece.len, w.copy_stream);
                } catch (const CudaFail&) {
                    helper_failed.store(1);
                    return;
                }
            }
        });
    }
    auto hand_out = [&](cudaEvent_t ev, const uint64_t (&to)[2]) {
        check(cudaEventRecord(ev, w.stream), "cudaEventRecord");
        for (int side = 0; side < 2; ++side) {
            const uint64_t off = side == 0 ? done[0] : done[1];
            if (to[side] <= off) continue;
            if (stage_out) {
                std::lock_guard<std::mutex> lock(qm);
                queue.push_back(Piece{ev, off, to[side] - off});
            } else {
                check(cudaStreamWaitEvent(w.copy_stream, ev, 0), "cudaStreamWaitEvent");
                download(off, to[side] - off, w.copy_stream);
            }
            done[side] = to[side];
        }
        qcv.notify_all();
    };
    const LevelHook level_hook = [&](uint32_t level) {
        if (level == early.level) {
            hand_out(w.early, early.first);
        }
    };
    TileParts parts;
    parts.cuts = early.cuts;
    parts.after_part = [&](uint32_t k) {
        if (k < early.upto.size()) {
            const uint64_t to[2] = {early.upto[k][0], early.upto[k][1]};
            hand_out(w.parts[k], to);
        }
    };
    bool again = false;
    rc = run(w, call, w.stream, w.input, device_width, w.blob, device_seconds, err, err_len,
        early.levels ? &level_hook : nullptr, early.cuts.empty() ? nullptr : &parts,
        overlap ? &input : nullptr, &again);
    if (uploader.joinable()) {
        uploader.join();
    }
    {
        std::lock_guard<std::mutex> lock(qm);
        closed = true;
    }
    qcv.notify_all();
    if (helper.joinable()) {
        helper.join();
    }
    check(cudaStreamSynchronize(w.copy_stream), "cudaStreamSynchronize");
    if (wide.load() != 0) {
        set_error(err, err_len, "input must contain every value from zero through size minus one");
        return kInvalidArgument;
    }
    if (rc != kOk) {
        return rc;
    }
    if (helper_failed.load()) {
        throw CudaFail{cudaErrorUnknown, "staged blob download"};
    }
    if (again) { // the pieces handed out belong to the first attempt
        done[0] = 0;
        done[1] = call.plan->section_offset[1];
    }
    // the rest: the tail of each section and whatever follows the output
    // section (the separate middle section)
    download(done[0], call.plan->section_offset[1] - done[0], w.stream);
    download(done[1], end - done[1], w.stream);
    check(cudaStreamSynchronize(w.stream), "cudaStreamSynchronize");
    return kOk;
}

} // namespace
} // namespace bpb200

using namespace bpb200;

extern "C" {

int bpb200_available(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        return 0;
    }
    int device = 0;
    return current_device_ok(&device);
}

const char* bpb200_backend_name(void) { return "b200"; }

int bpb200_encoded_size(uint64_t count, const bpb200_format* format, uint64_t* blob_bytes,
    char* err, size_t err_len) {
    Layout L;
    const Error e = make_layout(count, to_format(format), &L);
    if (!e.ok()) {
        set_error(err, err_len, e.message);
        return e.code;
    }
    *blob_bytes = L.end_offset;
    return kOk;
}

int bpb200_compress(const void* entries, uint64_t count, uint32_t entry_bytes,
    const bpb200_format* format, uint8_t* blob, uint64_t blob_len, double* device_seconds,
    char* err, size_t err_len) {
    return guarded(err, err_len, [&]() -> int {
        return compress_host(entries, count, entry_bytes, format, blob, blob_len,
            device_seconds, err, err_len);
    });
}

int bpb200_compress_device(const void* d_entries, uint64_t count, uint32_t entry_bytes,
    const bpb200_format* format, uint8_t* d_blob, uint64_t blob_len, void* stream,
    double* device_seconds, char* err, size_t err_len) {
    return guarded(err, err_len, [&]() -> int {
        int device = 0;
        if (!current_device_ok(&device)) {
            set_error(err, err_len, "b200 backend is unavailable");
            return kUnavailable;
        }
        if (const int bad = check_device_buffers(d_entries, entry_bytes, d_blob, err, err_len)) {
            return bad;
        }
        Lease lease(device);
        Workspace& w = *lease.w;
        Call call;
        int rc = prepare(count, entry_bytes, format, blob_len, w, &call, err, err_len);
        if (rc != kOk) {
            return rc;
        }
        // the work is queued on the caller's stream, after its earlier work
        return run(w, call, (cudaStream_t)stream, d_entries, entry_bytes, (uint32_t*)d_blob,
            device_seconds, err, err_len);
    });
}

int bpb200_compress_device_shard(const void* d_entries, uint64_t count, uint32_t entry_bytes,
    const bpb200_format* format, uint8_t* d_blob, uint64_t blob_len, uint32_t shard,
    uint32_t shards, void* stream, double* device_seconds, char* err, size_t err_len) {
    return guarded(err, err_len, [&]() -> int {
        int device = 0;
        if (!current_device_ok(&device)) {
            set_error(err, err_len, "b200 backend is unavailable");
            return kUnavailable;
        }
        if (!valid_shard(shard, shards)) {
            set_error(err, err_len, "shards must be a power of two and shard below it");
            return kInvalidArgument;
        }
        if (const int bad = check_device_buffers(d_entries, entry_bytes, d_blob, err, err_len)) {
            return bad;
        }
        Lease lease(device);
        Workspace& w = *lease.w;
        Call call;
        int rc = prepare(count, entry_bytes, format, blob_len, w, &call, err, err_len);
        if (rc != kOk) {
            return rc;
        }
        if (!set_shard(*call.plan, shard, shards)) {
            set_error(err, err_len, "permutation too small for that many shards");
            return kInvalidArgument;
        }
        return run(w, call, (cudaStream_t)stream, d_entries, entry_bytes, (uint32_t*)d_blob,
            device_seconds, err, err_len);
    });
}

void bpb200_set_profiling(int enabled) { g_profiling.store(enabled ? 1 : 0); }

int bpb200_get_tuning(uint64_t count, bpb200_tuning* out) {
    if (out == nullptr) return kInvalidArgument;
    const Tuning t = tuning_for(count);
    out->walk_blocks_per_sm = t.walk_blocks_per_sm;
    out->walk_max_log2 = t.walk_max_log2;
    out->jump_block_log2 = t.jump_block_log2;
    out->tile_max_log2 = t.tile_max_log2;
    return kOk;
}

int bpb200_set_tuning(const bpb200_tuning* forced) {
    std::lock_guard<std::mutex> lock(g_tuning_mutex);
    g_tuning_forced = forced != nullptr;
    if (forced != nullptr) {
        g_tuning_force = clamp_tuning(Tuning{forced->walk_blocks_per_sm, forced->walk_max_log2,
            forced->jump_block_log2, forced->tile_max_log2});
    }
    return kOk;
}

void bpb200_set_colouring(int union_find_only) {
    g_force_union_find.store(union_find_only == 2 ? 2 : (union_find_only ? 1 : 0));
}

int bpb200_describe(uint64_t count, const bpb200_format* format, uint32_t* depth,
    uint32_t* tile_level) {
    Layout L;
    const Error e = make_layout(count, to_format(format), &L);
    if (!e.ok()) {
        return e.code;
    }
    std::unique_ptr<Plan> p(new Plan);
    const uint64_t tile_max = 1ull << tuning_for(count).tile_max_log2;
    if (!make_plan(L, tile_max, p.get()).ok()) {
        return kLength;
    }
    TileShape shape;
    choose_tile(*p, &shape, tile_max);
    if (depth) *depth = p->depth;
    if (tile_level) *tile_level = p->tile_level;
    return kOk;
}

int bpb200_last_profile_launches(int* kinds, int* levels, double* seconds, int capacity) {
    const int n = (int)t_marks.size();
    for (int i = 0; i < n && i < capacity; ++i) {
        if (kinds) kinds[i] = t_marks[i].kind;
        if (levels) levels[i] = t_marks[i].level;
        if (seconds) seconds[i] = t_mark_seconds[i];
    }
    return n;
}

int bpb200_last_profile(double* seconds, uint32_t* launches, int kinds, uint32_t* total_launches) {
    const int n = kinds < kKernelKinds ? kinds : kKernelKinds;
    for (int k = 0; k < n; ++k) {
        if (seconds) seconds[k] = t_kernel_seconds[k];
        if (launches) launches[k] = t_kernel_counts[k];
    }
    if (total_launches) *total_launches = t_launches;
    return kKernelKinds;
}

void bpb200_shutdown(void) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    for (auto& w : g_pool) {
        if (!w->busy) {
            w->destroy();
        }
    }
    g_pool.erase(std::remove_if(g_pool.begin(), g_pool.end(),
                     [](const std::unique_ptr<Workspace>& w) { return w->device < 0; }),
        g_pool.end());
    destroy_rings();
}

int bpb200_probe_switch_bit(uint64_t count, const bpb200_format* format, int side,
    uint32_t level, uint64_t node, uint64_t pair, uint64_t* bit) {
    Layout L;
    if (!make_layout(count, to_format(format), &L).ok()) {
        return kInvalidArgument;
    }
    std::unique_ptr<Plan> p(new Plan);
    if (!make_plan(L, kTileMaxEntries, p.get()).ok()) {
        return kInvalidArgument;
    }
    if (level >= L.depth || node >= (1ull << level) || (side != 0 && side != 1)) {
        return kInvalidArgument;
    }
    const uint64_t size = node_size(p->levels[level], level, node);
    if (size <= p->leaf || pair >= size / 2) {
        return kInvalidArgument;
    }
    *bit = switch_bit(node_address(*p, side, level, node), pair);
    return kOk;
}

int bpb200_probe_scratch(uint64_t count, const bpb200_format* format, uint32_t shard,
    uint32_t shards, uint32_t* levels, uint32_t capacity, uint64_t* slots) {
    Layout L;
    if (!make_layout(count, to_format(format), &L).ok()) {
        return -kInvalidArgument;
    }
    std::unique_ptr<Plan> p(new Plan);
    const uint64_t tile_max = 1ull << tuning_for(count).tile_max_log2;
    if (!make_plan(L, tile_max, p.get()).ok()) {
        return -kInvalidArgument;
    }
    TileShape shape;
    choose_tile(*p, &shape, tile_max);
    if (!set_shard(*p, shard, shards)) {
        return -kInvalidArgument;
    }
    // as launch_levels
    uint32_t n = 0;
    auto reach = [&](uint32_t l) {
        if (n < capacity) levels[n] = l;
        ++n;
        return l;
    };
    uint32_t l = 0;
    while (l < p->tile_level) {
        const uint32_t stop = stage_stop(*p, l, p->tile_level);
        l = reach(stop != 0 ? stop : l + 1);
    }
    while (const uint32_t stop = few_tiles_stop(*p, l)) {
        l = reach(stop);
    }
    *slots = p->max_slots;
    return n <= capacity ? (int)n : -kLength;
}

int bpb200_probe_rank_bit(uint64_t count, const bpb200_format* format, uint32_t level,
    uint64_t node, int* section, uint64_t* bit) {
    Layout L;
    if (!make_layout(count, to_format(format), &L).ok()) {
        return kInvalidArgument;
    }
    std::unique_ptr<Plan> p(new Plan);
    if (!make_plan(L, kTileMaxEntries, p.get()).ok()) {
        return kInvalidArgument;
    }
    if (level > L.depth || node >= (1ull << level)) {
        return kInvalidArgument;
    }
    if (node_size(p->levels[level], level, node) > p->leaf) {
        return kInvalidArgument;
    }
    *bit = leaf_rank_bit(*p, level, node, section);
    return kOk;
}

} // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free entry point.
//
// Some callers cannot call cudaMalloc: processes whose device memory is
// owned by a pooling allocator that must account for every byte, and
// latency-critical paths that cannot afford the device-wide synchronisation
// cudaMalloc/cudaFree can imply.  For them,
// bpb200_compress_device_noalloc runs the same encode with all of its
// scratch (plan, status word, inverses, edges, stamps, ruler lists, colour
// bits, node descriptors) carved out of one file-scope device array
// of fixed size.  The array exists on every GPU that loads this library and
// stays allocated until the process exits.
// ---------------------------------------------------------------------------
namespace bpb200 {
namespace noalloc {

constexpr uint64_t kMaxEntries = 1ull << 18;          // largest permutation accepted
constexpr uint64_t kSlots = kMaxEntries + (1ull << 14); // level slots incl. padding
constexpr uint64_t kPairs = kSlots / 2 + (1ull << 13);
constexpr uint64_t kNodes = 1ull << 10;               // descriptors per global level

constexpr size_t kOffPlan = 0;
constexpr size_t kOffStatus = kOffPlan + up256(sizeof(Plan));
constexpr size_t kOffControl = kOffStatus + 256;
constexpr size_t kOffInv = kOffControl + up256(kMaxLevels * kCtlWords * 4);
constexpr size_t kOffInv2 = kOffInv + up256(kSlots * 4);
constexpr size_t kOffEdge = kOffInv2 + up256(kSlots * 4);
constexpr size_t kOffStamp = kOffEdge + up256(kSlots * 4);
constexpr size_t kOffXbits = kOffStamp + up256(kPairs * 4);
constexpr size_t kOffYbits = kOffXbits + up256((kPairs / 32 + 4) * 4);
constexpr size_t kOffAddr0 = kOffYbits + up256((kPairs / 32 + 4) * 4);
constexpr size_t kOffAddr1 = kOffAddr0 + up256(kNodes * sizeof(NodeAddress));
constexpr size_t kOffLists = kOffAddr1 + up256(kNodes * sizeof(NodeAddress));
constexpr size_t kBytes = kOffLists + place_lists(kPairs, nullptr, nullptr); // under 8 MB
static_assert(kBytes < (8u << 20), "allocation-free scratch stays under 8 MB");

} // namespace noalloc
} // namespace bpb200

// The scratch itself.  In host code this name is only a host-side stand-in,
// not a device address; the device address is obtained per device with
// cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char bpb200_noalloc_scratch[bpb200::noalloc::kBytes];

namespace bpb200 {
namespace noalloc {

constexpr int kMaxDevices = 64;
std::mutex g_mutex;                    // guards the two tables below
unsigned char* g_scratch[kMaxDevices]; // device address of the array, per device
Plan g_plan;                           // host staging of the plan (no heap, no pinning)

} // namespace noalloc
} // namespace bpb200

extern "C" int bpb200_compress_device_noalloc(const void* d_entries, uint64_t count,
    uint32_t entry_bytes, const bpb200_format* format, uint8_t* d_blob, uint64_t blob_len,
    void* stream, char* err, size_t err_len) {
    using namespace bpb200;
    return guarded(err, err_len, [&]() -> int {
        int device = 0;
        if (!current_device_ok(&device)) {
            set_error(err, err_len, "b200 backend is unavailable");
            return kUnavailable;
        }
        if (device < 0 || device >= noalloc::kMaxDevices) {
            set_error(err, err_len, "device ordinal out of range for the allocation-free entry point");
            return kRuntime;
        }
        if (count > noalloc::kMaxEntries) {
            set_error(err, err_len,
                "the allocation-free entry point accepts at most 262144 (2^18) entries");
            return kLength;
        }
        if (const int bad = check_device_buffers(d_entries, entry_bytes, d_blob, err, err_len)) {
            return bad;
        }
        // One host thread at a time stages the plan; device-side overlap of
        // two calls is the caller's to avoid (they would share the scratch).
        std::lock_guard<std::mutex> lock(noalloc::g_mutex);
        if (noalloc::g_scratch[device] == nullptr) {
            // first call on this device: resolve the array's device address
            // (callers make this first call before capturing any stream)
            void* ptr = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&ptr, bpb200_noalloc_scratch);
            if (e != cudaSuccess || ptr == nullptr) {
                set_error(err, err_len, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
                return kRuntime;
            }
            noalloc::g_scratch[device] = static_cast<unsigned char*>(ptr);
        }
        unsigned char* base = noalloc::g_scratch[device];
        Workspace w; // views into the static array; owns nothing
        w.h_plan = &noalloc::g_plan;
        Call call;
        const Tuning fixed = default_tuning(); // the scratch limits assume the compiled tile size
        int rc = prepare(count, entry_bytes, format, blob_len, w, &call, err, err_len, &fixed);
        if (rc != kOk) {
            return rc;
        }
        const Plan& p = *call.plan;
        const uint64_t nodes = p.tile_level > 0 ? (1ull << p.tile_level) : 0;
        if ((p.tile_level > 0 && (p.max_slots > noalloc::kSlots || p.max_pairs > noalloc::kPairs)) ||
            nodes > noalloc::kNodes) {
            set_error(err, err_len, "format needs more scratch than the allocation-free entry point holds");
            return kLength;
        }
        w.d_plan = reinterpret_cast<Plan*>(base + noalloc::kOffPlan);
        w.d_status = reinterpret_cast<uint32_t*>(base + noalloc::kOffStatus);
        w.control = reinterpret_cast<uint32_t*>(base + noalloc::kOffControl);
        w.inv[0] = reinterpret_cast<uint32_t*>(base + noalloc::kOffInv);
        w.inv[1] = reinterpret_cast<uint32_t*>(base + noalloc::kOffInv2);
        w.edge = reinterpret_cast<uint32_t*>(base + noalloc::kOffEdge);
        w.stamp = reinterpret_cast<uint32_t*>(base + noalloc::kOffStamp);
        w.xbits = reinterpret_cast<uint32_t*>(base + noalloc::kOffXbits);
        w.ybits = reinterpret_cast<uint32_t*>(base + noalloc::kOffYbits);
        w.addr[0] = reinterpret_cast<NodeAddress*>(base + noalloc::kOffAddr0);
        w.addr[1] = reinterpret_cast<NodeAddress*>(base + noalloc::kOffAddr1);
        place_lists(noalloc::kPairs, base + noalloc::kOffLists, &w.lists);
        cudaStream_t st = (cudaStream_t)stream;
        Header h{};
        h.bytes = (uint32_t)call.layout.header_bytes;
        write_header(call.layout, h.data);
        // Everything that must start cleared is cleared by the call's first
        // kernel.  A second pass as in run().
        const int colouring = g_force_union_find.load();
        bool union_find_only = colouring == 1;
        uint32_t status = 0;
        for (int pass = 0; pass < 2; ++pass) {
            Recorder rec; // timing disabled: no events are created
            rec.st = st;
            // one tile leaves its status in device memory, level kernels
            // have it copied there from where they gather it
            uint32_t* status_out = w.d_status + 1;
            if (entry_bytes == 4) {
                launch_levels<uint32_t>(w, rec, st, p, call.shape, call.tune, h,
                    (const uint32_t*)d_entries, (uint32_t*)d_blob, status_out, union_find_only);
            } else {
                launch_levels<uint64_t>(w, rec, st, p, call.shape, call.tune, h,
                    (const uint64_t*)d_entries, (uint32_t*)d_blob, status_out, union_find_only);
            }
            check(cudaMemcpyAsync(&status, status_out, 4, cudaMemcpyDeviceToHost, st), "status");
            check(cudaStreamSynchronize(st), "cudaStreamSynchronize");
            if (union_find_only || p.tile_level == 0 || (!gave_up(status) && colouring != 2)) {
                break;
            }
            union_find_only = true;
        }
        if (const int bad = status_code(status, err, err_len)) {
            return bad;
        }
        return kOk;
    });
}

// Batched and serving forms (share this file's pool, planning and launches).
#include "serve.inc"

// File form: streamed file -> device -> file (compress_file).
#include "file.inc"

// Batch lookup verifier (device twin of the reference's lookup).
#include "lookup.inc"

// Random-access roofline probe.
#include "probe.inc"
