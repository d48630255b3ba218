// Device graph, hierarchy and per-call context shared by the pipeline files.
#pragma once
#include "gp_device.cuh"

#include <atomic>
#include <thread>
#include <vector>

namespace gp {

constexpr int kInvalid = 0x7fffffff;  // SCLP_INVALID (src/coarsen.cu:292)

// A position among a level's entries.  A level holds up to 2^31 - 1 of them and
// a loop over a row's entries steps up to kEntryStep past the row's end, so
// such a loop's index and bounds are unsigned: as int, the last steps of a row
// that ends there would wrap to negative positions and read before the arrays.
using EntryPos = u32;
constexpr u32 kEntryStep = 4096;
static_assert(0x7fffffffu + 2 * kEntryStep < 0xffffffffu, "a step past the last row does not wrap");
// Pieces of `size` entries that a row of `degree` entries is cut into.
__host__ __device__ __forceinline__ int row_pieces(int degree, int size) {
    return static_cast<int>((static_cast<u32>(degree) + static_cast<u32>(size) - 1) / static_cast<u32>(size));
}

// A CSR level on the device (DeviceWeightedGraph, include/graph.hpp:148-171).
// ew == nullptr means unit edge weights.  The three metadata fields follow
// the reference's meaning exactly: maximum_degree is a bound (exact after an
// aggregation pass), incident_bound bounds every row's weight sum.
// Rows longer than kHeavyRow entries are split into chunks of at most
// kChunk entries so that row-parallel kernels give them many blocks instead
// of one serial warp (R-MAT hubs have 10^5 neighbours).
constexpr int kHeavyRow = 2048;
constexpr int kChunk = 2048;

struct DGraph {
    i64 n = 0, m = 0;
    int* off = nullptr;
    int* nbr = nullptr;
    u32* ew = nullptr;
    u32* vw = nullptr;
    bool implicit_unit = false;
    u64 maximum_degree = ~0ULL;
    bool has_heavy_rows = true;
    u64 incident_bound = ~0ULL;
    // Heavy rows (ascending) and their chunks; built by build_chunks().
    int* heavy = nullptr;
    i64 heavy_count = 0;
    int* chunk_row = nullptr;
    int* chunk_hidx = nullptr;  // index of the chunk's row in `heavy`
    int* chunk_begin = nullptr;
    int* heavy_chunk0 = nullptr;  // first chunk of each heavy row (chunks of a row are consecutive)
    i64 chunks = 0;
    i64 heavy_entries = 0;  // CSR entries in heavy rows
    int heavy_min = kHeavyRow;  // rows longer than this are the heavy (chunked) rows
};

// Chunk-parallel loop body helpers: the chunk's edge range.
__host__ __device__ __forceinline__ EntryPos chunk_end(const DGraph& g, int chunk, int row) {
    const EntryPos end = static_cast<EntryPos>(g.chunk_begin[chunk]) + kChunk;
    const EntryPos row_end = g.off[row + 1];
    return end < row_end ? end : row_end;
}

struct Hierarchy {
    std::vector<DGraph> levels;  // level 0 is the input
    std::vector<int*> maps;      // maps[i]: level i -> level i+1
};

// Thread-mapping thresholds.  They decide which kernel and how many threads
// handle a row, never a value: every choice computes the same exact integer
// sums, so results do not depend on them and gp_autotune may set them per
// workload.  The defaults are the fixed values this library was tuned with.
struct Mapping {
    int medium_degree = 256;    // coarsening: rows of 9..this, a warp and a 512-slot shared hash (<= 256)
    int large_narrow = 1024;    // coarsening: large rows up to this use a half-size shared table
    int build_short = 64;       // refinement: cache-build rows up to this, 8 lanes per row
    int rebuild_divisor = 100;  // refinement: rebuild the cache when moved entries exceed (n k size + 8 m) / this
    int on_demand_degree = 32;  // refinement: no cache when the maximum degree is at most this (0: never)
    // Refinement rows above these entry counts go through the block-per-chunk
    // kernels (2048-entry chunks) instead of a warp: on levels of at most
    // 65,536 vertices, at most 2^20 vertices, and larger ones.
    int refine_heavy_small = 256;
    int refine_heavy_mid = 512;
    int refine_heavy_large = 2048;
};

// Coarsening options, app/partition_main.cu:52-87 with no environment overrides.
struct CoarsenOptions {
    int parts = 4;
    u32 seed = 0;
    double stop_ratio = 0.90;
    int max_levels = 24;
    int cluster_size_factor = 256;
    bool pack_isolated = true;
    bool progressive = false;
    int fine_factor = 64, growth = 8;
    bool seed_matching = true, fast_path = true;
    int heavy_limit = 64;
    bool log = true;
    bool verify = false;  // GP_FLAG_VERIFY: strict per-level checks
    Mapping mapping;
};

// Device-resident scalars read back in batches through pinned memory.
constexpr int kScalars = 512;  // >= 2 * kMaxParts + headroom
// Copies `words` scalars into pinned host memory and then `sequence` into the
// word after the pinned scalars (gp_partition.cu).
void publish(cudaStream_t stream, const u64* from, u64* to, int words, u64* flag, u64 sequence);

struct Context {
    int device = 0;
    cudaStream_t stream = nullptr;
    Arena persist;  // hierarchy storage for one call
    Arena scratch;  // stack-disciplined temporaries
    u64* dev_scalars = nullptr;
    u64* host_scalars = nullptr;  // pinned: kScalars words and the number of the last fetch
    u64 fetched = 0;
    // Whether the device has room for the refinement's cluster; asked once per
    // context (-1: not yet).
    int refine_clusters = -1;
    cudaEvent_t ev[8] = {};
    // Kept host copies (GP_FLAG_KEEP_HIERARCHY).
    struct HostLevel {
        i64 n = 0, m = 0;
        std::vector<int> off, nbr, map;
        std::vector<u32> ew, vw;
        u64 meta[4] = {0, 0, 0, 0};
    };
    std::vector<HostLevel> kept;
    std::vector<int> initial_labels;

    // Copies `words` device scalars to host_scalars[at ...] and waits for them:
    // a kernel writes them to the pinned memory, then the call's number behind
    // them, for which the host polls (11 us a round trip against 15 us of a
    // copy and a stream synchronisation, and a V-cycle makes 100-500 of them).
    const u64* fetch(const u64* from, int words, int at = 0) {
        publish(stream, from, host_scalars + at, words, host_scalars + kScalars, ++fetched);
        wait_fetched();
        std::atomic_thread_fence(std::memory_order_acquire);
        return host_scalars + at;
    }
    // Waits the way the program chose for this device (cudaSetDeviceFlags), as
    // a stream synchronisation does: a program that blocks gets its core back.
    // Polling gives the core to another thread that wants it every microsecond
    // or two (batch workers share the cores with each other's METIS steps),
    // and asks the stream now and then, so a failed kernel ends the wait.
    void wait_fetched() {
        unsigned how = 0;
        GP_CUDA(cudaGetDeviceFlags(&how));
        how &= cudaDeviceScheduleMask;
        if (how == cudaDeviceScheduleBlockingSync) {
            GP_CUDA(cudaStreamSynchronize(stream));
            return;
        }
        const unsigned pauses = how == cudaDeviceScheduleYield ? 1 : how == cudaDeviceScheduleSpin ? kQueryPolls : 32;
        const volatile u64* flag = host_scalars + kScalars;
        for (unsigned polls = 1; *flag != fetched; ++polls) {
            cpu_pause();
            if (polls % pauses == 0) std::this_thread::yield();
            if (polls % kQueryPolls) continue;
            const cudaError_t e = cudaStreamQuery(stream);
            if (e == cudaSuccess) break;  // complete: the words are there
            if (e != cudaErrorNotReady) GP_CUDA(e);
            cudaGetLastError();  // an answer, not a failure: a launch check must not report it
        }
    }
    static constexpr unsigned kQueryPolls = 2048;
    static void cpu_pause() {
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
    }
    const u64* read_scalars(int count) { return fetch(dev_scalars, count); }
    void clear_scalars(int count) {
        GP_CUDA(cudaMemsetAsync(dev_scalars, 0, sizeof(u64) * count, stream));
    }
};

// Entry points of the pipeline stages.
// Rows longer than heavy_min entries become g's heavy rows, listed with their
// kChunk-entry chunks in `storage` (the context's persist arena by default).
void build_chunks(Context& ctx, DGraph& g, int heavy_min = kHeavyRow, Arena* storage = nullptr);
Hierarchy coarsen(Context& ctx, const DGraph& input, const CoarsenOptions& o);
void keep_levels(Context& ctx, const Hierarchy& h);

struct RefineOutcome {
    u64 cut = 0;
    u64 max_load = 0;
    int levels_refined = 0;
};
// Round budgets of one level's refinement (RefineOptions::max_rounds and
// exchange_rounds, include/refine.hpp:13-26; the pipeline uses 32 and 2).
struct RefineBudget {
    int rounds = 32;
    int exchange_rounds = 2;
};
// What one level's refinement did (the RefineStats fields of
// include/refine.hpp:28-53 that describe the moves, not the layout).
struct LevelStats {
    int rounds = 0, admission_iterations = 0, checkpoint_updates = 0;
    bool repair_failed = false;
    u64 proposals = 0, accepted = 0, initial_cut = 0, final_cut = 0, final_max_load = 0;
    u64 lp_gain = 0, lp_loss = 0, rebalance_gain = 0, rebalance_loss = 0, group_gain = 0, group_accepted = 0;
};
// Refines from the coarsest level down to level 0 (refine_hierarchy_impl,
// src/refine.cu:483-730); `labels` (device, level-0 sized) receives the result.
RefineOutcome uncoarsen(Context& ctx, Hierarchy& h, const std::vector<int>& coarse_labels, int k, double eps,
                        int* labels, bool log, bool verify, const Mapping& mapping);

// Refines one graph from `labels` (device, n entries, values in [0,k)) in
// place: refine_partition (src/refine.cu:470-481) on a device-resident graph
// whose metadata coarsen() has filled.  The part loads are measured first.
LevelStats refine_single(Context& ctx, const DGraph& g, int* labels, int k, double eps, const RefineBudget& budget,
                         bool log, bool verify, const Mapping& mapping);

// Device edge cut of labels (directed sum / 2); throws on an odd sum.
u64 device_cut(Context& ctx, const DGraph& g, const int* labels);

// GP_FLAG_VERIFY checks (gp_verify.cu); failures throw with `status` or GP_INTERNAL.
void verify_csr(Context& ctx, const DGraph& g, bool allow_self_loops, gp_status status);
void verify_level(Context& ctx, const DGraph& fine, const DGraph& coarse, const int* map, u64 cluster_cap);

}  // namespace gp
