// Evaluation of a labelling on a device-resident graph: the undirected cut
// and the part loads, the two quantities refine_cut_kernel and
// accumulate_part_weights_kernel (src/refine.cu:63-126) produce.  The
// reduction is deterministic (integer sums): every block writes its partial
// loads and partial cut to a scratch array, and one block sums the partials.
#include "gp_graph.h"
#include "gp_primitives.cuh"

#include <algorithm>
#include <mutex>

namespace gp {
namespace {

constexpr int kEvalBlocks = 148 * 4;
constexpr int kEvalThreads = 256;
constexpr int kEvalWarps = kEvalThreads / 32;
// Per block: k loads, the directed cut of its entries, the count of entries it
// skipped as invalid (a label outside [0,k), a neighbour outside [0,n) or an
// offset outside [0,m]).  The partials are column-major: value c of block b at
// partial[c * blocks + b].
constexpr int kEvalStride = kMaxParts + 2;
constexpr int kEvalWindow = 256;  // entries a warp reads per step, eight per lane

constexpr int kEvalRowCost = kEvalWindow / 32;  // a step reads 256 entries or ends 32 rows

// Rows finished within the first d units of the work, a row costing
// kEvalRowCost units and an entry one: a merge-path split (Merrill and Garland,
// "Merge-based Parallel Sparse Matrix-Vector Multiplication", 2016) whose row
// ends weigh what they cost here, found by the whole warp with 32 probes a
// step.  Always in [0, n], whatever the offsets.
__device__ __forceinline__ i64 work_split(const int* off, i64 n, i64 first, i64 d) {
    const int lane = threadIdx.x & 31;
    i64 lo = 0, hi = min(n, d / kEvalRowCost);
    while (lo < hi) {
        const i64 step = (hi - lo + 31) >> 5;
        const i64 at = lo + lane * step;
        const bool within = at < hi && (at + 1) * kEvalRowCost + (off[at + 1] - first) <= d;
        // The probes that hold are a prefix for monotone offsets; only that
        // prefix is used.
        const unsigned fails = ~__ballot_sync(0xffffffffu, within);
        const int holds = fails ? __ffs(fails) - 1 : 32;
        if (holds == 0) {
            hi = lo;
        } else {
            const i64 next = lo + holds * step;  // first probe that fails, if there is one
            lo += (holds - 1) * step + 1;
            if (next < hi) hi = next;
        }
    }
    return lo;
}
// Entries read within the first d units, `row` rows being finished: all of the
// open row's at most.
__device__ __forceinline__ i64 entries_within(const int* off, i64 n, i64 first, i64 entries, i64 d, i64 row) {
    const i64 row_end = row < n ? min(max(off[row + 1] - first, 0LL), entries) : entries;
    return min(max(d - row * kEvalRowCost, 0LL), row_end);
}

// Pass 1.  Loads: every thread takes four vertices at a time, 32 apart, and
// adds neighbouring ones of equal labels once, a warp of one label once.  Cut:
// every warp takes an equal share of the work over rows and entries, so neither
// a hub row nor a stretch of short rows falls to one warp; it reads 256 entries
// a step, eight gathers per lane in flight, next to the ends and labels of the
// next 32 rows, and finds each entry's row from the marks that non-empty rows
// leave at their first entry.  Bound by the label gathers: L1 works at 77% of
// its rate, L2 at 48%, DRAM at 12% (R-MAT scale 21).  R-MAT scale 22, k = 64
// (124 M entries): 0.59 ms with the reduction; a warp per row took 6.60 ms, its
// longest row alone setting the time, and shares of equal rows plus entries
// 1.14, half of the SMs' time idle at the end.  (Labels packed into bytes first
// gained nothing.)
// Every access is range-checked, so a malformed labelling or CSR cannot reach
// memory outside the caller's arrays or the block's shared tables.
__global__ void __launch_bounds__(kEvalThreads, 5) k_eval_partials(i64 n, i64 m, const int* off, const int* nbr,
                                                                   const u32* ew, const u32* vw, const int* labels,
                                                                   int k, u64* partial) {
    constexpr int U = kEvalWindow / 32;
    __shared__ u64 loads[kMaxParts];
    __shared__ u64 warp_cut[kEvalWarps];
    __shared__ u64 warp_bad[kEvalWarps];
    __shared__ signed char marks[kEvalWarps][kEvalWindow];
    for (int p = threadIdx.x; p < k; p += blockDim.x) loads[p] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 bad = 0;
    for (i64 base = static_cast<i64>(blockIdx.x) * kEvalThreads * 4; base < n;
         base += static_cast<i64>(gridDim.x) * kEvalThreads * 4) {
        int p[4];
        u64 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const i64 v = base + warp * 128 + j * 32 + lane;
            p[j] = -1;
            w[j] = 0;
            if (v < n) {
                const int begin = off[v], end = off[v + 1];
                if (begin < 0 || end < begin || end > m) ++bad;
                p[j] = labels[v];
                w[j] = vw ? vw[v] : 1u;
                if (static_cast<unsigned>(p[j]) >= static_cast<unsigned>(k)) {
                    p[j] = -1;
                    w[j] = 0;
                    ++bad;
                }
            }
        }
#pragma unroll
        for (int j = 1; j < 4; ++j)
            if (p[j] == p[j - 1]) {
                w[j] += w[j - 1];
                w[j - 1] = 0;
            }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!__any_sync(0xffffffffu, w[j] != 0)) continue;
            if (__all_sync(0xffffffffu, p[j] == __shfl_sync(0xffffffffu, p[j], 0))) {
                const u64 sum = warp_sum(w[j]);
                if (lane == 0 && p[j] >= 0) atomicAdd(loads + p[j], sum);
            } else if (w[j]) {
                atomicAdd(loads + p[j], w[j]);
            }
        }
    }
    u64 cut = 0;
    const i64 first = min(max(static_cast<i64>(off[0]), 0LL), m);
    const i64 entries = min(max(static_cast<i64>(off[n]), first), m) - first;
    const i64 units = n * kEvalRowCost + entries;
    const i64 warps = static_cast<i64>(gridDim.x) * kEvalWarps;
    const i64 share = max((units + warps - 1) / warps, static_cast<i64>(kEvalWindow));
    const i64 d0 = (static_cast<i64>(blockIdx.x) * kEvalWarps + warp) * share;
    if (d0 < units) {
        const i64 d1 = min(units, d0 + share);
        int row = static_cast<int>(work_split(off, n, first, d0));
        const int last_row = static_cast<int>(work_split(off, n, first, d1));
        i64 e = first + entries_within(off, n, first, entries, d0, row);
        const i64 last = first + entries_within(off, n, first, entries, d1, last_row);
        const int rows = static_cast<int>(n);
        signed char* mark = marks[warp];
        while (e < last && row <= last_row && row < rows) {
            // Positions below are relative to e.
            const int stop = static_cast<int>(min(last - e, static_cast<i64>(kEvalWindow)));
            const int* entry = nbr + e;
            int q[U];
#pragma unroll
            for (int j = 0; j < U; ++j) q[j] = j * 32 + lane < stop ? entry[j * 32 + lane] : 0;
            const int r = min(lane, rows - 1 - row) + row;
            const int row_end = lane < rows - row
                                    ? static_cast<int>(min(max(off[r + 1] - e, -1LL), kEvalWindow + 1LL))
                                    : stop;
            const int row_label = labels[r];
            // Entries of the 32 rows at hand; the ones past them are read
            // again with the next rows.
            const int reach = __shfl_sync(0xffffffffu, row_end, 31);
            const int until = min(reach, stop);
            int wrong = 0;
#pragma unroll
            for (int j = 0; j < U; ++j) {
                const bool in = j * 32 + lane < until;
                const bool good = static_cast<unsigned>(q[j]) < static_cast<unsigned>(rows);
                wrong += in && !good;
                q[j] = in && good ? labels[q[j]] : -1;
            }
            bad += wrong;
            if (__shfl_sync(0xffffffffu, row_end, 0) >= stop) {  // one row holds the whole window
                const int part = __shfl_sync(0xffffffffu, row_label, 0);
#pragma unroll
                for (int j = 0; j < U; ++j)
                    if (j * 32 + lane < until && q[j] != part) cut += edge_w(ew, e + j * 32 + lane);
            } else {
                const int before = __shfl_up_sync(0xffffffffu, row_end, 1);
                const int at = lane ? max(before, 0) : 0;
#pragma unroll
                for (int j = 0; j < U; ++j) mark[j * 32 + lane] = -1;
                __syncwarp();
                if (row_end > at && at < kEvalWindow) mark[at] = static_cast<signed char>(lane);
                __syncwarp();
                int carry = 0;
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    const int own = mark[j * 32 + lane];
                    const unsigned heads = __ballot_sync(0xffffffffu, own >= 0) & (0xffffffffu >> (31 - lane));
                    const int from = __shfl_sync(0xffffffffu, own, heads ? 31 - __clz(heads) : 0);
                    const int holder = heads ? from : carry;
                    carry = __shfl_sync(0xffffffffu, holder, 31);
                    const int part = __shfl_sync(0xffffffffu, row_label, holder);
                    if (j * 32 + lane < until && q[j] != part) cut += edge_w(ew, e + j * 32 + lane);
                }
                __syncwarp();
            }
            if (reach < stop) {
                row = rows - row > 32 ? row + 32 : rows;
                e += max(until, 0);
            } else {
                row += __popc(__ballot_sync(0xffffffffu, lane < rows - row && row_end <= stop));
                e += stop;
            }
        }
    }
    cut = warp_sum(cut);
    bad = warp_sum(bad);
    if (lane == 0) {
        warp_cut[warp] = cut;
        warp_bad[warp] = bad;
    }
    __syncthreads();
    u64* out = partial + blockIdx.x;
    for (int p = threadIdx.x; p < k; p += blockDim.x) out[static_cast<i64>(p) * gridDim.x] = loads[p];
    if (threadIdx.x == 0) {
        u64 c = 0, b = 0;
        for (int w = 0; w < kEvalWarps; ++w) {
            c += warp_cut[w];
            b += warp_bad[w];
        }
        out[static_cast<i64>(k) * gridDim.x] = c;
        out[static_cast<i64>(k + 1) * gridDim.x] = b;
    }
}

// Pass 2: sums the partials of all blocks, a warp per value.  (One thread per
// value walked the 592 blocks' partials one after another: most of the 61 us that
// judging a 256x256 grid took; it takes 22.)  With any invalid
// entry the cut output is UINT64_MAX (no real cut reaches it) and, when
// `invalid` is given, the count is stored there.
__global__ void __launch_bounds__(1024) k_eval_reduce(int blocks, int k, const u64* partial, u64* cut_out,
                                                      u64* loads_out, u64* invalid) {
    __shared__ u64 sums[2];
    const int lane = threadIdx.x & 31;
    for (int p = threadIdx.x >> 5; p <= k + 1; p += blockDim.x >> 5) {
        u64 s = 0;
        for (int b = lane; b < blocks; b += 32) s += partial[static_cast<i64>(p) * blocks + b];
        s = warp_sum(s);
        if (lane == 0) {
            if (p < k) loads_out[p] = s;
            else sums[p - k] = s;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *cut_out = sums[1] ? ~0ULL : sums[0] / 2;
        if (invalid) *invalid = sums[1];
    }
}

void check_evaluate_args(const gp_csr* g, const int32_t* labels, int32_t k, const uint64_t* cut_out,
                         const uint64_t* loads_out) {
    if (!g || !labels || !cut_out || !loads_out || !g->offsets || (g->m > 0 && !g->neighbors))
        fail(GP_INVALID_ARGUMENT, "graph, labels and outputs must not be NULL");
    if (g->n <= 0 || g->m < 0 || g->n > 0x7fffffff || g->m > 0x7fffffff)
        fail(GP_INVALID_ARGUMENT, "graph exceeds supported 32-bit CSR limits");
    if (k < 1 || k > kMaxParts) fail(GP_INVALID_ARGUMENT, "k must be in 1..128");
}

void launch_evaluate(const gp_csr* g, const int32_t* labels, int32_t k, uint64_t* cut_out, uint64_t* loads_out,
                     u64* partial, u64* invalid, cudaStream_t s) {
    // No more blocks than give every warp one window of entries.
    const int blocks = std::min(blocks_for(g->n * kEvalRowCost + g->m, kEvalWarps * kEvalWindow), kEvalBlocks);
    launch_ordinary(k_eval_partials, blocks, kEvalThreads, 0, s, static_cast<i64>(g->n), static_cast<i64>(g->m),
           g->offsets, g->neighbors, g->edge_weights, g->vertex_weights, labels, static_cast<int>(k), partial);
    launch_ordinary(k_eval_reduce, 1, 1024, 0, s, blocks, static_cast<int>(k), static_cast<const u64*>(partial),
           reinterpret_cast<u64*>(cut_out), reinterpret_cast<u64*>(loads_out), invalid);
}

template <class F>
gp_status guarded_eval(F&& f) {
    try {
        return f();
    } catch (const Failure& e) {
        set_error(e.what());
        return e.status;
    } catch (const std::exception& e) {
        set_error(e.what());
        return GP_INTERNAL;
    }
}

}  // namespace
}  // namespace gp

// ---------------------------------------------------------------------------
// Allocation-free variant.  Some callers cannot let a library call cudaMalloc:
// a framework whose caching allocator owns the whole device-memory budget (a
// raw cudaMalloc would bypass that budget and, on a full device, fail), or a
// serving loop that must not allocate or free device memory once it runs,
// because cudaMalloc/cudaFree may synchronise the device and stall the other
// streams.  gp_evaluate_device_static needs no context and no allocation: its
// per-block partial sums live in the fixed array below, which every GPU that
// loads this library holds until the process exits.
constexpr size_t kStaticScratchWords = static_cast<size_t>(gp::kEvalBlocks) * gp::kEvalStride;  // 616 KB
static __device__ __align__(256) unsigned long long g_eval_static_scratch[kStaticScratchWords];

namespace gp {
namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
u64* g_static_address[kMaxDevices] = {};

// Device address of the static scratch on the current device.  In host code
// the array's name is only a host-side stand-in, so the address is looked up
// once per device, with that device current, and cached.  The cache assumes
// the device's primary context (the one the runtime API uses) stays the same
// for the life of the process: after cudaDeviceReset, or under another
// context made current through the driver API, the cached address is stale.
u64* static_scratch_address() {
    int device = 0;
    GP_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= kMaxDevices) fail(GP_INVALID_ARGUMENT, "device ordinal beyond 63");
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (!g_static_address[device]) {
        void* address = nullptr;
        const cudaError_t err = cudaGetSymbolAddress(&address, g_eval_static_scratch);
        if (err != cudaSuccess) cudaGetLastError();  // handled here
        if (err != cudaSuccess || !address)
            fail(GP_CUDA_ERROR, std::string("cudaGetSymbolAddress(static scratch): ") + cudaGetErrorString(err));
        g_static_address[device] = static_cast<u64*>(address);
    }
    return g_static_address[device];
}
}  // namespace
}  // namespace gp

using namespace gp;

extern "C" gp_status gp_evaluate_device_static(const gp_csr* graph, const int32_t* labels, int32_t k,
                                               uint64_t* cut_out, uint64_t* loads_out, void* stream) {
    return guarded_eval([&]() -> gp_status {
        check_evaluate_args(graph, labels, k, cut_out, loads_out);
        // Every partial the reduction reads is rewritten by the first pass of
        // this call, so nothing in the shared array needs clearing first.
        u64* partial = static_scratch_address();
        launch_evaluate(graph, labels, k, cut_out, loads_out, partial, nullptr, static_cast<cudaStream_t>(stream));
        return GP_OK;
    });
}

// Context accessor defined in gp_partition.cu.
namespace gp { Context& context_of(gp_context* ctx); }

extern "C" gp_status gp_evaluate_device(gp_context* ctx, const gp_csr* graph, const int32_t* labels, int32_t k,
                                        uint64_t* cut_out, uint64_t* loads_out, void* stream) {
    return guarded_eval([&]() -> gp_status {
        if (!ctx) fail(GP_INVALID_ARGUMENT, "context is NULL");
        check_evaluate_args(graph, labels, k, cut_out, loads_out);
        Context& c = context_of(ctx);
        GP_CUDA(cudaSetDevice(c.device));
        cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : c.stream;
        ArenaScope scope(c.scratch);
        u64* partial = c.scratch.alloc<u64>(static_cast<size_t>(kEvalBlocks) * kEvalStride);
        launch_evaluate(graph, labels, k, cut_out, loads_out, partial, c.dev_scalars, s);
        // The partials live in the context arena: keep them until the
        // reduction has read them.
        GP_CUDA(cudaMemcpyAsync(c.host_scalars, c.dev_scalars, sizeof(u64), cudaMemcpyDeviceToHost, s));
        GP_CUDA(cudaStreamSynchronize(s));
        if (c.host_scalars[0])
            fail(GP_INVALID_ARGUMENT, std::to_string(c.host_scalars[0]) +
                                          " labels, neighbours or offsets out of range (labels must be in [0,k))");
        return GP_OK;
    });
}
