// Refinement of a small level in one launch: the initial capacity repair and
// every label-propagation round with its repair, by one thread-block cluster.
// Included by gp_refine.cu after the device functions it shares with the
// launch-per-step path.
//
// A round of a small level is a chain of a dozen dependent steps of a few
// microseconds each; as launches with host decisions in between, the chain
// takes 100-200 us whatever the level's size.  Here a step ends at the
// cluster's hardware barrier and every block takes the loop's decisions from
// the same counters, so a round costs the latency of its steps and their
// barriers: 8% of the issue slots are used and three quarters of the warps'
// time is spent at barriers (256x256 grid, k = 8).  The blocks of a cluster are
// always resident together, so clusters of concurrent contexts share the GPU
// without waiting for each other.
#pragma once

namespace gp {
namespace {

constexpr int kClusterBlocks = 16;     // one GPC; above the portable 8
constexpr int kClusterThreads = 512;
constexpr int kClusterHeavyCap = 512;  // rows a block sets aside for all its threads, per pass

// Loop state of a level, in global memory: where the kernel starts, and what
// it found.
enum ClusterStart : int {
    kStartLevel = 0,
    kStartAfterInitialRepair = 1,
    kStartAfterRoundRepair = 2,
    kStartInInitialRepair = 3,  // its next iteration
    kStartAfterPropagation = 4, // a round's label propagation is applied
    kStartInRoundRepair = 5,
};
enum ClusterStatus : int {
    kClusterDone = 0,
    kClusterInitialRepairFailed = 1,
    kClusterHostInitialRepair = 2,  // more listed donors than one block takes: the host
    kClusterHostRoundRepair = 3,    // completes this repair and starts the kernel again
    kClusterCutUnderflow = 4,
    kClusterCheck = 5,  // GP_FLAG_VERIFY: the host checks the batch just applied and starts the kernel again
};
struct ClusterLoop {
    u64 cut, best, feasible_start;
    int start, status;                // ClusterStart, ClusterStatus
    int rounds, stale, empty, moved;  // moved: a batch was applied since the best labels were saved
};
struct ClusterTotals {
    u64 proposals, accepted, lp_gain, lp_loss, rebalance_gain, rebalance_loss, repair_donors;
    u64 admission_iterations, checkpoint_updates;
};
struct ClusterState {
    ClusterLoop loop;
    ClusterTotals totals;
    u64 max_load;
    u64 listed, iterations;  // of a repair that the host completes or checks
};

template <class C>
struct ClusterLevel {
    i64 n;
    int k, max_rounds, heavy_min, region;  // region: list entries of one block
    bool check;  // stop after every batch (kClusterCheck)
    u64 capacity;
    double filter;
    const int* off;
    const int* nbr;
    const u32* ew;
    const u32* vw;
    int* labels;
    u64* loads;
    C* A;
    const C* totals;
    long long* gains;
    u64* proposal;
    unsigned char* locks;
    int* flags;
    int* targets;
    u32* state;
    Sample* samples;  // nullptr: unpriced
    double* prices;
    int* cand;    // kClusterBlocks regions
    int* movers;  // kClusterBlocks regions
    u32* plan;
    u64* class_weights;
    int* bound;
    u64* start;
    u64* list;
    u64* slack;
    u64* requests;
    int* saved_labels;
    u64* saved_loads;
    u64* ctl;  // 4 sets of 8 counters, zero at the first start
    ClusterState* io;
};

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
    int r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Counters of one batch (ctl set): added to by every block, read by all after
// a barrier, zeroed two batches ahead.
enum { kCtlMovers = 0, kCtlDelta = 1, kCtlListed = 2, kCtlDonors = 3, kCtlPlaced = 4, kCtlWords = 8 };

template <class C>
struct ClusterShared {
    AttemptParts<kClusterThreads> attempt;
    u64 load[kMaxParts], slack[kMaxParts], excess[kMaxParts], cdf[kMaxParts + 1], start[kMaxParts];
    double price[kMaxParts];
    long long diff[kMaxParts];
    int bound[kMaxParts];
    u64 scan[33];
    u32 scan32[33];
    int heavy[kClusterHeavyCap];
    ClusterTotals totals;  // added to by thread 0
    long long delta;
    u32 cand, movers, heavy_count, placed;
    u64 donors;
};

template <class C>
class ClusterRefiner {
public:
    __device__ ClusterRefiner(const ClusterLevel<C>& L, ClusterShared<C>& sm, unsigned char* raw)
        : L(L), sm(sm), raw(raw), rank(cluster_rank()), lane(threadIdx.x & 31), warp(threadIdx.x >> 5) {}

    __device__ void run() {
        for (int p = threadIdx.x; p < L.k; p += kClusterThreads) {
            sm.price[p] = L.prices ? L.prices[p] : 0.0;
            sm.diff[p] = 0;
        }
        if (threadIdx.x == 0) sm.totals = L.io->totals;
        st = L.io->loop;
        const int begin = st.start;
        iterations = static_cast<int>(L.io->iterations);
        refresh_loads();
        bool feasible = max_load <= L.capacity;
        st.status = kClusterDone;
        // Steps of the first round that are done already: none, the
        // propagation, some of the repair, the repair.
        const int done = begin == kStartAfterPropagation ? 1 : begin == kStartInRoundRepair ? 2
                         : begin == kStartAfterRoundRepair ? 3 : 0;
        if (!done) {
            if (begin != kStartAfterInitialRepair && !feasible) {
                feasible = repair(begin == kStartInInitialRepair);
                if (st.status == kClusterHostRoundRepair) st.status = kClusterHostInitialRepair;
                if (st.status == kClusterCheck) return stop(kStartInInitialRepair);
                if (st.status != kClusterDone) return finish();
                if (L.check) return stop(kStartAfterInitialRepair);
            }
            if (!feasible) {
                st.status = kClusterInitialRepairFailed;
                return finish();
            }
            st.feasible_start = st.best = st.cut;
            st.moved = 0;
            save();
        }
        for (int skip = done; skip || (st.rounds < L.max_rounds && st.stale < 3); skip = 0) {
            if (skip < 1) {
                ++st.rounds;
                const u64 count = lp_round();
                if (st.status != kClusterDone) return finish();
                if (!count) {
                    if (++st.empty >= 2) break;
                    ++st.stale;
                    continue;
                }
                st.empty = 0;
                feasible = max_load <= L.capacity;
                if (L.check) return stop(kStartAfterPropagation);
            }
            if (skip < 3 && !feasible) {
                feasible = repair(skip == 2);
                if (st.status == kClusterCheck) return stop(kStartInRoundRepair);
                if (st.status != kClusterDone) return finish();
                if (L.check) return stop(kStartAfterRoundRepair);
            }
            if (!feasible) break;
            if (L.samples) {
                for (int p = threadIdx.x; p < L.k; p += kClusterThreads) {
                    const Sample x = L.samples[p];
                    if (x.weight)
                        sm.price[p] = x.loss > 0 ? static_cast<double>(x.loss) / static_cast<double>(x.weight) : 0.0;
                }
                __syncthreads();
            }
            ++st.stale;
            if (st.cut < st.best) {
                if (st.best - st.cut > st.best / 1000) st.stale = 0;
                st.best = st.cut;
                st.moved = 0;
                save();
                if (threadIdx.x == 0) ++sm.totals.checkpoint_updates;
            }
        }
        finish();
    }

private:
    const ClusterLevel<C>& L;
    ClusterShared<C>& sm;
    unsigned char* raw;
    const int rank, lane, warp;
    ClusterLoop st;  // the same in every thread
    int listed = 0, iterations = 0;
    u64 max_load = 0;
    int batch = 0;
    static constexpr int kStep = kClusterBlocks * kClusterThreads;

    __device__ u64* counters(int b) const { return L.ctl + (b & 3) * kCtlWords; }
    __device__ void next_batch() {
        ++batch;
        // Set batch + 2 was last used two batches ago, before at least two
        // barriers that every block has passed.
        if (rank == 0 && threadIdx.x < kCtlWords) counters(batch + 2)[threadIdx.x] = 0;
    }
    __device__ void stop(int start) {
        st.status = kClusterCheck;
        st.start = start;
        finish();
    }
    // Ends the launch: a finished level goes back to its best labels (the
    // cache does not), and the state to global memory.
    __device__ void finish() {
        cluster_barrier();  // every block has read the counters and saved its share
        if (st.status == kClusterDone && st.moved) {
            for (i64 v = rank * kClusterThreads + threadIdx.x; v < L.n; v += kStep) {
                const int p = L.saved_labels[v];
                L.labels[v] = p;
                L.state[v] = static_cast<u32>(p);
            }
            u64 m = 0;
            for (int p = lane; p < L.k; p += 32) {
                const u64 x = __ldcg(L.saved_loads + p);
                m = x > m ? x : m;
                if (rank == 0 && warp == 0) L.loads[p] = x;
            }
            max_load = warp_max(m);
        }
        if (rank == 0) {
            for (int p = threadIdx.x; p < L.k; p += kClusterThreads)
                if (L.prices) L.prices[p] = sm.price[p];
            if (threadIdx.x < 4 * kCtlWords) L.ctl[threadIdx.x] = 0;
            if (threadIdx.x == 0)
                *L.io = ClusterState{st, sm.totals, max_load, static_cast<u64>(listed), static_cast<u64>(iterations)};
        }
    }
    // Part loads into shared memory, the largest into max_load.
    __device__ void refresh_loads() {
        u64 m = 0;
        for (int p = threadIdx.x; p < L.k; p += kClusterThreads) sm.load[p] = __ldcg(L.loads + p);
        __syncthreads();
        for (int p = lane; p < L.k; p += 32) m = sm.load[p] > m ? sm.load[p] : m;
        max_load = warp_max(m);
    }
    // Saves the labels and loads as the best ones.  The labels change next
    // two barriers later.
    __device__ void save() {
        for (i64 v = rank * kClusterThreads + threadIdx.x; v < L.n; v += kStep) L.saved_labels[v] = L.labels[v];
        if (rank == 0)
            for (int p = threadIdx.x; p < L.k; p += kClusterThreads) L.saved_loads[p] = sm.load[p];
    }
    __device__ void account(long long delta) {
        if (delta >= 0) {
            if (static_cast<u64>(delta) > st.cut) st.status = kClusterCutUnderflow;
            st.cut -= static_cast<u64>(delta);
        } else st.cut += static_cast<u64>(-delta);
    }

    // One label-propagation round (k_proposals, k_filter, k_compact_movers,
    // k_update and k_commit in three steps); the number of movers.
    __device__ u64 lp_round() {
        next_batch();
        const LpParams q = params();
        if (threadIdx.x == 0) sm.cand = sm.movers = 0;
        for (int p = threadIdx.x; p < L.k; p += kClusterThreads)
            sm.slack[p] = L.capacity - sm.load[p];  // every load fits between rounds
        __syncthreads();
        propose(q);
        cluster_barrier();
        if (L.samples && rank == 0)
            for (int p = threadIdx.x; p < L.k; p += kClusterThreads) L.samples[p] = Sample{0, 0};
        filter(q);
        if (threadIdx.x == 0 && sm.movers) atomicAdd(counters(batch) + kCtlMovers, static_cast<u64>(sm.movers));
        cluster_barrier();
        const int* mine = L.movers + static_cast<i64>(rank) * L.region;
        const int count = static_cast<int>(sm.movers);
        update(mine, count, 0, 1, true);
        cluster_barrier();
        const u64 total = __ldcg(counters(batch) + kCtlMovers);
        const long long delta = static_cast<long long>(__ldcg(counters(batch) + kCtlDelta));
        refresh_loads();
        settle(mine, count, 0, 1);
        if (total) {
            if (threadIdx.x == 0) {
                sm.totals.proposals += total;
                sm.totals.accepted += total;
                if (delta >= 0) sm.totals.lp_gain += static_cast<u64>(delta);
                else sm.totals.lp_loss += static_cast<u64>(-delta);
            }
            account(delta);
            st.moved = 1;
        }
        return total;
    }
    __device__ LpParams params() const {
        LpParams q{};
        q.n = L.n;
        q.k = L.k;
        q.capacity = L.capacity;
        q.filter = L.filter;
        q.off = L.off;
        q.nbr = L.nbr;
        q.ew = L.ew;
        q.vw = L.vw;
        q.labels = L.labels;
        q.loads = sm.load;
        q.prices = L.samples ? sm.price : nullptr;
        q.gains = L.gains;
        q.proposal = L.proposal;
        q.heavy_min = L.heavy_min;
        return q;
    }

    // k_proposals: 512 consecutive vertices a pass, eight lanes a row.
    __device__ void propose(const LpParams& q) {
        constexpr int W = 8, G = 32 / W;
        const int gid = lane / W, sub = lane % W, k = L.k;
        int* cand = L.cand + static_cast<i64>(rank) * L.region;
        for (i64 base = rank * kClusterThreads + warp * 32; base < L.n; base += kStep) {
            const i64 v = base + lane;
            int src = 0;
            u64 current = 0;
            bool act = false;
            if (v < L.n) {
                if (L.locks[v]) {
                    L.locks[v] = 0;
                } else {
                    src = L.labels[v];
                    current = L.A[v * k + src];
                    act = current != static_cast<u64>(L.totals[v]);
                }
                if (!act) L.proposal[v] = 0;
            }
            unsigned pending = __ballot_sync(0xffffffffu, act);
            while (pending) {
                unsigned mine = pending;
                for (int i = 0; i < gid; ++i) mine &= mine - 1;
                for (int i = 0; i < G; ++i) pending &= pending - 1;
                const int owner = mine ? __ffs(mine) - 1 : 0;
                const int osrc = __shfl_sync(0xffffffffu, src, owner);
                const u64 ocur = __shfl_sync(0xffffffffu, current, owner);
                const i64 vv = base + owner;
                int target = -1;
                u64 best = 0;
                double best_score = -DBL_MAX;
                if (mine) {
                    const C* row = L.A + vv * k;
                    const u64 weight = q.prices ? L.vw[vv] : 0;
                    for (int p0 = sub; p0 < k; p0 += 4 * W) {
                        C val[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) val[e] = p0 + e * W < k ? row[p0 + e * W] : C(0);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int p = p0 + e * W;
                            const u64 conn = val[e];
                            if (p == osrc || !conn) continue;
                            if (q.prices) {
                                const double cost =
                                    weight > sm.slack[p]
                                        ? __dmul_rn(sm.price[p], static_cast<double>(weight - sm.slack[p]))
                                        : 0.0;
                                const double score = __dsub_rn(static_cast<double>(conn), cost);
                                if (target < 0 || score > best_score) { target = p; best = conn; best_score = score; }
                            } else if (target < 0 || conn > best) {
                                target = p;
                                best = conn;
                            }
                        }
                    }
                }
#pragma unroll
                for (int d = W / 2; d; d >>= 1) {
                    const int ot = __shfl_xor_sync(0xffffffffu, target, d, W);
                    const u64 ob = __shfl_xor_sync(0xffffffffu, best, d, W);
                    const double os = __shfl_xor_sync(0xffffffffu, best_score, d, W);
                    if (ot >= 0) {
                        const bool greater = q.prices ? os > best_score : ob > best;
                        const bool equal = q.prices ? os == best_score : ob == best;
                        if (target < 0 || greater || (equal && ot < target)) { target = ot; best = ob; best_score = os; }
                    }
                }
                if (mine && sub == 0) {
                    const bool ok = target >= 0 && (best >= ocur || ocur - best < static_cast<u64>(q.filter * static_cast<double>(ocur)));
                    const long long gain = best >= ocur ? static_cast<long long>(best - ocur) : -static_cast<long long>(ocur - best);
                    if (ok) {
                        L.gains[vv] = gain;
                        cand[atomicAdd(&sm.cand, 1u)] = static_cast<int>(vv);
                    }
                    L.proposal[vv] = pack_proposal(osrc, ok ? target : -1, gain);
                }
            }
        }
    }

    // A candidate whose corrected gain stays non-negative becomes a mover of
    // this block and is marked in the packed state (k_compact_movers).
    __device__ void decide(const LpParams& q, int v, int s, int t, long long total) {
        bool keep = total >= 0;
        if (q.prices) {
            const u64 w = L.vw[v];
            const double adj = __dsub_rn(repair_cost(s, w, q.loads, q.capacity, q.prices),
                                         repair_cost(t, w, q.loads, q.capacity, q.prices));
            keep = __dadd_rn(static_cast<double>(total), adj) >= 0;
        }
        if (!keep) return;
        L.state[v] = static_cast<u32>(s) | (static_cast<u32>(t) << 8) | kMovingBit;
        L.movers[static_cast<i64>(rank) * L.region + atomicAdd(&sm.movers, 1u)] = v;
    }
    // k_filter over the block's candidates; rows above heavy_min by the block.
    __device__ void filter(const LpParams& q) {
        constexpr int W = 8, G = 32 / W;
        const int gid = lane / W, sub = lane % W;
        const int* cand = L.cand + static_cast<i64>(rank) * L.region;
        const int count = static_cast<int>(sm.cand);
        if (threadIdx.x == 0) sm.heavy_count = 0;
        __syncthreads();
        unsigned leaders = 0;
        for (int g = 0; g < G; ++g) leaders |= 1u << (g * W);
        for (int base = warp * G; base < count; base += kClusterThreads / W) {
            const int i = base + gid;
            const int v = i < count ? cand[i] : -1;
            const int begin = v >= 0 ? q.off[v] : 0, end = v >= 0 ? q.off[v + 1] : 0;
            const u64 own = v >= 0 ? q.proposal[v] : 0;
            const int s = static_cast<int>(own & 0xffu), t = static_cast<int>((own >> 8) & 0xffu);
            const long long gain = v >= 0 ? packed_gain(own, q.gains, v) : 0;
            bool mine = v >= 0;
            if (mine && end - begin > q.heavy_min) {
                u32 slot = kClusterHeavyCap;
                if (sub == 0) slot = atomicAdd(&sm.heavy_count, 1u);
                slot = __shfl_sync(0xffu << (lane & 24), slot, 0, W);  // all lanes of the row's group are here
                if (slot < kClusterHeavyCap) {
                    if (sub == 0) sm.heavy[slot] = v;
                    mine = false;
                }
            }
            __syncwarp();
            long long corr = mine && end - begin <= kFilterShort ? filter_entries(q, v, s, t, gain, begin + sub, end, W) : 0;
            for (unsigned rest = __ballot_sync(0xffffffffu, mine && end - begin > kFilterShort) & leaders; rest;
                 rest &= rest - 1) {
                const int leader = __ffs(rest) - 1;
                const int vv = __shfl_sync(0xffffffffu, v, leader), ss = __shfl_sync(0xffffffffu, s, leader),
                          tt = __shfl_sync(0xffffffffu, t, leader), b = __shfl_sync(0xffffffffu, begin, leader),
                          e = __shfl_sync(0xffffffffu, end, leader);
                const long long gg = __shfl_sync(0xffffffffu, gain, leader);
                const long long c = warp_sum(filter_entries(q, vv, ss, tt, gg, b + lane, e, 32));
                if (lane == leader) corr += c;
            }
#pragma unroll
            for (int d = W / 2; d; d >>= 1) corr += __shfl_xor_sync(0xffffffffu, corr, d, W);
            if (sub == 0 && mine) decide(q, v, s, t, gain + corr);
        }
        __syncthreads();
        const int heavy = min(static_cast<int>(sm.heavy_count), kClusterHeavyCap);
        for (int h = 0; h < heavy; ++h) {
            const int v = sm.heavy[h];
            const u64 own = q.proposal[v];
            const int s = static_cast<int>(own & 0xffu), t = static_cast<int>((own >> 8) & 0xffu);
            const long long gain = packed_gain(own, q.gains, v);
            const long long corr = block_sum(
                filter_entries(q, v, s, t, gain, q.off[v] + static_cast<int>(threadIdx.x), q.off[v + 1], kClusterThreads));
            if (threadIdx.x == 0) decide(q, v, s, t, gain + corr);
        }
        __syncthreads();
    }

    // What the leader of mover v (part s to part t) does beside the cache
    // update: its label, load change, lock and repair sample.
    __device__ void commit(int v, int s, int t, long long gain, bool lp) {
        const u64 w = L.vw[v];
        L.labels[v] = t;
        if (lp) L.locks[v] = 1;
        atomicAdd(reinterpret_cast<u64*>(sm.diff + s), 0ULL - w);
        atomicAdd(reinterpret_cast<u64*>(sm.diff + t), w);
        if (!lp && L.samples) {
            atomicAdd(reinterpret_cast<u64*>(&L.samples[s].loss), static_cast<u64>(-gain));
            atomicAdd(&L.samples[s].weight, w);
        }
    }
    // k_update and k_commit for list[first], list[first + stride * 64 groups],
    // ...: the cache and cut by the packed state, which stays as marked until
    // settle(); labels, loads and samples beside it.
    __device__ void update(const int* list, int count, int first_block, int blocks, bool lp) {
        constexpr int W = 8, G = 32 / W;
        const int gid = lane / W, sub = lane % W;
        if (threadIdx.x == 0) {
            sm.heavy_count = 0;
            sm.delta = 0;
        }
        __syncthreads();
        unsigned leaders = 0;
        for (int g = 0; g < G; ++g) leaders |= 1u << (g * W);
        long long total = 0;
        for (int base = (first_block * (kClusterThreads / 32) + warp) * G; base < count;
             base += blocks * (kClusterThreads / W)) {
            const int i = base + gid;
            const int v = i < count ? list[i] : -1;
            const int begin = v >= 0 ? L.off[v] : 0, end = v >= 0 ? L.off[v + 1] : 0;
            const u32 sv = v >= 0 ? L.state[v] : 0u;
            const int s = state_label(sv), t = static_cast<int>((sv >> 8) & 0xffu);
            bool mine = v >= 0;
            if (mine && end - begin > L.heavy_min) {
                u32 slot = kClusterHeavyCap;
                if (sub == 0) slot = atomicAdd(&sm.heavy_count, 1u);
                slot = __shfl_sync(0xffu << (lane & 24), slot, 0, W);  // all lanes of the row's group are here
                if (slot < kClusterHeavyCap) {
                    if (sub == 0) sm.heavy[slot] = v;
                    mine = false;
                }
            }
            __syncwarp();
            long long gain = mine && end - begin <= kUpdateShort
                                 ? update_entries(v, s, t, begin + sub, end, W, L.nbr, L.ew, L.state, L.k, L.A)
                                 : 0;
            for (unsigned rest = __ballot_sync(0xffffffffu, mine && end - begin > kUpdateShort) & leaders; rest;
                 rest &= rest - 1) {
                const int leader = __ffs(rest) - 1;
                const int vv = __shfl_sync(0xffffffffu, v, leader), ss = __shfl_sync(0xffffffffu, s, leader),
                          tt = __shfl_sync(0xffffffffu, t, leader), b = __shfl_sync(0xffffffffu, begin, leader),
                          e = __shfl_sync(0xffffffffu, end, leader);
                const long long g = warp_sum(update_entries(vv, ss, tt, b + lane, e, 32, L.nbr, L.ew, L.state, L.k, L.A));
                if (lane == leader) gain += g;
            }
#pragma unroll
            for (int d = W / 2; d; d >>= 1) gain += __shfl_xor_sync(0xffffffffu, gain, d, W);
            if (sub == 0 && mine) {
                total += gain;
                commit(v, s, t, gain, lp);
            }
        }
        __syncthreads();
        const int heavy = min(static_cast<int>(sm.heavy_count), kClusterHeavyCap);
        for (int h = 0; h < heavy; ++h) {
            const int v = sm.heavy[h];
            const u32 sv = L.state[v];
            const int s = state_label(sv), t = static_cast<int>((sv >> 8) & 0xffu);
            const long long gain =
                block_sum(update_entries(v, s, t, L.off[v] + static_cast<int>(threadIdx.x), L.off[v + 1], kClusterThreads,
                                         L.nbr, L.ew, L.state, L.k, L.A));
            if (threadIdx.x == 0) {
                total += gain;
                commit(v, s, t, gain, lp);
            }
        }
        total = warp_sum(total);
        if (lane == 0 && total) atomicAdd(reinterpret_cast<u64*>(&sm.delta), static_cast<u64>(total));
        __syncthreads();
        for (int p = threadIdx.x; p < L.k; p += kClusterThreads)
            if (sm.diff[p]) {
                atomicAdd(L.loads + p, static_cast<u64>(sm.diff[p]));
                sm.diff[p] = 0;
            }
        if (threadIdx.x == 0 && sm.delta) atomicAdd(counters(batch) + kCtlDelta, static_cast<u64>(sm.delta));
    }
    // After the barrier that ends an update: the movers' new labels in the
    // packed state.  Nothing reads the state before the next barrier.
    __device__ void settle(const int* list, int count, int first_block, int blocks) {
        for (int i = first_block * kClusterThreads + threadIdx.x; i < count; i += blocks * kClusterThreads) {
            const int v = list[i];
            L.state[v] = (L.state[v] >> 8) & 0xffu;
        }
    }

    // One capacity repair (the iterations of LevelRefiner::repair); whether
    // the parts fit at its end.  With more listed donors than one block
    // orders, leaves st.status at kClusterHostRoundRepair; between checked
    // iterations, at kClusterCheck.
    __device__ bool repair(bool resumed) {
        if (!resumed) iterations = 0;
        while (true) {
            next_batch();
            u64* ctl = counters(batch);
            receivers();
            destinations(ctl);
            cluster_barrier();
            bounds();
            cluster_barrier();
            collect(ctl);
            cluster_barrier();
            listed = static_cast<int>(__ldcg(ctl + kCtlListed));
            if (threadIdx.x == 0) sm.totals.repair_donors += __ldcg(ctl + kCtlDonors);
            if (listed > kAttemptCap) {
                st.status = kClusterHostRoundRepair;
                return false;
            }
            if (rank == 0) reserve(listed, ctl);
            cluster_barrier();
            const int placed = static_cast<int>(__ldcg(ctl + kCtlPlaced));
            update(L.movers, placed, rank, kClusterBlocks, false);
            cluster_barrier();
            const long long delta = static_cast<long long>(__ldcg(ctl + kCtlDelta));
            refresh_loads();
            settle(L.movers, placed, rank, kClusterBlocks);
            if (threadIdx.x == 0) {
                sm.totals.accepted += static_cast<u64>(placed);
                if (delta >= 0) sm.totals.rebalance_gain += static_cast<u64>(delta);
                else sm.totals.rebalance_loss += static_cast<u64>(-delta);
                ++sm.totals.admission_iterations;
            }
            if (placed) {
                account(delta);
                if (st.status != kClusterDone) return false;
                st.moved = 1;
            }
            ++iterations;
            const bool feasible = max_load <= L.capacity;
            if (feasible || placed == 0 || iterations >= 2 * L.k + 4) return feasible;
            if (L.check) {
                st.status = kClusterCheck;
                return false;
            }
        }
    }
    // k_slack: free room per part, its saturating prefix sums and the least
    // positive room; also the excess of the overloaded parts.
    __device__ void receivers() {
        const int p = threadIdx.x, k = L.k;
        __syncthreads();
        if (p < kMaxParts) {
            const u64 load = p < k ? sm.load[p] : L.capacity;
            const u64 room = load < L.capacity ? L.capacity - load : 0;
            sm.slack[p] = room;
            sm.excess[p] = load > L.capacity ? load - L.capacity : 0;
            u64 inc = room, least = room ? room : ~0ULL;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const u64 o = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc = saturating_add(inc, o);
                const u64 m = __shfl_xor_sync(0xffffffffu, least, d);
                least = m < least ? m : least;
            }
            if (lane == 31) sm.scan[warp] = inc;
            if (lane == 0) sm.scan[8 + warp] = least;
            sm.cdf[p] = inc;
        }
        if (threadIdx.x == 0) sm.donors = 0;
        __syncthreads();
        if (p < kMaxParts) {
            u64 before = 0;
            for (int w = 0; w < warp; ++w) before = saturating_add(before, sm.scan[w]);
            const u64 c = saturating_add(before, sm.cdf[p]);
            if (p < k) sm.cdf[p] = c;
            if (rank == 0 && p < k) {
                L.slack[p] = sm.slack[p];
                L.requests[p] = 0;
            }
            if (p == 0) {
                u64 m = ~0ULL;
                for (int w = 0; w < kMaxParts / 32; ++w) m = sm.scan[8 + w] < m ? sm.scan[8 + w] : m;
                sm.cdf[k] = m;
            }
        }
        __syncthreads();
    }
    // k_repair_dest: the donors' plans and class weights, eight lanes a row.
    __device__ void destinations(u64* ctl) {
        constexpr int W = 8, G = 32 / W;
        const int gid = lane / W, sub = lane % W, k = L.k;
        const int span = (k + W - 1) / W;
        u32 donors = 0;
        for (i64 base = rank * kClusterThreads + warp * 32; base < L.n; base += kStep) {
            const int own = base + lane < L.n ? L.labels[base + lane] : -1;
            unsigned pending = __ballot_sync(0xffffffffu, own >= 0 && sm.excess[own < 0 ? 0 : own] != 0);
            donors += __popc(pending);
            while (pending) {
                unsigned mine = pending;
                for (int q = 0; q < gid; ++q) mine &= mine - 1;
                for (int q = 0; q < G; ++q) pending &= pending - 1;
                const bool valid = mine != 0;
                const int owner = valid ? __ffs(mine) - 1 : 0;
                const int v = static_cast<int>(base) + owner;
                const int src = __shfl_sync(0xffffffffu, own, owner);
                const u64 w = valid ? L.vw[v] : 0;
                const C* row = L.A + static_cast<i64>(v) * k;
                const u64 current = valid ? static_cast<u64>(row[src]) : 0;
                const bool scan = valid && current != static_cast<u64>(L.totals[v]);
                int part = -1;
                u64 conn = 0, best_room = 0;
                if (scan) {
                    for (int p0 = sub; p0 < k; p0 += 4 * W) {
                        C val[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) val[e] = p0 + e * W < k ? row[p0 + e * W] : C(0);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int p = p0 + e * W;
                            if (p >= k || p == src) continue;
                            const u64 room = sm.slack[p];
                            if (w > room) continue;
                            const u64 value = val[e];
                            if (part < 0 || value > conn || (value == conn && room > best_room)) { part = p; conn = value; best_room = room; }
                        }
                    }
                }
#pragma unroll
                for (int d = W / 2; d; d >>= 1) {
                    const int op = __shfl_xor_sync(0xffffffffu, part, d, W);
                    const u64 oc = __shfl_xor_sync(0xffffffffu, conn, d, W);
                    const u64 orm = __shfl_xor_sync(0xffffffffu, best_room, d, W);
                    if (op >= 0 && (part < 0 || oc > conn || (oc == conn && (orm > best_room || (orm == best_room && op < part))))) {
                        part = op; conn = oc; best_room = orm;
                    }
                }
                if (!conn) part = -1;
                const bool ticket = valid && part < 0 && w > sm.cdf[k];
                const u32 hash = mix32(static_cast<u32>(v));
                if (__any_sync(0xffffffffu, ticket)) part = ticket_part<W>(ticket, part, src, w, hash, sub, span);
                if (valid && sub == 0) {
                    if (part < 0 && !ticket) {
                        conn = 0;
                        const u64 sum = sm.cdf[k - 1];
                        if (sum) {
                            const u64 t = static_cast<u64>(hash) % sum;
                            int lo = 0, hi = k;
                            while (lo < hi) { const int mid = (lo + hi) / 2; if (sm.cdf[mid] <= t) lo = mid + 1; else hi = mid; }
                            part = lo;
                        }
                    }
                    if (ticket) conn = 0;
                    const u32 word = make_plan(v, part, conn, current, w, sm.excess[src]);
                    L.plan[v] = word;
                    if (part >= 0) atomicAdd(L.class_weights + src * kBalanceWidth + plan_class(word), w);
                }
            }
        }
        if (lane == 0 && donors) atomicAdd(&sm.donors, static_cast<u64>(donors));
        __syncthreads();
        if (threadIdx.x == 0 && sm.donors) atomicAdd(ctl + kCtlDonors, sm.donors);
    }
    // The fallback ticket of k_repair_dest over the room of the parts that fit w.
    template <int W>
    __device__ int ticket_part(bool ticket, int part, int src, u64 w, u32 hash, int sub, int span) const {
        const int lo = sub * span, hi = min(L.k, lo + span);
        u64 mine = 0;
        if (ticket)
            for (int p = lo; p < hi; ++p)
                if (p != src && w <= sm.slack[p]) mine = saturating_add(mine, sm.slack[p]);
        u64 upto = mine;
#pragma unroll
        for (int d = 1; d < W; d <<= 1) {
            const u64 o = __shfl_up_sync(0xffffffffu, upto, d, W);
            if (sub >= d) upto = saturating_add(upto, o);
        }
        const u64 total = __shfl_sync(0xffffffffu, upto, W - 1, W);
        const u64 prev = __shfl_up_sync(0xffffffffu, upto, 1, W);
        const u64 before = sub == 0 ? 0 : prev;
        int found = -1;
        if (ticket && total) {
            u64 t = static_cast<u64>(hash) % total;
            if (t >= before && (t - before) < mine) {
                t -= before;
                for (int p = lo; p < hi; ++p)
                    if (p != src && w <= sm.slack[p]) {
                        if (t < sm.slack[p]) { found = p; break; }
                        t -= sm.slack[p];
                    }
            }
        }
#pragma unroll
        for (int d = W / 2; d; d >>= 1) found = max(found, __shfl_xor_sync(0xffffffffu, found, d, W));
        return ticket ? found : part;
    }
    // k_repair_bounds, a warp per part.
    __device__ void bounds() {
        constexpr int kPer = kBalanceWidth / 32;
        static_assert(kPer * 32 == kBalanceWidth, "equal classes per lane");
        for (int p = rank * (kClusterThreads / 32) + warp; p < L.k; p += kStep / 32) {
            const u64 excess = sm.excess[p];
            if (!excess) {
                if (lane == 0) L.bound[p] = -1;
                continue;
            }
            u64* row = L.class_weights + static_cast<i64>(p) * kBalanceWidth + lane * kPer;
            u64 w[kPer], local = 0;
#pragma unroll
            for (int j = 0; j < kPer; ++j) w[j] = __ldcg(row + j);
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                if (w[j]) row[j] = 0;
                local += w[j];
            }
            u64 inc = local;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const u64 o = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += o;
            }
            u64 before = inc - local;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int c = lane * kPer + j;
                if (before < excess && (c == kBalanceWidth - 1 || before + w[j] >= excess)) {
                    L.bound[p] = c;
                    L.start[p] = before;
                }
                before += w[j];
            }
        }
    }
    // k_repair_list.
    __device__ void collect(u64* ctl) {
        for (int p = threadIdx.x; p < L.k; p += kClusterThreads) {
            sm.bound[p] = __ldcg(L.bound + p);
            sm.start[p] = sm.bound[p] >= 0 ? __ldcg(L.start + p) : 0;
        }
        __syncthreads();
        for (i64 base = rank * kClusterThreads + warp * 32; base < L.n; base += kStep) {
            const i64 v = base + lane;
            const int last = v < L.n ? sm.bound[L.labels[v]] : -1;
            const u32 word = last >= 0 ? L.plan[v] : kNoPlan;
            const bool take = word != kNoPlan && plan_class(word) <= last;
            const unsigned mask = __ballot_sync(0xffffffffu, take);
            if (!mask) continue;
            u64 at = 0;
            if (lane == 0) at = atomicAdd(ctl + kCtlListed, static_cast<u64>(__popc(mask)));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(mask & ((1u << lane) - 1u));
            if (take) L.list[at] = (static_cast<u64>(repair_hash(static_cast<int>(v))) << 32) | static_cast<u64>(v);
        }
    }
    // k_repair_block and the marking of its movers in the packed state.
    __device__ void reserve(int listed, u64* ctl) {
        const AttemptDonors<C> donor(raw + kAttemptCap * sizeof(u64), kAttemptCap);
        for (int p = threadIdx.x; p < L.k; p += kClusterThreads) {
            sm.attempt.slack[p] = sm.slack[p];
            sm.attempt.requests[p] = 0;
            sm.attempt.base[p] = sm.start[p];
        }
        if (threadIdx.x == 0) sm.placed = 0;
        const int count = order_donors<C, kClusterThreads>(sm.attempt, donor, reinterpret_cast<u64*>(raw), L.list, listed,
                                                           L.labels, L.vw, L.k, L.plan, sm.bound, sm.load, L.capacity,
                                                           sm.scan32);
        run_attempts<C, 8, kClusterThreads>(sm.attempt, donor, count, 0, L.A, L.off, L.nbr, L.ew, L.labels, L.k, L.plan,
                                            L.targets, L.flags);
        __syncthreads();
        for (int j = threadIdx.x; j < count; j += kClusterThreads) {
            if (donor.state[j] != 1) continue;
            const int v = static_cast<int>(donor.v[j]);
            L.flags[v] = 0;
            L.state[v] = static_cast<u32>(donor.src[j]) | (static_cast<u32>(L.targets[v]) << 8) | kMovingBit;
            L.movers[atomicAdd(&sm.placed, 1u)] = v;
        }
        __syncthreads();
        if (threadIdx.x == 0) ctl[kCtlPlaced] = sm.placed;
    }
};

template <class C>
constexpr size_t cluster_smem() { return repair_block_smem<C>(); }

template <class C>
__global__ void __launch_bounds__(kClusterThreads, 1) k_refine_cluster(const __grid_constant__ ClusterLevel<C> L) {
    after_previous();
    __shared__ ClusterShared<C> sm;
    extern __shared__ __align__(16) unsigned char cluster_raw[];
    ClusterRefiner<C>(L, sm, cluster_raw).run();
}

}  // namespace
}  // namespace gp
