// Kept hierarchies of resident graphs (see gp_internal.h).  An entry owns the
// arena its levels live in; entries in use by a call are never dropped.
#pragma once
#include "gp_graph.h"

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <utility>
#include <vector>

namespace gp {

struct HierarchyCache {
    struct Key {
        uint64_t graph;
        int k;
        uint32_t seed, flags;
        bool operator<(const Key& o) const {
            return std::tie(graph, k, seed, flags) < std::tie(o.graph, o.k, o.seed, o.flags);
        }
    };
    struct Entry {
        Arena storage;
        Hierarchy h;
        u64 total = 0, directed = 0;
        int users = 0;
        u64 last_use = 0;
        // Recorded behind the kernels that wrote the levels, which may still
        // run when the entry is published: a call on another stream waits for
        // it on its own stream.
        cudaEvent_t built = nullptr;
        Entry() = default;
        Entry(const Entry&) = delete;
        Entry& operator=(const Entry&) = delete;
        ~Entry() { if (built) cudaEventDestroy(built); }
    };
    int device = 0;
    uint64_t budget = 0;
    std::mutex mu;
    std::map<Key, std::unique_ptr<Entry>> entries;
    u64 clock = 0;

    // The kept entry, in use by the caller, whose work on `stream` comes after
    // what built the entry; nullptr when there is none.
    Entry* find(const Key& key, cudaStream_t stream) {
        std::lock_guard<std::mutex> lock(mu);
        auto it = entries.find(key);
        if (it == entries.end()) return nullptr;
        GP_CUDA(cudaStreamWaitEvent(stream, it->second->built, 0));
        ++it->second->users;
        it->second->last_use = ++clock;
        return it->second.get();
    }
    // Keeps a complete `fresh` entry, in use by the caller and built by the
    // work enqueued on `stream`, and drops least recently used idle entries
    // while the total exceeds the budget.  When another call kept the same key
    // first, `fresh` is still the caller's and is freed at its release.
    // Returns the caller's entry.
    Entry* insert(const Key& key, std::unique_ptr<Entry> fresh, cudaStream_t stream) {
        GP_CUDA(cudaEventCreateWithFlags(&fresh->built, cudaEventDisableTiming));
        GP_CUDA(cudaEventRecord(fresh->built, stream));
        std::lock_guard<std::mutex> lock(mu);
        fresh->users = 1;
        fresh->last_use = ++clock;
        Entry* out = fresh.get();
        if (entries.count(key)) retired.push_back(std::move(fresh));
        else entries.emplace(key, std::move(fresh));
        evict();
        return out;
    }
    void release(Entry* e) {
        std::lock_guard<std::mutex> lock(mu);
        --e->users;
        evict();
        free_retired();
    }
    uint64_t bytes() const {
        uint64_t b = 0;
        for (auto& kv : entries) b += kv.second->storage.reserved();
        return b;
    }

private:
    std::vector<std::unique_ptr<Entry>> retired;  // duplicates, freed once idle
    void evict() {
        while (bytes() > budget) {
            auto victim = entries.end();
            for (auto it = entries.begin(); it != entries.end(); ++it)
                if (!it->second->users && (victim == entries.end() || it->second->last_use < victim->second->last_use))
                    victim = it;
            if (victim == entries.end()) break;  // everything is in use
            cudaSetDevice(device);
            entries.erase(victim);
        }
    }
    void free_retired() {
        for (auto& e : retired) if (e && !e->users) { cudaSetDevice(device); e.reset(); }
        retired.erase(std::remove(retired.begin(), retired.end(), nullptr), retired.end());
    }
};

}  // namespace gp
