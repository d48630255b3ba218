// A resident graph's arrays have arrived on every device when the server
// hands out the graph's id: the workers' streams do not wait for the copies.
#include "../../acc-gp_b200/csrc/gp_batch.cpp"
#include "fake_runtime.h"

struct gp_context {};

namespace gp {
void set_error(const std::string&) {}
const char* last_error() { return ""; }
gp_status validate_host_csr(const gp_csr*, bool) { return GP_OK; }
WorkerPool*& worker_pool(gp_context*) { static WorkerPool* none = nullptr; return none; }
int context_device(const gp_context*) { return 0; }
size_t context_reserved(const gp_context*) { return 0; }
void context_trim(gp_context*) {}
void copy_options(const gp_context*, gp_context*) {}
HierarchyCache* hierarchy_cache_create(int, uint64_t) { return nullptr; }
void hierarchy_cache_destroy(HierarchyCache*) {}
uint64_t hierarchy_cache_bytes(const HierarchyCache*) { return 0; }
gp_status partition_resident(gp_context*, HierarchyCache*, uint64_t, const gp_csr*, int32_t, double, uint32_t, uint32_t,
                             int32_t*, gp_stats*) { return GP_OK; }
}  // namespace gp
extern "C" {
gp_status gp_context_create(int, gp_context** out) { *out = new gp_context; return GP_OK; }
void gp_context_destroy(gp_context* c) { delete c; }
gp_status gp_partition(gp_context*, const gp_csr*, int32_t, double, uint32_t, uint32_t, int32_t*, gp_stats*) { return GP_OK; }
gp_status gp_partition_device(gp_context*, const gp_csr*, int32_t, double, uint32_t, uint32_t, int32_t*, void*, gp_stats*) {
    return GP_OK;
}
}

int main() {
    const int32_t offsets[4] = {0, 1, 2, 2}, neighbors[2] = {1, 0}, devices[2] = {0, 1};
    const uint32_t weights[3] = {1, 2, 3};
    const gp_csr graph{3, 2, offsets, neighbors, weights, nullptr};
    gp_server* server = nullptr;
    EXPECT(gp_server_create_devices(devices, 2, 1, 0, &server) == GP_OK);
    int32_t id = -1;
    calls.clear();
    EXPECT(gp_server_add_graph(server, &graph, &id) == GP_OK && id == 0);
    int copies = 0, waits = 0;
    for (const Call& c : calls) {
        if (c.name == "copy") ++copies;
        if (c.name == "synchronize") {
            ++waits;
            EXPECT(c.stream == nullptr && copies == 3 * waits);
        }
    }
    EXPECT(copies == 6 && waits == 2);
    runtime.synchronize = cudaErrorUnknown;
    runtime.last = cudaErrorUnknown;
    EXPECT(gp_server_add_graph(server, &graph, &id) != GP_OK && runtime.last == cudaSuccess);
    gp_server_destroy(server);
    return 0;
}
