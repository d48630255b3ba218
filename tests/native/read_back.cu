// A read-back that has to wait leaves no error behind, a failed stream ends
// it, it blocks where the program chose so, and a kernel that did not start
// fails its launch.
#include "../../acc-gp_b200/csrc/gp_graph.h"
#include "fake_runtime.h"

namespace gp {
thread_local u64 g_launches = 0;
thread_local KernelProfiler* g_profiler = nullptr;
bool KernelProfiler::matches(const void*) { return false; }
void KernelProfiler::before(cudaStream_t) {}
void KernelProfiler::after(cudaStream_t) {}
void publish(cudaStream_t s, const u64*, u64*, int, u64*, u64) { calls.push_back({"publish", s, nullptr}); }
}  // namespace gp

using namespace gp;

static void kernel(int) {}

template <class F>
static bool throws(F&& f) {
    try {
        f();
    } catch (const Failure&) {
        return true;
    }
    return false;
}

int main() {
    std::vector<u64> words(kScalars + 1, 0);
    Context ctx;
    ctx.stream = stream(3);
    ctx.host_scalars = words.data();
    auto arrive = [&] { words[kScalars] = ctx.fetched; };

    // Not ready three times, as an error that the runtime keeps; the next launch does not report it.
    int queries = 0;
    runtime.query = [&] {
        if (++queries == 3) arrive();
        return cudaErrorNotReady;
    };
    EXPECT(ctx.fetch(nullptr, 1, 7) == words.data() + 7);
    EXPECT(queries == 3 && runtime.last == cudaSuccess);
    EXPECT(!throws([&] { launch(kernel, 1, 32, 0, stream(3), 5); }));

    // The stream is done but the number is not seen: its work has ended, so the words are there.
    runtime.query = [] { return cudaSuccess; };
    EXPECT(!throws([&] { ctx.fetch(nullptr, 1); }));

    // A failed stream ends the wait.
    runtime.query = [] { return cudaErrorLaunchFailure; };
    EXPECT(throws([&] { ctx.fetch(nullptr, 1); }) && runtime.last == cudaSuccess);

    // A program that chose to block: no polling, and errors as before.
    for (unsigned how : {cudaDeviceScheduleSpin, cudaDeviceScheduleYield, cudaDeviceScheduleBlockingSync}) {
        runtime.flags = how | cudaDeviceMapHost;
        runtime.query = [&] { arrive(); return cudaErrorNotReady; };
        calls.clear();
        EXPECT(!throws([&] { ctx.fetch(nullptr, 1); }));
        EXPECT(calls.size() == 2 && calls[0].name == "publish" && calls[1].stream == stream(3));
        EXPECT(calls[1].name == (how == cudaDeviceScheduleBlockingSync ? "synchronize" : "query"));
    }
    runtime.synchronize = cudaErrorLaunchFailure;
    EXPECT(throws([&] { ctx.fetch(nullptr, 1); }));
    runtime.flags = cudaDeviceScheduleAuto;

    // A launch that returns an error fails, whether or not the runtime keeps it as the last one.
    runtime.launch = cudaErrorInvalidConfiguration;
    EXPECT(throws([&] { launch(kernel, 1, 32, 0, stream(3), 5); }));
    runtime.last = cudaErrorInvalidConfiguration;
    EXPECT(throws([&] { launch(kernel, 1, 32, 0, stream(3), 5); }) && runtime.last == cudaSuccess);
    runtime.launch = cudaSuccess;
    EXPECT(!throws([&] { launch(kernel, 1, 32, 0, stream(3), 5); }));
    return 0;
}
