// A kept hierarchy is published while the kernels that write its last level
// may still run on the stream that built it: a call that finds it has to wait
// on its own stream for an event recorded there.
#include "../../acc-gp_b200/csrc/gp_hierarchy_cache.h"
#include "fake_runtime.h"

int main() {
    gp::HierarchyCache cache;
    cache.budget = 1 << 30;
    const gp::HierarchyCache::Key key{1, 8, 0, 0};
    EXPECT(!cache.find(key, stream(1)) && calls.empty());
    auto* mine = cache.insert(key, std::make_unique<gp::HierarchyCache::Entry>(), stream(1));
    EXPECT(calls.size() == 1 && calls[0].name == "record" && calls[0].stream == stream(1));
    // Found by two other calls while its maker still uses it.
    for (size_t other : {2, 3}) {
        EXPECT(cache.find(key, stream(other)) == mine);
        EXPECT(calls.back().name == "wait" && calls.back().stream == stream(other) && calls.back().object == calls[0].object);
    }
    EXPECT(calls.size() == 3 && mine->users == 3);
    // A second maker of the same key keeps its own copy to itself.
    auto* second = cache.insert(key, std::make_unique<gp::HierarchyCache::Entry>(), stream(4));
    EXPECT(second != mine && calls.back().name == "record" && calls.back().stream == stream(4));
    EXPECT(cache.find(key, stream(5)) == mine && calls.back().object == calls[0].object);
    cache.release(second);
    for (int i = 0; i < 4; ++i) cache.release(mine);
    EXPECT(cache.entries.size() == 1 && mine->users == 0);
    return 0;
}
