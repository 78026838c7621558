// The shared-memory limits of sp3mm4amg_b200/csrc/smem_limit.h with a fake
// setter: a limit never shrinks, a failed setting is reported and not
// recorded, and with 8 threads the limit that a thread's launch would find is
// never below what that thread asked for.
#include "smem_limit.h"

#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

static std::atomic<size_t> g_limit[3];

struct FakeSet {
    int operator()(const void* f, size_t bytes) const {
        if (bytes > 1000) return 1;
        g_limit[reinterpret_cast<size_t>(f)].store(bytes);
        return 0;
    }
};

#define CHECK(x)                                                \
    do {                                                        \
        if (!(x)) {                                             \
            std::printf("failed: %s (line %d)\n", #x, __LINE__); \
            return 1;                                           \
        }                                                       \
    } while (0)

int main() {
    sp3mm::SmemLimits<FakeSet> L{FakeSet{}};
    const void* f1 = reinterpret_cast<const void*>(1);
    const void* f2 = reinterpret_cast<const void*>(2);
    CHECK(L.need(0, f1, 100) == 0 && g_limit[1] == 100);
    CHECK(L.need(0, f1, 60) == 0 && g_limit[1] == 100);
    CHECK(L.need(0, f2, 50) == 0 && g_limit[2] == 50 && g_limit[1] == 100);
    CHECK(L.need(0, f1, 2000) == 1 && g_limit[1] == 100);   // refused
    CHECK(L.need(0, f1, 70) == 0 && g_limit[1] == 100);
    g_limit[1] = 0;                                         // forgotten limits are set again
    CHECK(L.need(0, f1, 70) == 0 && g_limit[1] == 100);
    CHECK(L.need(1, f1, 40) == 0 && g_limit[1] == 40);      // per device

    sp3mm::SmemLimits<FakeSet> T{FakeSet{}};
    g_limit[1] = 0;
    std::atomic<int> low{0};
    std::vector<std::thread> th;
    for (int t = 0; t < 8; ++t)
        th.emplace_back([&, t] {
            for (int i = 0; i < 200000; ++i) {
                const size_t want = 100 + (t * 131 + i * 17) % 800;
                if (T.need(0, f1, want) != 0 || g_limit[1].load() < want) low.fetch_add(1);
            }
        });
    for (auto& t : th) t.join();
    CHECK(low.load() == 0);
    std::printf("ok\n");
    return 0;
}
