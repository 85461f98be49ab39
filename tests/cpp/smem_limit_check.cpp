// Host check of the kernels' dynamic shared-memory limit (crd_b200/csrc/smem_limit.hpp): it never falls, whatever order
// and thread the sizes come from, and a refused size is not remembered. Prints "smem limit ok" and exits 0, or names the
// first broken case and exits 1.

#include "smem_limit.hpp"

#include <atomic>
#include <cstdio>
#include <thread>

int main()
{
    crdfft::SmemLimits limits;
    int a = 0, b = 0, now = 0;
    auto set = [&](int v) { return now = v, 0; };
    limits.raise(&a, 190000, set);
    limits.raise(&a, 60000, set);
    if (now != 190000)
        return std::printf("a smaller launch lowered the limit to %d\n", now), 1;
    limits.raise(&b, 60000, set);
    if (now != 60000)
        return std::printf("another kernel got %d\n", now), 1;
    if (limits.raise(&a, 300000, [](int) { return 1; }) != 1)
        return std::printf("a refusal was not reported\n"), 1;
    limits.raise(&a, 50000, set);
    if (now != 190000)
        return std::printf("after a refusal the limit is %d\n", now), 1;

    // Two threads, as two plans of one kernel: whenever a call returns, the limit holds its size.
    std::atomic<int> limit{0}, broken{0};
    auto launches = [&](int bytes) {
        for (int i = 0; i < 100000; ++i)
        {
            limits.raise(&limit, bytes, [&](int v) { return limit.store(v), 0; });
            if (limit.load() < bytes)
                broken.fetch_add(1);
        }
    };
    std::thread t(launches, 190000);
    launches(60000);
    t.join();
    if (broken.load() != 0)
        return std::printf("%d launches found a limit below their size\n", broken.load()), 1;
    std::printf("smem limit ok\n");
    return 0;
}
