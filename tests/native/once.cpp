#include "slq_once.h"

#include <thread>
#include <vector>

// setup calls per device: `threads` threads go over the devices `rounds`
// times, the first `fails` calls of a device fail
extern "C" void once_calls(int devices, int threads, int rounds, int fails, int* calls)
{
    slq::DeviceOnce once;
    std::vector<std::atomic<int>> n(devices);
    std::vector<std::thread> pool;
    for (int t = 0; t < threads; ++t)
        pool.emplace_back([&] {
            for (int r = 0; r < rounds; ++r)
                for (int d = 0; d < devices; ++d)
                    once(d, [&] { return ++n[d] <= fails ? 1 : 0; });
        });
    for (auto& t : pool) t.join();
    for (int d = 0; d < devices; ++d) calls[d] = n[d];
}
