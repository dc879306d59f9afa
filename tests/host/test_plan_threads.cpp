// Threads that share one plan through the C ABI, each with the first use of lengths the others use too:
// run under the thread sanitizer, which reports any access of a plan's tables that is not ordered.
#include "bfly_b200.h"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <thread>
#include <vector>

int main(int argc, char** argv) {
    if (argc != 2) return 2;
    const std::string cfg = argv[1];
    bfly_context* ctx = nullptr;
    bfly_plan* plan = nullptr;
    if (bfly_context_create(&ctx) ||
        bfly_context_init(ctx, (cfg + "/b200_profile.json").c_str(), (cfg + "/b200_space.json").c_str(), "builtin") ||
        bfly_context_make_plan(ctx, 1024, 1, "r16_cta256_shared_fp32_stockham", &plan))
        return 3;
    const uint32_t lengths[] = {64, 128, 256, 60, 48, 37, 100, 512};
    std::vector<std::thread> threads;
    std::vector<int> bad(3, 0);
    std::atomic<int> waiting{3};
    for (int k = 0; k < 3; ++k)
        threads.emplace_back([&, k] {
            std::vector<float> x(2 * 1024, 1.f), y(2 * 1024);
            --waiting;
            while (waiting) std::this_thread::yield();   // every first use at once
            for (int round = 0; round < 2; ++round)
                for (uint32_t n : lengths) {
                    bad[k] += bfly_plan_exec_c2c_async(plan, x.data(), y.data(), n, 1, -1, 1.f, nullptr) != 0;
                    bad[k] += y[0] != (float)n;
                }
            uint64_t frames = 0;
            bad[k] += bfly_plan_exec_stft_async(plan, x.data(), y.data(), 64, 1, 128, 64, 0, nullptr, &frames, nullptr) != 0;
        });
    for (auto& t : threads) t.join();
    bfly_plan_destroy(plan);
    bfly_context_destroy(ctx);
    for (int b : bad)
        if (b) return 4;
    std::printf("all checks passed\n");
    return 0;
}
