// Which C2C kernel each plan candidate runs at 1024 and above, and the failures of the one-pass
// cluster route (its table's allocation, build and synchronisation, its launch), on the host runtime
// with direct_backend.cpp.
#include "backend.h"
#include "bfly/plan.hpp"

#include <cstdio>
#include <cstdlib>
#include <memory>
#include <string>
#include <vector>

namespace fake {
extern int allocations, releases, launches, syncs, failAllocation, failLaunch, failSync;
extern int lastE, lastCta, directTables;
extern uint32_t clusterUnavailable;
extern int longLaunches;
}  // namespace fake

#define CHECK(cond)                                                                    \
    do {                                                                               \
        if (!(cond)) {                                                                 \
            std::fprintf(stderr, "CHECK failed at %s:%d: %s\n", __FILE__, __LINE__, #cond); \
            std::exit(1);                                                              \
        }                                                                              \
    } while (0)

static std::unique_ptr<bfly::Plan> make(bfly::Context& context, uint32_t n, const std::string& id) {
    for (const bfly::Candidate& c : context.enumerate(n, 1))
        if (c.id == id) return c.state == bfly::State::Infeasible ? nullptr : context.makePlan(c);
    return nullptr;
}

int main(int argc, char** argv) {
    CHECK(argc == 2);
    const std::string cfg = argv[1];
    bfly::Context context;
    CHECK(context.init(cfg + "/b200_profile.json", cfg + "/b200_space.json", "builtin") == 0);
    std::vector<float> x(2 * 65536), y(2 * 65536);
    for (size_t i = 0; i < x.size(); ++i) x[i] = (float)(i % 7) - 3.f;

    auto runs = [&](const char* id, uint32_t planned, uint32_t n, int e, int cta) {
        auto p = make(context, planned, std::string(id) + "_shared_fp32_stockham");
        CHECK(p);
        fake::lastE = fake::lastCta = 0;
        CHECK(p->execC2C(x.data(), y.data(), n, 1, -1, 1.f, nullptr) == 0);
        CHECK(fake::lastE == e && (e == -3 || fake::lastCta == cta));
    };
    // every candidate that names a CTA size at 1024 runs it; r16 with 256 names the wide kernel
    runs("r8_cta128", 1024, 1024, 8, 128);
    runs("r8_cta256", 1024, 1024, 8, 256);
    runs("r8_cta512", 1024, 1024, 8, 512);
    runs("r16_cta128", 1024, 1024, 16, 128);
    runs("r16_cta512", 1024, 1024, 16, 512);
    runs("r16_cta256", 1024, 1024, 32, 64);
    runs("r16_cta256", 1024, 512, 16, 256);
    runs("r16_cta256", 1024, 2048, 16, 256);
    runs("r8_cta1024", 8192, 8192, 8, 1024);
    runs("r16_cta512", 8192, 8192, 32, 256);
    runs("r16_cta256", 1024, 8192, 32, 256);     // no variant of its own
    runs("r8_cta256", 1024, 8192, 32, 256);
    runs("r16_cta256", 1024, 32768, -3, 0);
    // a candidate without a kernel at 1024 is refused there, whatever it was made for
    for (const char* id : {"r8_cta1024_shared_fp32_stockham", "r16_cta1024_shared_fp32_stockham"}) {
        auto p = make(context, id[1] == '8' ? 8192 : 16384, id);
        CHECK(p && p->execC2C(x.data(), y.data(), 1024, 1, -1, 1.f, nullptr) == -8);
        CHECK(!make(context, 1024, id));
    }
    // no candidate of 32 values a thread, and no two of one length that run one kernel
    for (uint32_t n : {1024u, 8192u}) {
        std::vector<std::pair<int, int>> seen;
        for (const bfly::Candidate& c : context.enumerate(n, 1)) {
            CHECK(c.p.radix == 8 || c.p.radix == 16);
            if (c.state == bfly::State::Infeasible || c.f.schedule != "stockham") continue;
            auto p = context.makePlan(c);
            CHECK(p && p->execC2C(x.data(), y.data(), n, 1, -1, 1.f, nullptr) == 0);
            for (const auto& s : seen) CHECK(s != std::make_pair(fake::lastE, fake::lastCta));
            seen.push_back({fake::lastE, fake::lastCta});
        }
        CHECK(seen.size() == (n == 1024 ? 6u : 2u));
    }

    // the cluster route: one table per length, kept; every failure leaves nothing behind
    auto p = make(context, 1024, "r16_cta256_shared_fp32_stockham");
    CHECK(p);
    const auto call = [&](uint32_t n) { return p->execC2C(x.data(), y.data(), n, 1, 1, 0.5f, nullptr); };
    fake::failAllocation = fake::allocations + 1;
    CHECK(call(32768) == -2);
    fake::failAllocation = 0;
    int live = fake::allocations - fake::releases;
    fake::failLaunch = fake::launches + 1;   // the table's build
    CHECK(call(32768) == -2 && fake::allocations - fake::releases == live);
    fake::failLaunch = 0;
    fake::failSync = fake::syncs + 1;
    CHECK(call(32768) == -2 && fake::allocations - fake::releases == live);
    fake::failSync = 0;
    const int tables = fake::directTables;
    CHECK(call(32768) == 0 && fake::directTables == tables + 1 && fake::allocations - fake::releases == live + 1);
    CHECK(y[5] == -0.5f * x[5]);
    CHECK(call(32768) == 0 && fake::directTables == tables + 1 && fake::allocations - fake::releases == live + 1);
    fake::failLaunch = fake::launches + 1;
    CHECK(call(32768) == -5);
    fake::failLaunch = 0;
    CHECK(p->prepare(65536, 1) == 0 && fake::directTables == tables + 2);
    fake::lastE = 0;
    CHECK(p->runLong(x.data(), y.data(), 65536, 1, -1) == 0 && fake::lastE == -3 && y[7] == x[7]);
    CHECK(fake::directTables == tables + 2);
    // host requests of both kinds in one call
    std::vector<float> a(2 * 1024, 1.f), b(2 * 1024);
    const bfly::HostRequest reqs[2] = {{x.data(), y.data(), 65536, 1, 1, 2.f}, {a.data(), b.data(), 1024, 1, -1, 1.f}};
    CHECK(p->runMany(reqs, 2) == 0 && y[9] == -2.f * x[9] && b[0] == 1024.f);
    // a device that cannot hold the cluster of 65536: every entry takes the four-step kernels
    fake::clusterUnavailable = 65536;
    auto q = make(context, 1024, "r16_cta256_shared_fp32_stockham");
    CHECK(q);
    const int before = fake::directTables;
    for (int k = 0; k < 2; ++k) {
        fake::lastE = 0;
        if (k == 0) CHECK(q->execC2C(x.data(), y.data(), 65536, 1, -1, 1.f, nullptr) == 0);
        if (k == 1) CHECK(q->runLong(x.data(), y.data(), 65536, 1, -1) == 0 && q->runMany(reqs, 2) == 0);
        CHECK(fake::longLaunches > 0 && fake::lastE != -3 && fake::directTables == before);
        fake::longLaunches = 0;
    }
    CHECK(q->execC2C(x.data(), y.data(), 32768, 1, -1, 1.f, nullptr) == 0 && fake::lastE == -3);
    std::printf("all checks passed\n");
    return 0;
}
