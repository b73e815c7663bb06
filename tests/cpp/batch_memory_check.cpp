// The batch's host code on a stand-in for the CUDA runtime (fake_cudart.hpp):
// a batch whose curves' tables do not fit the device together runs all the
// same, the tables of some at a time.
#include <cstdio>
#include <cstdlib>
#include <exception>
#include <string>

#include "batch.hpp"
#include "fake_cudart.hpp"

using namespace rpg;

int main() {
    // six dense curves with launches of their own, 27 MB of tables each
    std::vector<BatchCurveSpec> curves(6);
    for (auto &c : curves) {
        c.coefficients = {"247747600", "-985905640", "567207969", "2396040466", "52485681", "-470135160", "82342800"};
        c.bound = 15'000;
        c.last = 400'000;
    }
    int wrong = 0;
    auto check = [&](const char *what, bool ok) {
        if (!ok) std::fprintf(stderr, "%s\n", what), ++wrong;
    };
    auto sieve_launches = [&](unsigned long long limit, const char *table_bytes) -> long long {
        fake::limit_allocations(limit);
        if (table_bytes) setenv("RPG_BATCH_TABLE_BYTES", table_bytes, 1);
        BatchStats stats;
        try {
            BatchEngine engine(0);
            engine.run(curves, &stats, false, false);
            engine.run(curves, &stats, false, true);
        } catch (const std::exception &e) {
            std::fprintf(stderr, "limit %llu: %s\n", limit, e.what());
            return -1;
        }
        release_pooled_engines(-1);
        unsetenv("RPG_BATCH_TABLE_BYTES");
        return (long long)stats.launches;
    };
    // three table launches per group, a sieve launch per curve, pre-verification
    check("one group", sieve_launches(~0ull, nullptr) == 3 + 6 + 1);
    check("groups by a limit", sieve_launches(~0ull, "60000000") == 3 * 3 + 6 + 1);
    check("a curve per group", sieve_launches(~0ull, "1") == 3 * 6 + 6 + 1);
    const long long small = sieve_launches(60'000'000, nullptr);
    check("groups where memory is short", small > 3 + 6 + 1 && small <= 3 * 6 + 6 + 1);
    fake::run_queued();
    check("stale sources", fake::stale_sources() == 0);
    if (!wrong) std::puts("all batches ran");
    return wrong ? 1 : 0;
}
