// The library's host code on a stand-in for the CUDA runtime (fake_cudart.hpp):
// the sources of its asynchronous uploads stay as they are until the streams
// have read them, in searches, sieves and batches, whichever launch fails.
#include <cstdio>
#include <exception>
#include <functional>

#include "batch.hpp"
#include "fake_cudart.hpp"
#include "search.hpp"
#include "sieve.hpp"

using namespace rpg;

int main() {
    const std::vector<std::string> sextic = {"-533746463", "2318474698", "1819918790", "-3268433658",
                                             "1978982371", "1087269120", "-559365050"};
    const std::vector<std::string> quintic = {"9", "1", "-7", "0", "3", "2"};
    auto spec = [](const std::vector<std::string> &f, long long bound, long long last, bool interval = false) {
        BatchCurveSpec c;
        c.coefficients = f;
        c.bound = bound;
        c.last = last;
        if (interval) {
            SearchInterval i;
            std::string error;
            parse_real("-0.5", "lower", i.lower, error);
            parse_real("2", "upper", i.upper, error);
            c.intervals = {i};
        }
        return c;
    };
    // narrow rows, launches of a curve's own, wide rows in an interval
    const std::vector<BatchCurveSpec> curves = {spec(sextic, 900, 60), spec(quintic, 80'000, 50),
                                                spec(sextic, 200'000, 40), spec(quintic, 80'000, 5'000, true)};
    auto sieve = [&](PlanKind plan, bool preverify) {
        SieveOptions o;
        o.plan = plan;
        o.preverify = preverify;
        Sieve s(sextic, 100'000, o);
        s.start(1, 1000, 100);
        BatchView view;
        while (s.next(view)) {}
    };
    const std::vector<std::function<void()>> calls = {
        [&] {
            SieveOptions o;
            o.plan = PlanKind::fast;
            o.preverify = true;
            Sieve s(sextic, 100'000, o);  // and gone before the streams have done anything
        },
        [&] { sieve(PlanKind::fast, true); },
        [&] { sieve(PlanKind::reference, false); },
        [&] {
            BatchEngine engine(0);
            engine.run(curves, nullptr, false, true);
            engine.run({curves[2], curves[0]}, nullptr, false, true);
        },
        [&] {  // an engine used again after a failed run
            BatchEngine engine(0);
            for (int i = 0; i < 2; ++i) try {
                    engine.run(curves, nullptr, false, i == 0);
                } catch (const std::exception &) {
                }
        },
    };
    int wrong = 0;
    for (std::size_t k = 0; k < calls.size(); ++k) {
        for (long long n = 0;; ++n) {
            fake::fail_launch(0);
            const long long before = fake::launches();
            fake::fail_launch(n);
            try {
                calls[k]();
            } catch (const std::exception &) {
            }
            fake::fail_launch(0);
            const bool failed = n > 0 && n <= fake::launches() - before;
            fake::run_queued();
            if (const long long stale = fake::stale_sources(); stale > wrong) {
                std::fprintf(stderr, "call %zu, launch %lld failing: %lld stale sources\n", k, n, stale - wrong);
                wrong = int(stale);
            }
            if (n > 0 && !failed) break;
        }
    }
    if (!wrong) std::puts("all sources kept");
    return wrong ? 1 : 0;
}
