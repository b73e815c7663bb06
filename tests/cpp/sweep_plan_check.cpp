// Host checks of the single-curve kernel's plans (csrc/plan.hpp, csrc/sweep.hpp),
// run by tests/test_sweep_plan_host.py.  Each argument is one check:
//   admitted H c0 c1 ..   the residue counts that a fast plan carries are those
//                         of its primes; prints the plan's primes and the
//                         swept words of denominators 1 .. 256
//   cost H c0 c1 ..       prints the modelled cost of the fast and the reference
//                         plan's sweep (SM cycles per denominator)
//   swept H last c0 ..    the words a batch's launch for denominators 1 .. last
//                         sweeps, in units of 16 words
//   memory H c0 c1 ..     a batch's admission estimate and table bytes for curves
//                         with launches of their own, by last denominator
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "batch.hpp"
#include "plan.hpp"
#include "sieve.hpp"
#include "sweep.hpp"

using namespace rpg;
using Coefficients = std::vector<std::string>;

static int admitted(long long bound, const Coefficients &f) {
    const FastPlan plan = single_curve_plan(f, bound, nullptr);
    int wrong = 0;
    for (const auto &a : plan.admitted) {
        std::printf("%d ", a.first);
        if (a.second != admitted_residues(a.first, f)) {
            std::fprintf(stderr, "prime %d: %d residues in the plan, %d admitted\n", a.first, a.second,
                         admitted_residues(a.first, f));
            ++wrong;
        }
    }
    const SweepCurve curve(f, bound, false, &plan, 0);
    std::printf("swept %llu\n", curve.swept_words(1, 256));
    return wrong;
}

static int cost(long long bound, const Coefficients &f) {
    const FastPlan plan = single_curve_plan(f, bound, nullptr);
    std::printf("%.6g %.6g\n", SweepCurve(f, bound, false, &plan, 1000).plan().cost,
                SweepCurve(f, bound, false, nullptr, 1000).plan().cost);
    return 0;
}

static int memory(long long bound, const Coefficients &f) {
    BatchCurveSpec c;
    c.coefficients = f;
    c.bound = bound;
    const double words = double(word_count64(bound));
    for (long long last : {1LL, 20LL, 1'000LL, 30'000LL, 400'000LL, 5'000'000LL, 2'000'000'000LL}) {
        c.last = last;
        // the batch's rule: rows of 2,048 words, or shorter ones with much work
        if (words < double(kBatchWideWords) && double(last) * (2.8e-3 * words - 0.9) <= 20000.0) continue;
        std::unique_ptr<SweepCurve> curve = batch_sweep_curve(c);
        SweepBuilder builder;
        builder.add(*curve);
        std::printf("%lld %llu ", last, (unsigned long long)builder.bytes());
        c.intervals.clear();
        std::printf("%llu ", BatchEngine::estimate_bytes(c));
        c.intervals.resize(9);  // more than the device takes: the whole row
        for (auto &i : c.intervals) i.lower_infinite = i.upper_infinite = true;
        std::printf("%llu\n", BatchEngine::estimate_bytes(c));
        c.intervals.clear();
    }
    return 0;
}

static int swept(long long bound, long long last, const Coefficients &f) {
    BatchCurveSpec c;
    c.coefficients = f;
    c.bound = bound;
    c.last = last;
    const std::unique_ptr<SweepCurve> curve = batch_sweep_curve(c);
    const long long words = sweep_words(bound, (long long)curve->plan().two * curve->plan().q);
    std::printf("%llu\n", curve->swept_words(1, last) / (unsigned long long)words *
                              (unsigned long long)((words + kSweepUnit - 1) / kSweepUnit * kSweepUnit));
    return 0;
}

int main(int argc, char **argv) {
    if (argc < 5) return 2;
    const long long bound = std::atoll(argv[2]);
    const Coefficients f(argv + 3, argv + argc);
    if (!std::strcmp(argv[1], "admitted")) return admitted(bound, f) ? 1 : 0;
    if (!std::strcmp(argv[1], "memory")) return memory(bound, f);
    if (!std::strcmp(argv[1], "swept")) return swept(bound, std::atoll(argv[3]), Coefficients(argv + 4, argv + argc));
    if (!std::strcmp(argv[1], "cost")) return cost(bound, f);
    return 2;
}
