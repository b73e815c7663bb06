// The tuner of the fast plan on a stand-in for the CUDA runtime
// (fake_cudart.hpp): it times each set of tested primes once.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "fake_cudart.hpp"
#include "plan.hpp"
#include "sieve.hpp"
#include "tune.hpp"

using namespace rpg;

int main(int argc, char **argv) {
    if (argc < 4) return 2;
    const long long bound = std::atoll(argv[1]);
    const std::vector<std::string> f(argv + 2, argv + argc);
    const TuneResult r = tune_fast_shape(f, bound, 1, 100, false, 0, 100);
    std::vector<std::vector<int>> sets;
    for (const auto &c : r.candidates) {
        const FastPlan plan = single_curve_plan(f, bound, nullptr, c.shape);
        std::vector<int> primes{plan.class_prime};
        for (const auto &slot : plan.slots) primes.insert(primes.end(), slot.begin(), slot.end());
        std::sort(primes.begin(), primes.end());
        sets.push_back(primes);
    }
    std::sort(sets.begin(), sets.end());
    const bool distinct = std::adjacent_find(sets.begin(), sets.end()) == sets.end();
    std::printf("%zu candidates, %s\n", sets.size(), distinct ? "distinct" : "some alike");
    return distinct && sets.size() >= 3 ? 0 : 1;
}
