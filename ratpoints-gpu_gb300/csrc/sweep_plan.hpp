// How the sieve kernel executes a plan: which primes become numerator
// classes, which become stage-1 rows, which are tested last.
//
// A plan (reference or fast, plan.hpp) fixes the tests a survivor passes, so
// any split of those tests gives the same survivors.  The kernel sweeps
// numerator classes a = r (mod two * Q), Q the product of the class primes:
// a class prime halves the swept words (only its admissible residues are
// swept) but shortens the classes, which must keep about 1,024 sites (16
// words of 64) to fill a half-warp.  Rows cost shared-memory reads per swept
// word and their copy per denominator; fewer rows let more words through to
// stage 2.  The split is the cheapest under a cost model of the kernel, in SM
// cycles per denominator.
#pragma once

#include <vector>

namespace rpg {

constexpr int kSweepRows = 12;            // stage-1 rows (at most)
constexpr int kSweepRowFactors = 4;       // primes per row
constexpr int kSweepUnit = 16;            // class words per half-warp
constexpr int kSweepSlots = 4;            // denominators in flight per CTA (at most)
constexpr int kSweepClassPrimes = 4;      // class primes (at most)
constexpr int kSweepMaxClasses = 640;     // admissible residues mod Q of one denominator (at most)
constexpr long long kSweepListBytes = 32; // bytes of a class-list entry

struct SweepPrime {
    int p = 0;
    int admitted = 0;       // residues x with f(x) a square mod p (at least one)
    int divided = 0;        // residues admitted where p | d
    bool optional = false;  // stage 2 tests it as well: it may be left out before
};

struct SweepInput {
    long long bound = 0;
    double denominators = 0;  // about how many the search has (0: not known)
    int two = 0;            // power of two whose classes the plan filters (0: no such filter, any may be used)
    double two_classes = 1; // mean classes mod two of a denominator that has any
    int two_max = 1;        // most of them
    std::vector<SweepPrime> primes;
    long long row_bytes = 0;  // most bytes of the rows' tables (0: no limit)
};

struct SweepPlan {
    int two = 1;                             // classes mod two * Q
    std::vector<int> class_primes;           // factors of Q
    int q = 1;                               // Q
    int two_max = 1;                         // most residues mod two of one denominator
    int q_max = 1;                           // most admissible residues mod Q of one denominator
    std::vector<std::vector<int>> rows;      // primes of each stage-1 row
    std::vector<int> moduli;                 // their products
    std::vector<int> late;                   // the plan's primes left for after stage 2
    int pairs = 1;                           // pairs of units an item sweeps side by side (1 or 2)
    int ctas = 2;                            // CTAs per SM
    int slots = 2;                           // denominators in flight per CTA
    int split = 0;                           // an item's residues mod two: 2^-split of the denominator's
    double cost = 0;                         // modelled SM cycles per denominator
};

// Staged words of a row: two periods (the sum of two offsets below m needs no
// wrap) and the 15 words a half-warp reads past its start.
constexpr int sweep_row_words(int m) { return 2 * m + kSweepUnit; }

// Class words of a class over numerators -H .. H for class modulus `mod`
// (a class may start one step before -H, see sieve_fast.cuh).
constexpr long long sweep_words(long long bound, long long mod) { return ((2 * bound + mod) / mod >> 6) + 1; }

// The kernel runs 24 warps per SM in two, three or four CTAs, one warp of each
// producing: more CTAs hand more denominators over at a time, fewer have room
// for more or longer rows.  Shared memory of a CTA: slots, the consumers'
// queues, and static arrays.
constexpr int kSweepWarps = 24;
constexpr int kSweepQueue = 64;                        // queued words per consumer warp
constexpr long long kSweepQueueBytes = 20 * kSweepQueue;
constexpr long long sweep_cta_bytes(int ctas) { return 228 * 1024 / ctas - 1024 - 4096; }
// A slot holds its denominator's lists as well, the one by d mod Q only up to
// kSweepSlotClasses entries; longer ones are read from L2 (an item reads one
// entry per half-warp for all its steps).
constexpr int kSweepSlotClasses = 64;
constexpr long long sweep_slot_bytes(long long row_words, int two_max, int q_max) {
    return row_words * 8 + kSweepListBytes * two_max + (q_max <= kSweepSlotClasses ? kSweepListBytes * q_max : 0);
}

SweepPlan plan_sweep(const SweepInput &in);

}  // namespace rpg
