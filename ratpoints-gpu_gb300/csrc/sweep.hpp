// One curve's sweep: its plan, its device tables and the sieve kernel's
// launches, for the single-curve sieve (sieve.cu) and the batch (batch.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "plan.hpp"
#include "sweep_plan.hpp"

namespace rpg {

namespace dev {
struct SweepTables;
struct PatternJob;
struct TableJob;
struct ListJob;
}  // namespace dev

// One launch: parameters first .. last (below 2^31), numerators
// a_lo .. a_hi (at most SweepCurve::tile() of them).  Device pointers: the
// survivor arrays (curve tags only with out_curve), their count, a zeroed work
// counter, the error word, and (optional) the counts of swept words and of the
// row bytes they read.
struct SweepLaunch {
    long long first = 0, last = 0;
    long long a_lo = 0, a_hi = 0;
    long long *out_a = nullptr;
    int *out_d = nullptr;
    int *out_curve = nullptr;
    int curve = 0;
    unsigned long long capacity = 0;
    unsigned long long *out_count = nullptr;
    unsigned long long *work = nullptr;
    unsigned long long *error = nullptr;
    unsigned long long *swept = nullptr;
};

class SweepCurve {
public:
    // fast null: the reference plan.  denominators: about how many the search
    // has (0: not known), weighed against the tables' build.  row_bytes: most
    // bytes of the rows' tables (0: no limit).  Host only.
    SweepCurve(const std::vector<std::string> &coefficients, long long bound, bool square, const FastPlan *fast,
               double denominators, long long row_bytes = 0);
    // What the curve adds to SweepBuilder::bytes(), at most, and the most that any
    // curve adds under the fast plan.
    std::size_t bytes() const;
    static unsigned long long most_bytes(long long bound, std::size_t coefficients, long long row_bytes);
    ~SweepCurve();
    SweepCurve(const SweepCurve &) = delete;
    SweepCurve &operator=(const SweepCurve &) = delete;

    const SweepPlan &plan() const { return plan_; }
    // Modelled work of a pass over `denominators` of them (SM cycles).
    double cost(double denominators) const { return plan_.cost * denominators / double(need_); }
    // Most numerators of one launch.
    long long tile() const { return tile_; }
    // Words a pass over parameters first .. last sweeps (64 sites each).
    unsigned long long swept_words(long long first, long long last) const;
    // Enqueues a launch on the current device (its tables built by a
    // SweepBuilder on a stream this one has waited for).
    void launch(const SweepLaunch &l, cudaStream_t stream) const;

private:
    friend class SweepBuilder;
    long long bound_ = 0, tile_ = 0;
    bool square_ = false;
    SweepPlan plan_;
    std::size_t table_bytes_ = 0;   // rows, patterns, lists, counts
    std::size_t smem_ = 0;
    std::unique_ptr<dev::SweepTables> tables_;  // pointers set by SweepBuilder::place
    // build inputs, offsets from the curve's table block (rows, patterns,
    // lists) or from its input block (residues, maps)
    std::vector<dev::PatternJob> patterns_;
    std::vector<dev::TableJob> jobs_;
    std::unique_ptr<dev::ListJob> list_;
    std::vector<unsigned char> input_;
    std::size_t list2_at_ = 0, listq_at_ = 0, count2_at_ = 0, countq_at_ = 0, rows_at_ = 0;
    std::vector<int> count2_;               // admissible residues mod two by d mod two
    std::vector<std::vector<int>> countq_;  // per class prime p: by d mod p
    std::vector<int> bad_primes_;           // denominator primes
    unsigned long long need_ = 1;           // denominators without survivors unless it divides them
};

// Builds the tables of one or more curves in one device allocation.
class SweepBuilder {
public:
    SweepBuilder();
    ~SweepBuilder();
    void add(SweepCurve &curve);
    // Device bytes, the part uploaded from the host (at the end) included.
    std::size_t bytes() const;
    std::size_t upload_bytes() const { return blob_.size(); }
    // Sets the curves' table addresses in the allocation at `arena`, uploads
    // the inputs and, in enqueue, launches the builds.  The upload reads this
    // object's array when the stream gets to it: the object outlives that.
    void place(unsigned char *arena, cudaStream_t stream);
    void enqueue(cudaStream_t stream) const;
    bool empty() const { return curves_.empty(); }

private:
    std::vector<SweepCurve *> curves_;
    std::vector<std::size_t> at_;           // table block of each curve
    std::size_t size_ = 0;
    std::vector<unsigned char> blob_;
    std::size_t patterns_at_ = 0, tables_at_ = 0, lists_at_ = 0;
    int pattern_jobs_ = 0, table_jobs_ = 0, list_jobs_ = 0;
    unsigned table_blocks_ = 0, list_blocks_ = 0;
    unsigned char *arena_ = nullptr;
};

}  // namespace rpg
