// Host driver of the device sieve: builds the per-curve tables on the GPU,
// launches the sieve over consecutive denominator batches on a CUDA stream,
// and hands each batch's survivors to the caller while later batches run.
//
// It replaces the reference's run_modular_sieve driver (src/sieve.cu:503-580):
// tables are built once per search instead of once per batch, device buffers
// are allocated once, survivor copies go through pinned memory, and up to two
// batches are in flight so host verification overlaps device work.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

namespace rpg {

enum class PlanKind : int { reference = 0, fast = 1 };

class CudaError : public std::runtime_error {
public:
    using std::runtime_error::runtime_error;
};

// A bounded wait inside a sieve kernel ran out; the launch's output is invalid.
class DeviceTimeout : public std::runtime_error {
public:
    using std::runtime_error::runtime_error;
};

void check_cuda(cudaError_t status, const char *what);

// Shape of a fast plan: how many rows its primes are packed into, and whether
// within the shared memory of two or three sets of them.  It selects the primes
// that survivors pass; which rows the kernel stages, and in how many slots, is
// the sweep plan's choice (sweep_plan.hpp).  rows 0: the cost model's choice.
struct FastShape {
    int rows = 0;
    int slots = 0;
};

struct SieveOptions {
    PlanKind plan = PlanKind::reference;
    bool square = false;            // parameters k give denominators k*k
    long long capacity = 1 << 22;   // survivors per device buffer
    int device = -1;                // -1: current device
    double denominators = 0;        // about how many the search has (0: not known)
    // Drop survivors that cannot be points on the device before the copy
    // (gcd and residue tests; see preverify.hpp).  Deliveries then hold a
    // subset of the modular survivors that still contains every point.
    bool preverify = false;
    // Fast plan only: a forced shape (rows > 0); otherwise a shape measured
    // earlier for curves of this kind (tune.hpp), when the tuning cache is
    // enabled and holds one, else the cost model's.
    FastShape fast_shape;
};

// One delivery of survivors.  Pointers stay valid until the next call to
// Sieve::next().  A batch whose survivors exceed one buffer arrives in several
// pieces; complete marks its last piece.
struct BatchView {
    long long first = 0, last = 0;   // parameter range of the batch
    const long long *a = nullptr;
    const int *d = nullptr;
    std::size_t count = 0;
    std::size_t modular = 0;         // modular survivors behind this piece (count, unless pre-verified)
    bool complete = true;
    float kernel_ms = 0.0f;          // event time of the launches behind this piece
};

struct SieveTimings {
    float table_ms = 0.0f;           // device table build (events)
    double table_wall_ms = 0.0;      // host + device table setup
    double plan_ms = 0.0;            // host plan work
    double workspace_ms = 0.0;       // allocations
    double sieve_ms = 0.0;           // sum of sieve launch event times
    unsigned long long launches = 0;
    unsigned long long reruns = 0;   // overflowed launches that were split
    unsigned long long h2d_bytes = 0;
    unsigned long long d2h_bytes = 0;
};

// cudaMalloc; before it fails for want of memory, what finished searches left
// for reuse is freed.
void *device_malloc(std::size_t bytes, const char *what);

// Frees the idle search pipelines (streams, events, survivor buffers, pinned
// staging, table memory) that finished sieves left for reuse on `device` (-1: every
// device).  A process that resets a device must call it first.
void release_pooled_pipelines(int device);

// The fast plan a single-curve sieve uses for a curve and numerator bound
// (host only): the autotuner's choice of primes; *max_classes (optional)
// receives the most classes of one denominator mod 64 times the class prime.
// A shape with rows > 0 fixes the row count (the rows filtering most) and the
// row sets instead of the cost model.
struct FastPlan;
FastPlan single_curve_plan(const std::vector<std::string> &coefficients, long long bound, int *max_classes,
                           FastShape shape = FastShape{});

// The fast plan a sieve chose for its curve (empty for the reference plan): the
// primes its survivors pass, wherever the sweep plan has them tested.
struct FastPlanInfo {
    int class_prime = 0;           // 1: none
    std::vector<int> primes;       // the others
    std::vector<int> moduli;       // their products that the planner packed them into
};

class Sieve {
public:
    Sieve(const std::vector<std::string> &coefficients, long long bound, const SieveOptions &options);
    ~Sieve();
    Sieve(const Sieve &) = delete;
    Sieve &operator=(const Sieve &) = delete;

    // Queue parameters [first, last] as consecutive batches of batch_size.
    void start(long long first, long long last, long long batch_size);
    // Waits for the table build, which runs on the sieve's own stream beside
    // the host; needed before launches on any other stream.
    void wait_tables() const;
    // Next piece in parameter order; false when every queued batch is delivered.
    bool next(BatchView &out);
    // Drop queued and in-flight work (e.g. after a first-point stop).
    void cancel();

    const SieveTimings &timings() const;
    long long words64() const;

    // Device-resident pass for benchmarks: sieve [first, last] in batches with
    // survivors counted on the device only; returns the survivor count.  The
    // caller times it with the events it records on stream().
    unsigned long long count_only(long long first, long long last, long long batch_size);
    cudaStream_t stream() const;

    // Work of a pass over parameters [first, last]: 64-site words swept by the
    // sieve kernel and shared-memory bytes read per swept word (stage 1).
    unsigned long long swept_words(long long first, long long last) const;
    unsigned smem_bytes_per_word() const;
    FastPlanInfo fast_plan_info() const;

    // Whether allocation-free launches take the rows: false only for very large
    // H (fast plan: more than 2^23 words of a class mod 64 q, q the plan's class
    // prime, reference plan: more than 2^30 words).
    bool allocation_free_rows() const;
    // Enqueue the sieve (one launch for nearly every curve) for parameters [first, last] (at most one batch
    // of 65536) on `stream`, writing survivors into caller-owned device arrays
    // and counting them in *out_count; `work` is a zeroed device counter the
    // launch uses for dynamic scheduling, and *error (a device word) becomes
    // nonzero if a bounded wait of the launch gives up.  Allocates nothing;
    // returns false if the rows are too long or the range is invalid.
    bool launch_into(long long first, long long last, long long *out_a, int *out_d,
                     unsigned long long capacity, unsigned long long *out_count,
                     unsigned long long *work, unsigned long long *error, cudaStream_t stream);
    int device() const;

private:
    struct Impl;
    std::unique_ptr<Impl> impl_;
};

}  // namespace rpg
