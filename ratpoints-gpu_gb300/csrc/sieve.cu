// Device sieve: the host driver of the single-curve sieve kernel and its table
// builds (sieve_fast.cuh) for sm_103a.
//
// Reference behaviour restated here:
//   - a site (a, d) survives the reference plan iff f(a/d) mod p is a square
//     for all 32 selected primes, the last word clipped at +H
//     (src/sieve.cu:141-172, 196-213, 221-388);
//   - survivors are (a, d) pairs, d = k or k*k (src/sieve.cu:179-181, 250-252).
//
// Both plans run on one kernel: the tables of a curve (stage-1 rows, class
// lists, candidate primes) are built once per search on the device, and each
// denominator batch is one persistent launch.
#include "sieve.hpp"
#include "batch.hpp"
#include "tune.hpp"

#include <algorithm>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <mutex>
#include <tuple>
#include <utility>

#include "plan.hpp"
#include "preverify.hpp"
#include "sweep.hpp"

namespace rpg {

void check_cuda(cudaError_t status, const char *what) {
    if (status != cudaSuccess)
        throw CudaError(std::string(what) + ": " + cudaGetErrorString(status));
}

void *device_malloc(std::size_t bytes, const char *what) {
    void *p = nullptr;
    cudaError_t status = cudaMalloc(&p, bytes);
    if (status == cudaErrorMemoryAllocation) {
        // the memory that finished searches left for reuse may be what is missing
        cudaGetLastError();
        release_pooled_pipelines(-1);
        release_pooled_engines(-1);
        status = cudaMalloc(&p, bytes);
    }
    check_cuda(status, what);
    return p;
}

// ---------------------------------------------------------------------------

namespace {

using Clock = std::chrono::steady_clock;
double ms_since(Clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(Clock::now() - t0).count();
}

template <typename T>
T *device_alloc(std::size_t count, const char *what) {
    return static_cast<T *>(device_malloc(std::max<std::size_t>(count, 1) * sizeof(T), what));
}

// Survivors per buffer before any growth.  A batch that overflows its buffer is
// run again, and dense curves leave 10^5 to 10^6 a batch (mostly multiples of
// points, which no estimate foresees): with 65,536, every search of one at H =
// 1e7, d <= 1e5 ran its first batch twice (49 instead of 29 ms).
constexpr long long kInitialSurvivors = 1 << 20;
constexpr long long kInitialHostSurvivors = 1 << 16;  // entries of the pinned host arrays

// The streams, events, survivor buffers, pinned staging and table memory of a
// finished search, kept for the next search on the same device so that it does
// not create and allocate them again (a search of a small box spent 0.16 of
// 0.6 ms allocating and freeing its tables).  Nothing in them outlives a
// search as content: every launch resets its counter words first, survivor
// arrays are written before they are read, and every table is built anew per
// search.
struct PooledPipeline {
    struct Buf {
        long long *a = nullptr, *pa = nullptr;
        int *d = nullptr, *pd = nullptr;
        long long cap = 0;
        unsigned long long *count = nullptr;
        cudaEvent_t begin = nullptr, end = nullptr, copied = nullptr;
    };
    int device = -1;
    cudaStream_t streams[4] = {};
    cudaEvent_t events[5] = {};
    Buf buf[2];
    unsigned char *arena = nullptr;
    std::size_t arena_bytes = 0;
    Preverifier *preverifier = nullptr;
    unsigned long long *h_count = nullptr;
    long long *h_a = nullptr;
    int *h_d = nullptr;
    long long host_capacity = 0;
};
constexpr std::size_t kPooledPipelines = 4;                   // per process
constexpr long long kPooledSurvivors = kInitialSurvivors;  // larger buffers are freed
constexpr std::size_t kPooledTables = std::size_t(64) << 20;  // bytes; larger tables are freed

// Never destroyed: static destructors may run after the CUDA runtime is gone.
std::mutex &pipeline_pool_mutex() {
    static auto *m = new std::mutex();
    return *m;
}
std::vector<PooledPipeline> &pipeline_pool() {
    static auto *pool = new std::vector<PooledPipeline>();
    return *pool;
}

}  // namespace

// Most admissible numerator classes of any denominator under the fast plan:
// 2-adic classes (by d mod 64) times residues mod the class prime q (by d mod q).
int max_admissible_classes(const std::vector<std::string> &coefficients, int q) {
    std::uint64_t classes[64];
    two_adic_classes(coefficients, classes);
    int most2 = 0;
    for (auto mask : classes) most2 = std::max(most2, __builtin_popcountll(mask));
    if (q <= 1) return std::max(1, most2);
    // d = 0 mod q: every r but 0; otherwise the residues r with f(r / d) a
    // square mod q, as many for every d
    const int most_q = std::max(q - 1, admitted_residues(q, coefficients));
    return std::max(1, most2 * most_q);
}

constexpr int kFastRowSlots = 3;  // most row sets the fast planner divides the budget by

// Staged row words per slot that the fast planner may spend: `slots` row sets
// (each row 96 words longer than its modulus), 12-warp queues and 32 bytes per
// class within half an SM's shared memory.  These are the planner's terms; the
// kernel stages the rows of the sweep plan made from its choice.
long long fast_row_budget(int max_classes, int slots) {
    const long long per_cta = 228 * 1024 / 2 - 1024 - 2048;
    const long long lists = ((long long)slots * max_classes * 32 + 7) / 8 * 8 + (long long)slots * (max_classes + 1) * 4;
    const long long queues = 11 * 64 * 16;
    return (per_cta - queues - lists) / (8LL * slots);
}

FastPlan single_curve_plan(const std::vector<std::string> &coefficients, long long bound, int *max_classes,
                           FastShape shape) {
    // The choice fixes the set of primes that survivors pass, not the rows that
    // the kernel stages (those are the sweep plan's): rows for two or three
    // row sets within the budget, three for rows of at most 2^20 words when
    // their primes filter within a quarter bit of the two-set plan's.
    const FastPlanner planner(coefficients, bound);
    const int classes = max_admissible_classes(coefficients, planner.class_prime());
    if (max_classes) *max_classes = classes;
    auto plan_for = [&](int slots) {
        const long long row_budget = fast_row_budget(classes, slots);
        FastPlan plan;
        for (int cap = kMaxModulus;;) {
            plan = shape.rows > 0 ? planner.plan(cap, std::min(shape.rows, kMaxFastSlots), row_budget, false)
                                  : planner.plan(cap, kMaxFastSlots, row_budget);
            int row_words = 0;
            for (int m : plan.moduli) row_words += (m + kFastRowExtension + 1) & ~1;
            if (row_words <= row_budget || cap <= 64) break;
            cap = cap * 7 / 8;
        }
        plan.row_slots = slots;
        return plan;
    };
    if (shape.rows > 0) return plan_for(shape.slots == kFastRowSlots ? kFastRowSlots : 2);
    const FastPlan two = plan_for(2);
    if (word_count64(bound) > (1LL << 20)) return two;
    const FastPlan three = plan_for(kFastRowSlots);
    return three.bits >= two.bits - 0.25 ? three : two;
}

struct Sieve::Impl {
    SieveOptions opt;
    long long bound = 0;
    int device = 0;
    // stream: table builds and the launches into buffer 0; stream2: the
    // launches into buffer 1, so that a launch's first CTAs take the SMs that
    // the previous launch's last CTAs leave idle; copy_stream: survivor
    // downloads; count_stream: each launch's counter words, so that their
    // small copy does not sit between two launches.
    cudaStream_t stream = nullptr, stream2 = nullptr, copy_stream = nullptr, count_stream = nullptr;
    cudaEvent_t fork_event = nullptr, join_event = nullptr;  // count_only across both launch streams
    // Device time of a search: launches on the two streams overlap, so each
    // batch adds the part of its [begin, end] interval after the previous
    // batch's end, both measured from an origin recorded at start().
    cudaEvent_t origin = nullptr;
    float last_end_ms = 0;
    // Around the table build on `stream`.  Nothing waits for it on the host:
    // stream2 waits on the device, and its time is read when the first
    // launch's results are there.
    cudaEvent_t tables_begin = nullptr, tables_end = nullptr;
    bool tables_timed = false;
    std::unique_ptr<SweepCurve> curve;
    std::unique_ptr<SweepBuilder> builder;  // its upload's source, until the tables are there
    unsigned char *arena = nullptr;  // its tables
    std::size_t arena_bytes = 0;
    mutable bool lent = false;       // launched on a caller's stream: the arena is freed, not pooled
    FastPlan fast_plan;
    long long capacity = 0;       // most survivors a buffer may grow to hold
    long long host_capacity = 0;  // entries of the pinned host arrays
    SieveTimings timings;

    struct Buffer {
        long long *a = nullptr;
        int *d = nullptr;
        long long *pa = nullptr;  // survivors kept by device pre-verification (same capacity)
        int *pd = nullptr;
        long long cap = 0;        // entries of a and d
        // [0] survivors, [1] work counter, [2] error word, [3] pre-verified survivors
        unsigned long long *count = nullptr;
        cudaEvent_t begin = nullptr, end = nullptr;
        cudaEvent_t copied = nullptr;  // the counter words are in pinned host memory
        long long first = 0, last = 0;
        bool busy = false;
    };
    Buffer buf[2];
    std::unique_ptr<Preverifier> preverifier;
    unsigned long long *h_count = nullptr;  // pinned, 4 words per buffer
    long long *h_a = nullptr;
    int *h_d = nullptr;

    bool in_flight = false;  // launched since the streams were last waited for

    // Batch queue.
    long long q_next = 0, q_last = -1, q_batch = 1;
    std::deque<int> order;  // buffers in flight, oldest first

    // Pieces of an overflowed batch still to deliver, in parameter/numerator order.
    struct Piece {
        long long first, last, a_lo, a_hi;
    };
    std::deque<Piece> pieces;
    long long piece_batch_first = 0, piece_batch_last = 0;

    ~Impl() { release(); }

    // Take a pooled pipeline of this device, if there is one.
    bool adopt_pipeline() {
        PooledPipeline p;
        {
            std::lock_guard<std::mutex> lock(pipeline_pool_mutex());
            auto &pool = pipeline_pool();
            auto it = std::find_if(pool.begin(), pool.end(),
                                   [&](const PooledPipeline &q) { return q.device == device; });
            if (it == pool.end()) return false;
            p = *it;
            pool.erase(it);
        }
        stream = p.streams[0];
        stream2 = p.streams[1];
        copy_stream = p.streams[2];
        count_stream = p.streams[3];
        fork_event = p.events[0];
        join_event = p.events[1];
        origin = p.events[2];
        tables_begin = p.events[3];
        tables_end = p.events[4];
        arena = p.arena;
        arena_bytes = p.arena_bytes;
        preverifier.reset(p.preverifier);
        for (int i = 0; i < 2; ++i) {
            Buffer &b = buf[i];
            const PooledPipeline::Buf &q = p.buf[i];
            b.a = q.a;
            b.d = q.d;
            b.pa = q.pa;
            b.pd = q.pd;
            b.cap = q.cap;
            b.count = q.count;
            b.begin = q.begin;
            b.end = q.end;
            b.copied = q.copied;
        }
        h_count = p.h_count;
        h_a = p.h_a;
        h_d = p.h_d;
        host_capacity = p.host_capacity;
        return true;
    }

    // Hand the pipeline to the pool if every stream finished without error
    // and the pool has room; release() then frees only what was not handed on.
    void offer_pipeline() {
        if (device < 0 || !stream || !stream2 || !copy_stream || !count_stream || !fork_event ||
            !join_event || !origin || !tables_begin || !tables_end || !h_count)
            return;
        for (cudaStream_t s : {stream, stream2, copy_stream, count_stream})
            if (cudaStreamSynchronize(s) != cudaSuccess) return;
        for (const auto &b : buf)
            if (!b.count || !b.begin || !b.end || !b.copied) return;
        {
            std::lock_guard<std::mutex> lock(pipeline_pool_mutex());
            if (pipeline_pool().size() >= kPooledPipelines) return;
        }
        for (auto &b : buf)
            if (b.cap > kPooledSurvivors) {
                cudaFree(b.a);
                cudaFree(b.d);
                cudaFree(b.pa);
                cudaFree(b.pd);
                b.a = b.pa = nullptr;
                b.d = b.pd = nullptr;
                b.cap = 0;
            }
        if (host_capacity > kPooledSurvivors) {
            cudaFreeHost(h_a);
            cudaFreeHost(h_d);
            h_a = nullptr;
            h_d = nullptr;
            host_capacity = 0;
        }
        if (lent || arena_bytes > kPooledTables) {
            cudaFree(arena);
            arena = nullptr;
            arena_bytes = 0;
        }
        PooledPipeline p;
        p.device = device;
        p.streams[0] = stream;
        p.streams[1] = stream2;
        p.streams[2] = copy_stream;
        p.streams[3] = count_stream;
        p.events[0] = fork_event;
        p.events[1] = join_event;
        p.events[2] = origin;
        p.events[3] = tables_begin;
        p.events[4] = tables_end;
        p.arena = arena;
        p.arena_bytes = arena_bytes;
        p.preverifier = preverifier.get();
        for (int i = 0; i < 2; ++i) {
            const Buffer &b = buf[i];
            PooledPipeline::Buf &q = p.buf[i];
            q.a = b.a;
            q.d = b.d;
            q.pa = b.pa;
            q.pd = b.pd;
            q.cap = b.cap;
            q.count = b.count;
            q.begin = b.begin;
            q.end = b.end;
            q.copied = b.copied;
        }
        p.h_count = h_count;
        p.h_a = h_a;
        p.h_d = h_d;
        p.host_capacity = host_capacity;
        {
            std::lock_guard<std::mutex> lock(pipeline_pool_mutex());
            if (pipeline_pool().size() >= kPooledPipelines) return;
            pipeline_pool().push_back(p);
        }
        stream = stream2 = copy_stream = count_stream = nullptr;
        fork_event = join_event = origin = tables_begin = tables_end = nullptr;
        arena = nullptr;
        arena_bytes = 0;
        (void)preverifier.release();
        for (auto &b : buf) b = Buffer{};
        h_count = nullptr;
        h_a = nullptr;
        h_d = nullptr;
        host_capacity = 0;
    }

    void release() {
        if (stream) cudaStreamSynchronize(stream);  // uploads read arrays of this object
        offer_pipeline();
        for (auto &b : buf) {
            cudaFree(b.a);
            cudaFree(b.d);
            cudaFree(b.pa);
            cudaFree(b.pd);
            cudaFree(b.count);
            if (b.begin) cudaEventDestroy(b.begin);
            if (b.end) cudaEventDestroy(b.end);
            if (b.copied) cudaEventDestroy(b.copied);
            b = Buffer{};
        }
        cudaFree(arena);
        arena = nullptr;
        arena_bytes = 0;
        preverifier.reset();
        if (h_count) cudaFreeHost(h_count);
        if (h_a) cudaFreeHost(h_a);
        if (h_d) cudaFreeHost(h_d);
        h_count = nullptr;
        h_a = nullptr;
        h_d = nullptr;
        if (stream) cudaStreamDestroy(stream);
        if (copy_stream) cudaStreamDestroy(copy_stream);
        if (count_stream) cudaStreamDestroy(count_stream);
        if (stream2) cudaStreamDestroy(stream2);
        if (fork_event) cudaEventDestroy(fork_event);
        if (join_event) cudaEventDestroy(join_event);
        for (cudaEvent_t e : {origin, tables_begin, tables_end})
            if (e) cudaEventDestroy(e);
        origin = tables_begin = tables_end = nullptr;
        stream = stream2 = copy_stream = count_stream = nullptr;
        fork_event = join_event = nullptr;
    }

    void init(const std::vector<std::string> &coefficients) {
        auto t0 = Clock::now();
        if (opt.device >= 0) check_cuda(cudaSetDevice(opt.device), "cudaSetDevice");
        check_cuda(cudaGetDevice(&device), "cudaGetDevice");
        if (!adopt_pipeline()) {
            check_cuda(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
            check_cuda(cudaStreamCreateWithFlags(&copy_stream, cudaStreamNonBlocking), "cudaStreamCreate");
            check_cuda(cudaStreamCreateWithFlags(&count_stream, cudaStreamNonBlocking), "cudaStreamCreate");
            check_cuda(cudaStreamCreateWithFlags(&stream2, cudaStreamNonBlocking), "cudaStreamCreate");
            check_cuda(cudaEventCreateWithFlags(&fork_event, cudaEventDisableTiming), "cudaEventCreate");
            check_cuda(cudaEventCreateWithFlags(&join_event, cudaEventDisableTiming), "cudaEventCreate");
            check_cuda(cudaEventCreate(&origin), "cudaEventCreate");
            check_cuda(cudaEventCreate(&tables_begin), "cudaEventCreate");
            check_cuda(cudaEventCreate(&tables_end), "cudaEventCreate");
        }
        // Survivor buffers start small (most searches have few survivors) and
        // grow on overflow up to the per-buffer capacity; past it a batch is
        // split.  RPG_SURVIVOR_CAPACITY fixes both at its value (at least 64,
        // one word's worth); tests use it to drive the split path.
        capacity = opt.capacity;
        long long initial = std::min<long long>(capacity, kInitialSurvivors);
        if (const char *env = std::getenv("RPG_SURVIVOR_CAPACITY")) initial = capacity = std::atoll(env);
        capacity = std::max<long long>(capacity, 64);
        initial = std::max<long long>(initial, 64);
        // A pooled buffer is kept if its capacity lies in [initial, capacity];
        // pa and pd, when present, always have the capacity of a and d.
        for (auto &b : buf) {
            if (b.cap < initial || b.cap > capacity || !b.a || !b.d) {
                cudaFree(b.a);
                cudaFree(b.d);
                cudaFree(b.pa);
                cudaFree(b.pd);
                b.a = b.pa = nullptr;
                b.d = b.pd = nullptr;
                b.cap = 0;
                b.a = device_alloc<long long>(std::size_t(initial), "cudaMalloc(survivors)");
                b.d = device_alloc<int>(std::size_t(initial), "cudaMalloc(survivors)");
                b.cap = initial;
            }
            if (opt.preverify && (!b.pa || !b.pd)) {
                cudaFree(b.pa);
                cudaFree(b.pd);
                b.pa = nullptr;
                b.pd = nullptr;
                b.pa = device_alloc<long long>(std::size_t(b.cap), "cudaMalloc(survivors)");
                b.pd = device_alloc<int>(std::size_t(b.cap), "cudaMalloc(survivors)");
            }
            if (!b.count) b.count = device_alloc<unsigned long long>(4, "cudaMalloc(count)");
            if (!b.begin) check_cuda(cudaEventCreate(&b.begin), "cudaEventCreate");
            if (!b.end) check_cuda(cudaEventCreate(&b.end), "cudaEventCreate");
            if (!b.copied)
                check_cuda(cudaEventCreateWithFlags(&b.copied, cudaEventDisableTiming), "cudaEventCreate");
            b.busy = false;
        }
        if (!h_count) check_cuda(cudaMallocHost(&h_count, 8 * sizeof(unsigned long long)), "cudaMallocHost");
        if (!h_a || !h_d) {
            const long long room = std::min(initial, kInitialHostSurvivors);
            if (h_a) cudaFreeHost(h_a);
            if (h_d) cudaFreeHost(h_d);
            h_a = nullptr;
            h_d = nullptr;
            host_capacity = 0;
            check_cuda(cudaMallocHost(&h_a, std::size_t(room) * sizeof(long long)), "cudaMallocHost");
            check_cuda(cudaMallocHost(&h_d, std::size_t(room) * sizeof(int)), "cudaMallocHost");
            host_capacity = room;
        }
        timings.workspace_ms += ms_since(t0);
        build_tables(coefficients);
    }

    // The curve's sweep plan, and its tables on the device.
    void build_tables(const std::vector<std::string> &coefficients) {
        auto t0 = Clock::now();
        const bool fast = opt.plan == PlanKind::fast;
        if (fast) {
            FastShape shape = opt.fast_shape;
            if (shape.rows <= 0) shape = tuned_fast_shape(coefficients, bound);
            fast_plan = single_curve_plan(coefficients, bound, nullptr, shape);
        }
        curve.reset(new SweepCurve(coefficients, bound, opt.square, fast ? &fast_plan : nullptr, opt.denominators));
        builder.reset(new SweepBuilder);
        builder->add(*curve);
        timings.plan_ms += ms_since(t0);
        auto t1 = Clock::now();
        if (arena_bytes < builder->bytes()) {
            cudaFree(arena);
            arena = nullptr;
            arena_bytes = 0;
            arena = device_alloc<unsigned char>(builder->bytes(), "cudaMalloc(sieve tables)");
            arena_bytes = builder->bytes();
        }
        timings.workspace_ms += ms_since(t1);
        check_cuda(cudaEventRecord(tables_begin, stream), "cudaEventRecord");
        builder->place(arena, stream);
        timings.h2d_bytes += builder->upload_bytes();
        builder->enqueue(stream);
        if (opt.preverify) {
            if (!preverifier) preverifier.reset(new Preverifier());
            preverifier->prepare({&coefficients}, stream);
            timings.h2d_bytes += preverifier->upload_bytes();
        }
        check_cuda(cudaEventRecord(tables_end, stream), "cudaEventRecord");
        check_cuda(cudaStreamWaitEvent(stream2, tables_end, 0), "cudaStreamWaitEvent");
        tables_timed = false;
        timings.table_wall_ms += ms_since(t0);
    }

    // Once a launch on the tables has completed: the device time of their build.
    void time_tables() {
        if (tables_timed) return;
        tables_timed = true;
        builder.reset();
        float ms = 0;
        cudaEventElapsedTime(&ms, tables_begin, tables_end);
        timings.table_ms += ms;
    }

    void launch_sweep(long long first, long long last, long long a_lo, long long a_hi, long long *out_a, int *out_d,
                      unsigned long long cap, unsigned long long *out_count, unsigned long long *work,
                      unsigned long long *error, cudaStream_t st) const {
        SweepLaunch l;
        l.first = first;
        l.last = last;
        l.a_lo = a_lo;
        l.a_hi = a_hi;
        l.out_a = out_a;
        l.out_d = out_d;
        l.capacity = cap;
        l.out_count = out_count;
        l.work = work;
        l.error = error;
        curve->launch(l, st);
    }

    cudaStream_t launch_stream(int which) const { return which ? stream2 : stream; }

    // Counting pass: survivors accumulate in buffer 0's counter across
    // launches; launch i runs on launch stream i mod 2 with that buffer's
    // work counter.
    void launch_counting(int which, long long first, long long last, long long a_lo, long long a_hi) {
        const cudaStream_t st = launch_stream(which);
        check_cuda(cudaMemsetAsync(buf[which].count + 1, 0, sizeof(unsigned long long), st),
                   "cudaMemsetAsync");
        launch_sweep(first, last, a_lo, a_hi, buf[0].a, buf[0].d, (unsigned long long)buf[0].cap, buf[0].count,
                     buf[which].count + 1, buf[0].count + 2, st);
        ++timings.launches;
    }

    bool one_launch() const { return 2 * bound + 1 <= curve->tile(); }

    void launch(int which, long long first, long long last, long long a_lo, long long a_hi) {
        Buffer &b = buf[which];
        b.first = first;
        b.last = last;
        b.busy = true;
        in_flight = true;
        const cudaStream_t st = launch_stream(which);
        check_cuda(cudaMemsetAsync(b.count, 0, 4 * sizeof(unsigned long long), st), "cudaMemsetAsync");
        check_cuda(cudaEventRecord(b.begin, st), "cudaEventRecord");
        launch_sweep(first, last, a_lo, a_hi, b.a, b.d, (unsigned long long)b.cap, b.count, b.count + 1, b.count + 2,
                     st);
        if (opt.preverify) {
            preverifier->launch(b.a, b.d, nullptr, b.count, (unsigned long long)b.cap, b.pa, b.pd, nullptr,
                               b.count + 3, nullptr, st);
            ++timings.launches;
        }
        check_cuda(cudaEventRecord(b.end, st), "cudaEventRecord");
        // The buffer is launched into again only after the host has waited
        // for b.copied, so this copy ends before the memset of its next launch.
        check_cuda(cudaStreamWaitEvent(count_stream, b.end, 0), "cudaStreamWaitEvent");
        check_cuda(cudaMemcpyAsync(h_count + 4 * which, b.count, 4 * sizeof(unsigned long long),
                                   cudaMemcpyDeviceToHost, count_stream),
                   "download survivor count");
        check_cuda(cudaEventRecord(b.copied, count_stream), "cudaEventRecord");
        timings.d2h_bytes += 4 * sizeof(unsigned long long);
        ++timings.launches;
    }

    // Launch queued batches into free buffers (pipelined path, rows that fit
    // one launch).  Rows of more than `tile` numerators go through pieces instead.
    void refill() {
        if (!one_launch() || !pieces.empty()) return;
        while (order.size() < 2 && q_next <= q_last) {
            const int which = buf[0].busy ? 1 : 0;
            if (buf[which].busy) break;
            const long long first = q_next;
            const long long last = std::min(q_last, first + q_batch - 1);
            q_next = last + 1;
            launch(which, first, last, -bound, bound);
            order.push_back(which);
        }
    }

    // Raise if a launch into buffer `which` reported a timed-out device wait.
    void check_error_word(int which) {
        unsigned long long err = 0;
        check_cuda(cudaMemcpy(&err, buf[which].count + 2, sizeof err, cudaMemcpyDeviceToHost),
                   "download error word");
        if (err) throw DeviceTimeout("sieve kernel: bounded wait for a row copy timed out");
    }

    // Device time a completed batch adds (see origin).
    float elapsed(const Buffer &b) {
        time_tables();
        float t0 = 0, t1 = 0;
        cudaEventElapsedTime(&t0, origin, b.begin);
        cudaEventElapsedTime(&t1, origin, b.end);
        const float ms = std::max(0.0f, t1 - std::max(t0, last_end_ms));
        last_end_ms = std::max(last_end_ms, t1);
        return ms;
    }

    void copy_out(int which, std::size_t n) {
        Buffer &b = buf[which];
        if (!n) return;
        check_cuda(cudaStreamWaitEvent(copy_stream, b.end, 0), "cudaStreamWaitEvent");
        check_cuda(cudaMemcpyAsync(h_a, opt.preverify ? b.pa : b.a, n * sizeof(long long),
                                   cudaMemcpyDeviceToHost, copy_stream),
                   "download survivors");
        check_cuda(cudaMemcpyAsync(h_d, opt.preverify ? b.pd : b.d, n * sizeof(int), cudaMemcpyDeviceToHost,
                                   copy_stream),
                   "download survivors");
        check_cuda(cudaStreamSynchronize(copy_stream), "download survivors");
        timings.d2h_bytes += n * (sizeof(long long) + sizeof(int));
    }

    // n modular survivors, of which kept (all, without pre-verification) are copied.
    void deliver(BatchView &out, int which, std::size_t n, std::size_t kept, float ms, long long first,
                 long long last, bool complete) {
        if (!opt.preverify) kept = n;
        host_room(kept);
        copy_out(which, kept);
        out.first = first;
        out.last = last;
        out.a = h_a;
        out.d = h_d;
        out.count = kept;
        out.modular = n;
        out.kernel_ms = ms;
        out.complete = complete;
    }

    // Wait until no launch of this search is on its way.
    void drain() {
        check_cuda(cudaStreamSynchronize(stream), "sieve stream");
        check_cuda(cudaStreamSynchronize(stream2), "sieve stream");
        for (auto &b : buf) b.busy = false;
        in_flight = false;
    }

    // Grow buffer `which` (idle) to hold n survivors if the capacity allows;
    // false if it is already as large as it may get.
    bool grow(int which, unsigned long long n) {
        Buffer &b = buf[which];
        if (b.cap >= capacity) return false;
        const long long cap = std::min<long long>(capacity, (long long)(n + n / 4 + 1024));
        const auto t0 = Clock::now();
        check_cuda(cudaStreamSynchronize(stream), "sieve stream");
        check_cuda(cudaStreamSynchronize(stream2), "sieve stream");
        cudaFree(b.a);
        cudaFree(b.d);
        cudaFree(b.pa);
        cudaFree(b.pd);
        b.a = b.pa = nullptr;
        b.d = b.pd = nullptr;
        b.cap = 0;
        b.a = device_alloc<long long>(std::size_t(cap), "cudaMalloc(survivors)");
        b.d = device_alloc<int>(std::size_t(cap), "cudaMalloc(survivors)");
        if (opt.preverify) {
            b.pa = device_alloc<long long>(std::size_t(cap), "cudaMalloc(survivors)");
            b.pd = device_alloc<int>(std::size_t(cap), "cudaMalloc(survivors)");
        }
        b.cap = cap;
        timings.workspace_ms += ms_since(t0);
        return true;
    }

    // Room in the pinned host arrays for n survivors (those that pass
    // pre-verification are far fewer than a buffer holds).
    void host_room(std::size_t n) {
        if (host_capacity >= (long long)n) return;
        const auto t0 = Clock::now();
        const long long room = (long long)(n + n / 4 + 1024);
        cudaFreeHost(h_a);
        cudaFreeHost(h_d);
        h_a = nullptr;
        h_d = nullptr;
        host_capacity = 0;
        check_cuda(cudaMallocHost(&h_a, std::size_t(room) * sizeof(long long)), "cudaMallocHost");
        check_cuda(cudaMallocHost(&h_d, std::size_t(room) * sizeof(int)), "cudaMallocHost");
        host_capacity = room;
        timings.workspace_ms += ms_since(t0);
    }

    // Queue a batch as pieces of at most a tile of numerators.
    void queue_pieces(long long first, long long last) {
        piece_batch_first = first;
        piece_batch_last = last;
        const long long tile = curve->tile();
        for (long long a = -bound;; a += tile) {
            const bool end = bound - a < tile;  // no overflow near the largest bounds
            pieces.push_back(Piece{first, last, a, end ? bound : a + tile - 1});
            if (end) break;
        }
    }

    // Split a piece into two halves (by parameter, else by numerator range,
    // down to the 64 numerators that the smallest buffer holds).
    void split_front(const Piece &p) {
        if (p.last > p.first) {
            const long long mid = p.first + (p.last - p.first) / 2;
            pieces.push_front(Piece{mid + 1, p.last, p.a_lo, p.a_hi});
            pieces.push_front(Piece{p.first, mid, p.a_lo, p.a_hi});
        } else if (p.a_hi - p.a_lo >= 64) {
            const long long mid = p.a_lo + (p.a_hi - p.a_lo) / 2;
            pieces.push_front(Piece{p.first, p.last, mid + 1, p.a_hi});
            pieces.push_front(Piece{p.first, p.last, p.a_lo, mid});
        } else {
            throw std::logic_error("survivor buffer cannot hold one word of survivors");
        }
    }

    // Run pieces one at a time (synchronously) until one fits a buffer.
    bool next_piece(BatchView &out) {
        while (!pieces.empty()) {
            const Piece p = pieces.front();
            pieces.pop_front();
            const int which = buf[0].busy ? 1 : 0;
            if (buf[which].busy) throw std::logic_error("no free survivor buffer");
            launch(which, p.first, p.last, p.a_lo, p.a_hi);
            check_cuda(cudaEventSynchronize(buf[which].copied), "sieve kernel");
            buf[which].busy = false;
            // the counter words came back with the launch: [2] is its error word
            if (h_count[4 * which + 2]) throw DeviceTimeout("sieve kernel: bounded wait for a row copy timed out");
            const unsigned long long n = h_count[4 * which], kept = h_count[4 * which + 3];
            const float ms = elapsed(buf[which]);
            timings.sieve_ms += ms;
            if (n > (unsigned long long)buf[which].cap) {
                ++timings.reruns;
                if (!grow(which, n)) split_front(p);
                else pieces.push_front(p);
                continue;
            }
            deliver(out, which, std::size_t(n), std::size_t(kept), ms, piece_batch_first, piece_batch_last,
                    pieces.empty());
            return true;
        }
        return false;
    }

    bool next(BatchView &out) {
        if (!pieces.empty()) return next_piece(out);
        if (order.empty() && !one_launch() && q_next <= q_last) {
            const long long first = q_next;
            const long long last = std::min(q_last, first + q_batch - 1);
            q_next = last + 1;
            queue_pieces(first, last);
            return next_piece(out);
        }
        refill();
        if (order.empty()) return false;
        const int which = order.front();
        order.pop_front();
        Buffer &b = buf[which];
        // The counter words were copied to pinned memory right after the launch.
        check_cuda(cudaEventSynchronize(b.copied), "sieve kernel");
        unsigned long long counts[4];
        for (int i = 0; i < 4; ++i) counts[i] = h_count[4 * which + i];
        if (counts[2]) throw DeviceTimeout("sieve kernel: bounded wait for a row copy timed out");
        const unsigned long long n = counts[0];
        const float ms = elapsed(b);
        timings.sieve_ms += ms;
        if (n > (unsigned long long)b.cap) {
            ++timings.reruns;
            b.busy = false;
            piece_batch_first = b.first;
            piece_batch_last = b.last;
            if (grow(which, n)) pieces.push_front(Piece{b.first, b.last, -bound, bound});
            else split_front(Piece{b.first, b.last, -bound, bound});
            return next_piece(out);
        }
        deliver(out, which, std::size_t(n), std::size_t(counts[3]), ms, b.first, b.last, true);
        b.busy = false;
        refill();
        return true;
    }
};

Sieve::Sieve(const std::vector<std::string> &coefficients, long long bound,
             const SieveOptions &options)
    : impl_(new Impl) {
    if (bound < 1) throw std::invalid_argument("numerator bound must be positive");
    // the fast kernel's queued positions a + H must stay below 2^47
    if (options.plan == PlanKind::fast && bound > (1LL << 45))
        throw std::invalid_argument("numerator bound too large for the fast plan (at most 2^45)");
    impl_->opt = options;
    impl_->bound = bound;
    try {
        impl_->init(coefficients);
    } catch (...) {
        impl_->release();
        throw;
    }
}

Sieve::~Sieve() = default;

void release_pooled_pipelines(int device) {
    std::vector<PooledPipeline> taken;
    {
        std::lock_guard<std::mutex> lock(pipeline_pool_mutex());
        auto &pool = pipeline_pool();
        for (auto it = pool.begin(); it != pool.end();) {
            if (device < 0 || it->device == device) {
                taken.push_back(*it);
                it = pool.erase(it);
            } else {
                ++it;
            }
        }
    }
    for (const auto &p : taken) {
        for (const auto &b : p.buf) {
            cudaFree(b.a);
            cudaFree(b.d);
            cudaFree(b.pa);
            cudaFree(b.pd);
            cudaFree(b.count);
            if (b.begin) cudaEventDestroy(b.begin);
            if (b.end) cudaEventDestroy(b.end);
            if (b.copied) cudaEventDestroy(b.copied);
        }
        cudaFree(p.arena);
        delete p.preverifier;
        if (p.h_count) cudaFreeHost(p.h_count);
        if (p.h_a) cudaFreeHost(p.h_a);
        if (p.h_d) cudaFreeHost(p.h_d);
        for (cudaEvent_t e : p.events)
            if (e) cudaEventDestroy(e);
        for (cudaStream_t s : p.streams)
            if (s) cudaStreamDestroy(s);
    }
}

void Sieve::start(long long first, long long last, long long batch_size) {
    if (first < 1 || last < first) throw std::invalid_argument("invalid denominator range");
    if (impl_->opt.square && last > 46340) throw std::invalid_argument("invalid denominator range");
    if (last > 2147483647LL) throw std::invalid_argument("invalid denominator range");
    cancel();
    check_cuda(cudaEventRecord(impl_->origin, impl_->stream), "cudaEventRecord");
    impl_->last_end_ms = 0;
    impl_->q_next = first;
    impl_->q_last = last;
    impl_->q_batch = std::max<long long>(1, batch_size);
}

bool Sieve::next(BatchView &out) { return impl_->next(out); }

void Sieve::cancel() {
    if (impl_->in_flight) impl_->drain();
    impl_->order.clear();
    impl_->pieces.clear();
    impl_->q_next = 0;
    impl_->q_last = -1;
}

const SieveTimings &Sieve::timings() const {
    wait_tables();
    return impl_->timings;
}

void Sieve::wait_tables() const {
    if (impl_->tables_timed) return;
    check_cuda(cudaEventSynchronize(impl_->tables_end), "class table build");
    impl_->time_tables();
}

unsigned long long Sieve::swept_words(long long first, long long last) const {
    return impl_->curve->swept_words(first, last);
}

FastPlanInfo Sieve::fast_plan_info() const {
    FastPlanInfo info;
    if (impl_->opt.plan != PlanKind::fast) return info;
    info.class_prime = impl_->fast_plan.class_prime;
    info.moduli = impl_->fast_plan.moduli;
    for (const auto &f : impl_->fast_plan.slots)
        for (int p : f) info.primes.push_back(p);
    return info;
}

int Sieve::device() const { return impl_->device; }

bool Sieve::allocation_free_rows() const {
    const long long sites = 2 * impl_->bound + 1;
    if (impl_->opt.plan == PlanKind::fast)
        return (sites / (64LL * impl_->fast_plan.class_prime) + 1 + 63) / 64 <= (1LL << 23);
    return word_count64(impl_->bound) <= (1LL << 30);
}

bool Sieve::launch_into(long long first, long long last, long long *out_a, int *out_d,
                        unsigned long long capacity, unsigned long long *out_count,
                        unsigned long long *work, unsigned long long *error, cudaStream_t stream) {
    const auto &I = *impl_;
    if (!allocation_free_rows() || last < first || last - first + 1 > (1 << 16)) return false;
    I.lent = true;
    // A launch per tile of numerators: one, but for curves that few primes
    // filter, whose classes are long.
    const long long tile = I.curve->tile();
    for (long long a = -I.bound;; a += tile) {
        const bool end = I.bound - a < tile;
        I.launch_sweep(first, last, a, end ? I.bound : a + tile - 1, out_a, out_d, capacity, out_count, work, error,
                       stream);
        if (end) return true;
        check_cuda(cudaMemsetAsync(work, 0, sizeof *work, stream), "cudaMemsetAsync");
    }
}

unsigned Sieve::smem_bytes_per_word() const { return unsigned(8 * impl_->curve->plan().moduli.size()); }
long long Sieve::words64() const { return sweep_words(impl_->bound, (long long)impl_->curve->plan().two * impl_->curve->plan().q); }
cudaStream_t Sieve::stream() const { return impl_->stream; }

unsigned long long Sieve::count_only(long long first, long long last, long long batch_size) {
    if (first < 1 || last < first) throw std::invalid_argument("invalid denominator range");
    cancel();
    auto &I = *impl_;
    // Launches share buffer 0's counter: survivors past capacity are counted,
    // not stored, so the total is exact while the stores stop early.
    auto &b = I.buf[0];
    check_cuda(cudaMemsetAsync(b.count, 0, 3 * sizeof(unsigned long long), I.stream),
               "cudaMemsetAsync");
    // the second launch stream starts after the reset and joins before the read
    check_cuda(cudaEventRecord(I.fork_event, I.stream), "cudaEventRecord");
    check_cuda(cudaStreamWaitEvent(I.stream2, I.fork_event, 0), "cudaStreamWaitEvent");
    int which = 0;
    for (long long f = first; f <= last; f += batch_size) {
        const long long l = std::min(last, f + batch_size - 1);
        const long long tile = I.curve->tile();
        for (long long a = -I.bound;; a += tile, which ^= 1) {
            const bool end = I.bound - a < tile;
            I.launch_counting(which, f, l, a, end ? I.bound : a + tile - 1);
            if (end) break;
        }
        which ^= 1;
    }
    check_cuda(cudaEventRecord(I.join_event, I.stream2), "cudaEventRecord");
    check_cuda(cudaStreamWaitEvent(I.stream, I.join_event, 0), "cudaStreamWaitEvent");
    unsigned long long total = 0;
    check_cuda(cudaMemcpyAsync(&total, b.count, sizeof total, cudaMemcpyDeviceToHost, I.stream),
               "download survivor count");
    check_cuda(cudaStreamSynchronize(I.stream), "sieve kernel");
    I.time_tables();
    I.check_error_word(0);
    return total;
}

}  // namespace rpg
