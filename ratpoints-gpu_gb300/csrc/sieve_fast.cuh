// The single-curve sieve kernel and its tables (reference and fast plan; see
// plan.hpp for what survives, sweep_plan.hpp for how the tests are split).
//
// Class layout.  With M = two * Q (Q the product of the class primes), a
// denominator d sweeps only the numerator classes a = r (mod M) whose
// residues are admissible: r mod two by d mod two (the 2-adic filter of the
// fast plan, every residue otherwise), r mod Q by d mod Q.  A class holds the
// sites a = a0 + M t; word w of it covers t = 64 w .. 64 w + 63, so words are
// S = 64 M apart.  S is invertible modulo a stage-1 modulus m (odd, prime to
// Q), so m's mask is periodic in w with period m and one table row per
// (m, d mod m) serves every class: word w of the class of a0 is row word
// a0 S^-1 + w (mod m).  Tables do not depend on H.
//
// A class is a pair: residue r2 mod two and residue rq mod Q.  Its a0 is
// abase + x2 + xq with x2, xq in [0, M) the CRT lifts (abase = -H - M for a
// whole row), so its row index is the sum of one term per residue, and the
// terms are few enough to be tabled once per search.  x2 + xq is not reduced
// modulo M: a class may start a step before the numerator range, and ends up to
// a step after it; emission drops those sites, the sweep needs no masks.
#pragma once

#include "plan.hpp"
#include "sieve_device.cuh"
#include "sweep_plan.hpp"

namespace rpg {
namespace dev {

constexpr int kOddPrimes = 96;             // odd primes below 512
constexpr int kFThreads = 12 * kWarpSize;  // largest CTA: warp 0 produces, the others sweep
constexpr int kFChunk = kWarpSize;         // work units per producer fetch (at most; one per lane)
constexpr int kFQueue = kSweepQueue;
constexpr int kFStage2Group = 6;           // stage-2 primes loaded together
constexpr int kFSegTable = 64;             // units of a class whose row offsets are tabled in shared memory
static_assert(kSweepQueueBytes == kFQueue * 20, "the planner budgets the kernel's queues");

// Arguments of one launch: parameters k_first .. k_first + k_count - 1
// (denominators k, or k * k when square), numerators a_lo .. a_hi, and the
// survivor output (structure of arrays, capacity entries).
struct SweepArgs {
    long long abase;     // a = abase + x2 + xq + S w + M j
    long long a_lo, a_hi;
    long long k_first;
    int k_count;
    int chunk;           // work units per producer fetch
    int part_shift;      // a denominator is 2^part_shift work units, each a share of its items
    int square;
    int segs;            // units of 16 words per class
    int shifted;         // the first class word is not word 0: row offsets take wlo
    int split;           // a group of units is 2^split items, each a range of the residues mod two
    long long *out_a;
    int *out_d;
    int *out_curve;              // curve tags (may be null)
    int curve;
    unsigned long long *out_count;
    unsigned long long capacity;
    unsigned long long *error;   // set nonzero if a bounded device wait ran out (may be null)
    unsigned long long *swept;   // class words swept and the row bytes they read (may be null)
};

struct SweepRow {                  // one stage-1 modulus
    long long offset;              // word offset of row 0 in the table
    unsigned long long magic;      // mod_u32 constant
    u32 m;                         // modulus (odd, prime to M)
    u32 length;                    // staged words of a row (sweep_row_words)
    u32 soff8;                     // byte offset of the row in a slot
    u32 wlo;                       // the launch's first class word, mod m
};

struct FastPrime {                 // one of the 36 reference candidates
    long long pattern;             // word offset of its pattern row 0
    long long offset;              // word offset of its class-layout row 0 (rows of length p), if tabled
    int p;
    u32 inv_stride;                // S^-1 mod p; 0: a class prime, which every swept site passes
    u32 inv_mod;                   // M^-1 mod p
    u32 base_mod;                  // abase mod p
    u32 magic;                     // magic40(p)
    int words;                     // words per pattern row
};

struct LatePrime {                 // a prime of the plan tested after stage 2
    long long pattern;
    unsigned long long magic;      // mod_u32 constant
    u32 p;
    u32 inv_mod;
    u32 base_mod;                  // abase mod p
    int words;
};
constexpr int kLatePrimes = kSweepRows * kSweepRowFactors + 1;  // every prime of a fast plan
constexpr int kFLateGroup = 4;     // late primes loaded together

// Entry of the lists by d mod two and by d mod Q: one admissible residue, its
// CRT lift x and its term of the row index of each modulus, in bytes
// (8 (x S^-1 mod m); by d mod Q with -H - M: 8 ((x - H - M) S^-1 mod m)).
struct SweepClass {
    unsigned short start8[kSweepRows];
    u32 x;
    u32 pad;
};
static_assert(sizeof(SweepClass) == kSweepListBytes, "class lists are copied by TMA");
static_assert(kMaxModulus * 8 < 65536, "row offsets fit 16 bits");

struct SweepTables {
    const SweepClass *listq;       // [Q][q_max]
    const SweepClass *list2;       // [two][two_max]
    const int *count2;             // [two]
    const int *countq;             // [Q]
    const u64 *rows;               // stage-1 and candidate tables, pattern rows
    int nbad, nlate;
    int tabled;                    // the largest candidates have class-layout tables
    int two_mask;                  // two - 1
    u32 q;                         // Q
    unsigned long long q_magic;    // mod_u32 constant of Q
    unsigned long long segs_magic; // ceil(2^64 / segs)
    int two_max, q_max;
    long long stride;              // S = 64 M
    int class_mod;                 // M
    int row_words;                 // staged row words of a slot
    int slots;
    SweepRow row[kSweepRows];
    FastPrime prime[kCandidatePrimes];
    // denominator primes: p | k iff k x <= y (mod 2^32), x = p^-1 mod 2^32 and
    // y = floor((2^32 - 1) / p)
    uint2 bad[kOddPrimes];
    LatePrime late[kLatePrimes + kFLateGroup];  // padded with its last
    uint2 need;                    // d has survivors only if d x <= y (mod 2^32): a divisor d must have
};

// A denominator in flight: written by the producer warp, read by the others.
struct FastSlot {
    long long d;                   // denominator; -1: no more work
    int n2;                        // residues mod two
    int units;                     // units of 16 class words: residues mod Q times segs
    int first, items;              // sweep items of the work unit: first .. items - 1
    int rot;                       // items handed out in this CTA before these, mod the consumer count
    const SweepClass *list;        // residues mod Q in global memory
};

// The 64 bits from position k of a pattern row.
__device__ __forceinline__ u64 pattern_window(const u64 *row, u32 k) {
    const u64 lo = __ldg(row + (k >> 6)), hi = __ldg(row + (k >> 6) + 1);
    const u32 sh = k & 63u;
    return sh ? (lo >> sh) | (hi << (64 - sh)) : lo;
}

// One group of stage 2: candidates ci0, ci0-1, .., ci0-COUNT+1 (descending),
// each tested on the words whose denominator it does not divide; ndiv counts
// the candidates that divide it.  The group's words are loaded together, from
// class-layout tables (TABLED) or as windows of the pattern rows.
template <int COUNT, bool TABLED>
__device__ __forceinline__ void fast_stage2_group(const SweepTables &T, int ci0, u32 hi, u32 lo, u32 d,
                                                  u64 &m, int &ndiv) {
    u64 rows[COUNT];
    bool skip[COUNT];
#pragma unroll
    for (int t = 0; t < COUNT; ++t) {
        const FastPrime &P = T.prime[ci0 - t];
        const u32 p = u32(P.p);
        const u32 rho = mod_small(d, p, P.magic);
        u32 r = mod_small(hi, p, P.magic);
        r = mod_small((r << 16) | lo, p, P.magic);  // pos mod p
        r += P.base_mod;                            // a mod p
        if (r >= p) r -= p;
        const u32 u = mod_small(r * (TABLED ? P.inv_stride : P.inv_mod), p, P.magic);
        skip[t] = rho == 0;
        ndiv += skip[t] ? 1 : 0;
        rows[t] = ~u64(0);
        if (m != 0 && P.inv_stride != 0)
            rows[t] = TABLED ? __ldg(T.rows + P.offset + (long long)rho * p + u)
                             : pattern_window(T.rows + P.pattern + (long long)rho * P.words, u);
    }
#pragma unroll
    for (int t = 0; t < COUNT; ++t) m &= skip[t] ? ~u64(0) : rows[t];
}

// Stage 2 for up to 32 queued words (one per lane), then emission.  Its table
// reads are uncoalesced, one L1 cycle per lane that asks: lanes whose word is
// already empty do not (after six primes one word in sixty is left).  A queued
// word carries its denominator and the position pos = a - abase of its bit 0:
// its sites are a = abase + pos + M j.  For prime p they are the 64 bits from
// position (a mod p) M^-1 mod p of pattern row d mod p, or, tabled, the word
// (a mod p) S^-1 mod p of class-layout row d mod p.
// A word meets the reference's selection, the 32 largest of the 36
// candidates that do not divide d: the 32 largest candidates (the first six,
// which nearly every word meets, from tables when the curve has them; the
// others four at a time in a loop that is not unrolled, which keeps the
// kernel's code compact; the warp stops once its words are empty), skipping
// those dividing d, then, one at a time and only for words where some of those
// divided d, the four smallest until 32 have been tested.  The few words left meet the late
// primes and drop the sites outside the launch's numerators.
__device__ __forceinline__ void fast_drain(const u64 *qmask, const u64 *qpos, const u32 *qd, int start, int n,
                                           const SweepTables &T, const SweepArgs &A) {
    const int lane = threadIdx.x & 31;
    u64 m = 0, pos = 0;
    u32 d = 1;  // lanes past n hold no word: any denominator keeps their row indices in range
    if (lane < n) {
        m = qmask[start + lane];
        pos = qpos[start + lane];
        d = qd[start + lane];
    }
    __syncwarp();
    const u32 hi = u32(pos >> 16), lo = u32(pos & 0xFFFF);
    static_assert(kCandidatePrimes == 36 && kSelectedPrimes == 32, "stage-2 group schedule");
    int ndiv = 0;  // of the candidates tested so far, those dividing d
    int g = 0;
    if (T.tabled) {
        fast_stage2_group<kFStage2Group, true>(T, kCandidatePrimes - 1, hi, lo, d, m, ndiv);
        g = kFStage2Group;
    }
    constexpr int kLater = 4;  // primes per later group
    static_assert((kSelectedPrimes - kFStage2Group) % kLater == 2 && kSelectedPrimes % kLater == 0, "group schedule");
    if (T.tabled && __any_sync(kFullMask, m != 0)) {
        fast_stage2_group<2, false>(T, kCandidatePrimes - 1 - g, hi, lo, d, m, ndiv);
        g += 2;
    }
#pragma unroll 1
    for (; g < kSelectedPrimes; g += kLater) {
        if (!__any_sync(kFullMask, m != 0)) break;
        fast_stage2_group<kLater, false>(T, kCandidatePrimes - 1 - g, hi, lo, d, m, ndiv);
    }
    // candidates 3, 2, 1, 0 make up for the larger ones that divide d
#pragma unroll
    for (int ci = 3; ci >= 0; --ci) {
        if (!__any_sync(kFullMask, m != 0 && ndiv > 0)) break;
        const FastPrime &P = T.prime[ci];
        const u32 p = u32(P.p);
        const u32 rho = mod_small(d, p, P.magic);
        if (m != 0 && ndiv > 0 && rho != 0) {
            u32 r = mod_small(hi, p, P.magic);
            r = mod_small((r << 16) | lo, p, P.magic);
            r += P.base_mod;
            if (r >= p) r -= p;
            const u32 u = mod_small(r * P.inv_mod, p, P.magic);
            if (P.inv_stride != 0) m &= pattern_window(T.rows + P.pattern + (long long)rho * P.words, u);
            --ndiv;  // one of the 32 taken by a smaller candidate
        }
    }
    if (!__any_sync(kFullMask, m != 0)) return;
    const long long a0 = A.abase + (long long)pos;
    const long long M = T.class_mod;
    if (m) {
        // four at a time: the chain of one is long, and the survivors of a
        // small search all meet every late prime (padded with repeats)
        for (int l = 0; l < T.nlate && m; l += kFLateGroup) {
            u64 rows[kFLateGroup];
#pragma unroll
            for (int t = 0; t < kFLateGroup; ++t) {
                const LatePrime &P = T.late[l + t];
                u32 r = mod_u32(hi, P.p, P.magic);
                r = mod_u32((r << 16) | lo, P.p, P.magic) + P.base_mod;
                if (r >= P.p) r -= P.p;
                const u32 k = mod_u32(r * P.inv_mod, P.p, P.magic);
                rows[t] = pattern_window(T.rows + P.pattern + (long long)mod_u32(d, P.p, P.magic) * P.words, k);
            }
#pragma unroll
            for (int t = 0; t < kFLateGroup; ++t) m &= rows[t];
        }
        if (a0 < A.a_lo || a0 + 63 * M > A.a_hi) {  // ends of the numerator range
            for (u64 rest = m; rest; rest &= rest - 1) {
                const int j = __ffsll((long long)rest) - 1;
                const long long a = a0 + M * j;
                if (a < A.a_lo || a > A.a_hi) m &= ~(u64(1) << j);
            }
        }
    }
    u32 cnt = __popcll(m);
    if (!__any_sync(kFullMask, cnt != 0)) return;
    u32 incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        u32 v = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += v;
    }
    const u32 total = __shfl_sync(kFullMask, incl, 31);
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(A.out_count, (unsigned long long)total);
    base = __shfl_sync(kFullMask, base, 0);
    unsigned long long at = base + incl - cnt;
    while (m) {
        const int bit = __ffsll((long long)m) - 1;
        m &= m - 1;
        if (at < A.capacity) {
            A.out_a[at] = a0 + M * bit;
            A.out_d[at] = int(d);
            if (A.out_curve) A.out_curve[at] = A.curve;
        }
        ++at;
    }
}

__device__ __forceinline__ void lds_u64(u32 a, u32 &lo, u32 &hi) {
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(a));
}
__device__ __forceinline__ void lds_u32x4(u32 a, u32 (&v)[4]) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(a));
}

// The row terms of N rows: 16-bit values two to a word.
template <int N>
__device__ __forceinline__ void load_starts16(u32 a, u32 (&v)[N]) {
    u32 x[6];
    if (N > 4) {
        u32 y[4];
        lds_u32x4(a, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = y[i];
    } else {
        lds_u64(a, x[0], x[1]);
    }
    if (N > 8) lds_u64(a + 16, x[4], x[5]);
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = r % 2 ? x[r / 2] >> 16 : x[r / 2] & 0xFFFFu;
}

// Warp-specialized persistent CTAs.  Warp 0 produces: it takes work units from
// the launch's counter, drops denominators without classes or with a
// denominator prime, and for each live one fills a slot by TMA with the NS
// stage-1 rows of d mod m and the class lists of d mod two and d mod Q.  The
// other warps sweep filled slots.  An item is a group of U pairs of units (16
// words of one residue mod Q each, one per half-warp) against the residues mod
// two: the units' row addresses stay in registers, a step adds one residue's
// terms (a broadcast read shared by the pairs) and ANDs one word per lane, row
// and pair.  Items go round-robin over the consumer warps, across
// denominators; no barrier spans the CTA and every wait is bounded.
//
// What bounds it: the shared-memory pipe.  A row's word for a warp (two
// conflict-free 128-byte halves) takes two of its cycles, whatever the layout,
// so a swept word costs NS / 16 cycles of an SM.  The class primes halve the
// words per prime down to classes of 16 words; everything else keeps the
// pipe's other work and the instructions small:
//   - rows are staged as two periods, so that the sum of two row offsets below
//     m needs no wrap: 61 instead of 115 instructions per step of ten rows,
//     1.95 instead of 2.49 ms per 65,536 denominators of a curve of degree 6
//     at H = 5e6, the pipe busy in 93 instead of 71 % of its cycles;
//   - a broadcast 128-bit shared read takes two cycles, a 64-bit one one: the
//     terms of a residue are packed to 16 bits (two cycles for eight rows,
//     three for twelve) and shared by U = 2 pairs (1.81 -> 1.75 ms); read from
//     kernel parameters instead, they cost more instructions than they saved
//     cycles (2.07 ms);
//   - a unit without a partner is split over both half-warps by residues: at
//     H = 20,000, where a class is one unit, 400,000 denominators of four
//     curves take 0.42, 0.25, 0.48 and 0.81 ms instead of 0.53, 0.28, 0.66 and
//     1.10;
//   - the 24 warps of an SM form two, three or four CTAs: with four, a curve of
//     240 words per denominator (H = 3e5) takes 0.22 instead of 0.29 ms per
//     131,072 denominators, each CTA's producer being serial.
template <int NS, int U>
__global__ void __launch_bounds__(kFThreads, 2) fast_sieve_kernel(const __grid_constant__ SweepTables T,
                                                                  const __grid_constant__ SweepArgs A,
                                                                  unsigned long long *work) {
    extern __shared__ __align__(16) unsigned char smem[];
    const u32 list2_at = u32(T.row_words) * 8u;
    const u32 listq_at = list2_at + u32(T.two_max) * u32(sizeof(SweepClass));
    const bool listq_staged = T.q_max <= kSweepSlotClasses;
    const u32 slot_bytes = listq_at + (listq_staged ? u32(T.q_max) * u32(sizeof(SweepClass)) : 0u);
    u64 *qmask = reinterpret_cast<u64 *>(smem + T.slots * slot_bytes);
    const int consumers = int(blockDim.x) / kWarpSize - 1;
    u64 *qpos = qmask + consumers * kFQueue;
    u32 *qd = reinterpret_cast<u32 *>(qpos + consumers * kFQueue);

    __shared__ FastSlot slot[kSweepSlots];
    __shared__ __align__(16) unsigned short s_seg[kFSegTable][16];  // row offsets of unit seg of a class
    __shared__ __align__(8) unsigned long long s_full[kSweepSlots];
    __shared__ __align__(8) unsigned long long s_empty[kSweepSlots];

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int slots = T.slots;
    if (threadIdx.x == 0) {
        for (int b = 0; b < slots; ++b) {
            mbar_init(smem_addr(&s_full[b]), 1);
            mbar_init(smem_addr(&s_empty[b]), u32(consumers));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < min(A.segs, kFSegTable) * NS; i += int(blockDim.x)) {
        const int seg = i / NS, r = i % NS;
        s_seg[seg][r] = (unsigned short)(8u * mod_u32(T.row[r].wlo + u32(kSweepUnit * seg), T.row[r].m, T.row[r].magic));
    }
    __syncthreads();

    if (warp == 0) {
        // ---- producer ----
        // A chunk's work units (parameter, share of its items) are classified
        // one per lane, the next chunk's fetch already issued; the live ones go
        // to the slots in order.
        int b = 0, round = 0;      // slot of the next fill, and how often it has been filled
        bool failed = false;
        unsigned long long swept = 0;  // class words handed out
        int rot = 0;               // sweep items handed out so far, mod the consumer count
        const SweepRow R = T.row[lane < NS ? lane : 0];  // the row this lane copies
        const int chunk_size = A.chunk;
        const long long unit_count = (long long)A.k_count << A.part_shift;
        unsigned long long next_chunk = 0;
        if (lane == 0) next_chunk = atomicAdd(work, (unsigned long long)chunk_size);
        // waits until slot b is released by every consumer (false: gave up)
        auto acquire_slot = [&]() -> bool {
            return round == 0 || mbar_wait(smem_addr(&s_empty[b]), u32(round - 1) & 1u);
        };
        for (;;) {
            const long long chunk = (long long)__shfl_sync(kFullMask, next_chunk, 0);
            if (chunk >= unit_count) break;
            if (lane == 0) next_chunk = atomicAdd(work, (unsigned long long)chunk_size);
            const long long idx = chunk + lane;
            const bool valid = lane < chunk_size && idx < unit_count;
            const long long k = A.k_first + (valid ? idx >> A.part_shift : 0);
            const u32 du = A.square ? u32(k) * u32(k) : u32(k);
            const u32 dq = mod_u32(du, T.q, T.q_magic);
            int n2 = 0, nq = 0;
            if (valid) {
                n2 = __ldg(T.count2 + (du & u32(T.two_mask)));
                nq = __ldg(T.countq + dq);
            }
            // Denominator primes: for p | d and p !| a, F(a, d) = c_n a^n
            // (mod p), which is not a square when c_n is not and n is even, so
            // d holds no points.  p | k^2 iff p | k.
            bool hit = false;
#pragma unroll 4
            for (int i = 0; i < T.nbad; ++i) hit |= u32(k) * T.bad[i].x <= T.bad[i].y;
            if (hit || du * T.need.x > T.need.y) nq = 0;
            const int units = nq * A.segs;
            const int all = ((units + 2 * U - 1) / (2 * U)) << A.split;
            const int part = int(idx) & ((1 << A.part_shift) - 1);
            const int first = int((long long)all * part >> A.part_shift);
            const int items = int((long long)all * (part + 1) >> A.part_shift);  // first: fewer items than parts
            const int turn = int(unsigned(items - first) % unsigned(consumers));
            const bool mine = n2 > 0 && nq > 0 && first < items;
            if (valid && n2 > 0 && nq > 0 && part == 0)  // the whole denominator's; this share may be empty
                swept += (unsigned long long)units * unsigned(n2) * kSweepUnit;
            u32 live = __ballot_sync(kFullMask, mine);
            while (live) {
                const int j = __ffs(live) - 1;
                live &= live - 1;
                const u32 d = __shfl_sync(kFullMask, du, j);
                const u32 full = smem_addr(&s_full[b]);
                const u32 at8 = smem_addr(smem) + u32(b) * slot_bytes;
                const u32 rho = mod_u32(d, R.m, R.magic);
                const u64 *const row = T.rows + R.offset + (long long)rho * R.length;
                const u32 bytes2 = __shfl_sync(kFullMask, u32(n2) * u32(sizeof(SweepClass)), j);
                const u32 bytesq = __shfl_sync(kFullMask, u32(nq) * u32(sizeof(SweepClass)), j);
                const u32 dq_j = __shfl_sync(kFullMask, dq, j);
                const int turn_j = __shfl_sync(kFullMask, turn, j);
                if (!acquire_slot()) {
                    failed = true;
                    break;
                }
                if (lane == j) {
                    FastSlot &S = slot[b];
                    S.d = d;
                    S.units = units;
                    S.n2 = n2;
                    S.first = first;
                    S.items = items;
                    S.rot = rot;
                    S.list = T.listq + (long long)dq * T.q_max;
                    mbar_arrive_expect_tx(full, u32(T.row_words) * 8u + bytes2 + (listq_staged ? bytesq : 0u));
                }
                rot += turn_j;
                if (rot >= consumers) rot -= consumers;
                // the consumers' reads of this slot's previous contents are
                // ordered before the asynchronous copies that overwrite them
                fence_proxy_async_shared();
                __syncwarp();
                if (lane < NS) {
                    bulk_copy_to_shared(at8 + R.soff8, row, R.length * 8u, full);
                } else if (lane == 30) {
                    bulk_copy_to_shared(at8 + list2_at, T.list2 + (long long)(d & u32(T.two_mask)) * T.two_max,
                                        bytes2, full);
                } else if (lane == 31 && listq_staged) {
                    bulk_copy_to_shared(at8 + listq_at, T.listq + (long long)dq_j * T.q_max,
                                        bytesq, full);
                }
                if (++b == slots) {
                    b = 0;
                    ++round;
                }
            }
            if (failed) break;
        }
        if (A.swept) {
            for (int o = 16; o > 0; o >>= 1) swept += __shfl_xor_sync(kFullMask, swept, o);
            if (lane == 0) {
                atomicAdd(A.swept, swept);
                atomicAdd(A.swept + 1, swept * 8ull * NS);
            }
        }
        if (!failed) {
            // no more work: an empty slot fill tells the consumers to finish
            if (acquire_slot()) {
                if (lane == 0) {
                    slot[b].d = -1;
                    __threadfence_block();
                    mbar_arrive(smem_addr(&s_full[b]));
                }
            } else {
                failed = true;
            }
        }
        if (failed) {
            if (A.error && lane == 0) atomicOr(A.error, 1ull);
            // let the copies already issued land (bounded) before leaving
            for (int t = 0; t < slots; ++t) {
                const int fills = round + (t < b ? 1 : 0);
                if (lane == 0 && fills > 0) mbar_wait(smem_addr(&s_full[t]), u32(fills - 1) & 1u);
            }
        }
        return;
    }

    // ---- consumers ----
    // Consumer cw sweeps the items i of a fill with (i - first + rot) mod
    // consumers = cw, rot carried across denominators by the producer.
    const int cw = warp - 1;
    u64 *wq_mask = qmask + cw * kFQueue;
    u64 *wq_pos = qpos + cw * kFQueue;
    u32 *wq_d = qd + cw * kFQueue;
    u32 phase = 0;   // bit b: parity of slot b's next fill
    int b = 0;
    int qn = 0;      // queued words (kept across denominators)
    const u32 lane_word8 = u32(lane & (kSweepUnit - 1)) * 8u;
    for (;;) {
        if (!mbar_wait(smem_addr(&s_full[b]), (phase >> b) & 1u)) {  // bounded wait
            if (A.error && lane == 0) atomicOr(A.error, 1ull);
            return;
        }
        phase ^= 1u << b;
        const FastSlot &S = slot[b];
        if (S.d < 0) {  // the producer has no more work
            __syncwarp();
            if (qn > 0) fast_drain(wq_mask, wq_pos, wq_d, 0, qn, T, A);
            return;
        }
        const int total_items = S.items;
        int item = cw - S.rot;
        if (item < 0) item += consumers;
        item += S.first;
        if (item < total_items) {
            const u32 d = u32(S.d);
            const u32 slot_addr = smem_addr(smem) + u32(b) * slot_bytes;
            const u32 words_addr = slot_addr + lane_word8;
            const int units = S.units, n2 = S.n2;
            for (; item < total_items; item += consumers) {
                const int group = item >> A.split;
                const int range = (n2 + (1 << A.split) - 1) >> A.split;
                const int e0 = (item & ((1 << A.split) - 1)) * range;
                int steps = min(range, n2 - e0);
                // A last group that is at most half full (of short classes the
                // only one): both half-warps take each of its units, with half
                // of the residues each.
                const bool alone = units - 2 * U * group <= U;
                const int half = lane >> 4;
                // this half-warp's units, 16 words of one residue mod Q each:
                // the addresses of their first words in the staged rows
                u32 o[U][NS];
                u64 pos0[U];
                bool valid[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    int unit = 2 * U * group + (alone ? u : 2 * u + half);
                    valid[u] = unit < units;
                    if (!valid[u]) unit = 0;
                    int s = unit, seg = 0;
                    if (A.segs > 1) {
                        s = int(__umul64hi(u64(unit), T.segs_magic));
                        seg = unit - s * A.segs;
                    }
                    u32 xq;
                    if (listq_staged) {
                        const u32 entry = slot_addr + listq_at + u32(s) * u32(sizeof(SweepClass));
                        u32 pad;
                        load_starts16<NS>(entry, o[u]);
                        lds_u64(entry + 2 * kSweepRows, xq, pad);
                    } else {
                        const uint4 *entry = reinterpret_cast<const uint4 *>(S.list + s);
                        const uint4 e0 = __ldg(entry), e1 = __ldg(entry + 1);
                        const u32 e[6] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y};
#pragma unroll
                        for (int r = 0; r < NS; ++r) o[u][r] = r % 2 ? e[r / 2] >> 16 : e[r / 2] & 0xFFFFu;
                        xq = e1.z;
                    }
                    if (A.segs > 1 || A.shifted) {
                        u32 g[NS];
                        if (A.segs <= kFSegTable) {
                            load_starts16<NS>(smem_addr(s_seg[seg]), g);
                        } else {
#pragma unroll
                            for (int r = 0; r < NS; ++r)
                                g[r] = 8u * mod_u32(T.row[r].wlo + u32(kSweepUnit * seg), T.row[r].m, T.row[r].magic);
                        }
#pragma unroll
                        for (int r = 0; r < NS; ++r) {
                            const u32 v = o[u][r] + g[r];
                            o[u][r] = min(v, v - 8u * T.row[r].m);  // unsigned: wraps into [0, 8 m)
                        }
                    }
#pragma unroll
                    for (int r = 0; r < NS; ++r) o[u][r] += words_addr + T.row[r].soff8;
                    pos0[u] = u64(xq) + u64(T.stride) * u64(kSweepUnit * seg + (lane & (kSweepUnit - 1)));
                }
                u32 a_addr = slot_addr + list2_at + u32(e0) * u32(sizeof(SweepClass));
                int i = 0, end = steps;
                int own = valid[0] ? steps : 0;  // U == 1: steps in which this lane's words count
                if (alone && steps > 0) {
                    // of an odd number the middle one is both halves' and
                    // counts in the second, which has it first
                    const int low = steps >> 1;
                    steps -= low;
                    end = U == 1 ? steps : low;
                    own = half ? steps : low;
                    if (half) a_addr += u32(low) * u32(sizeof(SweepClass));
                }
                // U == 2: the steps in which both halves count, then the middle
                // residue's; with U == 1 a comparison with own is cheaper
                for (;;) {
#pragma unroll 1
                    for (; i < end; ++i, a_addr += u32(sizeof(SweepClass))) {
                        u32 t[NS];
                        load_starts16<NS>(a_addr, t);
                        u32 al[U], ah[U];
                        bool hit[U];
                        u32 bb[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            u32 lo[NS], hi[NS];
#pragma unroll
                            for (int r = 0; r < NS; ++r) lds_u64(o[u][r] + t[r], lo[r], hi[r]);
                            al[u] = lo[0];
                            ah[u] = hi[0];
#pragma unroll
                            for (int r = 1; r + 1 < NS; r += 2) {
                                al[u] = and3(al[u], lo[r], lo[r + 1]);
                                ah[u] = and3(ah[u], hi[r], hi[r + 1]);
                            }
                            if (NS % 2 == 0) {
                                al[u] &= lo[NS - 1];
                                ah[u] &= hi[NS - 1];
                            }
                            hit[u] = (al[u] | ah[u]) != 0 && (U == 1 ? i < own : valid[u]);
                            bb[u] = __ballot_sync(kFullMask, hit[u]);
                        }
                        u32 any = bb[0];
                        if (U > 1) any |= bb[U - 1];
                        if (!any) continue;
                        u32 x2, pad;
                        lds_u64(a_addr + 2 * kSweepRows, x2, pad);
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            if (!bb[u]) continue;
                            const int to = qn + __popc(bb[u] & lanemask_lt());
                            if (hit[u]) {
                                wq_mask[to] = (u64(ah[u]) << 32) | al[u];
                                wq_pos[to] = pos0[u] + x2;
                                wq_d[to] = d;
                            }
                            qn += __popc(bb[u]);
                            if (qn >= 32) {
                                __syncwarp();
                                fast_drain(wq_mask, wq_pos, wq_d, qn - 32, 32, T, A);
                                qn -= 32;
                            }
                        }
                    }
                    if (U == 1 || end >= steps) break;
                    end = steps;
#pragma unroll
                    for (int u = 0; u < U; ++u) valid[u] = valid[u] && half;
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_addr(&s_empty[b]));  // this warp is done with slot b
        b = b + 1 == slots ? 0 : b + 1;
    }
}

}  // namespace dev
}  // namespace rpg
