// Batched many-curve sieve (batch.hpp): device kernels and host driver.
#include "batch.hpp"

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <system_error>
#include <thread>

#include "exact.hpp"
#include "plan.hpp"
#include "preverify.hpp"
#include "sieve.hpp"
#include "sieve_device.cuh"
#include "sweep.hpp"
#include "tune.hpp"

namespace rpg {
namespace dev {

constexpr int kWideSlots = 6;                      // stage-1 moduli of a wide curve (padded)
constexpr int kWK = 4;                             // words per lane per step (lanes 32 apart)
constexpr int kWWarps = 12;                        // warp 0 produces, the others sweep
constexpr int kWThreads = kWWarps * kWarpSize;
constexpr int kWConsumers = kWWarps - 1;
constexpr int kWSlotCount = 2;                     // denominators in flight per CTA
constexpr int kWSteps = 4;
constexpr int kWItemWords = kWarpSize * kWK * kWSteps;  // class words per sweep item
constexpr int kWExt = kWarpSize * (kWK - 1);            // row extension
constexpr int kWMaxSmemWords = 6000;                    // staged row words per slot (two
                                                        // slots, 2 CTAs per SM)
constexpr int kQueue = 64;
constexpr long long kMaxClassWords = 1LL << 23;         // class words of a row (sweep-item arithmetic)
constexpr int kAdmQ = 16;                               // residue words for class primes <= 13
constexpr int kNarrowSlots = 8;
constexpr int kNK = 4;                                  // consecutive row words per lane (long ranges)
constexpr int kNShortWords = 96;                        // ranges up to this many words: one word per lane
// Words with several sites that a drain of stage 2 puts back; with more it loops
// over their sites.  6, 12, 18, 31: high-degree batch 19.9, 19.0, 18.9, 18.8 ms,
// 384 small curves 1.95, 1.85, 1.82, 1.81, a curve with sites everywhere 5.55,
// 5.56, 5.59, 6.05.
constexpr int kNarrowMore = 18;
constexpr int kNarrowQueue = 64;                        // queued words per warp
constexpr int kNWarps = 8;
constexpr int kNThreads = kNWarps * kWarpSize;
constexpr int kNarrowTableWords = 7680;                 // sum of m (m + kNK - 1) per curve
constexpr int kAffWords = kCandidatePrimes * 8;         // the 36 candidate bitmasks
constexpr int kRefWords = 8;                            // u64 words of a bitmask over [0, 512)
constexpr int kMaxFactors = 4;
constexpr int kMaxIntervals = 8;                        // more: sweep the whole row


// The odd primes below 512 with ceil(2^64 / p) (mod_u32): a curve's
// denominator primes are a bit mask over this table.
constexpr int kOddPrimes = 96;
struct OddPrime {
    u32 p;
    u32 inverse;                   // p^-1 mod 2^32: p | n iff n inverse <= (2^32 - 1) / p (mod 2^32)
    unsigned long long magic;
};

struct Modulus {                   // one stage-1 modulus of a wide curve (class layout)
    long long offset;              // word offset of row 0 in the table pool
    unsigned long long magic;      // mod_u32 constant (all ones for m = 1)
    int m;
    int length;                    // row length in words (m + kWExt, even)
    int smem_offset;               // word offset of the staged row
    u32 inv_stride;                // S^-1 mod m
    u32 neg_h;                     // (-H) mod m
    u32 step;                      // (32 kWK) mod m
};

struct WideCurve {
    long long bound;               // H
    long long stride;              // S = 64 M: numerator step between words of a class
    long long count_q;             // 2H = count_q M + count_r
    long long aff;                 // u64 offset of the 36 candidate bitmasks
    long long cls;                 // index of the curve's ClassStart[M] block
    Modulus mod[kWideSlots];
    u64 admissible[64 + kAdmQ];    // 2-adic classes by d mod 64, residues mod q by d mod q
    int count_r;
    int class_prime;               // q (1: 2-adic classes only)
    int class_mod;                 // M = 64 q
    int smem_words;
    int square;
    int index;                     // position in the caller's curve list
    int rows;                      // stage-1 moduli in use (the others are padding)
    u64 denom_primes[2];           // bit i: odd prime i of the OddPrime table is a denominator prime
    unsigned short neg_h[kCandidatePrimes];   // (-H) mod p
    unsigned short m_mod[kCandidatePrimes];   // M mod p
    unsigned char crt[13 * 13];    // [r64 mod q][rq] -> t with r = r64 + 64 t (mod 64 q)
    unsigned char mod_q[64];       // r64 mod q
    int nint;                      // x intervals (at least one)
    double lo[kMaxIntervals];      // ascending lower bounds (-inf: none)
    double hi[kMaxIntervals];      // upper bounds (+inf: none)
};

struct NarrowCurve {
    long long bound;
    long long tables;              // word offset of the curve's table block (even)
    long long aff;
    unsigned long long magic[kNarrowSlots];
    u64 dense2[64];                // by d mod 64: bit j set iff a = -H + j (mod 64) may hold points
    int table_words;               // even
    int square;
    int index;
    int rows;                      // stage-1 moduli in use (the others are padding)
    u64 denom_primes[2];           // bit i: odd prime i of the OddPrime table is a denominator prime
    int m[kNarrowSlots];           // moduli (1: padding)
    int off[kNarrowSlots];         // word offset of each table inside the block
    int len[kNarrowSlots];         // row length m + kNK - 1 (rows repeat their first words)
    u32 shift[kNarrowSlots];       // (-H) 64^-1 mod m: table word of row word 0
    u32 step[kNarrowSlots];        // (32 kNK) mod m
    unsigned short neg_h[kCandidatePrimes];
    int nint;
    double lo[kMaxIntervals];
    double hi[kMaxIntervals];
};

static_assert(sizeof(WideCurve) % 4 == 0 && sizeof(NarrowCurve) % 4 == 0, "u32 copies");

struct BatchItem {
    long long first;               // first parameter k
    int curve;                     // descriptor index
    int count;                     // parameters in this item
    int range;                     // which numerator range of each denominator (wide items, see x_range)
    int pad;
};

// Numerator ranges of denominator d for x in the curve's intervals: each
// interval [lo, hi] gives a in [floor(lo d) - 1, ceil(hi d) + 1] (widened by
// one so that double rounding never drops a site; the host applies the exact
// interval test), clipped to [-H, H]; overlapping ranges are merged.  Sets
// [L, U] to the first of the disjoint ascending ranges from interval i on, and
// i to the interval after it; false if there is none.
__device__ __forceinline__ bool next_x_range(const double *lo, const double *hi, int nint, long long H, double d,
                                             int &i, long long &L, long long &U) {
    const double h = double(H);
    bool any = false;
    for (; i < nint; ++i) {
        const double x = floor(lo[i] * d) - 1.0;
        const double y = ceil(hi[i] * d) + 1.0;
        const long long l = !(x > -h) ? -H : (x > h ? H + 1 : (long long)x);
        const long long u = !(y < h) ? H : (y < -h ? -H - 1 : (long long)y);
        if (l > u) continue;
        if (any && l > U + 1) break;
        if (!any) {
            any = true;
            L = l;
            U = u;
        } else if (u > U) {
            U = u;
        }
    }
    return any;
}

// The want-th of them.
__device__ __forceinline__ bool x_range(const double *lo, const double *hi, int nint, long long H,
                                        long long d, int want, long long &L, long long &U) {
    for (int i = 0, n = 0; next_x_range(lo, hi, nint, H, double(d), i, L, U); ++n)
        if (n == want) return true;
    return false;
}

struct AffineSpec {                // bitmask of x in [0, p) with f(x) a square mod p
    long long out;                 // u64 offset of the 8-word output
    long long residues;            // offset of c_0 .. c_n mod p
    int p, n;
};

struct PatternSpec {               // q x q words: bit j of word (rho, u) tests x = (s u + t j) mod q
    long long offset;
    long long aff;
    int q, lead_ok, s, t;
};

struct CompositeSpec {             // m rows of `length` words: AND of the factor patterns
    long long offset;
    long long pattern[kMaxFactors];
    int m, length, nf;
    int q[kMaxFactors];
};

struct BatchOut {
    long long *a;
    int *d;
    int *curve;
    unsigned long long *count;
    unsigned long long capacity;
    unsigned long long *error;
};

struct Candidates {
    int p[kCandidatePrimes];
    u32 magic[kCandidatePrimes];
};

// ---------------------------------------------------------------------------
// Table construction

__global__ void affine_kernel(const AffineSpec *specs, long long nspecs,
                              const unsigned short *residues, const u64 *square_masks, u64 *out) {
    const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (id >= nspecs * kRefWords) return;
    const AffineSpec S = specs[id / kRefWords];
    const int k = int(id % kRefWords);
    const int p = S.p;
    const unsigned short *c = residues + S.residues;
    const u64 *sq = square_masks + (long long)p * kRefWords;
    u64 word = 0;
    for (int b = 0; b < 64; ++b) {
        const int x = 64 * k + b;
        if (x >= p) break;
        int v = c[S.n];
        for (int i = S.n - 1; i >= 0; --i) v = (v * x + c[i]) % p;
        if ((sq[v >> 6] >> (v & 63)) & 1) word |= u64(1) << b;
    }
    out[S.out + k] = word;
}

// Index of the last spec whose offset is <= id (specs sorted by offset).
template <typename Spec>
__device__ __forceinline__ int find_spec(const Spec *specs, int nspecs, long long id) {
    int lo = 0, hi = nspecs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (specs[mid].offset <= id) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

constexpr int kPatternWords = 4;  // words per thread (see composite_kernel)

__global__ void pattern_kernel(const PatternSpec *specs, int nspecs, const u64 *affine,
                               const unsigned short *inv_table, u64 *patterns, long long total) {
    const long long base = (long long)blockIdx.x * blockDim.x * kPatternWords + threadIdx.x;
    if (base >= total) return;
    int s = find_spec(specs, nspecs, base);
    for (int i = 0; i < kPatternWords; ++i) {
        const long long id = base + (long long)i * blockDim.x;
        if (id >= total) break;
        while (s + 1 < nspecs && specs[s + 1].offset <= id) ++s;
        const PatternSpec S = specs[s];
        const int q = S.q;
        const int rel = int(id - S.offset);
        const int rho = rel / q;
        const int u = rel % q;
        const u64 *aff = affine + S.aff;
        const int inv = rho ? inv_table[q * kMaximumPrime + rho] : 0;
        int x = (S.s * u) % q;
        u64 word = 0;
        for (int j = 0; j < 64; ++j) {
            bool ok;
            if (rho == 0) {
                ok = x != 0 && S.lead_ok;  // q | d: q !| a, and c_n a square mod q for even degree
            } else {
                const int y = (x * inv) % q;
                ok = (__ldg(aff + (y >> 6)) >> (y & 63)) & 1;
            }
            if (ok) word |= u64(1) << j;
            x += S.t;
            if (x >= q) x -= q;
        }
        patterns[id] = word;
    }
}

// kCompositeWords words per thread, a block's threads interleaved (stores
// stay coalesced): one binary search over the specs per thread, then the
// spec index only moves forward.
constexpr int kCompositeWords = 16;

__global__ void composite_kernel(const CompositeSpec *specs, int nspecs, const u64 *patterns,
                                 u64 *rows, long long total) {
    const long long base = (long long)blockIdx.x * blockDim.x * kCompositeWords + threadIdx.x;
    if (base >= total) return;
    int s = find_spec(specs, nspecs, base);
    for (int i = 0; i < kCompositeWords; ++i) {
        const long long id = base + (long long)i * blockDim.x;
        if (id >= total) break;
        while (s + 1 < nspecs && specs[s + 1].offset <= id) ++s;
        const CompositeSpec &S = specs[s];
        const long long rel = id - S.offset;
        const int rho = int(rel / S.length);
        const int u = int(rel % S.length) % S.m;
        u64 word = ~u64(0);
        for (int f = 0; f < S.nf; ++f) {
            const int q = S.q[f];
            word &= __ldg(patterns + S.pattern[f] + (rho % q) * q + (u % q));
        }
        rows[id] = word;
    }
}

// ---------------------------------------------------------------------------
// Stage 2 and emission

// Warp-collective emission of sites a = base + step j for the set bits j of m.
__device__ __forceinline__ void emit(u64 m, long long base, long long step, long long d, int curve,
                                     const BatchOut &out) {
    const int lane = threadIdx.x & 31;
    const u32 cnt = __popcll(m);
    if (!__any_sync(kFullMask, cnt != 0)) return;
    u32 incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 v = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += v;
    }
    const u32 total = __shfl_sync(kFullMask, incl, 31);
    unsigned long long pos = 0;
    if (lane == 0) pos = atomicAdd(out.count, (unsigned long long)total);
    pos = __shfl_sync(kFullMask, pos, 0) + incl - cnt;
    while (m) {
        const int j = __ffsll((long long)m) - 1;
        m &= m - 1;
        if (pos < out.capacity) {
            out.a[pos] = base + step * j;
            out.d[pos] = int(d);
            out.curve[pos] = curve;
        }
        ++pos;
    }
}

// Denominator primes: for p | d and p !| a, F(a, d) = c_n a^n (mod p), not a
// square when c_n is not and n is even, so a denominator with such a prime
// factor holds no points.  True if k (d = k or k^2: p | k^2 iff p | k) has a
// prime factor in the curve's mask (the loop is uniform over the warp).
__device__ __forceinline__ bool has_denominator_prime(u32 k, u64 mask0, u64 mask1, const OddPrime *odd) {
    bool hit = false;
    for (int w = 0; w < 2; ++w)
        for (u64 m = w ? mask1 : mask0; m; m &= m - 1) {
            const int i = 64 * w + __ffsll((long long)m) - 1;
            hit |= mod_u32(k, __ldg(&odd[i].p), __ldg(&odd[i].magic)) == 0;
        }
    return hit;
}

// ---------------------------------------------------------------------------
// Wide rows with x intervals: class layout, warp-specialized like the
// single-curve kernel (which sweeps the wide rows without intervals).  Warp 0
// produces denominators into two slots: it takes work items (curve, parameter
// range, numerator range) from the device queue, skips parameters without
// admissible classes or with a denominator prime, lays out the classes clipped
// to the numerator range in shared memory, and copies the curve's stage-1 rows
// into the slot by TMA.  The other warps sweep each filled slot's items and
// release it; queued words carry a private context (curve, d), so they wait
// past later denominators and curves.  No barrier spans the CTA.

// One class of one denominator in the numerator range being swept: class
// words [wbase, wbase + words); the first word drops its `first` low bits,
// the last keeps its `last` low bits; start[sl] is the row index of class word
// wbase for modulus sl.
struct WideRun {
    int wbase;
    int words;
    unsigned short ofs;            // (r + H) mod M: the class's least a is -H + ofs
    unsigned char first;
    unsigned char last;            // 1..64
    unsigned short start[kWideSlots];
};

// Per curve and class residue r mod M (precomputed on the host): the row
// index of class word 0 for each modulus, (a0 S^-1) mod m with a0 = -H + ofs.
struct ClassStart {
    unsigned short start[kWideSlots];
    unsigned short ofs;            // (r + H) mod M
    unsigned short pad;
};
static_assert(sizeof(ClassStart) == 16, "one 16-byte load per class");

// A denominator in flight: written by the producer warp, read by the others.
struct WideSlot {
    long long d;                   // -1: no more work
    const WideRun *runs;           // the denominator's class runs (shared memory)
    const int *prefix;             // sweep-item prefix of the runs
    unsigned long long magic[kWideSlots];  // the curve's stage-1 moduli: mod_u32 constants,
    u32 m[kWideSlots];             //   moduli,
    u32 step8[kWideSlots];         //   8 ((32 kWK) mod m): byte advance per step,
    u32 soff[kWideSlots];          //   byte offsets of the staged rows
    int curve;
    int nclass;
    int next;                      // sweep-item counter
};

// A denominator a consumer warp still has queued words of.
constexpr int kWCtx = 8;
struct WideCtx {
    int d;
    int curve;
};

// Stage 2 and emission for up to 32 queued words.  A queued word carries its
// context (bits 56..58) and the position pos = a + H of its bit 0 (bits
// 0..55); its sites are a = -H + pos + M j.  A word meets the reference's
// selection, the 32 largest of the 36 candidates that do not divide its d:
// the candidates go largest first, the same one for the whole warp, each
// skipped where it divides d, until every word has met 32 or is empty.  The
// curve's descriptor and bitmasks are read through the read-only cache.
__device__ __forceinline__ void wide_drain(const u64 *qmask, const u64 *qpos, int start, int n,
                                           const WideCurve *curves, const u64 *affine,
                                           const Candidates &cand, const unsigned short *inv_table,
                                           const WideCtx *ctx, const BatchOut &out) {
    const int lane = threadIdx.x & 31;
    u64 m = 0, pos = 0;
    if (lane < n) {
        m = qmask[start + lane];
        pos = qpos[start + lane];
    }
    __syncwarp();
    const WideCtx &X = ctx[int(pos >> 56) & (kWCtx - 1)];
    const WideCurve *Cg = curves + (lane < n ? X.curve : 0);
    const u64 p56 = pos & ((u64(1) << 56) - 1);
    const u32 hi = u32(p56 >> 16), lo = u32(p56 & 0xFFFF);
    const u64 *aff = affine + __ldg(&Cg->aff);
    const u32 d = lane < n ? u32(X.d) : 1u;
    // the 32 largest candidates that do not divide d, largest first
    int tested = 0;
    for (int ci = kCandidatePrimes - 1; ci >= 0; --ci) {
        if (!__any_sync(kFullMask, m != 0 && tested < kSelectedPrimes)) break;
        const u32 p = u32(cand.p[ci]), magic = cand.magic[ci];
        const u32 rho = mod_small(d, p, magic);
        if (m != 0 && tested < kSelectedPrimes && rho != 0) {
            ++tested;
            const u32 dinv = __ldg(inv_table + p * kMaximumPrime + rho);
            u32 r = mod_small(hi, p, magic);
            r = mod_small((r << 16) | lo, p, magic);  // pos mod p
            r += __ldg(&Cg->neg_h[ci]);               // a mod p
            if (r >= p) r -= p;
            const u32 x0 = mod_small(r * dinv, p, magic);
            const u32 dx = mod_small(u32(__ldg(&Cg->m_mod[ci])) * dinv, p, magic);
            const u64 *bits = aff + ci * kRefWords;
            u64 rest = m;
            while (rest) {
                const int j = __ffsll((long long)rest) - 1;
                rest &= rest - 1;
                const u32 x = mod_small(x0 + u32(j) * dx, p, magic);
                if (!((__ldg(bits + (x >> 6)) >> (x & 63)) & 1)) m &= ~(u64(1) << j);
            }
        }
    }
    const bool any = __any_sync(kFullMask, m != 0);
    if (!any) return;
    emit(m, -__ldg(&Cg->bound) + (long long)p56, __ldg(&Cg->class_mod), X.d, __ldg(&Cg->index), out);
}

// Producer layout for curves with x intervals: denominator d's admissible
// classes clipped to the item's numerator range, into runs / prefix in
// shared memory (the whole warp; 32 classes per pass).
__device__ __forceinline__ int wide_layout(const WideCurve &C, const ClassStart *cstart, u32 du,
                                           long long d, int range, WideRun *runs, int *prefix) {
    const int lane = threadIdx.x & 31;
    const int q = C.class_prime;
    const int M = C.class_mod;
    const u64 classes2 = C.admissible[du & 63];
    const u64 classesq = q > 1 ? C.admissible[64 + int(du % u32(q))] : u64(1);
    const int nq = __popcll(classesq);
    const int nclass = __popcll(classes2) * nq;
    long long lo_a = 0, hi_a = -1;
    x_range(C.lo, C.hi, C.nint, C.bound, d, range, lo_a, hi_a);
    int carry = 0;
    for (int base = 0; base < nclass; base += 32) {
        const int c = base + lane;
        int nitems_c = 0;
        if (c < nclass) {
            const int r64 = nth_bit64(classes2, c / nq);
            int r = r64;
            if (q > 1) {
                const int rq = nth_bit64(classesq, c % nq);
                r = r64 + 64 * int(C.crt[C.mod_q[r64] * 13 + rq]);
            }
            const ClassStart cs = cstart[r];
            const int ofs = cs.ofs;
            // sites of class r: a = -H + ofs + M t, t in [0, count); those in
            // [lo_a, hi_a] are t in [t_lo, t_hi]
            const long long count = C.count_q + (ofs <= C.count_r ? 1 : 0);
            const long long a0 = -C.bound + ofs;
            const long long below = lo_a - a0;
            const long long t_lo = below <= 0 ? 0 : (below + M - 1) / M;
            const long long above = hi_a - a0;
            const long long t_hi = above < 0 ? -1 : min(count - 1, above / M);
            WideRun run;
            run.ofs = (unsigned short)ofs;
            if (t_lo <= t_hi) {
                run.wbase = int(t_lo >> 6);
                run.words = int((t_hi >> 6) - (t_lo >> 6) + 1);
                run.first = (unsigned char)(t_lo & 63);
                run.last = (unsigned char)((t_hi & 63) + 1);
            } else {
                run.wbase = 0;
                run.words = 0;
                run.first = 0;
                run.last = 64;
            }
#pragma unroll
            for (int sl = 0; sl < kWideSlots; ++sl)
                run.start[sl] = (unsigned short)mod_u32(u32(cs.start[sl]) + u32(run.wbase), u32(C.mod[sl].m),
                                                        C.mod[sl].magic);
            runs[c] = run;
            nitems_c = (run.words + kWItemWords - 1) / kWItemWords;
        }
        int incl = nitems_c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= o) incl += v;
        }
        if (c < nclass) prefix[c] = carry + incl - nitems_c;
        carry += __shfl_sync(kFullMask, incl, 31);
    }
    if (lane == 0) prefix[nclass] = carry;
    return nclass;
}

__global__ void __launch_bounds__(kWThreads, 2)
    wide_kernel(const WideCurve *__restrict__ curves, const BatchItem *__restrict__ items,
                int nitems, const u64 *__restrict__ pool, const u64 *__restrict__ affine,
                const ClassStart *__restrict__ class_starts, const unsigned short *__restrict__ inv_table, const OddPrime *__restrict__ odd,
                Candidates cand, BatchOut out, int row_stride, int max_classes, unsigned long long *work,
                unsigned long long *swept) {
    extern __shared__ __align__(16) u64 smem[];
    u64 *qmask = smem + kWSlotCount * row_stride;
    u64 *qpos = qmask + kWConsumers * kQueue;
    WideRun *runs0 = reinterpret_cast<WideRun *>(qpos + kWConsumers * kQueue);  // [slots][max_classes]
    int *prefix0 = reinterpret_cast<int *>(runs0 + kWSlotCount * max_classes);  // [slots][prefix stride]
    const int pstride = (max_classes + 1);
    __shared__ WideSlot slot[kWSlotCount];
    __shared__ WideCtx s_ctx[kWConsumers][kWCtx];
    __shared__ unsigned long long s_swept[kWConsumers][2];
    __shared__ __align__(8) unsigned long long s_full[kWSlotCount];
    __shared__ __align__(8) unsigned long long s_empty[kWSlotCount];

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int b = 0; b < kWSlotCount; ++b) {
            mbar_init(smem_addr(&s_full[b]), 1);
            mbar_init(smem_addr(&s_empty[b]), kWConsumers);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < kWConsumers * kWCtx; i += kWThreads) {
        s_ctx[i / kWCtx][i % kWCtx].d = 1;
        s_ctx[i / kWCtx][i % kWCtx].curve = 0;
    }
    __syncthreads();

    if (warp == 0) {
        // ---- producer ----
        // Work items come from the device queue with the next item's index
        // fetched ahead; lane j classifies parameter j of each 32 of an item,
        // and the live denominators go to the slots in order.  Lanes
        // 0 .. kWideSlots-1 copy one row each.
        int b = 0;
        int uses[kWSlotCount] = {};  // fills of each slot so far
        bool failed = false;
        int next_item = 0;
        if (lane == 0) next_item = int(atomicAdd(work, 1ull));
        auto acquire_slot = [&]() -> bool {
            int used = 0;
#pragma unroll
            for (int t = 0; t < kWSlotCount; ++t) used = t == b ? uses[t] : used;
            return used == 0 || mbar_wait(smem_addr(&s_empty[b]), u32(used - 1) & 1u);
        };
        for (;;) {
            const int idx = __shfl_sync(kFullMask, next_item, 0);
            if (idx >= nitems) break;
            if (lane == 0) next_item = int(atomicAdd(work, 1ull));
            const BatchItem item = items[idx];
            const WideCurve &C = curves[item.curve];
            const int q = C.class_prime;
            const unsigned long long magic_q = (~0ull) / u32(q) + 1;
            const u64 bad0 = C.denom_primes[0], bad1 = C.denom_primes[1];
            for (int base = 0; base < item.count && !failed; base += kWarpSize) {
                const bool valid = base + lane < item.count;
                const long long k = item.first + base + (valid ? lane : 0);
                const long long dd = C.square ? k * k : k;
                const u32 dv = u32(dd);
                const int dq = q > 1 ? int(mod_u32(dv, u32(q), magic_q)) : 0;
                bool live = false;
                if (valid) {
                    long long L, U;
                    live = C.admissible[dv & 63] != 0 && (q == 1 || C.admissible[64 + dq] != 0) &&
                           x_range(C.lo, C.hi, C.nint, C.bound, dd, item.range, L, U);
                }
                if (bad0 | bad1) live = live && !has_denominator_prime(u32(k), bad0, bad1, odd);
                for (u32 todo = __ballot_sync(kFullMask, live); todo; todo &= todo - 1) {
                    const int j = __ffs(todo) - 1;
                    const long long d = __shfl_sync(kFullMask, dd, j);
                    if (!acquire_slot()) {
                        failed = true;
                        break;
                    }
                    WideSlot &S = slot[b];
                    const u32 full = smem_addr(&s_full[b]);
                    const u32 du = u32(d);
                    if (lane < kWideSlots) {
                        const Modulus &Md = C.mod[lane];
                        S.magic[lane] = Md.magic;
                        S.m[lane] = u32(Md.m);
                        S.step8[lane] = 8u * Md.step;
                        S.soff[lane] = 8u * u32(Md.smem_offset);
                    }
                    WideRun *runs = runs0 + b * max_classes;
                    int *prefix = prefix0 + b * pstride;
                    const int nclass = wide_layout(C, class_starts + C.cls, du, d, item.range, runs, prefix);
                    __syncwarp();
                    if (lane == 0) {
                        S.runs = runs;
                        S.prefix = prefix;
                        S.nclass = nclass;
                        S.d = d;
                        S.curve = item.curve;
                        S.next = 0;
                        __threadfence_block();
                        mbar_arrive_expect_tx(full, u32(C.smem_words) * 8u);
                    }
                    __syncwarp();
                    if (lane < kWideSlots) {
                        // the consumers' reads of this slot's previous contents are
                        // ordered before the asynchronous copies that overwrite them
                        fence_proxy_async_shared();
                        const Modulus &Md = C.mod[lane];
                        const u32 rho = mod_u32(du, u32(Md.m), Md.magic);
                        bulk_copy_to_shared(smem_addr(smem + b * row_stride) + u32(Md.smem_offset) * 8u,
                                            pool + Md.offset + (long long)rho * Md.length,
                                            u32(Md.length) * 8u, full);
                    }
#pragma unroll
                    for (int t = 0; t < kWSlotCount; ++t) uses[t] += t == b ? 1 : 0;
                    b = b + 1 == kWSlotCount ? 0 : b + 1;
                }
            }
            if (failed) break;
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
            if (out.error && lane == 0) atomicOr(out.error, 1ull);
            // let the copies already issued land (bounded) before leaving
#pragma unroll
            for (int t = 0; t < kWSlotCount; ++t)
                if (lane == 0 && uses[t] > 0) mbar_wait(smem_addr(&s_full[t]), u32(uses[t] - 1) & 1u);
        }
        return;
    }

    // ---- consumers ----
    const int cw = warp - 1;
    u64 *wq_mask = qmask + cw * kQueue;
    u64 *wq_pos = qpos + cw * kQueue;
    WideCtx *ctx = s_ctx[cw];
    u32 phase = 0;
    int b = 0;
    int qn = 0;      // queued words (kept across denominators and curves)
    int seq = 0;     // slot fills this warp has taken
    int oldest = 0;  // oldest context that may still have queued words
    auto drain_all = [&]() {
        while (qn > 0) {
            const int nd = qn < 32 ? qn : 32;
            __syncwarp();
            wide_drain(wq_mask, wq_pos, qn - nd, nd, curves, affine, cand, inv_table, ctx, out);
            qn -= nd;
        }
    };
    // class words this warp sweeps, and the stage-1 shared-memory bytes
    // they read (8 per word and row of the curve), kept in shared memory
    unsigned long long *my_swept = s_swept[cw];
    if (lane == 0) my_swept[0] = my_swept[1] = 0;
    for (;;) {
        if (!mbar_wait(smem_addr(&s_full[b]), (phase >> b) & 1u)) {  // bounded wait
            if (out.error && lane == 0) atomicOr(out.error, 1ull);
            return;
        }
        phase ^= 1u << b;
        const WideSlot &S = slot[b];
        if (S.d < 0) {
            drain_all();
            if (lane == 0) {
                atomicAdd(swept, my_swept[0]);
                atomicAdd(swept + 1, my_swept[1]);
            }
            return;
        }
        // context kc replaces the one taken kWCtx fills ago: its queued words go first
        const int kc = seq & (kWCtx - 1);
        if (qn > 0 && seq - oldest >= kWCtx) drain_all();
        if (qn == 0) oldest = seq;
        __syncwarp();
        if (lane == 0) {
            ctx[kc].d = int(S.d);
            ctx[kc].curve = S.curve;
        }
        __syncwarp();
        const u64 tag = u64(kc) << 56;
        const WideCurve &C = curves[S.curve];
        const unsigned char *sbase = reinterpret_cast<const unsigned char *>(smem + b * row_stride);
        const u64 stride = u64(C.stride);
        const u32 rows = u32(__ldg(&C.rows));
        const WideRun *runs = S.runs;
        const int *prefix = S.prefix;
        const int nclass = S.nclass;
        u32 step8[kWideSlots], mod8[kWideSlots];
        const unsigned char *slot_base[kWideSlots];
#pragma unroll
        for (int sl = 0; sl < kWideSlots; ++sl) {
            step8[sl] = S.step8[sl];
            mod8[sl] = 8u * S.m[sl];
            slot_base[sl] = sbase + S.soff[sl];
        }
        const int total_items = prefix[nclass];
        int c = 0;  // this warp's items of a slot only increase: so do their classes
        for (;;) {
            int sweep = 0;
            if (lane == 0) sweep = atomicAdd(const_cast<int *>(&S.next), 1);
            sweep = __shfl_sync(kFullMask, sweep, 0);
            if (sweep >= total_items) break;
            // class index: largest c with prefix[c] <= sweep, from the last one on
            for (int base = c; base < nclass; base += 32) {
                const int cc = base + lane;
                const u32 bb = __ballot_sync(kFullMask, cc < nclass && prefix[cc] <= sweep);
                if (bb) c = base + 31 - __clz(bb);
                if (bb != kFullMask) break;
            }
            const int w0 = (sweep - prefix[c]) * kWItemWords;
            const WideRun run = runs[c];
            const int wt = run.words;
            if (lane == 0) {
                const u32 words = u32(min(kWItemWords, wt - w0));
                my_swept[0] += words;
                my_swept[1] += 8ull * words * rows;
            }
            const u64 first_mask = ~u64(0) << run.first;
            const u64 last_mask = run.last >= 64 ? ~u64(0) : ((u64(1) << run.last) - 1);
            const u64 pos0 = u64(run.ofs) + stride * u64(run.wbase);
            u32 o[kWideSlots];
#pragma unroll
            for (int sl = 0; sl < kWideSlots; ++sl)
                o[sl] = 8u * mod_u32(u32(run.start[sl]) + u32(w0 + lane), S.m[sl], S.magic[sl]);
#pragma unroll 1
            for (int step = 0; step < kWSteps; ++step) {
                const int ws = w0 + step * kWarpSize * kWK;
                if (ws >= wt) break;
                // a class's last step often covers fewer than kWK groups of
                // 32 words (short rows): the groups past its end are skipped
                const int nk = min(kWK, (wt - ws + kWarpSize - 1) / kWarpSize);
                u64 acc[kWK];
#pragma unroll
                for (int kk = 0; kk < kWK; ++kk)
                    acc[kk] = kk < nk ? *reinterpret_cast<const u64 *>(slot_base[0] + o[0] + 256 * kk) : 0;
#pragma unroll
                for (int sl = 1; sl < kWideSlots; ++sl) {
#pragma unroll
                    for (int kk = 0; kk < kWK; ++kk)
                        if (kk < nk) acc[kk] &= *reinterpret_cast<const u64 *>(slot_base[sl] + o[sl] + 256 * kk);
                }
#pragma unroll
                for (int sl = 0; sl < kWideSlots; ++sl) {
                    // advance (32 kWK) mod m words; unsigned min wraps into [0, m)
                    const u32 t = o[sl] + step8[sl];
                    o[sl] = min(t, t - mod8[sl]);
                }
                const u64 any = acc[0] | acc[1] | acc[2] | acc[3];
                if (!__ballot_sync(kFullMask, any != 0)) continue;
#pragma unroll
                for (int kk = 0; kk < kWK; ++kk) {
                    if (kk >= nk) break;
                    const int w = ws + kWarpSize * kk + lane;
                    u64 a = acc[kk];
                    if (w == 0) a &= first_mask;
                    if (w == wt - 1) a &= last_mask;
                    const bool live_word = a != 0 && w < wt;
                    const u32 bb = __ballot_sync(kFullMask, live_word);
                    if (bb) {
                        const int at = qn + __popc(bb & lanemask_lt());
                        if (live_word) {
                            wq_mask[at] = a;
                            wq_pos[at] = tag | (pos0 + stride * u64(w));
                        }
                        qn += __popc(bb);
                        if (qn >= 32) {
                            __syncwarp();
                            wide_drain(wq_mask, wq_pos, qn - 32, 32, curves, affine, cand, inv_table, ctx, out);
                            qn -= 32;
                            if (qn == 0) oldest = seq;
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_addr(&s_empty[b]));  // this warp is done with slot b
        ++seq;
        b = b + 1 == kWSlotCount ? 0 : b + 1;
    }
}

// ---------------------------------------------------------------------------
// Narrow rows: dense layout, one warp per denominator, whole tables in shared memory.

// Stage 2 and emission for up to 32 queued words of one curve, each with its
// denominator: the 32 largest of the 36 candidates that do not divide it,
// largest first.  Returns how many of the words it put back, from `start` on.
// Most words have one site, and one site per lane is what a candidate tests in
// one go: the words take their lowest, four candidates at a time with all their
// loads in flight, and those with more go back to the queue.  With a loop over
// each word's bits per candidate, which is left for words full of sites, a drain
// took 840 instructions and 60 % of the time of a batch of high-degree curves
// in intervals.
__device__ __forceinline__ int narrow_drain(u64 *qmask, u32 *qword, u32 *qd, int start, int n,
                                            const NarrowCurve &C, const Candidates &cand, const u64 *s_aff,
                                            const unsigned short *inv_table, const BatchOut &out) {
    const int lane = threadIdx.x & 31;
    u64 m = 0;
    u32 w = 0, d = 1;
    if (lane < n) {
        m = qmask[start + lane];
        w = qword[start + lane];
        d = qd[start + lane];
    }
    __syncwarp();
    const u32 more = __ballot_sync(kFullMask, (m & (m - 1)) != 0);
    if (__popc(more) <= kNarrowMore) {
        constexpr int kGroup = 4;
        static_assert(kCandidatePrimes % kGroup == 0, "whole groups");
        const u64 rest = m & (m - 1);
        if (rest) {
            const int at = start + __popc(more & lanemask_lt());
            qmask[at] = rest;
            qword[at] = w;
            qd[at] = d;
        }
        const u32 site = 64u * w + (m ? u32(__ffsll((long long)m) - 1) : 0u);  // a + H
        bool alive = m != 0;
        int tested = 0;
#pragma unroll 1
        for (int ci = kCandidatePrimes - 1; ci >= 0; ci -= kGroup) {
            if (!__any_sync(kFullMask, alive && tested < kSelectedPrimes)) break;
            bool ok = true;
#pragma unroll
            for (int t = 0; t < kGroup; ++t) {
                const u32 p = u32(cand.p[ci - t]), magic = cand.magic[ci - t];
                const u32 rho = mod_small(d, p, magic);
                const bool meets = alive && tested < kSelectedPrimes && rho != 0;
                const u32 dinv = meets ? __ldg(inv_table + p * kMaximumPrime + rho) : 0;
                u32 r = C.neg_h[ci - t] + mod_small(site, p, magic);  // a mod p
                if (r >= p) r -= p;
                const u32 x = mod_small(r * dinv, p, magic);
                tested += meets ? 1 : 0;
                ok &= !meets || ((s_aff[(ci - t) * kRefWords + (x >> 6)] >> (x & 63)) & 1) != 0;
            }
            alive = alive && ok;
        }
        emit(alive ? u64(1) : 0, -C.bound + (long long)site, 1, (long long)d, C.index, out);
        __syncwarp();
        return __popc(more);
    }
    int tested = 0;
    for (int ci = kCandidatePrimes - 1; ci >= 0; --ci) {
        if (!__any_sync(kFullMask, m != 0 && tested < kSelectedPrimes)) break;
        const u32 p = u32(cand.p[ci]), magic = cand.magic[ci];
        const u32 rho = mod_small(d, p, magic);
        if (m != 0 && tested < kSelectedPrimes && rho != 0) {
            ++tested;
            const u32 dinv = __ldg(inv_table + p * kMaximumPrime + rho);
            u32 r = C.neg_h[ci] + mod_small(64u * mod_small(w, p, magic), p, magic);  // a mod p
            if (r >= p) r -= p;
            const u32 x0 = mod_small(r * dinv, p, magic);
            const u64 *bits = s_aff + ci * kRefWords;
            u64 rest = m;
            while (rest) {
                const int j = __ffsll((long long)rest) - 1;
                rest &= rest - 1;
                const u32 x = mod_small(x0 + u32(j) * dinv, p, magic);
                if (!((bits[x >> 6] >> (x & 63)) & 1)) m &= ~(u64(1) << j);
            }
        }
    }
    emit(m, -C.bound + 64LL * w, 1, (long long)d, C.index, out);
    return 0;
}

// A CTA takes items (curve, parameters; all numerator ranges) and keeps the curve's
// stage-1 tables in shared memory.  A warp fetches up to 32 parameters and
// classifies one per lane (2-adic masks, denominator primes, numerator range),
// then sweeps the live ones in turn; live words of all of them share its
// queue, so that stage 2 runs with full warps.
//
// What bounds it is instruction issue (72 % of the slots): with the range of x
// (fp64, 16 cycles an instruction on this chip), the denominator primes and the
// selection of stage 2's primes worked out by a whole warp per denominator, 96
// curves of degree 12 to 40, 1e5 denominators in three intervals each, took 41.5
// ms; classified by lanes 21.4 (60 % of it stage 2: a range of 347 words sends
// 43 there), with stage 2 by sites 18.9; 384 quartics and cubics up to H =
// 30,000 2.10 and 1.82.  The curve's constants stay in shared memory: held in
// registers they spill (+10 %).  Rows long enough to sweep 64 words without a
// wrap, one CTA of 24 warps per SM, have no bank conflicts (a quarter of the
// reads here) but wait for each other at an item's end: 22.4 and 2.25 ms.
__global__ void __launch_bounds__(kNThreads, 3)
    narrow_kernel(const NarrowCurve *__restrict__ curves, const BatchItem *__restrict__ items,
                  int nitems, const u64 *__restrict__ pool, const u64 *__restrict__ affine,
                  const unsigned short *__restrict__ inv_table, const OddPrime *__restrict__ odd,
                  Candidates cand, BatchOut out, unsigned long long *work, unsigned long long *swept) {
    extern __shared__ __align__(16) u64 smem[];
    __shared__ NarrowCurve C;
    __shared__ int s_item;
    __shared__ int s_next;
    __shared__ int s_abort;
    __shared__ int s_nbad;
    __shared__ uint2 s_bad[kOddPrimes];  // the curve's denominator primes: p^-1 mod 2^32, (2^32 - 1) / p
    // (k lane) mod m for k = 1 and kNK, 32 mod m
    __shared__ unsigned char s_lane1[kNarrowSlots][kWarpSize], s_lane4[kNarrowSlots][kWarpSize];
    __shared__ u32 s_step32[kNarrowSlots];
    __shared__ __align__(8) unsigned long long s_bar;

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const u64 *tab = smem;
    const u64 *s_aff = smem + kNarrowTableWords;  // the curve's 36 candidate bitmasks
    u64 *queues = smem + kNarrowTableWords + kAffWords;
    u64 *wq_mask = queues + warp * kNarrowQueue;
    u32 *wq_word = reinterpret_cast<u32 *>(queues + kNWarps * kNarrowQueue) + warp * kNarrowQueue;
    u32 *wq_d = wq_word + kNWarps * kNarrowQueue;
    const u32 bar = smem_addr(&s_bar);
    u32 phase = 0;
    int cur = -1;
    // row words this warp sweeps and the stage-1 shared-memory bytes they read
    unsigned long long swept_words = 0, swept_bytes = 0, counted = 0;
    // lane s mod 8 works out modulus s of a denominator: its constants
    const int my = lane & (kNarrowSlots - 1);
    u32 my_m = 1, my_shift = 0, my_off = 0, my_len = 1;
    unsigned long long my_magic = ~0ull;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    for (;;) {
        if (threadIdx.x == 0) {
            s_item = int(atomicAdd(work, 1ull));
            s_next = 0;
        }
        __syncthreads();
        const int it = s_item;
        if (it >= nitems) break;
        const BatchItem item = items[it];
        if (item.curve != cur) {
            const u32 *src = reinterpret_cast<const u32 *>(curves + item.curve);
            u32 *dst = reinterpret_cast<u32 *>(&C);
            for (int i = threadIdx.x; i < int(sizeof(NarrowCurve) / 4); i += kNThreads) dst[i] = src[i];
            cur = item.curve;
            __syncthreads();
            for (int t = threadIdx.x; t < kNarrowSlots * kWarpSize; t += kNThreads) {
                const int s = t / kWarpSize, l = t % kWarpSize;
                s_lane1[s][l] = (unsigned char)(u32(l) % u32(C.m[s]));
                s_lane4[s][l] = (unsigned char)(u32(kNK * l) % u32(C.m[s]));
            }
            if (threadIdx.x < kNarrowSlots) s_step32[threadIdx.x] = u32(kWarpSize) % u32(C.m[threadIdx.x]);
            const u64 bad0 = C.denom_primes[0], bad1 = C.denom_primes[1];
            if (int(threadIdx.x) < kOddPrimes) {
                const int i = int(threadIdx.x), b = i & 63;
                if (((i < 64 ? bad0 : bad1) >> b) & 1) {
                    const int rank = __popcll((i < 64 ? bad0 : bad1) & ((u64(1) << b) - 1)) + (i < 64 ? 0 : __popcll(bad0));
                    s_bad[rank] = make_uint2(odd[i].inverse, 0xFFFFFFFFu / odd[i].p);
                }
            }
            my_m = u32(C.m[my]);
            my_magic = C.magic[my];
            my_shift = C.shift[my];
            my_off = u32(C.off[my]);
            my_len = u32(C.len[my]);
            if (threadIdx.x == 0) {
                s_nbad = __popcll(bad0) + __popcll(bad1);
                fence_proxy_async_shared();
                mbar_arrive_expect_tx(bar, u32(C.table_words + kAffWords) * 8u);
                bulk_copy_to_shared(smem_addr(smem), pool + C.tables, u32(C.table_words) * 8u, bar);
                bulk_copy_to_shared(smem_addr(smem + kNarrowTableWords), affine + C.aff,
                                    u32(kAffWords) * 8u, bar);
            }
            if (!mbar_wait(bar, phase)) {
                s_abort = 1;
                if (out.error) atomicOr(out.error, 1ull);
            }
            phase ^= 1u;
            __syncthreads();
            if (s_abort) {
                if (threadIdx.x == 0) mbar_wait(bar, phase ^ 1u);
                return;
            }
        }
        // parameters per fetch: a lane each, but every warp gets some
        const int fetch = max(1, min(kWarpSize, (item.count + 2 * kNWarps - 1) / (2 * kNWarps)));
        const int nbad = s_nbad;
        int qn = 0;
        for (;;) {
            int idx0 = 0;
            if (lane == 0) idx0 = atomicAdd(&s_next, fetch);
            idx0 = __shfl_sync(kFullMask, idx0, 0);
            if (idx0 >= item.count) break;
            const bool valid = lane < fetch && idx0 + lane < item.count;
            const long long k = item.first + idx0 + (valid ? lane : 0);
            const u32 dd = C.square ? u32(k) * u32(k) : u32(k);
            bool live = valid && C.dense2[dd & 63] != 0;
            bool hit = false;
#pragma unroll 4
            for (int i = 0; i < nbad; ++i) hit |= u32(k) * s_bad[i].x <= s_bad[i].y;
            live = live && !hit;
            for (int interval = 0;;) {
                // the denominators' next numerator range, a in [L, U]: words
                // [w_lo, w_hi], the first keeping its bits from L on, the last up to U
                long long L = -C.bound, U = C.bound;
                bool here = live;
                if (C.nint > 0)
                    here = live && next_x_range(C.lo, C.hi, C.nint, C.bound, double(dd), interval, L, U);
                u32 todo = __ballot_sync(kFullMask, here);
                if (!todo) break;
                const u32 first = u32(L + C.bound), last = u32(U + C.bound);
                for (; todo; todo &= todo - 1) {
                    const int j = __ffs(todo) - 1;
                    const u32 d = __shfl_sync(kFullMask, dd, j);
                    const u32 lo_j = __shfl_sync(kFullMask, first, j), hi_j = __shfl_sync(kFullMask, last, j);
                    const int w_lo = int(lo_j >> 6), w_hi = int(hi_j >> 6);
                    const u64 first_mask = ~u64(0) << (lo_j & 63), last_mask = ~u64(0) >> (63 - (hi_j & 63));
                    const u64 mask2 = C.dense2[d & 63];
                    swept_words += u32(w_hi - w_lo + 1);
                    // per modulus: the table word of row d mod m and the row index of word w_lo
                    const u32 mine = (my_off + mod_u32(d, my_m, my_magic) * my_len) |
                                     (mod_u32(my_shift + u32(w_lo), my_m, my_magic) << 16);
                    static_assert(kNarrowTableWords < 65536, "table words fit 16 bits");
                    u32 base[kNarrowSlots], at[kNarrowSlots];
#pragma unroll
                    for (int s = 0; s < kNarrowSlots; ++s) {
                        const u32 v = __shfl_sync(kFullMask, mine, s);
                        base[s] = v & 0xFFFFu;
                        at[s] = v >> 16;
                    }
                    // Short ranges: lane l takes word w0 + l of each 32-word step.
                    // Others: words w0 + kNK l .. w0 + kNK l + kNK - 1 of each
                    // 128-word step: rows repeat their first kNK - 1 words, so the
                    // kNK words of a lane never wrap and one index per modulus
                    // advances.
                    const bool wide = w_hi - w_lo >= kNShortWords;
#pragma unroll
                    for (int s = 0; s < kNarrowSlots; ++s) {
                        const u32 t = at[s] + u32(wide ? s_lane4[s][lane] : s_lane1[s][lane]);
                        at[s] = min(t, t - u32(C.m[s]));
                    }
                    for (int w0 = w_lo;;) {
                        u64 acc[kNK];
                        int w = w0 + lane;
                        if (wide) {
#pragma unroll
                            for (int k4 = 0; k4 < kNK; ++k4) acc[k4] = mask2;
#pragma unroll
                            for (int s = 0; s < kNarrowSlots; ++s) {
                                const u64 *row = tab + base[s] + at[s];
#pragma unroll
                                for (int k4 = 0; k4 < kNK; ++k4) acc[k4] &= row[k4];
                                const u32 t = at[s] + C.step[s];
                                at[s] = min(t, t - u32(C.m[s]));
                            }
                            w = w0 + kNK * lane;
                            if (w0 == w_lo || w0 + kWarpSize * kNK - 1 > w_hi) {  // the range's first or last step
#pragma unroll
                                for (int k4 = 0; k4 < kNK; ++k4) {
                                    if (w + k4 > w_hi) acc[k4] = 0;
                                    if (w + k4 == w_lo) acc[k4] &= first_mask;
                                    if (w + k4 == w_hi) acc[k4] &= last_mask;
                                }
                            }
                        } else {
                            acc[0] = mask2;
#pragma unroll
                            for (int k4 = 1; k4 < kNK; ++k4) acc[k4] = 0;
#pragma unroll
                            for (int s = 0; s < kNarrowSlots; ++s) {
                                acc[0] &= tab[base[s] + at[s]];
                                const u32 t = at[s] + s_step32[s];
                                at[s] = min(t, t - u32(C.m[s]));
                            }
                            if (w > w_hi) acc[0] = 0;
                            if (w == w_lo) acc[0] &= first_mask;
                            if (w == w_hi) acc[0] &= last_mask;
                        }
                        // queue the live words, those of one k4 after another: one
                        // copy of stage 2, or the kernel outgrows the instruction cache
                        int left = wide ? kNK : 1;
                        if (wide && !__any_sync(kFullMask, (acc[0] | acc[1] | acc[2] | acc[3]) != 0)) left = 0;
#pragma unroll 1
                        for (; left; --left) {
                            const u64 word = acc[0];
                            const u32 b = __ballot_sync(kFullMask, word != 0);
                            if (word) {
                                const int pos = qn + __popc(b & lanemask_lt());
                                wq_mask[pos] = word;
                                wq_word[pos] = u32(w);
                                wq_d[pos] = d;
                            }
                            qn += __popc(b);
                            while (qn >= 32) {
                                __syncwarp();
                                qn -= 32;
                                qn += narrow_drain(wq_mask, wq_word, wq_d, qn, 32, C, cand, s_aff, inv_table, out);
                            }
                            acc[0] = acc[1];
                            acc[1] = acc[2];
                            acc[2] = acc[3];
                            acc[3] = 0;
                            ++w;
                        }
                        w0 += wide ? kWarpSize * kNK : kWarpSize;
                        if (w0 > w_hi) break;
                    }
                }
                if (C.nint == 0) break;
            }
        }
        // the queue's words are this curve's: stage 2 before the next item
        while (qn) {
            __syncwarp();
            const int n = min(qn, kWarpSize);
            qn -= n;
            qn += narrow_drain(wq_mask, wq_word, wq_d, qn, n, C, cand, s_aff, inv_table, out);
        }
        swept_bytes += 8ull * u32(C.rows) * (swept_words - counted);
        counted = swept_words;
        __syncthreads();
    }
    if (lane == 0) {
        atomicAdd(swept, swept_words);
        atomicAdd(swept + 1, swept_bytes);
    }
}

}  // namespace dev

// ---------------------------------------------------------------------------
// Host driver

namespace {

using Clock = std::chrono::steady_clock;
double ms_since(Clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(Clock::now() - t0).count();
}

// Grow-only device array: kept across runs, reallocated only when a run
// needs more room than it has.
template <typename T>
struct DeviceArray {
    T *p = nullptr;
    std::size_t cap = 0;
    DeviceArray() = default;
    DeviceArray(const DeviceArray &) = delete;
    DeviceArray &operator=(const DeviceArray &) = delete;
    ~DeviceArray() { cudaFree(p); }
    void ensure(std::size_t count, const char *what) {
        count = std::max<std::size_t>(count, 1);
        if (count <= cap) return;
        cudaFree(p);
        p = nullptr;
        cap = 0;
        p = static_cast<T *>(device_malloc(count * sizeof(T), what));
        cap = count;
    }
    std::size_t bytes() const { return cap * sizeof(T); }
    void free() {
        cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    void upload(const std::vector<T> &v, cudaStream_t s, unsigned long long &bytes, const char *what) {
        ensure(v.size(), what);
        if (!v.empty())
            check_cuda(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s),
                       what);
        bytes += v.size() * sizeof(T);
    }
};

// Host threads that share the per-curve work of batched runs (any number of
// runs at a time).  They are started as work arrives, wait for more, and end
// after a second without any: starting 16 threads for each of a run's four
// loops took longer than the loops of a small batch.
class Workers {
public:
    struct Job {
        std::function<void(std::size_t)> fn;
        std::size_t n = 0;
        std::atomic<std::size_t> next{0};
        int running = 0;  // threads inside, the caller apart (guarded by the mutex)
        std::exception_ptr error;
    };

    // The process's instance; a child made by fork, which has none of its
    // threads, gets a new one.  Never destroyed: its threads may outlive main.
    static Workers &get() {
        static std::mutex *creation = new std::mutex();
        static Workers *instance = nullptr;
        std::lock_guard<std::mutex> lock(*creation);
        if (!instance || instance->pid_ != getpid()) instance = new Workers();
        return *instance;
    }

    // fn(i) for i in [0, n), the caller taking part; rethrows the first exception.
    void run(std::size_t n, std::function<void(std::size_t)> fn) {
        const auto job = std::make_shared<Job>();
        job->fn = std::move(fn);
        job->n = n;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            jobs_.push_back(job);
            const std::size_t wanted = std::min<std::size_t>(n - 1, limit_);
            try {
                while (threads_ < wanted) {
                    std::thread(&Workers::loop, this).detach();
                    ++threads_;
                }
            } catch (const std::system_error &) {
                // no more threads to be had: those there are, and the caller, do the work
            }
        }
        wake_.notify_all();
        work(*job);
        std::unique_lock<std::mutex> lock(mutex_);
        const auto it = std::find(jobs_.begin(), jobs_.end(), job);
        if (it != jobs_.end()) jobs_.erase(it);
        done_.wait(lock, [&] { return job->running == 0; });
        if (job->error) std::rethrow_exception(job->error);
    }

private:
    Workers() : pid_(getpid()), limit_(std::min(std::max(std::thread::hardware_concurrency(), 1u), 64u) - 1) {}

    void work(Job &job) {
        for (std::size_t i; (i = job.next.fetch_add(1)) < job.n;) {
            try {
                job.fn(i);
            } catch (...) {
                std::lock_guard<std::mutex> lock(mutex_);
                if (!job.error) job.error = std::current_exception();
            }
        }
    }

    void loop() {
        std::unique_lock<std::mutex> lock(mutex_);
        while (wake_.wait_for(lock, std::chrono::seconds(1), [&] { return !jobs_.empty(); })) {
            const std::shared_ptr<Job> job = jobs_.front();
            if (job->next.load() >= job->n) {
                jobs_.pop_front();  // nothing of it left to take
                continue;
            }
            ++job->running;
            lock.unlock();
            work(*job);
            lock.lock();
            --job->running;
            done_.notify_all();
        }
        --threads_;
    }

    const pid_t pid_;
    const std::size_t limit_;
    std::size_t threads_ = 0;
    std::mutex mutex_;
    std::condition_variable wake_, done_;
    std::deque<std::shared_ptr<Job>> jobs_;
};

// Runs fn(i) for i in [0, n) on the host's threads; rethrows the first exception.
template <typename F>
void parallel_for(std::size_t n, F &&fn) {
    if (n < 2 || std::thread::hardware_concurrency() <= 1) {
        for (std::size_t i = 0; i < n; ++i) fn(i);
        return;
    }
    Workers::get().run(n, std::function<void(std::size_t)>(std::ref(fn)));
}

long long gcd_ll(long long a, long long b) {
    if (a < 0) a = -a;
    while (b) {
        const long long t = a % b;
        a = b;
        b = t;
    }
    return a;
}

bool is_small_prime(int n) {
    if (n < 2) return false;
    for (int f = 2; f * f <= n; ++f)
        if (n % f == 0) return false;
    return true;
}

unsigned long long host_magic(int m) {
    return m == 1 ? ~0ull : (~0ull) / (unsigned long long)m + 1;
}

// Position of the odd prime p in the list of odd primes (3 -> 0, 5 -> 1, ...).
int odd_prime_index(int p) {
    int i = 0;
    for (int f = 3; f < p; f += 2) i += is_small_prime(f) ? 1 : 0;
    return i;
}

// Bit i set iff the i-th odd prime p below 512 (p != skip) is a denominator
// prime of the curve: even degree and c_n a nonzero non-square mod p (a
// denominator divisible by one holds no points).
void denominator_prime_mask(const std::vector<std::string> &coefficients, int skip, dev::u64 out[2]) {
    out[0] = out[1] = 0;
    if ((coefficients.size() - 1) % 2) return;
    int i = 0;
    for (int p = 3; p < kMaximumPrime; p += 2) {
        if (!is_small_prime(p)) continue;
        const int lc = decimal_mod(coefficients.back(), p);
        if (p != skip && lc != 0 && !square_mod(lc, p)) out[i >> 6] |= dev::u64(1) << (i & 63);
        ++i;
    }
}

bool lead_is_square(const std::vector<std::string> &coefficients, int q) {
    const int n = int(coefficients.size()) - 1;
    if (n % 2) return true;  // odd degree: F(a, d) = d (...) vanishes mod q | d
    const int lc = decimal_mod(coefficients.back(), q);
    for (int v = 0; v < q; ++v)
        if ((v * v) % q == lc) return true;
    return false;
}

int round_even(long long v) { return int((v + 1) & ~1LL); }

// A rational bound as a double (leading 18 digits of numerator and
// denominator), +-inf beyond 1e300: the device widens every range by one site,
// far more than this rounding can move a bound that matters (|x d| <= 2^36).
double approx_value(const Rational &r) {
    auto split = [](const BigInt &v, double &mant, long &exp10) {
        std::string t = v.to_string();
        const bool neg = !t.empty() && t[0] == '-';
        if (neg) t.erase(0, 1);
        const std::size_t keep = std::min<std::size_t>(t.size(), 18);
        mant = std::stod(t.substr(0, keep));
        exp10 = long(t.size() - keep);
        if (neg) mant = -mant;
    };
    double mn, md;
    long en, ed;
    split(r.num, mn, en);
    split(r.den, md, ed);
    if (mn == 0) return 0.0;
    const long e = en - ed;
    if (e > 300) return mn > 0 ? HUGE_VAL : -HUGE_VAL;
    if (e < -300) return 0.0;
    return mn / md * std::pow(10.0, double(e));
}

// The intervals as ascending (lo, hi) doubles for the device ranges; false
// when there are none or more than the device takes (then rows are swept whole).
bool device_intervals(const std::vector<SearchInterval> &intervals, int &nint, double *lo, double *hi) {
    nint = 0;
    if (intervals.empty() || intervals.size() > std::size_t(dev::kMaxIntervals)) return false;
    std::vector<std::pair<double, double>> v;
    for (const auto &iv : intervals)
        v.push_back({iv.lower_infinite ? -HUGE_VAL : approx_value(iv.lower),
                     iv.upper_infinite ? HUGE_VAL : approx_value(iv.upper)});
    std::sort(v.begin(), v.end());
    for (const auto &p : v) {
        lo[nint] = p.first;
        hi[nint] = p.second;
        ++nint;
    }
    return true;
}

struct CurveWork {
    bool ok = false;
    bool wide = false;
    std::unique_ptr<ExactPolynomial> poly;
    FastPlan plan;
    long long words = 0;       // dense 64-site words per row
    long long swept = 0;       // words a denominator sweeps after interval narrowing (estimate)
    long long count = 0;       // parameters
    dev::u64 adm2[64] = {};    // 2-adic admissible classes by d mod 64
    int classes = 1;           // wide curves: most numerator classes of one denominator
    std::unique_ptr<FastPlanner> planner;  // wide curves, until planned
    std::unique_ptr<SweepCurve> sweep;     // curves swept by launches of their own
    std::vector<unsigned short> cand_residues;  // c_i mod p for the 36 candidates, candidate-major
    dev::u64 denom_primes[2] = {};             // the curve's denominator primes (no class prime removed)
};

// Words of one denominator's row that the sieve sweeps: the whole row, or with
// x intervals the interval numerators at a middle denominator (each interval
// [lo, hi] covers about (hi - lo) d / 64 words).  Picks the kernel shape.
long long swept_row_words(const BatchCurveSpec &c, long long first, long long last, long long words) {
    if (c.intervals.empty() || c.intervals.size() > std::size_t(dev::kMaxIntervals)) return words;
    const double dmid = 0.5 * double(first) + 0.5 * double(std::max(first, last));
    const double d = c.square ? dmid * dmid : dmid;
    double total = 0;
    for (const auto &iv : c.intervals) {
        if (iv.lower_infinite || iv.upper_infinite) return words;
        const double len = approx_value(iv.upper) - approx_value(iv.lower);
        if (len < 0) continue;
        total += std::min(double(words), len * d / 64.0 + 2.0);
    }
    return std::min(words, (long long)std::ceil(total));
}

// Whether a curve gets sieve launches of its own (sweep.hpp) instead of work
// items of the batched kernels.  Rows of at least kBatchWideWords words always
// do; shorter ones from 322 words on, with denominators enough.  Kernel time of
// 400,000 denominators, mean of six random sextics, narrow kernel and sweep: H =
// 5,000 0.21 and 0.22 ms, 10,000 0.28 and 0.21, 20,000 0.40 and 0.21, 65,000
// 1.04 and 0.23; of 40,000 at H = 20,000 0.10 and 0.04, of 4,000 at 65,000 0.045
// and 0.025.  A launch of a curve's own needs its sweep plan (some 0.1 ms of a
// host core) and tables (0.03 ms), which the narrow kernel shares better among
// many small curves.  The line is flat: with 0.7 for 0.9 or 8,000 for 20,000,
// bursts of requests and batches change by 4 % at most, either way.
// Curves with x intervals stay in the kernels that sweep only those.
bool swept_alone(const BatchCurveSpec &c, bool wide, long long words, long long count) {
    if (!c.intervals.empty() && c.intervals.size() <= std::size_t(dev::kMaxIntervals)) return false;
    if (wide) return true;
    return double(count) * (2.8e-3 * double(words) - 0.9) > 20000.0;
}

// Narrow plan: every odd prime up to kBatchNarrowModulus that filters at
// least 0.15 bit, strongest first, each joining the slot whose product stays
// within the cap (smallest product first) or opening a new slot, while the
// tables (m rows of m + kNK - 1 words per slot) fit shared memory.
FastPlan narrow_plan(const std::vector<std::string> &coefficients) {
    std::vector<std::pair<double, int>> strength;
    for (int q = 3; q <= kBatchNarrowModulus; q += 2) {
        if (!is_small_prime(q)) continue;
        const double rate = pass_rate(q, coefficients);
        const double bits = rate > 0 ? -std::log2(rate) : 8.0;
        if (bits >= 0.15) strength.push_back({bits, q});
    }
    std::sort(strength.begin(), strength.end(), [](const auto &a, const auto &b) {
        return a.first != b.first ? a.first > b.first : a.second < b.second;
    });
    auto words = [](long long m) { return m * (m + dev::kNK - 1); };
    FastPlan plan;
    long long used = 0;
    for (const auto &sq : strength) {
        const int q = sq.second;
        int join = -1;
        for (std::size_t i = 0; i < plan.moduli.size(); ++i)
            if (plan.moduli[i] * q <= kBatchNarrowModulus &&
                (join < 0 || plan.moduli[i] < plan.moduli[std::size_t(join)]))
                join = int(i);
        if (join >= 0) {
            const long long m = plan.moduli[std::size_t(join)];
            const long long grown = used - words(m) + words(m * q);
            if (grown + dev::kNK * (dev::kNarrowSlots - long(plan.moduli.size())) >
                dev::kNarrowTableWords - 1)  // one word may pad the block to an even length
                continue;
            used = grown;
            plan.moduli[std::size_t(join)] *= q;
            plan.slots[std::size_t(join)].push_back(q);
        } else {
            if (int(plan.moduli.size()) == dev::kNarrowSlots) continue;
            const long long grown = used + words(q);
            if (grown + dev::kNK * (dev::kNarrowSlots - long(plan.moduli.size()) - 1) >
                dev::kNarrowTableWords - 1)
                continue;
            used = grown;
            plan.moduli.push_back(q);
            plan.slots.push_back({q});
        }
        plan.bits += sq.first;
    }
    return plan;
}

// Wide plan: moduli capped so that tables stay small against the curve's
// work, and the staged rows fit the shared-memory budget.
// Staged row words a wide curve may use (both buffers together) so that a
// CTA stays within a third of an SM's shared memory: static arrays, queues,
// and two sets of class runs and item prefixes for max_classes classes.
long long wide_row_budget(int max_classes) {
    const long long per_cta = 228 * 1024 / 2 - 1024;
    const long long fixed = 6 * 1024 +  // static shared memory of the kernel (5 KB) and slack
                            (long long)dev::kWConsumers * dev::kQueue * 16 +
                            (long long)dev::kWSlotCount * max_classes * 32 +
                            (long long)dev::kWSlotCount * ((max_classes + 4) & ~3) * 4;
    return std::max(2LL * 64, (per_cta - fixed) / 8);
}

// Admissible residues mod the class prime q by d mod q: bit r of out[dq] is
// set iff f(r / dq) is a square mod q, or (q | d) r != 0 and c_n is a square.
void class_prime_residues(const std::vector<std::string> &coefficients, int q, dev::u64 *out) {
    const auto aff = affine_mask(q, coefficients);
    const bool lead = lead_is_square(coefficients, q);
    for (int dq = 0; dq < q; ++dq) {
        out[dq] = 0;
        const int inverse = dq == 0 ? 0 : int(mod_inverse(dq, q));
        for (int r = 0; r < q; ++r) {
            const bool ok = dq == 0 ? (r != 0 && lead) : aff[(r * inverse) % q] != 0;
            if (ok) out[dq] |= dev::u64(1) << r;
        }
    }
}

// Most numerator classes of any one denominator of a wide curve: admissible
// 2-adic classes times admissible residues of the class prime.
int wide_classes(const std::vector<std::string> &coefficients, const dev::u64 adm2[64], int q) {
    int most2 = 0, mostq = 1;
    for (int dd = 0; dd < 64; ++dd) most2 = std::max(most2, __builtin_popcountll(adm2[dd]));
    if (q > 1) {
        dev::u64 admq[13];
        class_prime_residues(coefficients, q, admq);
        mostq = 0;
        for (int dq = 0; dq < q; ++dq) mostq = std::max(mostq, __builtin_popcountll(admq[dq]));
    }
    return most2 * std::max(1, mostq);
}

// max_classes: the most classes of a denominator of any wide curve in the
// launch, which sizes the slots' class arrays and so the share of shared
// memory left for rows.
FastPlan wide_plan(const FastPlanner &planner, long double work, int max_classes) {
    int cap = int(std::min<long double>(kMaxModulus, std::max<long double>(64, std::sqrt(work / 48.0L))));
    // two slots of staged rows
    const long long smem_budget =
        std::min<long long>(dev::kWMaxSmemWords, wide_row_budget(max_classes) / dev::kWSlotCount);
    for (;;) {
        FastPlan plan = planner.plan(cap, dev::kWideSlots, 1LL << 40, false);
        long long smem = 0;
        for (int sl = 0; sl < dev::kWideSlots; ++sl) {
            const int m = sl < int(plan.moduli.size()) ? plan.moduli[sl] : 1;
            smem += round_even(m + dev::kWExt);
        }
        if (smem <= smem_budget || cap <= 64) return plan;
        cap = cap * 7 / 8;
    }
}

}  // namespace

namespace {

// Everything one batched run launches: per-curve descriptors, table specs
// and work items, built on the host from the curves' plans.
struct BatchPlan {
    std::vector<CurveWork> work;
    std::vector<std::size_t> sweeps;           // curves with launches of their own
    std::vector<dev::WideCurve> wide;
    std::vector<dev::NarrowCurve> narrow;
    std::vector<dev::AffineSpec> aspecs;
    std::vector<unsigned short> residues;
    std::vector<dev::PatternSpec> pspecs;
    std::vector<dev::CompositeSpec> cspecs;
    std::vector<dev::BatchItem> wide_items, narrow_items;
    std::vector<dev::ClassStart> class_starts;
    long long aff_words = 0, pattern_words = 0, row_words = 0;
    int wide_smem_words = 0;
    int wide_max_classes = 1;   // most classes of a denominator of any wide curve

    // Empty, with the arrays' memory kept for the next run.
    void clear() {
        work.clear(), sweeps.clear(), wide.clear(), narrow.clear(), aspecs.clear(), residues.clear();
        pspecs.clear(), cspecs.clear(), wide_items.clear(), narrow_items.clear(), class_starts.clear();
        aff_words = pattern_words = row_words = 0;
        wide_smem_words = 0;
        wide_max_classes = 1;
    }
    std::size_t bytes() const {
        auto of = [](const auto &v) { return v.capacity() * sizeof(v[0]); };
        return of(work) + of(sweeps) + of(wide) + of(narrow) + of(aspecs) + of(residues) + of(pspecs) + of(cspecs) +
               of(wide_items) + of(narrow_items) + of(class_starts);
    }
};

// Validation and per-curve plans (one curve per task), then descriptors,
// table specs and work items in the order the kernels take them.  Curves
// marked in `solo` are validated and planned, but given no denominators.
void build_plan(const std::vector<BatchCurveSpec> &curves, const std::vector<char> &solo,
                std::vector<BatchCurveResult> &results, BatchPlan &P, BatchStats &stats, int items_per_kernel) {
    P.work.resize(curves.size());
    parallel_for(curves.size(), [&](std::size_t i) {
        const BatchCurveSpec &c = curves[i];
        BatchCurveResult &r = results[i];
        CurveWork &cw = P.work[i];
        const long long first = solo[i] ? 1 : c.first, last = solo[i] ? 0 : c.last;
        try {
            if (c.coefficients.size() < 2) throw std::invalid_argument("polynomial must have degree >= 1");
            if (c.bound < 1) throw std::invalid_argument("numerator bound must be positive");
            if (first < 1) throw std::invalid_argument("denominators start at 1");
            if (last > (c.square ? 46340LL : 2147483647LL))
                throw std::invalid_argument("denominator range too large for 32-bit denominators");
            if (c.bound > (1LL << 33))
                throw std::invalid_argument("numerator bound too large for the batched search");
            cw.poly.reset(new ExactPolynomial(c.coefficients));
            if (!cw.poly->is_squarefree()) {
                r.status = 6;
                r.error = "polynomial is not squarefree";
                return;
            }
            cw.words = word_count64(c.bound);
            cw.count = last >= first ? last - first + 1 : 0;
            cw.swept = swept_row_words(c, first, last, cw.words);
            cw.wide = cw.swept >= kBatchWideWords;
            if (cw.count > 0 && swept_alone(c, cw.wide, cw.words, cw.count)) {
                cw.sweep = batch_sweep_curve(c, &cw.plan);
                cw.ok = true;
                return;
            }
            two_adic_classes(c.coefficients, cw.adm2);
            if (cw.wide) {
                cw.planner.reset(new FastPlanner(c.coefficients, c.bound, true, kFastPrimeLimit));
                cw.classes = wide_classes(c.coefficients, cw.adm2, cw.planner->class_prime());
            } else {
                cw.plan = narrow_plan(c.coefficients);
            }
            denominator_prime_mask(c.coefficients, 1, cw.denom_primes);
            {
                const auto &cps = candidate_primes();
                cw.cand_residues.reserve(kCandidatePrimes * c.coefficients.size());
                for (int ci = 0; ci < kCandidatePrimes; ++ci)
                    for (const auto &coef : c.coefficients)
                        cw.cand_residues.push_back((unsigned short)decimal_mod(coef, cps[ci]));
            }
            cw.ok = true;
        } catch (const std::exception &e) {
            r.status = 1;
            r.error = e.what();
        }
    });
    // wide plans: one row budget for the launch, from the largest class count
    // of its curves (each slot holds its denominator's classes)
    int max_classes = 1;
    for (std::size_t i = 0; i < curves.size(); ++i)
        if (P.work[i].ok && P.work[i].wide && !P.work[i].sweep) max_classes = std::max(max_classes, P.work[i].classes);
    parallel_for(curves.size(), [&](std::size_t i) {
        CurveWork &cw = P.work[i];
        if (!cw.ok) return;
        if (cw.wide && !cw.sweep) {
            cw.plan = wide_plan(*cw.planner, (long double)cw.words * cw.count, max_classes);
            cw.planner.reset();
        }
        results[i].wide = cw.wide;
        results[i].class_prime = cw.plan.class_prime;
        results[i].moduli = cw.plan.moduli;
    });

    const auto &cands = candidate_primes();
    // largest work first, so that the persistent kernels end on small items
    std::vector<std::size_t> order;
    for (std::size_t i = 0; i < curves.size(); ++i) {
        const CurveWork &cw = P.work[i];
        if (!cw.ok || cw.count <= 0) continue;
        if (!cw.sweep) {
            order.push_back(i);
            continue;
        }
        P.sweeps.push_back(i);
        stats.rectangle_sites += (long double)(2 * curves[i].bound + 1) * (long double)cw.count;
        stats.denominators += (unsigned long long)cw.count;
        stats.words += (unsigned long long)(cw.words * cw.count);
        stats.curves += 1;
        stats.wide_curves += cw.wide ? 1 : 0;
    }
    // the longest first, so that the device is shared to the end
    std::stable_sort(P.sweeps.begin(), P.sweeps.end(), [&](std::size_t a, std::size_t b) {
        return P.work[a].sweep->cost(double(P.work[a].count)) > P.work[b].sweep->cost(double(P.work[b].count));
    });
    std::stable_sort(order.begin(), order.end(), [&](std::size_t a, std::size_t b) {
        return (long double)P.work[a].words * P.work[a].count >
               (long double)P.work[b].words * P.work[b].count;
    });
    // items: large enough that building and fetching them stays cheap, small
    // enough that a small batch still spreads over the device (about
    // items_per_kernel items per kernel): up to 2^21 row words (wide) and 2^18
    // swept words (narrow), at least one denominator per warp; one set per
    // numerator range
    long double wide_work = 0, narrow_work = 0;
    for (std::size_t i : order) {
        const CurveWork &cw = P.work[i];
        (cw.wide ? wide_work : narrow_work) += (long double)(cw.wide ? cw.words : cw.swept) * cw.count;
    }
    const long long wide_item =
        (long long)std::min<long double>(1LL << 21, std::max<long double>(1LL << 14, wide_work / items_per_kernel));
    const long long narrow_item =
        (long long)std::min<long double>(1LL << 18, std::max<long double>(1LL << 12, narrow_work / items_per_kernel));
    auto item_chunk = [&](const CurveWork &cw) -> long long {
        return cw.wide ? std::max(1LL, std::min<long long>(1 << 16, wide_item / cw.words))
                       : std::max<long long>(dev::kNWarps,
                                             std::min<long long>(1 << 16, narrow_item / std::max(1LL, cw.swept)));
    };
    // Where each curve's part of every array begins, so that the curves are
    // described in parallel (one after another they took half the planning of
    // a batch of 384 small searches).
    struct Place {
        std::size_t curve, aspec, residue, pspec, cspec, item, descriptor, cls;
        long long aff, pattern, row;
    };
    std::vector<Place> places;
    places.reserve(order.size());
    {
        std::size_t pspecs = 0, cspecs = 0, wide_items = 0, narrow_items = 0, wide = 0, narrow = 0, cls = 0;
        std::size_t aspecs = 0, residues = 0;
        for (std::size_t i : order) {
            const CurveWork &cw = P.work[i];
            places.push_back({i, aspecs, residues, pspecs, cspecs, cw.wide ? wide_items : narrow_items,
                              cw.wide ? wide : narrow, cls, P.aff_words, P.pattern_words, P.row_words});
            std::size_t primes = 0;
            for (const auto &slot : cw.plan.slots)
                for (int q : slot) {
                    ++primes;
                    P.pattern_words += (long long)q * q;
                }
            const int slots = cw.wide ? dev::kWideSlots : dev::kNarrowSlots;
            for (int sl = 0; sl < slots; ++sl) {
                const long long m = sl < int(cw.plan.moduli.size()) ? cw.plan.moduli[std::size_t(sl)] : 1;
                P.row_words += m * (cw.wide ? round_even(m + dev::kWExt) : m + dev::kNK - 1);
            }
            P.row_words += P.row_words % 2;  // 16-byte aligned bulk copies
            P.aff_words += (long long)(std::size_t(kCandidatePrimes) + primes) * dev::kRefWords;
            aspecs += std::size_t(kCandidatePrimes) + primes;
            residues += (std::size_t(kCandidatePrimes) + primes) * curves[i].coefficients.size();
            pspecs += primes;
            cspecs += std::size_t(slots);
            const long long chunk = item_chunk(cw);
            const std::size_t parts = std::size_t((cw.count + chunk - 1) / chunk);
            if (cw.wide) {
                if ((2 * curves[i].bound) / (64LL * cw.plan.class_prime) / 64 + 2 >= dev::kMaxClassWords)
                    throw std::invalid_argument("numerator bound too large for the batched search");
                wide_items += parts * curves[i].intervals.size();  // at most kMaxIntervals: swept_alone
                cls += 64 * std::size_t(cw.plan.class_prime);
                ++wide;
            } else {
                narrow_items += parts;
                ++narrow;
            }
            stats.rectangle_sites += (long double)(2 * curves[i].bound + 1) * (long double)cw.count;
            stats.denominators += (unsigned long long)cw.count;
            stats.words += (unsigned long long)(cw.words * cw.count);
            stats.curves += 1;
            stats.wide_curves += cw.wide ? 1 : 0;
        }
        P.wide.resize(wide);
        P.narrow.resize(narrow);
        P.aspecs.resize(aspecs);
        P.residues.resize(residues);
        P.pspecs.resize(pspecs);
        P.cspecs.resize(cspecs);
        P.wide_items.resize(wide_items);
        P.narrow_items.resize(narrow_items);
        P.class_starts.resize(cls);
    }
    parallel_for(places.size(), [&](std::size_t k) {
        Place at = places[k];
        const std::size_t i = at.curve;
        const BatchCurveSpec &c = curves[i];
        CurveWork &cw = P.work[i];
        const FastPlan &plan = cw.plan;
        auto add_affine = [&](int p, const unsigned short *residues) {
            dev::AffineSpec A{};
            A.out = at.aff;
            A.residues = (long long)at.residue;
            A.p = p;
            A.n = int(c.coefficients.size()) - 1;
            std::copy(residues, residues + c.coefficients.size(), &P.residues[at.residue]);
            at.residue += c.coefficients.size();
            P.aspecs[at.aspec++] = A;
            at.aff += dev::kRefWords;
            return A.out;
        };
        const long long H = c.bound;
        const long long aff_base = at.aff;
        // the 36 candidate bitmasks, residues computed with the plan
        for (int ci = 0; ci < kCandidatePrimes; ++ci)
            add_affine(cands[ci], &cw.cand_residues[std::size_t(ci) * c.coefficients.size()]);
        // per-prime patterns of this curve's stage-1 factors
        const long long M = cw.wide ? 64LL * plan.class_prime : 1;
        const long long S = cw.wide ? 64LL * M : 64;
        long long pattern_of[kFastPrimeLimit];
        std::vector<unsigned short> residues(c.coefficients.size());
        for (const auto &slot : plan.slots)
            for (int q : slot) {
                for (std::size_t j = 0; j < residues.size(); ++j)
                    residues[j] = (unsigned short)decimal_mod(c.coefficients[j], q);
                dev::PatternSpec Q{};
                Q.offset = at.pattern;
                Q.aff = add_affine(q, residues.data());
                Q.q = q;
                Q.lead_ok = lead_is_square(c.coefficients, q) ? 1 : 0;
                Q.s = int(S % q);
                Q.t = int(M % q);
                P.pspecs[at.pspec++] = Q;
                pattern_of[q] = at.pattern;
                at.pattern += (long long)q * q;
            }
        auto add_composite = [&](int sl, int length) {
            dev::CompositeSpec T{};
            T.offset = at.row;
            if (sl < int(plan.moduli.size())) {
                T.m = plan.moduli[sl];
                T.nf = int(plan.slots[sl].size());
                for (int f = 0; f < T.nf; ++f) {
                    T.q[f] = plan.slots[sl][f];
                    T.pattern[f] = pattern_of[T.q[f]];
                }
            } else {
                T.m = 1;  // padding: a row of ones
                T.nf = 0;
            }
            T.length = length < 0 ? T.m : length;
            P.cspecs[at.cspec++] = T;
            at.row += (long long)T.m * T.length;
            return T;
        };
        if (cw.wide) {
            dev::WideCurve C{};
            const int q = plan.class_prime;
            C.bound = H;
            C.stride = S;
            C.count_q = (2 * H) / M;
            C.count_r = int((2 * H) % M);
            C.class_prime = q;
            C.class_mod = int(M);
            C.square = c.square ? 1 : 0;
            C.index = int(i);
            C.rows = int(plan.moduli.size());
            // the class prime's classes already leave q | d without sites
            C.denom_primes[0] = cw.denom_primes[0] & ~(q > 1 ? dev::u64(1) << odd_prime_index(q) : 0);
            C.denom_primes[1] = cw.denom_primes[1];
            C.aff = aff_base;
            int smem = 0;
            for (int sl = 0; sl < dev::kWideSlots; ++sl) {
                const int m = sl < int(plan.moduli.size()) ? plan.moduli[sl] : 1;
                const dev::CompositeSpec T = add_composite(sl, round_even(m + dev::kWExt));
                dev::Modulus &Md = C.mod[sl];
                Md.offset = T.offset;
                Md.magic = host_magic(m);
                Md.m = m;
                Md.length = T.length;
                Md.smem_offset = smem;
                smem += T.length;
                Md.inv_stride = m > 1 ? dev::u32(mod_inverse(S % m, m)) : 0;
                Md.neg_h = dev::u32((m - H % m) % m);
                Md.step = dev::u32((dev::kWarpSize * dev::kWK) % m);
            }
            C.smem_words = smem;
            std::copy(cw.adm2, cw.adm2 + 64, C.admissible);
            if (q > 1) {
                class_prime_residues(c.coefficients, q, C.admissible + 64);
                const int inv64 = int(mod_inverse(64 % q, q));
                for (int a = 0; a < q; ++a)
                    for (int rq = 0; rq < q; ++rq)
                        C.crt[a * 13 + rq] = (unsigned char)(((rq - a + q) % q) * inv64 % q);
            }
            for (int r64 = 0; r64 < 64; ++r64) C.mod_q[r64] = (unsigned char)(q > 1 ? r64 % q : 0);
            // class starts for every residue r mod M: ofs = (r + H) mod M, and per
            // modulus the row index ((-H + ofs) S^-1) mod m of class word 0
            C.cls = (long long)at.cls;
            for (long long r = 0; r < M; ++r) {
                dev::ClassStart cs{};
                const long long ofs = (r + H % M) % M;
                cs.ofs = (unsigned short)ofs;
                for (int sl = 0; sl < dev::kWideSlots; ++sl) {
                    const dev::Modulus &Md = C.mod[sl];
                    const long long m = Md.m;
                    cs.start[sl] = (unsigned short)((Md.neg_h + ofs) % m * Md.inv_stride % m);
                }
                P.class_starts[at.cls++] = cs;
            }
            for (int ci = 0; ci < kCandidatePrimes; ++ci) {
                const int p = cands[ci];
                C.neg_h[ci] = (unsigned short)((p - H % p) % p);
                C.m_mod[ci] = (unsigned short)(M % p);
            }
            device_intervals(c.intervals, C.nint, C.lo, C.hi);
            const long long chunk = item_chunk(cw);
            for (int range = 0; range < C.nint; ++range)
                for (long long f = c.first; f <= c.last; f += chunk)
                    P.wide_items[at.item++] = {f, int(at.descriptor), int(std::min(chunk, c.last - f + 1)), range, 0};
            P.wide[at.descriptor] = C;
        } else {
            dev::NarrowCurve &C = P.narrow[at.descriptor];
            C.bound = H;
            C.square = c.square ? 1 : 0;
            C.index = int(i);
            C.rows = int(plan.moduli.size());
            C.denom_primes[0] = cw.denom_primes[0];
            C.denom_primes[1] = cw.denom_primes[1];
            C.aff = aff_base;
            C.tables = at.row;
            int used = 0;
            for (int sl = 0; sl < dev::kNarrowSlots; ++sl) {
                const int m = sl < int(plan.moduli.size()) ? plan.moduli[sl] : 1;
                const dev::CompositeSpec T = add_composite(sl, m + dev::kNK - 1);
                C.m[sl] = m;
                C.off[sl] = used;
                C.len[sl] = T.length;
                used += m * T.length;
                C.magic[sl] = host_magic(m);
                const long long inv64 = m > 1 ? mod_inverse(64 % m, m) : 0;
                C.shift[sl] = dev::u32(((m - H % m) % m) * inv64 % m);
                C.step[sl] = dev::u32((dev::kWarpSize * dev::kNK) % m);
            }
            used += used % 2;
            if (used > dev::kNarrowTableWords) throw std::logic_error("narrow tables exceed shared memory");
            C.table_words = used;
            // dense layout: bit j of a word holds a = -H + 64 w + j, so a = j - H (mod 64)
            const dev::u64 *by_class = cw.adm2;
            const int h64 = int(H % 64);
            for (int dd = 0; dd < 64; ++dd)  // bit j = class bit (j - H) mod 64: a rotation
                C.dense2[dd] = h64 ? (by_class[dd] << h64) | (by_class[dd] >> (64 - h64)) : by_class[dd];
            for (int ci = 0; ci < kCandidatePrimes; ++ci) {
                const int p = cands[ci];
                C.neg_h[ci] = (unsigned short)((p - H % p) % p);
            }
            device_intervals(c.intervals, C.nint, C.lo, C.hi);
            const long long chunk = item_chunk(cw);
            for (long long f = c.first; f <= c.last; f += chunk)
                P.narrow_items[at.item++] = {f, int(at.descriptor), int(std::min(chunk, c.last - f + 1)), 0, 0};
        }
    });
    for (const auto &C : P.wide) P.wide_smem_words = std::max(P.wide_smem_words, round_even(C.smem_words));
    for (const auto &at : places)
        if (P.work[at.curve].wide) P.wide_max_classes = std::max(P.wide_max_classes, P.work[at.curve].classes);
    stats.wide_items = P.wide_items.size();
    stats.narrow_items = P.narrow_items.size();
    stats.table_words = (unsigned long long)P.row_words;
}

}  // namespace

namespace {

// Curve-independent tables: inverses and squares modulo every prime below
// 512, made once per process.
struct FixedTables {
    std::vector<unsigned short> inverses;
    std::vector<dev::u64> squares;
    std::vector<dev::OddPrime> odd;
};
const FixedTables &fixed_tables() {
    static const FixedTables tables = [] {
        FixedTables t;
        t.inverses.assign(std::size_t(kMaximumPrime) * kMaximumPrime, 0);
        t.squares.assign(std::size_t(kMaximumPrime) * dev::kRefWords, 0);
        for (int p = 2; p < kMaximumPrime; ++p) {
            if (!is_small_prime(p)) continue;
            modular_inverses(p, &t.inverses[std::size_t(p) * kMaximumPrime]);
            for (int v = 0; v < p; ++v) {
                const int sq = v * v % p;
                t.squares[std::size_t(p) * dev::kRefWords + sq / 64] |= dev::u64(1) << (sq % 64);
            }
        }
        for (int p = 3; p < kMaximumPrime; p += 2)
            if (is_small_prime(p)) {
                dev::u32 inverse = dev::u32(p);  // Newton's iteration, right in 3 bits to start with
                for (int i = 0; i < 4; ++i) inverse *= 2u - dev::u32(p) * inverse;
                t.odd.push_back({dev::u32(p), inverse, host_magic(p)});
            }
        if (t.odd.size() != std::size_t(dev::kOddPrimes)) throw std::logic_error("odd prime table");
        return t;
    }();
    return tables;
}

}  // namespace

struct BatchEngine::Impl {
    int device = 0;
    int sms = 0;
    cudaStream_t stream = nullptr, side = nullptr;
    // the sweeps' launches go round-robin over these and `stream`, so that
    // the short ones share the device
    static constexpr int kSweepStreams = 7;
    cudaStream_t sweep_stream[kSweepStreams] = {};
    cudaEvent_t sweep_join[kSweepStreams] = {};
    cudaEvent_t ev[6] = {};    // tables, wide kernel, narrow kernel (start, end)
    cudaEvent_t fork = nullptr, join = nullptr;
    // device counters of a run: survivors, wide and narrow work items, error
    // word, survivors kept by pre-verification, words swept, stage-1
    // shared-memory bytes read
    static constexpr int kCounters = 7;
    unsigned long long *h_counters = nullptr;
    unsigned long long capacity = 0;  // survivors of a run (grows)
    BatchPlan plan;                   // of the run; its memory is kept
    bool failed = false;              // a run is under way, or ended with an exception
    dev::Candidates cand{};
    DeviceArray<dev::WideCurve> d_wide;
    DeviceArray<dev::NarrowCurve> d_narrow;
    DeviceArray<dev::BatchItem> d_witems, d_nitems;
    DeviceArray<dev::AffineSpec> d_aspecs;
    DeviceArray<dev::PatternSpec> d_pspecs;
    DeviceArray<dev::CompositeSpec> d_cspecs;
    DeviceArray<dev::ClassStart> d_cls;
    DeviceArray<unsigned short> d_res, d_inv;
    DeviceArray<dev::u64> d_sq, d_aff, d_patterns, d_rows;
    DeviceArray<dev::OddPrime> d_odd;
    // [0] survivors [1] wide work [2] narrow work [3] error [4] pre-verified survivors
    // [5] swept words [6] their row bytes, then a work counter per sweep
    DeviceArray<unsigned long long> d_counters;
    DeviceArray<unsigned char> d_sweep_tables;
    DeviceArray<long long> d_a, d_pa;        // survivors, and those kept by pre-verification
    DeviceArray<int> d_d, d_c, d_pd, d_pc;
    DeviceArray<unsigned long long> d_curve_modular;  // per-curve modular survivors
    Preverifier pre;
    // Curves with launches of their own (of plan.sweeps), whose tables share
    // d_sweep_tables; the builders hold the uploads' sources.
    struct SweepGroup {
        std::size_t begin = 0, end = 0;
        std::unique_ptr<SweepBuilder> tables;
    };
    std::vector<SweepGroup> sweep_groups;

    Impl() {  // on the current device
        check_cuda(cudaGetDevice(&device), "cudaGetDevice");
        check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device),
                   "cudaDeviceGetAttribute");
        check_cuda(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
        check_cuda(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking), "cudaStreamCreate");
        for (auto &s : sweep_stream) check_cuda(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "cudaStreamCreate");
        for (auto &e : sweep_join) check_cuda(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
        for (auto &e : ev) check_cuda(cudaEventCreate(&e), "cudaEventCreate");
        check_cuda(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming), "cudaEventCreate");
        check_cuda(cudaEventCreateWithFlags(&join, cudaEventDisableTiming), "cudaEventCreate");
        check_cuda(cudaMallocHost(&h_counters, 8 * sizeof(unsigned long long)), "cudaMallocHost");
        const auto &cands = candidate_primes();
        for (int ci = 0; ci < kCandidatePrimes; ++ci) {
            cand.p[ci] = cands[ci];
            cand.magic[ci] = dev::magic40(dev::u32(cands[ci]));
        }
        const FixedTables &fixed = fixed_tables();
        unsigned long long bytes = 0;
        d_inv.upload(fixed.inverses, stream, bytes, "upload inverses");
        d_sq.upload(fixed.squares, stream, bytes, "upload squares");
        d_odd.upload(fixed.odd, stream, bytes, "upload odd primes");
        d_counters.ensure(kCounters, "cudaMalloc(batch counters)");
        check_cuda(cudaStreamSynchronize(stream), "batch engine setup");
    }

    // The survivor capacity of an engine's first run.  RPG_BATCH_CAPACITY
    // overrides it (tests use a small one to exercise the rerun after an
    // overflow).
    static unsigned long long first_capacity() {
        if (const char *env = std::getenv("RPG_BATCH_CAPACITY"))
            return (unsigned long long)std::max(1LL, std::atoll(env));
        return 1ull << 20;
    }

    // Waits for every stream; true if all finished without error.
    bool wait() {
        bool ok = true;
        for (cudaStream_t s : {stream, side}) ok = cudaStreamSynchronize(s) == cudaSuccess && ok;
        for (cudaStream_t s : sweep_stream) ok = cudaStreamSynchronize(s) == cudaSuccess && ok;
        return ok;
    }

    // True if nothing of it is in flight and every stream finished without error.
    bool idle() { return !failed && wait(); }

    // Frees the largest arrays until at most `limit` bytes are held on the
    // device, and the host's plan if it holds more than an eighth of that.
    void trim(std::size_t limit) {
        sweep_groups.clear();
        plan.clear();
        if (plan.bytes() > limit / 8) plan = BatchPlan{};
        std::vector<std::pair<std::size_t, std::function<void()>>> arrays;
        std::size_t total = 0;
        auto add = [&](auto &x) {
            arrays.push_back({x.bytes(), [&x] { x.free(); }});
            total += x.bytes();
        };
        add(d_wide), add(d_narrow), add(d_witems), add(d_nitems), add(d_aspecs), add(d_pspecs), add(d_cspecs);
        add(d_cls), add(d_res), add(d_aff), add(d_patterns), add(d_rows), add(d_counters), add(d_sweep_tables);
        add(d_a), add(d_pa), add(d_d), add(d_c), add(d_pd), add(d_pc), add(d_curve_modular);
        std::sort(arrays.begin(), arrays.end(), [](const auto &x, const auto &y) { return x.first > y.first; });
        for (auto &x : arrays) {
            if (total <= limit) break;
            x.second();
            total -= x.first;
        }
    }

    ~Impl() {
        if (stream) cudaStreamSynchronize(stream);
        if (side) cudaStreamSynchronize(side);
        for (auto &s : sweep_stream)
            if (s) {
                cudaStreamSynchronize(s);
                cudaStreamDestroy(s);
            }
        for (auto &e : sweep_join)
            if (e) cudaEventDestroy(e);
        for (auto &e : ev)
            if (e) cudaEventDestroy(e);
        if (fork) cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
        if (h_counters) cudaFreeHost(h_counters);
        if (stream) cudaStreamDestroy(stream);
        if (side) cudaStreamDestroy(side);
    }

    // Groups the plan's sweeps, in their order, so that the tables of a group
    // take at most `limit` bytes (or are one curve's); the bytes of the largest.
    std::size_t group_sweeps(std::size_t limit) {
        sweep_groups.clear();
        std::size_t largest = 0, used = 0;
        for (std::size_t j = 0; j < plan.sweeps.size(); ++j) {
            SweepCurve &curve = *plan.work[plan.sweeps[j]].sweep;
            if (sweep_groups.empty() || used + curve.bytes() > limit) {
                sweep_groups.push_back({j, j, std::unique_ptr<SweepBuilder>(new SweepBuilder)});
                used = 0;
            }
            used += curve.bytes();
            sweep_groups.back().tables->add(curve);
            sweep_groups.back().end = j + 1;
        }
        for (const auto &g : sweep_groups) largest = std::max(largest, g.tables->bytes());
        return largest;
    }

    // Groups the sweeps and gets the memory for their tables: nearly always one
    // group.  Tables of 13 to 40 MB a curve (searches long enough to gain from
    // them) fill the device with 7,000 to 20,000 curves, so there is a limit,
    // and a lower one if that much is not to be had.  RPG_BATCH_TABLE_BYTES sets
    // it (tests use a small one).
    void ensure_sweep_tables() {
        std::size_t limit = std::size_t(64) << 30;
        if (const char *env = std::getenv("RPG_BATCH_TABLE_BYTES")) limit = std::size_t(std::max(1LL, std::atoll(env)));
        for (;;) {
            const std::size_t bytes = group_sweeps(limit);
            try {
                if (bytes) d_sweep_tables.ensure(bytes, "cudaMalloc(sieve tables)");
                return;
            } catch (const CudaError &) {
                if (sweep_groups.size() == plan.sweeps.size()) throw;
                cudaGetLastError();
                limit = std::min(limit, bytes) / 2;
            }
        }
    }

    void ensure_output(unsigned long long cap) {
        d_a.ensure(cap, "cudaMalloc(batch survivors)");
        d_d.ensure(cap, "cudaMalloc(batch survivors)");
        d_c.ensure(cap, "cudaMalloc(batch survivors)");
        d_pa.ensure(cap, "cudaMalloc(batch survivors)");
        d_pd.ensure(cap, "cudaMalloc(batch survivors)");
        d_pc.ensure(cap, "cudaMalloc(batch survivors)");
    }

    std::vector<BatchCurveResult> run(const std::vector<BatchCurveSpec> &curves, BatchStats *stats_out,
                                      bool use_graph, bool preverify, int items_per_kernel);
};

std::vector<BatchCurveResult> BatchEngine::Impl::run(const std::vector<BatchCurveSpec> &curves,
                                                     BatchStats *stats_out, bool use_graph, bool preverify,
                                                     int items_per_kernel) {
    const auto started = Clock::now();
    BatchStats stats;
    if (items_per_kernel <= 0) {
        items_per_kernel = tuned_batch_items(curves);
        stats.items_from_cache = items_per_kernel > 0;
        if (items_per_kernel <= 0) items_per_kernel = kDefaultBatchItems;
    }
    stats.items_per_kernel = items_per_kernel;
    std::vector<BatchCurveResult> results(curves.size());
    check_cuda(cudaSetDevice(device), "cudaSetDevice");
    // what a run that failed left on its way reads the plan's arrays
    if (failed) wait();
    failed = true;  // until the end
    // Curves with huge rows fill the device on their own: batching gains them
    // nothing, and the single-curve kernel (row count compiled in, stage 2
    // from class-layout tables) sweeps them faster.  They are validated with
    // the others, then searched one by one in a thread beside the batched
    // kernels.
    std::vector<std::size_t> solo;
    std::vector<char> is_solo(curves.size(), 0);
    for (std::size_t i = 0; i < curves.size(); ++i)
        if (curves[i].last >= curves[i].first && curves[i].bound >= 1 &&
            word_count64(curves[i].bound) >= kBatchSoloWords) {
            solo.push_back(i);
            is_solo[i] = 1;
        }
    BatchPlan &P = plan;
    P.clear();
    const auto t_plan = Clock::now();
    build_plan(curves, is_solo, results, P, stats, items_per_kernel);
    stats.plan_ms = ms_since(t_plan);
    const std::vector<CurveWork> &work = P.work;
    std::exception_ptr solo_error;
    std::thread solo_thread;
    struct Joiner {
        std::thread &t;
        ~Joiner() {
            if (t.joinable()) t.join();
        }
    } joiner{solo_thread};
    if (!solo.empty())
        solo_thread = std::thread([&] {
            try {
                check_cuda(cudaSetDevice(device), "cudaSetDevice");
                for (std::size_t i : solo) {
                    if (results[i].status != 0) continue;
                    const BatchCurveSpec &c = curves[i];
                    SearchOptions o;
                    o.coefficients = c.coefficients;
                    o.numerator_bound = c.bound;
                    o.first = c.first;
                    o.last = c.last;
                    o.intervals = c.intervals;
                    o.include_infinity = false;  // added below with the batched curves'
                    o.devices = {device};
                    o.square = c.square;
                    o.plan = PlanKind::fast;
                    o.device_preverify = preverify;
                    PointSearch search(o);
                    std::vector<PointPair> found;
                    const SearchMetrics m = search.run([&](const PointPair &p) {
                        found.push_back(p);
                        return true;
                    });
                    results[i].points = std::move(found);
                    results[i].survivors = m.modular_survivors;
                    results[i].wide = true;
                    results[i].solo = true;
                }
            } catch (...) {
                solo_error = std::current_exception();
            }
        });

    if (!P.wide.empty() || !P.narrow.empty() || !P.sweeps.empty()) {
        d_wide.upload(P.wide, stream, stats.h2d_bytes, "upload wide curves");
        d_narrow.upload(P.narrow, stream, stats.h2d_bytes, "upload narrow curves");
        d_witems.upload(P.wide_items, stream, stats.h2d_bytes, "upload work items");
        d_nitems.upload(P.narrow_items, stream, stats.h2d_bytes, "upload work items");
        d_aspecs.upload(P.aspecs, stream, stats.h2d_bytes, "upload bitmask specs");
        d_pspecs.upload(P.pspecs, stream, stats.h2d_bytes, "upload pattern specs");
        d_cspecs.upload(P.cspecs, stream, stats.h2d_bytes, "upload table specs");
        d_res.upload(P.residues, stream, stats.h2d_bytes, "upload residues");
        d_cls.upload(P.class_starts, stream, stats.h2d_bytes, "upload class starts");
        d_aff.ensure(std::size_t(P.aff_words), "cudaMalloc(batch bitmasks)");
        d_patterns.ensure(std::size_t(P.pattern_words), "cudaMalloc(batch patterns)");
        d_rows.ensure(std::size_t(P.row_words), "cudaMalloc(batch tables)");
        ensure_output(capacity);
        d_counters.ensure(kCounters + P.sweeps.size(), "cudaMalloc(batch counters)");
        if (preverify) {
            std::vector<const std::vector<std::string> *> coefs(curves.size(), nullptr);
            for (std::size_t i = 0; i < curves.size(); ++i)
                if (work[i].ok) coefs[i] = &curves[i].coefficients;
            pre.prepare(coefs, stream, [](std::size_t n, const std::function<void(std::size_t)> &fn) {
                parallel_for(n, fn);
            });
            stats.h2d_bytes += pre.upload_bytes();
            d_curve_modular.ensure(std::max<std::size_t>(1, curves.size()), "cudaMalloc(batch counters)");
        }
        ensure_sweep_tables();  // last: it may do with less
        // more groups than one: their tables are uploaded and built in turn
        const bool in_turn = sweep_groups.size() > 1;
        auto upload_tables = [&](const SweepGroup &g) {
            g.tables->place(d_sweep_tables.p, stream);
            stats.h2d_bytes += g.tables->upload_bytes();
        };
        if (sweep_groups.size() == 1) upload_tables(sweep_groups[0]);

        const int wide_smem_words = P.wide_smem_words;
        const int wide_max_classes = P.wide_max_classes;
        const std::size_t wide_smem = std::size_t(dev::kWSlotCount) * std::size_t(wide_smem_words) * 8 +
                                      std::size_t(dev::kWConsumers) * dev::kQueue * 16 +
                                      std::size_t(dev::kWSlotCount) * std::size_t(wide_max_classes) *
                                          sizeof(dev::WideRun) +
                                      std::size_t(dev::kWSlotCount) * std::size_t(wide_max_classes + 1) * 4;
        const std::size_t narrow_smem = std::size_t(dev::kNarrowTableWords + dev::kAffWords) * 8 +
                                        std::size_t(dev::kNWarps) * dev::kNarrowQueue * 16;
        int wide_grid = 0, narrow_grid = 0;
        if (!P.wide.empty()) {
            int per_sm = 0;
            check_cuda(cudaFuncSetAttribute(dev::wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            int(wide_smem)),
                       "cudaFuncSetAttribute");
            check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::wide_kernel,
                                                                     dev::kWThreads, wide_smem),
                       "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
            wide_grid = std::max(1, std::min<int>(sms * std::max(1, per_sm), int(P.wide_items.size())));
        }
        if (!P.narrow.empty()) {
            int per_sm = 0;
            check_cuda(cudaFuncSetAttribute(dev::narrow_kernel,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, int(narrow_smem)),
                       "cudaFuncSetAttribute");
            check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::narrow_kernel,
                                                                     dev::kNThreads, narrow_smem),
                       "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
            narrow_grid = std::max(1, std::min<int>(sms * std::max(1, per_sm), int(P.narrow_items.size())));
        }

        // external records become event nodes when the stream is captured
        bool capturing = false;
        auto record = [&](cudaEvent_t e, cudaStream_t s) {
            check_cuda(capturing ? cudaEventRecordWithFlags(e, s, cudaEventRecordExternal)
                                 : cudaEventRecord(e, s),
                       "cudaEventRecord");
        };
        auto enqueue_sieve = [&]() {
            const dev::BatchOut out{d_a.p, d_d.p, d_c.p, d_counters.p, capacity, d_counters.p + 3};
            check_cuda(cudaMemsetAsync(d_counters.p, 0, (kCounters + P.sweeps.size()) * sizeof(unsigned long long),
                                       stream),
                       "cudaMemsetAsync");
            if (preverify)
                check_cuda(cudaMemsetAsync(d_curve_modular.p, 0, curves.size() * sizeof(unsigned long long), stream),
                           "cudaMemsetAsync");
            check_cuda(cudaEventRecord(fork, stream), "cudaEventRecord");
            check_cuda(cudaStreamWaitEvent(side, fork, 0), "cudaStreamWaitEvent");
            record(ev[2], stream);
            if (wide_grid) {
                dev::wide_kernel<<<wide_grid, dev::kWThreads, wide_smem, stream>>>(
                    d_wide.p, d_witems.p, int(P.wide_items.size()), d_rows.p, d_aff.p, d_cls.p, d_inv.p, d_odd.p, cand, out, wide_smem_words, wide_max_classes,
                    d_counters.p + 1, d_counters.p + 5);
                check_cuda(cudaGetLastError(), "wide_kernel launch");
            }
            for (const SweepGroup &g : sweep_groups) {
                if (in_turn) {  // after the launches of the group before
                    upload_tables(g);
                    g.tables->enqueue(stream);
                    check_cuda(cudaEventRecord(fork, stream), "cudaEventRecord");
                }
                const int streams = int(std::min<std::size_t>(kSweepStreams, g.end - g.begin));
                for (int k = 0; k < streams; ++k)
                    check_cuda(cudaStreamWaitEvent(sweep_stream[k], fork, 0), "cudaStreamWaitEvent");
                for (std::size_t j = g.begin; j < g.end; ++j) {
                    const std::size_t i = P.sweeps[j];
                    SweepLaunch l;
                    l.first = curves[i].first;
                    l.last = curves[i].last;
                    l.a_lo = -curves[i].bound;
                    l.a_hi = curves[i].bound;
                    l.out_a = d_a.p;
                    l.out_d = d_d.p;
                    l.out_curve = d_c.p;
                    l.curve = int(i);
                    l.capacity = capacity;
                    l.out_count = d_counters.p;
                    l.work = d_counters.p + kCounters + j;
                    l.error = d_counters.p + 3;
                    l.swept = d_counters.p + 5;
                    const int k = int((j - g.begin) % std::size_t(kSweepStreams + 1));
                    work[i].sweep->launch(l, k < streams ? sweep_stream[k] : stream);
                }
                for (int k = 0; k < streams; ++k) {
                    check_cuda(cudaEventRecord(sweep_join[k], sweep_stream[k]), "cudaEventRecord");
                    check_cuda(cudaStreamWaitEvent(stream, sweep_join[k], 0), "cudaStreamWaitEvent");
                }
            }
            record(ev[3], stream);
            record(ev[4], side);
            if (narrow_grid) {
                dev::narrow_kernel<<<narrow_grid, dev::kNThreads, narrow_smem, side>>>(
                    d_narrow.p, d_nitems.p, int(P.narrow_items.size()), d_rows.p, d_aff.p, d_inv.p,
                    d_odd.p, cand, out, d_counters.p + 2, d_counters.p + 5);
                check_cuda(cudaGetLastError(), "narrow_kernel launch");
            }
            record(ev[5], side);
            check_cuda(cudaEventRecord(join, side), "cudaEventRecord");
            check_cuda(cudaStreamWaitEvent(stream, join, 0), "cudaStreamWaitEvent");
            if (preverify)
                pre.launch(d_a.p, d_d.p, d_c.p, d_counters.p, capacity, d_pa.p, d_pd.p, d_pc.p, d_counters.p + 4,
                           d_curve_modular.p, stream);
            check_cuda(cudaMemcpyAsync(h_counters, d_counters.p, kCounters * sizeof(unsigned long long),
                                       cudaMemcpyDeviceToHost, stream),
                       "download batch counters");
        };
        auto enqueue_all = [&]() {
            record(ev[0], stream);
            const long long aff_threads = (long long)P.aspecs.size() * dev::kRefWords;
            if (aff_threads) {
                dev::affine_kernel<<<unsigned((aff_threads + 255) / 256), 256, 0, stream>>>(
                    d_aspecs.p, (long long)P.aspecs.size(), d_res.p, d_sq.p, d_aff.p);
                check_cuda(cudaGetLastError(), "affine_kernel launch");
            }
            if (P.pattern_words) {
                dev::pattern_kernel<<<unsigned((P.pattern_words + 256 * dev::kPatternWords - 1) /
                                               (256 * dev::kPatternWords)),
                                      256, 0, stream>>>(
                    d_pspecs.p, int(P.pspecs.size()), d_aff.p, d_inv.p, d_patterns.p, P.pattern_words);
                check_cuda(cudaGetLastError(), "pattern_kernel launch");
            }
            if (P.row_words) {
                dev::composite_kernel<<<unsigned((P.row_words + 256 * dev::kCompositeWords - 1) /
                                                 (256 * dev::kCompositeWords)),
                                        256, 0, stream>>>(
                    d_cspecs.p, int(P.cspecs.size()), d_patterns.p, d_rows.p, P.row_words);
                check_cuda(cudaGetLastError(), "composite_kernel launch");
            }
            if (sweep_groups.size() == 1) sweep_groups[0].tables->enqueue(stream);
            record(ev[1], stream);
            enqueue_sieve();
        };
        if (use_graph && !in_turn) {  // a graph has no uploads in it
            cudaGraph_t graph = nullptr;
            cudaGraphExec_t exec = nullptr;
            check_cuda(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal),
                       "cudaStreamBeginCapture");
            capturing = true;
            try {
                enqueue_all();
            } catch (...) {
                capturing = false;
                cudaStreamEndCapture(stream, &graph);
                if (graph) cudaGraphDestroy(graph);
                throw;
            }
            capturing = false;
            check_cuda(cudaStreamEndCapture(stream, &graph), "cudaStreamEndCapture");
            const cudaError_t inst = cudaGraphInstantiate(&exec, graph, 0);
            cudaGraphDestroy(graph);
            check_cuda(inst, "cudaGraphInstantiate");
            const cudaError_t launched = cudaGraphLaunch(exec, stream);
            const cudaError_t synced = cudaStreamSynchronize(stream);
            cudaGraphExecDestroy(exec);
            check_cuda(launched, "cudaGraphLaunch");
            check_cuda(synced, "batch graph");
            stats.graph = true;
        } else {
            enqueue_all();
            check_cuda(cudaStreamSynchronize(stream), "batch sieve");
        }
        stats.launches += (P.aspecs.empty() ? 0 : 1) + (P.pattern_words ? 1 : 0) + (P.row_words ? 1 : 0) +
                          (wide_grid ? 1 : 0) + (narrow_grid ? 1 : 0) + (preverify ? 1 : 0) +
                          3 * sweep_groups.size() + P.sweeps.size();
        auto elapsed = [&](int a, int b) {
            float ms = 0;
            cudaEventElapsedTime(&ms, ev[a], ev[b]);
            return double(ms);
        };
        stats.table_ms = elapsed(0, 1);
        stats.wide_ms = elapsed(2, 3);
        stats.narrow_ms = elapsed(4, 5);
        stats.sieve_ms = std::max(elapsed(2, 3), elapsed(2, 5));
        if (h_counters[3]) throw DeviceTimeout("batched sieve: a bounded wait for a table copy timed out");
        while (h_counters[0] > capacity) {  // survivors did not fit: run again with room for all
            capacity = h_counters[0] + (h_counters[0] >> 3) + 1024;
            ensure_output(capacity);
            enqueue_sieve();
            check_cuda(cudaStreamSynchronize(stream), "batch sieve");
            stats.sieve_ms += std::max(elapsed(2, 3), elapsed(2, 5));
            stats.launches += (wide_grid ? 1 : 0) + (narrow_grid ? 1 : 0) + (preverify ? 1 : 0) +
                              (in_turn ? 3 * sweep_groups.size() : 0) + P.sweeps.size();
            if (h_counters[3]) throw DeviceTimeout("batched sieve: a bounded wait timed out");
        }
        stats.survivors = h_counters[0];
        stats.swept_words = h_counters[5];
        stats.smem_bytes = h_counters[6];
        // survivors for the host: those kept by pre-verification, or all
        const std::size_t n = std::size_t(preverify ? h_counters[4] : h_counters[0]);
        stats.host_candidates = n;
        std::vector<long long> ha(n);
        std::vector<int> hd(n), hc(n);
        std::vector<unsigned long long> curve_modular(preverify ? curves.size() : 0);
        if (n) {
            check_cuda(cudaMemcpyAsync(ha.data(), preverify ? d_pa.p : d_a.p, n * sizeof(long long),
                                       cudaMemcpyDeviceToHost, stream),
                       "download batch survivors");
            check_cuda(cudaMemcpyAsync(hd.data(), preverify ? d_pd.p : d_d.p, n * sizeof(int),
                                       cudaMemcpyDeviceToHost, stream),
                       "download batch survivors");
            check_cuda(cudaMemcpyAsync(hc.data(), preverify ? d_pc.p : d_c.p, n * sizeof(int),
                                       cudaMemcpyDeviceToHost, stream),
                       "download batch survivors");
        }
        if (!curve_modular.empty())
            check_cuda(cudaMemcpyAsync(curve_modular.data(), d_curve_modular.p,
                                       curve_modular.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                       stream),
                       "download batch survivor counts");
        check_cuda(cudaStreamSynchronize(stream), "download batch survivors");
        stats.d2h_bytes += n * (sizeof(long long) + 2 * sizeof(int)) + kCounters * sizeof(unsigned long long) +
                           curve_modular.size() * sizeof(unsigned long long);

        // ---- exact verification per curve, in single-search order ----
        const auto t_verify = Clock::now();
        std::vector<std::vector<std::size_t>> by_curve(curves.size());
        for (std::size_t s = 0; s < n; ++s) by_curve[std::size_t(hc[s])].push_back(s);
        parallel_for(curves.size(), [&](std::size_t i) {
            if (!work[i].ok) return;
            BatchCurveResult &r = results[i];
            const ExactPolynomial &poly = *work[i].poly;
            std::vector<PointPair> found;
            std::string root;
            for (std::size_t s : by_curve[i]) {
                if (gcd_ll(ha[s], hd[s]) != 1) continue;
                if (poly.square_root(ha[s], hd[s], root)) found.push_back(PointPair{ha[s], root, hd[s]});
            }
            std::sort(found.begin(), found.end(), [](const PointPair &a, const PointPair &b) {
                return a.denominator != b.denominator ? a.denominator < b.denominator
                                                      : a.numerator < b.numerator;
            });
            SearchOptions filter;
            filter.intervals = curves[i].intervals;
            for (auto &p : found)
                if (filter.accepts(p.numerator, p.denominator)) r.points.push_back(std::move(p));
            r.survivors = preverify ? curve_modular[i] : by_curve[i].size();
        });
        stats.verify_ms = ms_since(t_verify);
    }
    // the point at infinity first, as a single search reports it
    parallel_for(curves.size(), [&](std::size_t i) {
        if (!work[i].ok || !curves[i].include_infinity || is_solo[i]) return;
        std::string root;
        if (work[i].poly->square_root(1, 0, root))
            results[i].points.insert(results[i].points.begin(), PointPair{1, root, 0});
    });
    if (solo_thread.joinable()) solo_thread.join();
    if (solo_error) std::rethrow_exception(solo_error);
    for (std::size_t i : solo)
        if (results[i].status == 0) {
            const BatchCurveSpec &c = curves[i];
            const long long count = c.last - c.first + 1;
            ++stats.solo_curves;
            ++stats.curves;
            ++stats.wide_curves;
            stats.survivors += results[i].survivors;
            stats.denominators += (unsigned long long)count;
            stats.rectangle_sites += (long double)(2 * c.bound + 1) * (long double)count;
        }
    // the point at infinity first, as a single search reports it
    parallel_for(solo.size(), [&](std::size_t j) {
        const std::size_t i = solo[j];
        if (!work[i].ok || !curves[i].include_infinity) return;
        std::string root;
        if (work[i].poly->square_root(1, 0, root))
            results[i].points.insert(results[i].points.begin(), PointPair{1, root, 0});
    });
    failed = false;
    for (const auto &r : results) stats.points += r.points.size();
    stats.wall_ms = ms_since(started);
    if (stats_out) *stats_out = stats;
    return results;
}

// The device resources of engines that are gone, kept for the next engine on
// the same device: creating and freeing nine streams, the events and some
// twenty arrays took about 3 of the 13 ms of a batch of 384 small searches.  Every
// run uploads, clears or builds all that it reads but the tables that are the
// same for all curves.  Never destroyed: static destructors may run after the
// CUDA runtime is gone.
struct BatchEnginePool {
    static constexpr std::size_t kEngines = 4;                     // per process
    static constexpr std::size_t kBytes = std::size_t(512) << 20;  // device memory kept by each
    std::mutex mutex;
    std::vector<std::unique_ptr<BatchEngine::Impl>> idle;

    static BatchEnginePool &get() {
        static auto *pool = new BatchEnginePool();
        return *pool;
    }
    std::unique_ptr<BatchEngine::Impl> take(int device) {
        std::lock_guard<std::mutex> lock(mutex);
        for (auto it = idle.rbegin(); it != idle.rend(); ++it)
            if ((*it)->device == device) {
                std::unique_ptr<BatchEngine::Impl> engine = std::move(*it);
                idle.erase(std::next(it).base());
                return engine;
            }
        return nullptr;
    }
    // Destroys what it does not keep (outside the lock).
    void give(std::unique_ptr<BatchEngine::Impl> engine) {
        if (!engine->idle()) return;
        engine->trim(kBytes);
        std::lock_guard<std::mutex> lock(mutex);
        if (idle.size() < kEngines) idle.push_back(std::move(engine));
    }
};

BatchEngine::BatchEngine(int device) {
    if (device >= 0) check_cuda(cudaSetDevice(device), "cudaSetDevice");
    int current = 0;
    check_cuda(cudaGetDevice(&current), "cudaGetDevice");
    impl_ = BatchEnginePool::get().take(current);
    if (!impl_) impl_.reset(new Impl());
    // a pooled engine keeps the room that an earlier run grew to
    impl_->capacity = Impl::first_capacity();
    if (!std::getenv("RPG_BATCH_CAPACITY")) impl_->capacity = std::max<unsigned long long>(impl_->capacity, impl_->d_a.cap);
}

BatchEngine::~BatchEngine() {
    try {
        if (impl_) BatchEnginePool::get().give(std::move(impl_));
    } catch (...) {  // no memory for the pool's list: the engine is freed
    }
}

void release_pooled_engines(int device) {
    std::vector<std::unique_ptr<BatchEngine::Impl>> taken;
    auto &pool = BatchEnginePool::get();
    std::lock_guard<std::mutex> lock(pool.mutex);
    for (auto &engine : pool.idle)
        if (device < 0 || engine->device == device) taken.push_back(std::move(engine));
    pool.idle.erase(std::remove(pool.idle.begin(), pool.idle.end(), nullptr), pool.idle.end());
}

std::vector<BatchCurveResult> BatchEngine::run(const std::vector<BatchCurveSpec> &curves,
                                               BatchStats *stats, bool use_graph, bool preverify,
                                               int items_per_kernel) {
    return impl_->run(curves, stats, use_graph, preverify, items_per_kernel);
}

std::unique_ptr<SweepCurve> batch_sweep_curve(const BatchCurveSpec &c, FastPlan *plan) {
    FastPlan own = single_curve_plan(c.coefficients, c.bound, nullptr);
    std::unique_ptr<SweepCurve> sweep(new SweepCurve(c.coefficients, c.bound, c.square, &own,
                                                     double(c.last) - double(c.first) + 1.0, kBatchRowBytes));
    if (plan) *plan = std::move(own);
    return sweep;
}

int BatchEngine::device() const { return impl_->device; }

unsigned long long BatchEngine::estimate_bytes(const BatchCurveSpec &c) {
    const long long words = word_count64(std::max(1LL, c.bound));
    const long long count = c.last >= c.first ? c.last - c.first + 1 : 0;
    // a search of its own beside the batch (huge rows), with its survivor
    // buffers, or launches of its own
    if (words >= kBatchSoloWords)
        return SweepCurve::most_bytes(c.bound, c.coefficients.size(), 0) + (50ull << 20);
    if (count > 0 && swept_alone(c, words >= kBatchWideWords, words, count))
        return SweepCurve::most_bytes(c.bound, c.coefficients.size(), kBatchRowBytes);
    long long table;
    if (words >= kBatchWideWords) {
        const double cap = std::min<double>(kMaxModulus, std::max(64.0, std::sqrt(double(words) * count / 48.0)));
        table = (long long)(6.0 * cap * (cap + dev::kWExt));
    } else {
        table = dev::kNarrowTableWords;
    }
    // tables, bitmasks, patterns, descriptor and items (8-byte words)
    return (unsigned long long)(table + 2 * dev::kAffWords + 6 * 127 * 127 + 1024 +
                                std::max(1LL, count * std::max(1LL, (long long)c.intervals.size()) /
                                                  64)) * 8ull;
}

std::vector<BatchCurveResult> batch_search(const std::vector<BatchCurveSpec> &curves, int device,
                                           BatchStats *stats, bool use_graph, bool preverify) {
    BatchEngine engine(device);
    return engine.run(curves, stats, use_graph, preverify);
}

}  // namespace rpg
