// Plans, tables and launches of the sieve kernel (sweep.hpp).
#include "sweep.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <stdexcept>

#include "sieve.hpp"
#include "sieve_device.cuh"
#include "sieve_fast.cuh"

namespace rpg {
namespace dev {

// ---------------------------------------------------------------------------
// Table builds.  Offsets in the jobs are bytes from the allocation's start.

// Pattern rows of one prime q: for each rho = d mod q, bit k of row rho tests
// the sites with a = k step (mod q), step = M mod q, for k in [0, q + 64) and
// up to the end of its `words` words (the sequence has period q).  A word of
// sites a, a + M, .. is then the 64 bits from position (a mod q) M^-1 mod q.
// The test: f(a / rho) a square mod q; for rho = 0 by lead (0: no site, 1: a
// not divisible by q, 2: every site).
struct PatternJob {
    std::size_t out;
    std::size_t residues;          // c_0 .. c_n mod q (unsigned short)
    int n;
    int q;
    int words;                     // ceil((q + 64) / 64) + 1
    int lead;
    int step;                      // M mod q
    int pad;
};

constexpr int kPatternBlocks = 4;  // blocks per prime, each every fourth row
constexpr int kBuildThreads = 256;

// Bound by its shared-memory lookups, one per bit; residues advance by
// additions (no division per bit), and the curve enters only as its
// coefficients mod q: 33 -> 8 us for the 60 primes of one curve.
__global__ void __launch_bounds__(kBuildThreads) pattern_kernel(unsigned char *arena, std::size_t jobs) {
    __shared__ unsigned char s_square[512], s_affine[512];
    __shared__ unsigned short s_inverse[512];
    const PatternJob J = reinterpret_cast<const PatternJob *>(arena + jobs)[blockIdx.x / kPatternBlocks];
    const int part = int(blockIdx.x % kPatternBlocks);
    const int q = J.q, t = int(threadIdx.x);
    const unsigned short *c = reinterpret_cast<const unsigned short *>(arena + J.residues);
    for (int v = t; v < q; v += kBuildThreads) s_square[v] = 0;
    __syncthreads();
    for (int v = t; 2 * v <= q; v += kBuildThreads) s_square[v * v % q] = 1;
    __syncthreads();
    for (int x = t; x < q; x += kBuildThreads) {
        int v = c[J.n];
        for (int i = J.n - 1; i >= 0; --i) v = (v * x + c[i]) % q;
        s_affine[x] = s_square[v];
        // x^(q-2): the inverse (0 for x = 0)
        int inv = 1, b = x;
        for (int e = q - 2; e; e >>= 1) {
            if (e & 1) inv = inv * b % q;
            b = b * b % q;
        }
        s_inverse[x] = (unsigned short)(x ? inv : 0);
    }
    __syncthreads();
    u64 *out = reinterpret_cast<u64 *>(arena + J.out);
    const int rows = (q - part + kPatternBlocks - 1) / kPatternBlocks;
    for (int i = t; i < rows * J.words; i += kBuildThreads) {
        const int rho = part + kPatternBlocks * (i / J.words), w = i % J.words;
        int x = int((long long)(64 * w % q) * J.step % q);  // a mod q
        u64 word = 0;
        if (rho == 0) {
            for (int j = 0; j < 64; ++j) {
                if (J.lead == 2 || (J.lead == 1 && x != 0)) word |= u64(1) << j;
                x += J.step;
                if (x >= q) x -= q;
            }
        } else {
            const int inv = s_inverse[rho], dy = J.step * inv % q;
            int y = x * inv % q;
            for (int j = 0; j < 64; ++j) {
                word |= u64(s_affine[y]) << j;
                y += dy;
                if (y >= q) y -= q;
            }
        }
        out[(long long)rho * J.words + w] = word;
    }
}

// Class-layout rows of one modulus m: bit j of word u of row rho = AND over
// the prime factors q of the test of sites a = S u + M j: the window from
// position S u M^-1 = 64 u (mod q) of q's pattern row rho mod q.  Words
// u >= m repeat word u - m.
struct TableJob {
    std::size_t out;
    std::size_t pattern[kSweepRowFactors];
    int m, nf, length;
    int q[kSweepRowFactors];
    int words[kSweepRowFactors];
    unsigned block0;               // first block: one per row rho
};

constexpr int kTableThreads = 128;

// One block per row: the row's pattern rows stay in L1, and each word is
// computed once and stored for both periods.  Bound by the stores.
__global__ void __launch_bounds__(kTableThreads) class_table_kernel(unsigned char *arena, std::size_t jobs, int njobs) {
    const TableJob *table = reinterpret_cast<const TableJob *>(arena + jobs);
    int lo = 0, hi = njobs - 1;  // last job with block0 <= blockIdx.x
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (table[mid].block0 <= blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const TableJob &J = table[lo];
    const int rho = int(blockIdx.x - J.block0);
    const int m = J.m, nf = J.nf, length = J.length;
    u64 *row = reinterpret_cast<u64 *>(arena + J.out) + (long long)rho * length;
    const u64 *pattern[kSweepRowFactors];
    int q[kSweepRowFactors];
#pragma unroll
    for (int f = 0; f < kSweepRowFactors; ++f) {
        q[f] = f < nf ? J.q[f] : 1;
        pattern[f] = f < nf ? reinterpret_cast<const u64 *>(arena + J.pattern[f]) + (rho % q[f]) * J.words[f] : nullptr;
    }
    for (int u = int(threadIdx.x); u < m; u += kTableThreads) {
        u64 word = ~u64(0);
#pragma unroll
        for (int f = 0; f < kSweepRowFactors; ++f)
            if (f < nf) {
                const u32 k = u32(64 * u) % u32(q[f]);
                const u64 a = pattern[f][k >> 6], b = pattern[f][(k >> 6) + 1];
                word &= k & 63u ? (a >> (k & 63u)) | (b << (64 - (k & 63u))) : a;
            }
        for (int v = u; v < length; v += m) row[v] = word;
    }
}

// The class lists: block b < Q writes the entries of denominators d = b
// (mod Q), block Q + b those of d = b (mod two).  A residue r mod Q is
// admissible if every class prime p admits it: byte r d^-1 mod p of its map of
// the x with f(x) a square, or, where p | d, by `divided`; a residue mod two if
// bit r of adm2[d mod two] is set.  (A map by d mod p and r mod p, p^2 bytes
// made on the host, took 0.4 ms for a prime of 331.)
struct ListJob {
    std::size_t adm[kSweepClassPrimes], inverses[kSweepClassPrimes], adm2;
    std::size_t list2, listq, count2, countq;
    int two, q, two_max, q_max, nprimes, nrows;
    int p[kSweepClassPrimes];
    int divided[kSweepClassPrimes];  // p | d: 0 admits none, 1 all but 0, 2 all
    u32 lift2, liftq;              // 1 mod two and 0 mod Q; 0 mod two and 1 mod Q (below M)
    u32 h2, hq;                    // H mod two, H mod Q
    u32 m[kSweepRows], inv_stride[kSweepRows], base[kSweepRows];  // base: (-H - M) mod m
    unsigned block0;
    int pad;
};

__global__ void __launch_bounds__(kBuildThreads) class_list_kernel(unsigned char *arena, std::size_t jobs, int njobs) {
    __shared__ int s_count[kBuildThreads / 32];
    __shared__ int s_base;
    const ListJob *lists = reinterpret_cast<const ListJob *>(arena + jobs);
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (lists[mid].block0 <= blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const ListJob &S = lists[lo];
    const int block = int(blockIdx.x - S.block0);
    const bool second = block >= S.q;
    const int dres = second ? block - S.q : block;
    const int n = second ? S.two : S.q;
    const int room = second ? S.two_max : S.q_max;
    const u32 M = u32(S.two) * u32(S.q);
    SweepClass *out = reinterpret_cast<SweepClass *>(arena + (second ? S.list2 : S.listq)) + (long long)dres * room;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ u32 s_inverse[kSweepClassPrimes];  // d^-1 mod p, 0 where p | d
    if (threadIdx.x == 0) s_base = 0;
    if (!second && int(threadIdx.x) < S.nprimes) {
        const int i = int(threadIdx.x);
        s_inverse[i] = reinterpret_cast<const unsigned short *>(arena + S.inverses[i])[dres % S.p[i]];
    }
    __syncthreads();
    for (int r0 = 0; r0 < n; r0 += kBuildThreads) {
        const int r = r0 + int(threadIdx.x);
        bool ok = r < n;
        if (second) {
            ok = ok && ((reinterpret_cast<const u64 *>(arena + S.adm2)[dres] >> (r & 63)) & 1);
        } else {
            for (int i = 0; i < S.nprimes && ok; ++i) {
                const u32 p = u32(S.p[i]), rp = u32(r) % p, inverse = s_inverse[i];
                ok = inverse ? arena[S.adm[i] + rp * inverse % p] != 0
                             : S.divided[i] > (rp == 0 ? 1 : 0);
            }
        }
        const u32 vote = __ballot_sync(kFullMask, ok);
        if (lane == 0) s_count[warp] = __popc(vote);
        __syncthreads();
        int at = s_base + __popc(vote & lanemask_lt());
        for (int w = 0; w < warp; ++w) at += s_count[w];
        if (ok && at < room) {
            SweepClass C{};
            const u32 v = u32(r) + (second ? S.h2 : S.hq);
            C.x = u32(u64(second ? S.lift2 : S.liftq) * (v % u32(n)) % M);
            for (int i = 0; i < S.nrows; ++i) {
                const u32 m = S.m[i];
                C.start8[i] = (unsigned short)(8u * ((C.x + (second ? 0u : S.base[i])) % m * S.inv_stride[i] % m));
            }
            out[at] = C;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 0; w < kBuildThreads / 32; ++w) s_base += s_count[w];
        __syncthreads();
    }
    if (threadIdx.x == 0) reinterpret_cast<int *>(arena + (second ? S.count2 : S.countq))[dres] = s_base;
}

}  // namespace dev

namespace {

unsigned long long magic_of(long long m) { return m == 1 ? ~0ull : (~0ull) / (unsigned long long)m + 1; }
long long mod_of(long long v, long long m) { return ((v % m) + m) % m; }

std::size_t aligned(std::size_t bytes) { return (bytes + 255) & ~std::size_t(255); }

const void *kernel_ptr(int rows, int pairs) {
    switch (2 * rows + pairs) {
#define RPG_FAST_PTR(n)                                                                     \
    case 2 * n + 1: return reinterpret_cast<const void *>(&dev::fast_sieve_kernel<n, 1>);   \
    case 2 * n + 2: return reinterpret_cast<const void *>(&dev::fast_sieve_kernel<n, 2>);
        RPG_FAST_PTR(1) RPG_FAST_PTR(2) RPG_FAST_PTR(3) RPG_FAST_PTR(4) RPG_FAST_PTR(5) RPG_FAST_PTR(6)
        RPG_FAST_PTR(7) RPG_FAST_PTR(8) RPG_FAST_PTR(9) RPG_FAST_PTR(10) RPG_FAST_PTR(11) RPG_FAST_PTR(12)
#undef RPG_FAST_PTR
    default: throw std::logic_error("no sieve kernel for this row count");
    }
}

int multiprocessors() {
    int device = 0, sms = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    return sms;
}

// The odd primes below 512 with p^-1 mod 2^32 (Newton's iteration) and
// floor((2^32 - 1) / p).
struct OddPrime {
    int p;
    dev::u32 inverse, limit;
};
const std::vector<OddPrime> &odd_primes() {
    static const std::vector<OddPrime> primes = [] {
        std::vector<OddPrime> out;
        for (int p = 3; p < kMaximumPrime; p += 2) {
            bool prime = true;
            for (int f = 3; f * f <= p && prime; f += 2) prime = p % f != 0;
            if (!prime) continue;
            dev::u32 inverse = dev::u32(p);  // right in 3 bits
            for (int i = 0; i < 4; ++i) inverse *= 2u - dev::u32(p) * inverse;
            out.push_back({p, inverse, 0xFFFFFFFFu / dev::u32(p)});
        }
        return out;
    }();
    return primes;
}

// 64^-1 modulo candidate i.
int inverse64(int i) {
    static const std::vector<int> inverses = [] {
        std::vector<int> out;
        for (int p : candidate_primes()) out.push_back(int(mod_inverse(64 % p, p)));
        return out;
    }();
    return inverses[std::size_t(i)];
}

}  // namespace

SweepCurve::~SweepCurve() = default;

SweepCurve::SweepCurve(const std::vector<std::string> &coefficients, long long bound, bool square, const FastPlan *fast,
                       double denominators, long long row_bytes)
    : bound_(bound), square_(square), tables_(new dev::SweepTables{}), list_(new dev::ListJob{}) {
    dev::SweepTables &T = *tables_;
    dev::ListJob &L = *list_;
    const int n = int(coefficients.size()) - 1;
    auto lead_of = [&](int p) {
        return n % 2 == 1 || square_mod(decimal_mod(coefficients.back(), p), p) ? 1 : 0;
    };
    std::vector<char> strict(kMaximumPrime, 0);
    SweepInput in;
    in.bound = bound;
    in.denominators = denominators;
    in.row_bytes = row_bytes;
    dev::u64 adm2[64];
    for (auto &v : adm2) v = ~dev::u64(0);
    if (fast) {
        two_adic_classes(coefficients, adm2);
        in.two = 64;
        int total = 0, live = 0;
        for (auto v : adm2) {
            const int c = __builtin_popcountll(v);
            total += c;
            live += c > 0;
            in.two_max = std::max(in.two_max, c);
        }
        in.two_classes = live ? double(total) / live : 1.0;
    }
    // A prime p mod which no f(x) is a square leaves only denominators that p
    // divides: a divisor d needs (`need_`), not a row, whose filtering there
    // would be overrated.  The plan's own test where p | d comes last.
    std::vector<int> late_primes;
    auto needed = [&](int p) {
        const unsigned long long product = need_ * (unsigned long long)p;
        need_ = product > 0xFFFFFFFFull ? 0xFFFFFFFFull : product;
    };
    if (fast)
        for (const auto &known : fast->admitted) {
            const int p = known.first, count = known.second;
            strict[std::size_t(p)] = 1;
            if (count == 0) {
                needed(p);
                late_primes.push_back(p);
            } else {
                in.primes.push_back({p, count, lead_of(p) ? p - 1 : 0, false});
            }
        }
    // The 32 largest candidates are always selected where they do not divide
    // d, so stage 1 may test them as well: all of the reference plan's, and
    // those of a fast plan whose own rows filter weakly (13 bits are usual) or
    // whose long rows take several class primes away from them (shorter
    // searches save the planning time).
    const auto &cands = candidate_primes();
    if (!fast || fast->bits < 12.5 || bound >= 4'000'000 || in.primes.size() < 4)
        for (int i = kCandidatePrimes - kSelectedPrimes; i < kCandidatePrimes; ++i)
            if (!strict[std::size_t(cands[i])]) {
                const int count = admitted_residues(cands[i], coefficients);
                if (count == 0) needed(cands[i]);
                in.primes.push_back({cands[i], std::max(1, count), cands[i], true});
            }
    in.denominators /= double(need_);
    plan_ = plan_sweep(in);
    late_primes.insert(late_primes.end(), plan_.late.begin(), plan_.late.end());

    const int q = plan_.q;
    const long long M = (long long)plan_.two * q;
    const long long S = 64LL * M;
    std::size_t size = 0;
    auto take = [&](std::size_t bytes) {
        const std::size_t at = size;
        size += aligned(bytes);
        return at;
    };
    auto put = [&](const void *data, std::size_t bytes) {
        const std::size_t at = input_.size();
        input_.resize(at + ((bytes + 15) & ~std::size_t(15)));
        if (bytes) std::memcpy(input_.data() + at, data, bytes);
        return at;
    };
    // pattern rows per (prime, rho = 0 rule)
    auto pattern_of = [&](int p, int lead) -> const dev::PatternJob & {
        for (const auto &J : patterns_)
            if (J.q == p && J.lead == lead) return J;
        dev::PatternJob J{};
        std::vector<unsigned short> residues;
        for (const auto &c : coefficients) residues.push_back((unsigned short)decimal_mod(c, p));
        J.residues = put(residues.data(), residues.size() * sizeof(unsigned short));
        J.n = n;
        J.q = p;
        J.words = (p + 64 + 63) / 64 + 1;
        J.lead = lead;
        J.step = int(M % p);
        J.out = take(std::size_t(p) * std::size_t(J.words) * 8);
        patterns_.push_back(J);
        return patterns_.back();
    };
    L.two = plan_.two;
    L.q = q;
    L.two_max = plan_.two_max;
    L.q_max = plan_.q_max;
    L.nprimes = int(plan_.class_primes.size());
    L.nrows = int(plan_.moduli.size());
    L.lift2 = dev::u32(plan_.two == 1 ? 0 : (long long)q * mod_inverse(q % plan_.two, plan_.two) % M);
    L.liftq = dev::u32(q == 1 ? 0 : (long long)plan_.two * mod_inverse(plan_.two % q, q) % M);
    L.h2 = dev::u32(bound % plan_.two);
    L.hq = dev::u32(bound % q);
    // Offsets in T count words from the curve's table block.
    int row_words = 0;
    for (std::size_t r = 0; r < plan_.moduli.size(); ++r) {
        dev::TableJob J{};
        const int m = plan_.moduli[r];
        J.m = m;
        J.nf = int(plan_.rows[r].size());
        for (int i = 0; i < J.nf; ++i) {
            const int p = plan_.rows[r][std::size_t(i)];
            const dev::PatternJob &P = pattern_of(p, strict[std::size_t(p)] ? lead_of(p) : 2);
            J.q[i] = p;
            J.pattern[i] = P.out;
            J.words[i] = P.words;
        }
        J.length = sweep_row_words(m);
        J.out = take(std::size_t(m) * std::size_t(J.length) * 8);
        jobs_.push_back(J);
        dev::SweepRow &R = T.row[r];
        R.offset = (long long)(J.out / 8);
        R.magic = magic_of(m);
        R.m = dev::u32(m);
        R.length = dev::u32(J.length);
        R.soff8 = dev::u32(8 * row_words);
        row_words += J.length;
        L.m[r] = dev::u32(m);
        L.inv_stride[r] = dev::u32(mod_inverse(S % m, m));
        L.base[r] = dev::u32(mod_of(-(bound % m) - M, m));
    }
    // The six largest candidates get class-layout tables (11 MB) where the
    // search is long enough to gain from one read per word instead of two.
    T.tabled = denominators <= 0 || plan_.cost * in.denominators > 2.0e8 ? 1 : 0;
    for (int i = 0; i < kCandidatePrimes; ++i) {
        const int p = cands[i];
        dev::FastPrime &P = T.prime[i];
        P.p = p;
        P.magic = dev::magic40(dev::u32(p));
        if (q % p == 0) continue;  // a class prime: the swept classes pass it
        // rows with p | d go unused (stage 2 skips such p) unless the plan has p
        const dev::PatternJob &J = pattern_of(p, strict[std::size_t(p)] ? lead_of(p) : 2);
        P.pattern = (long long)(J.out / 8);
        P.words = J.words;
        P.inv_mod = dev::u32(mod_inverse(M % p, p));
        P.inv_stride = dev::u32((long long)P.inv_mod * inverse64(i) % p);  // S = 64 M
        if (T.tabled && i >= kCandidatePrimes - dev::kFStage2Group) {
            dev::TableJob K{};
            K.m = K.length = p;
            K.nf = 1;
            K.q[0] = p;
            K.pattern[0] = J.out;
            K.words[0] = J.words;
            K.out = take(std::size_t(p) * std::size_t(p) * 8);
            jobs_.push_back(K);
            P.offset = (long long)(K.out / 8);
        }
    }
    if (late_primes.size() > std::size_t(dev::kLatePrimes)) throw std::logic_error("more late primes than a plan has");
    for (int p : late_primes) {
        const dev::PatternJob &J = pattern_of(p, lead_of(p));
        T.late[T.nlate++] = {(long long)(J.out / 8), magic_of(p), dev::u32(p), dev::u32(mod_inverse(M % p, p)), 0, J.words};
    }
    if (T.nlate)
        for (int t = 0; t < dev::kFLateGroup; ++t) T.late[T.nlate + t] = T.late[T.nlate - 1];
    // admissible residues of the class primes by d mod p
    for (int i = 0; i < L.nprimes; ++i) {
        const int p = plan_.class_primes[std::size_t(i)];
        const auto aff = affine_mask(p, coefficients);
        std::vector<unsigned short> inv(static_cast<std::size_t>(p));
        modular_inverses(p, inv.data());
        L.p[i] = p;
        L.divided[i] = !strict[std::size_t(p)] ? 2 : lead_of(p) ? 1 : 0;
        L.adm[i] = put(aff.data(), aff.size());
        L.inverses[i] = put(inv.data(), inv.size() * sizeof(unsigned short));
        std::vector<int> counts(std::size_t(p), int(std::count_if(aff.begin(), aff.end(), [](auto v) { return v != 0; })));
        counts[0] = L.divided[i] == 2 ? p : L.divided[i] * (p - 1);
        countq_.push_back(std::move(counts));
    }
    const dev::u64 two_bits = plan_.two == 64 ? ~dev::u64(0) : (dev::u64(1) << plan_.two) - 1;
    for (int dd = 0; dd < plan_.two; ++dd) count2_.push_back(__builtin_popcountll(adm2[dd] & two_bits));
    L.adm2 = put(adm2, sizeof adm2);
    L.list2 = list2_at_ = take(std::size_t(plan_.two) * std::size_t(plan_.two_max) * sizeof(dev::SweepClass));
    L.listq = listq_at_ = take(std::size_t(q) * std::size_t(plan_.q_max) * sizeof(dev::SweepClass));
    L.count2 = count2_at_ = take(std::size_t(plan_.two) * sizeof(int));
    L.countq = countq_at_ = take(std::size_t(q) * sizeof(int));
    table_bytes_ = size;
    // Denominator primes (fast plan): p < 512 with c_n not a square mod p, for
    // even degree.  A denominator divisible by one holds no points: p !| a
    // (gcd) gives F(a, d) = c_n a^n (mod p), a non-square.  The producer skips
    // such denominators.
    if (fast && n % 2 == 0)
        for (const auto &o : odd_primes()) {
            const int lc = decimal_mod(coefficients.back(), o.p);
            if (lc == 0 || square_mod(lc, o.p)) continue;
            T.bad[bad_primes_.size()] = make_uint2(o.inverse, o.limit);
            bad_primes_.push_back(o.p);
        }
    T.nbad = int(bad_primes_.size());
    dev::u32 inverse = dev::u32(need_);
    for (int i = 0; i < 4; ++i) inverse *= 2u - dev::u32(need_) * inverse;
    T.need = make_uint2(inverse, dev::u32(0xFFFFFFFFull / need_));
    T.two_mask = plan_.two - 1;
    T.q = dev::u32(q);
    T.q_magic = magic_of(q);
    T.two_max = plan_.two_max;
    T.q_max = plan_.q_max;
    T.stride = S;
    T.class_mod = int(M);
    T.row_words = row_words;
    T.slots = plan_.slots;
    smem_ = std::size_t(plan_.slots) * std::size_t(sweep_slot_bytes(row_words, plan_.two_max, plan_.q_max)) +
            std::size_t(kSweepQueueBytes) * std::size_t(kSweepWarps / plan_.ctas - 1);
    // queued positions stay below 2^46 and class words below 2^23
    tile_ = S * std::min<long long>(1LL << 23, (1LL << 45) / S);
}

std::size_t SweepCurve::bytes() const {
    return table_bytes_ + input_.size() + patterns_.size() * sizeof(dev::PatternJob) + jobs_.size() * sizeof(dev::TableJob) +
           sizeof(dev::ListJob) + 1024;  // alignment
}

unsigned long long SweepCurve::most_bytes(long long bound, std::size_t coefficients, long long row_bytes) {
    // rows as wide as two slots' worth of a CTA allow, by the plan's largest modulus
    if (row_bytes <= 0) row_bytes = sweep_cta_bytes(2) * kMaxModulus;
    // pattern rows of every odd prime below 512, the six largest candidates'
    // tables, and a job and the coefficients' residues for each of them
    static const unsigned long long tables = [] {
        unsigned long long sum = 0;
        for (const auto &o : odd_primes())
            sum += std::size_t(o.p) * std::size_t((o.p + 64 + 63) / 64 + 1) * 8 + 256 + sizeof(dev::PatternJob) +
                   sizeof(dev::TableJob) + 16;
        const auto &cands = candidate_primes();
        for (int i = kCandidatePrimes - dev::kFStage2Group; i < kCandidatePrimes; ++i)
            sum += (unsigned long long)cands[std::size_t(i)] * (unsigned long long)cands[std::size_t(i)] * 8 + 256;
        return sum;
    }();
    unsigned long long bytes =
        (unsigned long long)row_bytes + tables + odd_primes().size() * coefficients * sizeof(unsigned short);
    // class lists: Q at most 8,192, and small enough for classes of ten words
    const long long q = std::max(1LL, std::min<long long>(8192, bound / (320 * 64) + 1));
    bytes += (unsigned long long)std::min(32LL << 20, q * std::min<long long>(q, kSweepMaxClasses) * kSweepListBytes);
    bytes += 64 * 64 * kSweepListBytes + 65536;  // the list mod two, counts, maps, alignment
    return bytes;
}

unsigned long long SweepCurve::swept_words(long long first, long long last) const {
    if (last < first) return 0;
    // Parameters per residue mod M, then the classes of each residue.
    const long long M = (long long)plan_.two * plan_.q;
    std::vector<unsigned long long> per_residue(std::size_t(M), 0);
    auto residue = [&](long long k) { return square_ ? (k % M) * (k % M) % M : k % M; };
    if (bad_primes_.empty() && need_ == 1) {
        for (long long t = 0; t < M; ++t) {
            const long long lo = first + ((t - first % M) % M + M) % M;  // first k >= first, k = t (mod M)
            if (lo <= last) per_residue[std::size_t(residue(t))] += (unsigned long long)((last - lo) / M + 1);
        }
    } else {
        // parameters k without a denominator prime factor, by segments
        constexpr long long kSegment = 1LL << 22;
        std::vector<unsigned char> skip;
        for (long long lo = first; lo <= last; lo += kSegment) {
            const long long hi = std::min(last, lo + kSegment - 1);
            skip.assign(std::size_t(hi - lo + 1), 0);
            for (int p : bad_primes_)
                for (long long k = lo + ((p - lo % p) % p); k <= hi; k += p) skip[std::size_t(k - lo)] = 1;
            for (long long k = lo; k <= hi; ++k)
                if (!skip[std::size_t(k - lo)] && (square_ ? k * k : k) % (long long)need_ == 0) per_residue[std::size_t(residue(k))] += 1;
        }
    }
    unsigned long long total = 0;
    for (long long r = 0; r < M; ++r) {
        unsigned long long classes = (unsigned long long)count2_[std::size_t(r % plan_.two)];
        for (std::size_t i = 0; i < countq_.size(); ++i)
            classes *= (unsigned long long)countq_[i][std::size_t(r % plan_.class_primes[i])];
        total += per_residue[std::size_t(r)] * classes;
    }
    return total * (unsigned long long)sweep_words(bound_, M);
}

void SweepCurve::launch(const SweepLaunch &l, cudaStream_t stream) const {
    const long long M = tables_->class_mod, S = tables_->stride;
    const long long w_lo = (l.a_lo + bound_) / S;
    const int grid = multiprocessors() * plan_.ctas;
    dev::SweepArgs A{};
    A.abase = -bound_ - M + S * w_lo;
    A.a_lo = l.a_lo;
    A.a_hi = l.a_hi;
    A.k_first = l.first;
    A.k_count = int(l.last - l.first + 1);
    // Few denominators with much to sweep are split into shares of their
    // items, so that every CTA gets several (the tail of a launch is at most
    // one of them per CTA), while a share stays well above the copy of its
    // rows: 4,001 denominators of 6.8e5 words took 20 instead of 15 ms whole.
    // A fetch takes work worth about 2^15 cycles.
    double cost = plan_.cost * (double(l.a_hi) - double(l.a_lo) + 1.0) / (2.0 * double(bound_) + 1.0);
    while (A.part_shift < 6 && ((long long)A.k_count << A.part_shift) < 32LL * grid && cost > 40000.0) {
        ++A.part_shift;
        cost *= 0.5;
    }
    const long long shares = (long long)A.k_count << A.part_shift;
    A.chunk = int(std::max<long long>(
        1, std::min<long long>({dev::kFChunk, shares / (4LL * grid), (long long)(32768.0 / cost)})));
    A.square = square_ ? 1 : 0;
    const long long words = ((l.a_hi - A.abase) / M >> 6) + 1;
    A.segs = int((words + kSweepUnit - 1) / kSweepUnit);
    A.shifted = w_lo != 0;
    A.split = A.segs > 64 ? 0 : plan_.split;
    A.out_a = l.out_a;
    A.out_d = l.out_d;
    A.out_curve = l.out_curve;
    A.curve = l.curve;
    A.out_count = l.out_count;
    A.capacity = l.capacity;
    A.error = l.error;
    A.swept = l.swept;
    dev::SweepTables T = *tables_;
    T.segs_magic = A.segs == 1 ? 0 : magic_of(A.segs);
    for (std::size_t r = 0; r < plan_.moduli.size(); ++r) T.row[r].wlo = dev::u32(w_lo % plan_.moduli[r]);
    for (auto &P : T.prime) P.base_mod = dev::u32(mod_of(A.abase, P.p));
    for (int l = 0; T.nlate && l < T.nlate + dev::kFLateGroup; ++l)
        T.late[l].base_mod = dev::u32(mod_of(A.abase, (long long)T.late[l].p));
    const int blocks = int(std::min<long long>(grid, (shares + A.chunk - 1) / A.chunk));
    unsigned long long *work = l.work;
    void *params[] = {&T, &A, &work};
    const void *kernel = kernel_ptr(int(plan_.moduli.size()), plan_.pairs);
    check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sweep_cta_bytes(2))),
               "cudaFuncSetAttribute");
    check_cuda(cudaLaunchKernel(kernel, dim3(unsigned(blocks)),
                                dim3(unsigned(kSweepWarps / plan_.ctas * dev::kWarpSize)), params, smem_, stream),
               "sieve kernel launch");
}

// ---------------------------------------------------------------------------

SweepBuilder::SweepBuilder() = default;
SweepBuilder::~SweepBuilder() = default;

void SweepBuilder::add(SweepCurve &curve) {
    curves_.push_back(&curve);
    at_.push_back(size_);
    size_ += curve.table_bytes_;
}

std::size_t SweepBuilder::bytes() const {
    std::size_t inputs = 0, patterns = 0, tables = 0;
    for (const SweepCurve *c : curves_) {
        inputs += c->input_.size();
        patterns += c->patterns_.size();
        tables += c->jobs_.size();
    }
    return size_ + aligned(inputs) + aligned(patterns * sizeof(dev::PatternJob)) + aligned(tables * sizeof(dev::TableJob)) +
           aligned(curves_.size() * sizeof(dev::ListJob));
}

void SweepBuilder::place(unsigned char *arena, cudaStream_t stream) {
    arena_ = arena;
    std::vector<dev::PatternJob> patterns;
    std::vector<dev::TableJob> tables;
    std::vector<dev::ListJob> lists;
    blob_.clear();
    table_blocks_ = list_blocks_ = 0;
    for (std::size_t i = 0; i < curves_.size(); ++i) {
        SweepCurve &c = *curves_[i];
        const std::size_t block = at_[i], input = size_ + blob_.size();
        blob_.insert(blob_.end(), c.input_.begin(), c.input_.end());
        for (dev::PatternJob J : c.patterns_) {
            J.out += block;
            J.residues += input;
            patterns.push_back(J);
        }
        for (dev::TableJob J : c.jobs_) {
            J.out += block;
            for (int f = 0; f < J.nf; ++f) J.pattern[f] += block;
            J.block0 = table_blocks_;
            table_blocks_ += unsigned(J.m);
            tables.push_back(J);
        }
        dev::ListJob L = *c.list_;
        for (int k = 0; k < L.nprimes; ++k) {
            L.adm[k] += input;
            L.inverses[k] += input;
        }
        L.adm2 += input;
        L.list2 += block;
        L.listq += block;
        L.count2 += block;
        L.countq += block;
        L.block0 = list_blocks_;
        list_blocks_ += unsigned(L.q + L.two);
        lists.push_back(L);
        dev::SweepTables &T = *c.tables_;
        T.rows = reinterpret_cast<const dev::u64 *>(arena + block);
        T.list2 = reinterpret_cast<const dev::SweepClass *>(arena + block + c.list2_at_);
        T.listq = reinterpret_cast<const dev::SweepClass *>(arena + block + c.listq_at_);
        T.count2 = reinterpret_cast<const int *>(arena + block + c.count2_at_);
        T.countq = reinterpret_cast<const int *>(arena + block + c.countq_at_);
    }
    auto append = [&](const void *data, std::size_t bytes) {
        blob_.resize(aligned(blob_.size()));
        const std::size_t at = size_ + blob_.size();
        blob_.resize(blob_.size() + bytes);
        if (bytes) std::memcpy(blob_.data() + (at - size_), data, bytes);
        return at;
    };
    patterns_at_ = append(patterns.data(), patterns.size() * sizeof(dev::PatternJob));
    tables_at_ = append(tables.data(), tables.size() * sizeof(dev::TableJob));
    lists_at_ = append(lists.data(), lists.size() * sizeof(dev::ListJob));
    pattern_jobs_ = int(patterns.size());
    table_jobs_ = int(tables.size());
    list_jobs_ = int(lists.size());
    check_cuda(cudaMemcpyAsync(arena + size_, blob_.data(), blob_.size(), cudaMemcpyHostToDevice, stream),
               "upload table inputs");
}

void SweepBuilder::enqueue(cudaStream_t stream) const {
    dev::pattern_kernel<<<unsigned(pattern_jobs_ * dev::kPatternBlocks), dev::kBuildThreads, 0, stream>>>(arena_,
                                                                                                       patterns_at_);
    check_cuda(cudaGetLastError(), "pattern_kernel launch");
    dev::class_table_kernel<<<table_blocks_, dev::kTableThreads, 0, stream>>>(arena_, tables_at_, table_jobs_);
    check_cuda(cudaGetLastError(), "class_table_kernel launch");
    dev::class_list_kernel<<<list_blocks_, dev::kBuildThreads, 0, stream>>>(arena_, lists_at_, list_jobs_);
    check_cuda(cudaGetLastError(), "class_list_kernel launch");
}

}  // namespace rpg
