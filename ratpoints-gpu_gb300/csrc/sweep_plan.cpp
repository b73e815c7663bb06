#include "sweep_plan.hpp"

#include <algorithm>
#include <cmath>

namespace rpg {

namespace {

struct Weighed {
    int p;
    int admitted, divided;
    bool optional;
    double bits;
};

struct ClassChoice {
    int two = 1;
    double two_classes = 1;
    int two_max = 1;
    int count = 0;
    int index[kSweepClassPrimes];  // into the primes
    int q = 1;
    double q_mean = 1;
    int q_max = 1;
    double pairs = 1, steps = 1, fill = 1;  // per live denominator
    double rough = 0;
};

// Cost model, fitted to GB300 (SM cycles): a step (a warp's two units of 16
// words through all rows) takes two cycles of the shared-memory pipe per row,
// a copied row one per 80 bytes, a live word about five (queue); a step's
// instructions, those of a live word (queue, stage 2), of an item's set-up
// and of each consumer's visit to a slot share four issue slots per cycle; a
// denominator's rows and lists arrive from L2 at about 50 B/clk; the producer
// of a CTA takes about 1,800 cycles per denominator.
constexpr double kStepIssue = 18, kRowIssue = 4.2, kLiveIssue = 45, kItemIssue = 90, kVisitIssue = 60,
                 kFillIssue = 250, kFillCycles = 1800;

double cost_of(const ClassChoice &c, int rows, double bits, double staged_bytes, int ctas) {
    const double live = c.steps * 32.0 * c.fill * (1.0 - std::pow(1.0 - std::exp2(-bits), 64.0));
    const double a_reads = (rows <= 8 ? 2.0 : 3.0) / (c.pairs >= 6.0 ? 2.0 : 1.0);
    const double smem = (c.steps * (2.0 * rows + a_reads) + staged_bytes / 80.0 + live * 5.0) / 0.95;
    const double issue = (c.steps * (kStepIssue + kRowIssue * rows) + live * kLiveIssue + std::max(1.0, c.pairs) * kItemIssue +
                          kVisitIssue * (kSweepWarps / ctas - 1) + kFillIssue) /
                         4.0 / 0.8;
    const double l2 = staged_bytes / 50.0;
    const double fill = kFillCycles / ctas;
    return std::cbrt(smem * smem * smem + issue * issue * issue + l2 * l2 * l2 + fill * fill * fill);
}

// How items are cut: pairs of units side by side (1 or 2) and ranges of the
// residues mod two.  More items keep more consumer warps busy on the slots in
// flight, each costs a set-up (about 2.5 steps of one pair).  Two pairs share
// the residue's terms but a set-up and a part-filled last group weigh double:
// with 23 residues and 3 pairs a denominator one pair takes 2.08 ms where two
// took 2.28, with 40 and 16 two take 9.9 ms where one takes 10.5.
void choose_items(const ClassChoice &c, SweepPlan &plan) {
    const int consumers = kSweepWarps / plan.ctas - 1;
    double best = 0;
    for (int pairs = 1; pairs <= 2; ++pairs)
        for (int split = 0; split <= 3 && (1 << split) <= c.two; ++split) {
            const double ranges = double(1 << split);
            // a denominator's last group of two pairs is often not full
            const double groups = std::max(1.0, pairs == 1 ? c.pairs : (c.pairs + 0.6) / 2.0);
            const double items = groups * ranges;
            const double busy = std::min(double(consumers), std::max(1.0, double(plan.slots - 1)) * items);
            const double steps = (pairs == 1 ? c.pairs : 1.95 * (c.pairs + 0.25) / 2.0) * c.two_classes;
            const double cost = (steps + items * (pairs == 1 ? 2.5 : 3.5)) / busy;
            if (best > 0 && cost >= best) continue;
            best = cost;
            plan.pairs = pairs;
            plan.split = split;
        }
}

}  // namespace

SweepPlan plan_sweep(const SweepInput &in) {
    std::vector<Weighed> primes;
    for (const auto &s : in.primes)
        primes.push_back({s.p, s.admitted, s.divided, s.optional,
                          -std::log2(double(s.admitted) / s.p)});
    std::sort(primes.begin(), primes.end(), [](const Weighed &a, const Weighed &b) {
        const double da = a.bits / std::log2(double(a.p)), db = b.bits / std::log2(double(b.p));
        return da != db ? da > db : a.p < b.p;
    });
    const int n = int(primes.size());

    // ---- class primes: the two cheapest choices at eight rows of 12 bits ----
    constexpr int kKeep = 2;
    ClassChoice best[kKeep];
    int kept = 0;
    auto offer = [&](ClassChoice c) {
        const long long mod = (long long)c.two * c.q;
        const double words = double(sweep_words(in.bound, mod));
        const double segs = std::ceil(words / kSweepUnit);
        // consecutive units pair up, also across residues; one left over
        // takes half the steps of a pair
        c.pairs = std::max(0.5, c.q_mean * segs / 2.0);
        c.steps = c.pairs * c.two_classes;
        c.fill = words / (segs * kSweepUnit);
        c.rough = cost_of(c, 8, 12.0, 16384.0 + kSweepListBytes * c.q_mean, 2);
        int at = kept;
        while (at > 0 && best[at - 1].rough > c.rough) --at;
        if (at >= kKeep) return;
        if (kept < kKeep) ++kept;
        for (int i = kept - 1; i > at; --i) best[i] = best[i - 1];
        best[at] = c;
    };
    const double sites = 2.0 * double(in.bound) + 1.0;
    auto extend = [&](auto &&self, ClassChoice c, int from) -> void {
        offer(c);
        if (c.count == kSweepClassPrimes) return;
        for (int i = from; i < n; ++i) {
            const Weighed &w = primes[std::size_t(i)];
            if (w.bits < 0.3) continue;
            const long long q = (long long)c.q * w.p;
            if (sites / (double(c.two) * double(q)) < 640.0) continue;  // classes of ten words at least
            const long long q_max = (long long)c.q_max * std::max(w.admitted, w.divided);
            if (q > 8192 || q_max > kSweepMaxClasses || q * q_max * kSweepListBytes > (32LL << 20)) continue;
            ClassChoice next = c;
            next.index[next.count++] = i;
            next.q = int(q);
            next.q_max = int(q_max);
            next.q_mean = c.q_mean * w.admitted;
            self(self, next, i + 1);
        }
    };
    if (in.two > 0) {
        ClassChoice c;
        c.two = in.two;
        c.two_classes = in.two_classes;
        c.two_max = in.two_max;
        extend(extend, c, 0);
    } else {
        for (int two = 1; two <= 64; two *= 2) {
            ClassChoice c;
            c.two = two;
            c.two_classes = c.two_max = two;
            extend(extend, c, 0);
        }
    }

    // ---- rows: primes in order of bits per bit of size, packed into products
    // below a cap (each into the row with the most headroom that takes it,
    // else a new row); every cap and row count is priced ----
    static const int caps[] = {1500, 1050, 740, 512, 360, 250, 170, 110};
    struct Packing {
        int count = 0;
        int modulus[kSweepRows];
        int factors[kSweepRows];
        int factor[kSweepRows][kSweepRowFactors];
        double bits = 0;
    };
    SweepPlan out;
    bool found = false;
    for (int k = 0; k < kept; ++k) {
        const ClassChoice &c = best[k];
        bool used[512] = {};
        for (int i = 0; i < c.count; ++i) used[primes[std::size_t(c.index[i])].p] = true;
        int largest = caps[0] + 1;  // of the moduli packed at the previous cap
        for (int cap : caps) {
            if (largest <= cap) continue;  // the same packings
            largest = 0;
            for (int rows = std::min(3, n); rows <= kSweepRows; ++rows) {
                Packing p;
                for (const auto &w : primes) {
                    if (used[w.p] || w.p > cap || w.bits < 0.25) continue;
                    int target = -1, headroom = -1;
                    for (int i = 0; i < p.count; ++i) {
                        if (p.factors[i] == kSweepRowFactors) continue;
                        const long long product = (long long)p.modulus[i] * w.p;
                        if (product <= cap && int(cap - product) > headroom) {
                            headroom = int(cap - product);
                            target = i;
                        }
                    }
                    if (target < 0) {
                        if (p.count == rows) continue;
                        target = p.count++;
                        p.modulus[target] = 1;
                        p.factors[target] = 0;
                    }
                    p.modulus[target] *= w.p;
                    p.factor[target][p.factors[target]++] = w.p;
                    p.bits += w.bits;
                }
                if (p.count < rows && rows > 3) break;  // no more primes for another row
                if (p.count == 0) continue;
                for (int i = 0; i < p.count; ++i) largest = std::max(largest, p.modulus[i]);
                long long words = 0;
                for (int i = 0; i < p.count; ++i) words += sweep_row_words(p.modulus[i]);
                const long long slot = sweep_slot_bytes(words, c.two_max, c.q_max);
                double cost = 0;
                int ctas = 0, slots = 0;
                for (int n_ctas = 2; n_ctas <= 4; ++n_ctas) {
                    const long long room = sweep_cta_bytes(n_ctas) - kSweepQueueBytes * (kSweepWarps / n_ctas - 1);
                    if (slot > room) break;
                    const double staged = double(words) * 8.0 + kSweepListBytes * (c.q_mean + c.two_classes);
                    double v = cost_of(c, p.count, p.bits, staged, n_ctas);
                    // two slots hide less of the copies, one none of them
                    if (2 * slot > room) v += staged / 100.0 + 800.0;
                    else if (3 * slot > room) v *= 1.03;
                    if (ctas && v >= cost) continue;
                    cost = v;
                    ctas = n_ctas;
                    slots = int(std::min<long long>(kSweepSlots, room / slot));
                }
                if (!ctas) continue;
                double build = 0;  // words of the rows' tables
                for (int i = 0; i < p.count; ++i) build += double(p.modulus[i]) * sweep_row_words(p.modulus[i]);
                if (in.row_bytes > 0 && build * 8.0 > double(in.row_bytes)) continue;
                // their build, about three words per SM cycle over the
                // device, shared by the denominators
                if (in.denominators > 0) cost += build / 3.0 / in.denominators;
                if (found && cost >= out.cost) continue;
                found = true;
                out.cost = cost;
                out.two = c.two;
                out.two_max = c.two_max;
                out.q = c.q;
                out.q_max = c.q_max;
                out.class_primes.clear();
                for (int i = 0; i < c.count; ++i) out.class_primes.push_back(primes[std::size_t(c.index[i])].p);
                out.rows.clear();
                out.moduli.assign(p.modulus, p.modulus + p.count);
                for (int i = 0; i < p.count; ++i) out.rows.emplace_back(p.factor[i], p.factor[i] + p.factors[i]);
                out.ctas = ctas;
                out.slots = slots;
                choose_items(c, out);
            }
        }
    }
    if (!found) {  // no prime filters: one row of a small prime all the same
        const ClassChoice &c = best[0];
        out.two = c.two;
        out.two_max = c.two_max;
        out.q = c.q;
        out.q_max = c.q_max;
        for (int i = 0; i < c.count; ++i) out.class_primes.push_back(primes[std::size_t(c.index[i])].p);
        double bits = 0;
        for (const auto &w : primes)
            if (out.moduli.empty() &&
                std::find(out.class_primes.begin(), out.class_primes.end(), w.p) == out.class_primes.end()) {
                out.moduli.push_back(w.p);
                out.rows.push_back({w.p});
                bits = w.bits;
            }
        out.slots = 2;
        out.cost = cost_of(c, 1, bits, double(sweep_row_words(out.moduli[0])) * 8.0 +
                           kSweepListBytes * (c.q_mean + c.two_classes), out.ctas);
    }
    bool placed[512] = {};
    for (int p : out.class_primes) placed[p] = true;
    for (const auto &r : out.rows)
        for (int p : r) placed[p] = true;
    for (const auto &w : primes)
        if (!w.optional && !placed[w.p]) out.late.push_back(w.p);
    return out;
}

}  // namespace rpg
