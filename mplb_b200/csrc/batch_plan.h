// How batched cavities are held in shared memory for many steps
// (batch_resident.cuh): plain host arithmetic.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <map>
#include <vector>

namespace mplb {

// A strip of a cavity: rows [row0, row0 + rows) are computed, rows
// [vrow0, vrow0 + vrows) (counted from row0) are stored.
struct ResidentItem {
    int cav;
    int n;
    int base;        // element offset of the cavity, in 128-byte units
    int row0, rows;
    int vrow0, vrows;
    int rows_per_cta;
    int whole;       // the strip is the whole cavity: stored where it is read
};

// Nodes of a CTA whose slots fill 1 / 2^halves of an SM: its 233,472 bytes of
// shared memory hold 2^halves CTAs, each with 1 KB of its own besides its slots
// (9 values of 4 or 8 bytes a node).
constexpr int kSmemOfSm = 228 * 1024, kSmemOfCta = 1024;
constexpr int ResidentSlots(bool f64, int halves) {
    return (halves == 0 ? 6400 : halves == 1 ? 3200 : 1584) / (f64 ? 2 : 1);
}
constexpr int ResidentSmem(bool f64, int halves) {
    return 9 * ResidentSlots(f64, halves) * (f64 ? 8 : 4);
}
constexpr bool ResidentFits(bool f64) {
    for (int h = 0; h < 3; h++)
        if ((ResidentSmem(f64, h) + kSmemOfCta) << h > kSmemOfSm) return false;
    return true;
}
static_assert(ResidentFits(false) && ResidentFits(true),
              "an SM holds the CTAs of every form");

// Nodes a thread advances at once, and so the nodes of a warp.
constexpr int kResidentGroup32 = 64;
constexpr int kResidentGroup64 = 32;

// Sides up to here are held in strips: rows of up to an eighth of the slots
// (strips of larger cavities would be mostly overlap).
inline int ResidentMaxSide(bool f64) { return ResidentSlots(f64, 0) / 8; }

// Resident strips launched together: the same cluster size, slots and block.
struct ResidentClass {
    int halves, ranks, warps;
    int max_steps;      // per launch
    bool whole;         // every strip is a whole cavity
    long long work;     // nodes computed per step
    std::vector<ResidentItem> items;
    int first = 0;      // of its items in the list of all
};

// Cluster sizes of the plans, and which of them, in which form, the device can
// hold at all: part of a GPU (fewer SMs in its GPCs, less shared memory left) may
// have no place for some that a whole B200 has.
constexpr int kResidentRanks[] = {1, 2, 3, 4, 5, 6, 8, 9};
constexpr int kNumResidentRanks = 8;
inline int ResidentRankIndex(int ranks) {
    int r = 0;
    while (kResidentRanks[r] != ranks) r++;
    return r;
}
struct ResidentHeld {
    bool at[3][kNumResidentRanks];   // [halves][index of the ranks]
    ResidentHeld() {
        for (auto& h : at) std::fill(h, h + kNumResidentRanks, true);
    }
};

// How the cavities of one side are held in shared memory; score infinite: not
// at all.
struct ResidentPlan {
    int halves = 0, ranks = 1;
    int strips = 1, overlap = 0;
    double score = INFINITY;
};

// The best plan for cavities of side n when an SM has `load` nodes of the
// active cavities to advance per step: the fewest SM cycles per node while
// the GPU is full, the shortest step of one strip while it is not.  The
// constants are measured on a B200: `fixed` is the part of a step that does
// not shrink with its nodes (barrier, one pass' latency), `reload` the
// reading and writing of a strip in steps of it, and the last table the share
// of the SMs that clusters of that size can fill (a GPC's SMs are not always
// a multiple of it).  Sweeps of every plan at sides 64-256 found none more than
// 6 % faster than the one chosen here.
inline ResidentPlan PlanResident(int n, bool f64, double load,
                                 const ResidentHeld& held) {
    static const double kFill[] = {1.0, 1.0, 0.91, 0.89, 0.88, 0.89, 0.81,
                                   0.91};
    const double reload = f64 ? 1.3 : 2.5;
    ResidentPlan best;
    for (int halves = 0; halves < 3; halves++) {
        const int cap = ResidentSlots(f64, halves);
        const double share = 1.0 / (1 << halves);
        for (int r = 0; r < kNumResidentRanks; r++) {
            if (!held.at[halves][r]) continue;
            const int ranks = kResidentRanks[r];
            const int most = ranks * (cap / n);   // rows of a strip
            const double fixed = ranks > 1 ? 400 : 250;
            auto consider = [&](int strips, int overlap, int rows) {
                const double per_cta = (double)((rows + ranks - 1) / ranks) * n;
                const double steps = strips > 1 ? overlap + 1 : 64;
                const double cost = strips * ranks *
                                    (per_cta + share * fixed) *
                                    (1.0 + reload / steps) /
                                    ((double)n * n * kFill[r]);
                const double time = (per_cta + fixed) * (1.0 + reload / steps);
                const double score =
                    std::max(cost * load, time) + 0.1 * cost * load;
                if (score >= best.score) return;
                best.halves = halves;
                best.ranks = ranks;
                best.strips = strips;
                best.overlap = overlap;
                best.score = score;
            };
            if (most >= n) {
                consider(1, 0, n);
                continue;
            }
            for (int overlap : {3, 5, 7, 11, 15, 23}) {
                const int inner = most - 2 * overlap;
                if (inner < 1) break;
                const int strips =
                    std::max(2, (n - 2 * overlap + inner - 1) / inner);
                const int valid = (n - 2 * overlap + strips - 1) / strips;
                // the last strip takes what the others leave
                if (n - overlap - (strips - 1) * valid < 1) continue;
                consider(strips, overlap, valid + 2 * overlap);
            }
        }
    }
    return best;
}

// Resident strips of the cavities `active` of the sides `sides` (base: their
// element offsets in 128-byte units) on a GPU of `sms` SMs, the longest class
// first, the longest strips of a class first; none if a cavity does not fit in
// what the device holds.
inline std::vector<ResidentClass> PlanStrips(const std::vector<int>& active,
                                             const std::vector<int>& sides,
                                             const std::vector<int>& base,
                                             bool f64, int sms,
                                             const ResidentHeld& held) {
    std::vector<ResidentClass> classes;
    double nodes = 0;
    for (int c : active) {
        const double n = sides[c];
        if (n > ResidentMaxSide(f64)) return classes;
        nodes += n * n;
    }
    const int group = f64 ? kResidentGroup64 : kResidentGroup32;
    std::map<int, ResidentPlan> plans;
    for (int c : active) {
        const int n = sides[c];
        auto at = plans.find(n);
        if (at == plans.end())
            at = plans.emplace(n, PlanResident(n, f64, nodes / sms, held))
                     .first;
        const ResidentPlan& p = at->second;
        if (std::isinf(p.score)) return {};
        const int valid = (n - 2 * p.overlap + p.strips - 1) / p.strips;
        // the same block for all strips of a cavity: they read each other's
        // rows of the launch before, so they stay in one class
        const int tall = p.strips == 1 ? n : valid + 2 * p.overlap;
        const int groups =
            ((tall + p.ranks - 1) / p.ranks * n + group - 1) / group;
        const int most = 24 >> p.halves;
        const int passes = (groups + most - 1) / most;
        const int warps = std::max(2, (groups + passes - 1) / passes);
        const int max_steps = p.strips == 1 ? 128 : p.overlap + 1;
        for (int j = 0; j < p.strips; j++) {
            ResidentItem it{};
            it.cav = c;
            it.n = n;
            it.base = base[c];
            it.whole = p.strips == 1;
            const int v0 = j == 0 ? 0 : p.overlap + j * valid;
            const int v1 = j + 1 == p.strips ? n : p.overlap + (j + 1) * valid;
            it.row0 = std::max(0, v0 - p.overlap);
            it.rows = std::min(n, v1 + p.overlap) - it.row0;
            it.vrow0 = v0 - it.row0;
            it.vrows = v1 - v0;
            it.rows_per_cta = (it.rows + p.ranks - 1) / p.ranks;
            ResidentClass* cls = nullptr;
            for (ResidentClass& k : classes)
                if (k.halves == p.halves && k.ranks == p.ranks &&
                    k.warps == warps && k.max_steps == max_steps)
                    cls = &k;
            if (!cls) {
                ResidentClass k{};
                k.halves = p.halves;
                k.ranks = p.ranks;
                k.warps = warps;
                k.max_steps = max_steps;
                k.whole = it.whole != 0;
                classes.push_back(k);
                cls = &classes.back();
            }
            cls->items.push_back(it);
            cls->work += (long long)it.rows * n;
        }
    }
    std::sort(classes.begin(), classes.end(),
              [](const ResidentClass& x, const ResidentClass& y) {
                  return x.work > y.work;
              });
    int first = 0;
    for (ResidentClass& k : classes) {
        std::stable_sort(k.items.begin(), k.items.end(),
                         [](const ResidentItem& x, const ResidentItem& y) {
                             return x.rows_per_cta * x.n >
                                    y.rows_per_cta * y.n;
                         });
        k.first = first;
        first += (int)k.items.size();
    }
    return classes;
}

}  // namespace mplb
