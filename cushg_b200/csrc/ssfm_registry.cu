// ssfm_registry.cu — lookup of the compiled fused-march variants and the autotuner's
// choices (see ssfm_variants.h).
#include <algorithm>
#include <functional>
#include <mutex>
#include <queue>
#include <vector>

#include "../../include/shg.h"
#include "ssfm_variants.h"

namespace shg {

namespace {

std::mutex g_mu;
// Chosen plain variants, one per (precision, n); from: the number of runs from which the choice
// also holds against the variants for few runs.
struct Choice {
    const PlainVariant* v;
    int from;
};
std::vector<Choice> g_chosen;

// f(variant) until it returns true; with `few` also the variants kept for few runs
template <typename F>
void for_each_variant(F&& f, bool few = false) {
    const VariantTable tables[] = {variants_f32_small(), variants_f32_128(), variants_f32_192(), variants_f32_256(),
                                   variants_f64_small(), variants_f64_large(), variants_thermal(),
                                   variants_multipass(), variants_split(), variants_split64(), variants_wide()};
    const int k = (int)(sizeof(tables) / sizeof(tables[0])) - (few ? 0 : 3);
    for (int t = 0; t < k; ++t)
        for (int i = 0; i < tables[t].count; ++i)
            if (f(&tables[t].v[i])) return;
}

// Plain runs that have the device to themselves: the faster variant by the number of runs, where it is
// not the default (cluster 0: the wide march, one run over the whole GPU).  With few runs the SMs are
// idle unless a run spreads over many of them, and what bounds a step is the chain of one thread; a
// wider split costs more exchange between CTAs, so once the device is full the narrow ones win.  The
// lines lie where the measured times cross, which is where a variant's clusters no longer fit at once.
// us per step at the first and last count of a row (parts of the step count's start-up included) /
// of the default there:
//   FP32 32: 1-28 3.4-4.8 / 5.3-5.8.  48: 1-14 3.9-4.9 / 11, 15-100 7.3-12.0 / 11-12.
//   64: 1-14 4.1-5.0 / 14.1, 15-104 7.8-14.0 / 14.2-15.2.  96: 1-7 5.6-5.7 / 30.5, 8-48 10-19 /
//   31, 49-72 24 / 31.  128: 1-2 6.3-6.7 / 29.8, 3-7 7.5 / 29.8, 8-48 12-27 / 30.5, 73-108 44 / 61.
//   192: 1-9 7.2-23 / 37.6, 10-15 26 / 37.4 (16: 39.8 / 37.4), 37-48 58-61 / 74 (51: 79.9 / 75).
//   256: 1-4 8.4-18 / 24, 5-7 21-21.3 / 21-23.6 (8: 34 / 23.4).
//   512: 1 14.4 / 29.2 (multi-pass)
//   FP64 32: 1-28 3.5-5.5 / 6.8-7.1, 29-60 5.8-6.9 / 7.3.  48: 1-14 4.2-8.0 / 8.3, 101-148 17.5 /
//   16-22.  64: 1-14 4.9-9.3 / 15, 15-48 9.9-14.7 / 15.5, 73-108 20.5 / 26.  96: 1-6 6.2-8.6 / 32.4,
//   7-48 13-32 / 33.  128: 1-3 6.5-8.3 / 19.1, 4-7 11 / 19.1.  192: 1-6 8.5-21 / 25.8.
//   256: 1-4 9.7-24 / 34, 5-7 33.7 / 33.6-36.6 (8: 66.8 / 37.6).  512: 1 19.0 / 39.3 (multi-pass)
// us1, us: of one run on the row's variant, and of upto of them.  beside: the runs that count as a full
// device in a batch with other classes, where that is not upto (0: the row is for its class alone).
struct FewRow { int precision, n, upto, cluster, threads; double us1, us; int beside = -1; };
const FewRow kFew[] = {
    {32, 32, 28, 16, 64, 2.9, 4.1},      {32, 48, 14, 16, 96, 3.5, 4.3},      {32, 48, 100, 4, 96, 6.5, 10.6},
    {32, 64, 14, 16, 128, 3.6, 4.5},     {32, 64, 104, 4, 128, 7.1, 12.6},    {32, 64, 148, 1, 512, 13.2, 14.6},
    {32, 96, 7, 16, 288, 5.2, 5.3},      {32, 96, 48, 8, 288, 9.5, 18.3},     {32, 96, 72, 2, 192, 23.0, 23.2},
    {32, 128, 2, 0, 0, 5.9, 6.2},        {32, 128, 7, 16, 256, 7.0, 7.0},     {32, 128, 48, 8, 256, 11.0, 25.4},
    {32, 128, 72, 2, 512, 29.0, 30.1},   {32, 128, 108, 4, 256, 20.0, 59.2},  {32, 192, 9, 0, 0, 6.8, 22.9},
    {32, 192, 15, 8, 192, 26.2, 26.4, 16}, {32, 192, 36, 4, 384, 36.1, 37.4}, {32, 192, 48, 8, 192, 26.2, 60.6, 56},
    {32, 256, 4, 0, 0, 8.0, 18.6},       {32, 256, 7, 16, 256, 20.6, 21.0, 6}, {32, 512, 1, 0, 0, 14.7, 14.7},
    {64, 32, 28, 16, 64, 3.0, 4.7},      {64, 32, 60, 4, 128, 4.8, 6.0},      {64, 48, 14, 16, 160, 3.9, 7.6},
    {64, 48, 100, 4, 96, 7.6, 14.4},     {64, 48, 148, 1, 288, 15.8, 16.0},   {64, 64, 14, 16, 256, 4.5, 8.8},
    {64, 64, 48, 4, 128, 9.4, 13.9},     {64, 64, 72, 2, 256, 14.3, 15.1},    {64, 64, 108, 4, 128, 9.4, 23.6},
    {64, 96, 6, 0, 0, 5.9, 8.9},         {64, 96, 48, 8, 288, 12.8, 30.7},    {64, 128, 3, 0, 0, 6.2, 7.9},
    {64, 128, 7, 16, 512, 10.8, 10.8},   {64, 192, 6, 0, 0, 8.0, 21.2},       {64, 192, 7, 16, 192, 24.9, 25.3, 0},
    {64, 256, 4, 0, 0, 9.5, 24.6},       {64, 256, 7, 16, 256, 33.1, 33.4, 0}, {64, 512, 1, 0, 0, 19.5, 19.5},
};

}  // namespace

FewRuns few_runs_variant(int precision, int n, int runs, int level, bool alone, const PlainVariant* own) {
    for (const FewRow& r : kFew) {
        if (r.precision != precision || r.n != n) continue;
        if (r.beside == 0 && !alone && !(own && own->cluster == r.cluster && own->threads == r.threads)) continue;
        if (level > 0) {
            --level;
            continue;
        }
        if (own && r.cluster == 0) continue;
        const PlainVariant* v = nullptr;
        for_each_variant([&](const PlainVariant* c) {
            if (c->precision == precision && c->n == n && !c->thermal && c->cluster == r.cluster &&
                (r.cluster ? c->threads == r.threads : c->fit != nullptr))
                v = c;
            return v != nullptr;
        }, true);
        int fit = 0;
        if (v && v->fit && v->fit(&fit) != cudaSuccess) {
            cudaGetLastError();  // the device cannot hold the launch: the next row, the default can
            continue;
        }
        const double at = r.upto > 1 ? std::min(1.0, (runs - 1.0) / (r.upto - 1.0)) : 0.0;
        return {v, alone || r.beside <= 0 ? r.upto : r.beside, r.us1 + (r.us - r.us1) * at, r.cluster == 0};
    }
    return {nullptr, 0, 0.0, false};
}

const PlainVariant* find_split(int precision, int n, int cluster, int threads) {
    const PlainVariant* v = nullptr;
    for_each_variant([&](const PlainVariant* c) {
        if (c->precision == precision && c->n == n && !c->thermal && c->cluster == cluster && c->threads == threads) v = c;
        return v != nullptr;
    });
    return v;
}

// 64 x 64 FP32 runs past the rows of kFew, by the modelled time of the two splits.  One CTA of 512
// threads per run: 13.3 us per step, 148 runs at a time, the longest first.  4-CTA clusters, five CTAs to
// an SM: 17.8 us per step of the longest run, and 0.099 us per step of all of them together.  Over 152 to 600
// runs of equal, nearly equal, uniform, log-uniform and two lengths the choice was at most 4 %
// slower than the other.  ms on one CTA / on clusters: 160 equal runs of 149 steps 3.95 / 2.65, 300 5.93 /
// 4.48, 600 9.95 / 8.73; 296 (two full waves) of 60 steps 1.77 / 1.93; 160 of 99-399 steps 5.24 / 6.45, 300 of
// 20-250 3.35 / 4.17.
//   Beside larger sides the clusters' CTAs hold up clusters that need a whole SM: 160 runs of 64 x 64 and
// 8 of 128 x 128 (61 slices) took 2.73 ms against 1.90, with two of 256 x 256 3.2 against 2.0, a sweep of
// 256 runs over 64-256 75.2 against 74.1.  With up to three runs of 96 x 96 or 128 x 128 beside 149-450
// equal ones they were never slower (three of 96 x 96 beside 160: 1.87 against 2.70), with four
// sometimes (128 x 128: 2.66 against 1.87).
const PlainVariant* many_small_variant(std::vector<int> steps64, int runs_to_128, int runs_above) {
    constexpr int kPlaces = 148;
    if ((int)steps64.size() <= kPlaces || runs_to_128 > 3 || runs_above > 0) return nullptr;
    std::sort(steps64.begin(), steps64.end(), [](int a, int b) { return a > b; });
    std::priority_queue<long long, std::vector<long long>, std::greater<long long>> ends;  // of the places' queues
    for (int i = 0; i < kPlaces; ++i) ends.push(0);
    long long total = 0, last = 0;
    for (int st : steps64) {
        const long long e = ends.top() + st;
        ends.pop();
        ends.push(e);
        last = std::max(last, e);
        total += st;
    }
    const double clusters = std::max(17.8 * steps64[0], 0.099 * (double)total);
    return clusters < 13.3 * (double)last ? find_split(32, 64, 4, 128) : nullptr;
}

// 256 x 256 FP32 runs of a larger batch beside smaller ones.  The multi-pass march that these runs take
// by themselves is a row of launches, and each of them waits for places that the persistent CTAs of 128 x 128
// and 192 x 192 runs hold; 16-CTA clusters hold theirs.  While the device is not full the batch lasts
// as long as its longest run, and the clusters win: sweeps of 16-48 runs over 64-256 (100-400
// slices) took 1.0-1.17 times as long on the multi-pass march, of 64-128 runs 0.79-0.98.  `share` is the part
// of the device that the batch's clusters fill, 14 of these runs to a device; the line lies at 1.5 (1.46
// 1.12, 1.51 1.00, 1.72 0.95), and at 1 where a tenth and more of it is runs that a guard promotes to FP64,
// whose clusters go first (guarded sweeps of 16-48 runs: up to 1 1.0-1.3, above 0.79-1.13).  With only 64 x 64 runs beside, whose CTAs leave by themselves, the
// multi-pass march is as fast or faster; beside less than a tenth of the others it is from 11 runs on
// (8 runs and one of 128 x 128 1.25, 10 and one 1.07, 13 and one 0.87); with 14 runs or more the clusters
// leave no place for the others, and where another class has more work it goes first and holds theirs.
const PlainVariant* mixed_256_variant(int runs, double work, double others_work, double others_share, double promoted_share) {
    const double share = runs / 14.0 + others_share;
    if (others_share <= 0.0 || runs > 13 || share > (promoted_share < 0.1 ? 1.5 : 1.0) || others_work > work) return nullptr;
    if (runs > 10 && others_share < 0.1) return nullptr;
    return default_variant(32, 256, 0, SHG_MARCH_FUSED);
}

const PlainVariant* find_plain_variant(int precision, int n, int thermal, int march) {
    if (march == SHG_MARCH_AUTO && !thermal) {
        std::lock_guard<std::mutex> lk(g_mu);
        for (const Choice& c : g_chosen)
            if (c.v->precision == precision && c.v->n == n) return c.v;
    }
    return default_variant(precision, n, thermal, march);
}

const PlainVariant* default_variant(int precision, int n, int thermal, int march) {
    const int th = thermal ? 1 : 0;
    const PlainVariant *fused = nullptr, *multi = nullptr;
    for_each_variant([&](const PlainVariant* v) {
        if (v->precision == precision && v->n == n && v->thermal == th) {
            if (v->mp && !multi) multi = v;
            if (!v->mp && !fused) fused = v;
        }
        return false;
    });
    if (march == SHG_MARCH_FUSED) return fused;
    if (march == SHG_MARCH_MULTIPASS) return multi;
    // automatic, for batches too large for the marches for few runs: thermal runs and
    // 256 x 256 plain ones on the multi-pass kernels where they are built, whose launches spread each
    // step over the whole GPU (a 16-CTA cluster per 256 x 256 run covers 112 of the 148 SMs at most:
    // 8 / 72 runs FP32 34.5 -> 24.0 / 175 -> 120 us per step, FP64 66 -> 38 / 362 -> 225; a sweep of
    // 256 runs over sides 64-256 73.8 -> 68.6 ms); smaller sides, which fill it with clusters, on the
    // fused march
    if (multi && (th || n >= 256)) return multi;
    return fused ? fused : multi;
}

bool plain_choice_rules(int precision, int n, int runs) {
    std::lock_guard<std::mutex> lk(g_mu);
    for (const Choice& c : g_chosen)
        if (c.v->precision == precision && c.v->n == n) return runs >= c.from;
    return false;
}

int plain_candidates(int precision, int n, const PlainVariant** out, int max) {
    int k = 0;
    for_each_variant([&](const PlainVariant* v) {
        if (v->precision == precision && v->n == n && !v->thermal && k < max) out[k++] = v;
        return false;
    });
    return k;
}

void clear_plain_choices() {
    std::lock_guard<std::mutex> lk(g_mu);
    g_chosen.clear();
}

void clear_plain_choice(int precision, int n) {
    std::lock_guard<std::mutex> lk(g_mu);
    for (size_t i = 0; i < g_chosen.size(); ++i)
        if (g_chosen[i].v->precision == precision && g_chosen[i].v->n == n) {
            g_chosen.erase(g_chosen.begin() + i);
            return;
        }
}

void set_plain_choice(const PlainVariant* v, int from) {
    std::lock_guard<std::mutex> lk(g_mu);
    for (Choice& c : g_chosen)
        if (c.v->precision == v->precision && c.v->n == v->n) {
            c = {v, from};
            return;
        }
    g_chosen.push_back({v, from});
}

}  // namespace shg
