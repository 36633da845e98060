// ssfm_variants.h — registry of the compiled variants of the SSFM marches.
//
// A variant of the fused march fixes the precision, the grid side N, the cluster split C (CTAs per
// instance), the threads per CTA and the CTAs per SM the register budget targets; the multi-pass and
// wide marches have one variant each where they are built.  Each (precision, N) has a default
// variant, variants for few runs, and possibly alternatives with another split, which the tuners time.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

#include "shg_internal.h"

namespace shg {

// Launch of `count` instances from `descs`.  queue != nullptr: a persistent launch of at
// most as many clusters as fit on the device, fed by the work queue *queue (an int the
// caller zeroes, stream-ordered, before the launch).  queue == nullptr: one cluster per
// instance.
using PlainLaunch = cudaError_t (*)(const InstDesc* descs, int count, int* queue, cudaStream_t stream);

// Launch of a multi-pass march (ssfm_multipass.cuh): device and host copies of the
// descriptors (the host sequences the per-step launches from the step counts).
using MpLaunch = cudaError_t (*)(const InstDesc* dev_descs, const InstDesc* host_descs, int count,
                                 cudaStream_t stream);

struct PlainVariant {
    int precision;  // 32 or 64
    int n;          // grid side
    int cluster;    // CTAs per instance (0: multi-pass, the planes in global memory)
    int threads;    // threads per CTA (multi-pass: of the row pass)
    int minb;       // CTAs per SM the register budget targets
    int thermal;    // 1: thermal pass (per-voxel optics, Q emission)
    size_t smem;    // dynamic shared memory per CTA (multi-pass: of the row pass)
    PlainLaunch launch;  // fused cluster march, or null
    MpLaunch mp;         // multi-pass or wide march, or null
    cudaError_t (*fit)(int* instances) = nullptr;  // instances resident on the device at once
};

// Run `count` instances through variant v (either kind); queue as for PlainLaunch.
inline cudaError_t run_variant(const PlainVariant* v, const InstDesc* dev_descs, const InstDesc* host_descs, int count,
                               int* queue, cudaStream_t stream) {
    return v->mp ? v->mp(dev_descs, host_descs, count, stream) : v->launch(dev_descs, count, queue, stream);
}

struct VariantTable {
    const PlainVariant* v;
    int count;
};

// per translation unit tables (ssfm_v_*.cu)
VariantTable variants_f32_small();
VariantTable variants_f32_128();
VariantTable variants_f32_192();
VariantTable variants_f32_256();
VariantTable variants_f64_small();
VariantTable variants_f64_large();
VariantTable variants_thermal();
VariantTable variants_multipass();
VariantTable variants_split();  // this and the next two: not among the batch tuner's choices
VariantTable variants_split64();
VariantTable variants_wide();

// The variant the drivers use for (precision, n, thermal) under march preference `march`
// (SHG_MARCH_*) where the number of runs does not say otherwise: automatic = the one a tuner or
// shg_set_schedule chose, else the default (ssfm_registry.cu: the first compiled fused variant, or the
// multi-pass one); fused / multi-pass = the default of that kind.  Null if none is built.
const PlainVariant* find_plain_variant(int precision, int n, int thermal = 0, int march = 0);
// The wide march (ssfm_wide.cuh) of thermal passes of (precision, n) if it is the faster one for
// `count` runs that have the device to themselves, else null.
const PlainVariant* wide_thermal_variant(int precision, int n, int count);
// Plain runs of (precision, n): the level-th variant for few runs, from the widest on; v is null past the
// last.  alone: with no other class.  own, if given: no wide march (a cooperative launch, which has the
// device to itself while it runs) but the next row, the class's own variant among them.
struct FewRuns {
    const PlainVariant* v;
    int upto;   // the number of runs up to which it is the fastest, or that fill the device beside other classes
    double us;  // per step, of `runs` runs
    bool wide;
};
FewRuns few_runs_variant(int precision, int n, int runs, int level, bool alone, const PlainVariant* own = nullptr);
// The variant of the 64 x 64 FP32 runs of a larger batch with these step counts, beside `runs_to_128`
// runs of the sides above 64 up to 128 and `runs_above` of larger ones; null: the default.
const PlainVariant* many_small_variant(std::vector<int> steps64, int runs_to_128, int runs_above);
// The variant of the `runs` 256 x 256 FP32 runs of a larger batch: work is their point-steps, others_work the
// most that a class of 128 x 128 or 192 x 192 runs has, others_share the part of the device that those classes'
// clusters fill, promoted_share the FP64 ones' part of it; null: the default.
const PlainVariant* mixed_256_variant(int runs, double work, double others_work, double others_share, double promoted_share);
// find_plain_variant without the choices below.
const PlainVariant* default_variant(int precision, int n, int thermal, int march);
// Every compiled plain variant of (precision, n) but those for few runs; returns how many.
int plain_candidates(int precision, int n, const PlainVariant** out, int max);
// The one of them with this split; null if there is none.
const PlainVariant* find_split(int precision, int n, int cluster, int threads);
// Make v the variant find_plain_variant returns for its plain (precision, n).  Against the variants for
// few runs it holds in calls with at least `from` runs of the class: 0 where a caller pins it, the
// number of runs it was measured with where a tuner chose it, so that tuning a large batch leaves
// the single runs of its classes as they were.
void set_plain_choice(const PlainVariant* v, int from);
// Whether such a choice rules a call with `runs` runs of the class.
bool plain_choice_rules(int precision, int n, int runs);
void clear_plain_choice(int precision, int n);
// forget every choice: later runs use the compiled defaults
void clear_plain_choices();

}  // namespace shg
