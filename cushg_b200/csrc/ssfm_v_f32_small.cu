// ssfm_v_f32_small.cu — FP32 variants of the fused march for grid sides 32-96.  The first variant of
// each side is the default.  32, 48 and 96 run a thread per field and point pair, as a step's time is
// a thread's chain even on a full device.  Per step, 148 runs / 300 runs, against one thread for both
// fields: 32 6.6 / 14.1 (9.7 / 20.1) us, 48 12.7 / 28.5 (15.0 / 41.4), 96 32.5 (45.0).  64 alone gains
// the same way in 4-CTA clusters (34.5 against 44.6 at 300 runs), but in a sweep beside other sides
// those wait for four free places, and two split CTAs per SM slow the others down: 256 instances of
// 64-256 take 75.2 and 76.9 ms against 74.1.
#include "ssfm_launch.cuh"

namespace shg {

static const PlainVariant kTable[] = {
    SHG_SPLIT_VARIANT(float, 32, 32, 1, 256, 2),
    SHG_VARIANT(float, 32, 32, 1, 128, 1, false),
    SHG_SPLIT_VARIANT(float, 32, 48, 1, 288, 2),
    SHG_VARIANT(float, 32, 48, 1, 192, 1, false),
    SHG_VARIANT(float, 32, 64, 1, 512, 1, false),
    SHG_SPLIT_VARIANT(float, 32, 64, 4, 128, 5),
    SHG_VARIANT(float, 32, 64, 1, 256, 2, false),
    SHG_SPLIT_VARIANT(float, 32, 96, 1, 384, 1),
    SHG_VARIANT(float, 32, 96, 1, 192, 1, false),
};

VariantTable variants_f32_small() { return {kTable, (int)(sizeof(kTable) / sizeof(kTable[0]))}; }

}  // namespace shg
