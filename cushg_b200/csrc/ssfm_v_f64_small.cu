// ssfm_v_f64_small.cu — FP64 variants of the fused march for grid sides 32-96, the default of each
// side first, with a thread per field and point pair.  Per step, 148 runs / 300 runs, against one
// thread for both fields: 32 9.0 / 19.6 (12.1 / 24.9) us, 48 22.0 / 36.8 (19.9 / 56.1), 64 25.9 / 59.9
// (26.4 / 60.1), 96 66.2 (73.9).
#include "ssfm_launch.cuh"

namespace shg {

static const PlainVariant kTable[] = {
    SHG_SPLIT_VARIANT(double, 64, 32, 1, 256, 2),
    SHG_VARIANT(double, 64, 32, 1, 128, 1, false),
    SHG_SPLIT_VARIANT(double, 64, 48, 4, 96, 4),
    SHG_SPLIT_VARIANT(double, 64, 48, 1, 288, 2),
    SHG_VARIANT(double, 64, 48, 1, 192, 1, false),
    // 64: two-CTA clusters at two per SM
    SHG_SPLIT_VARIANT(double, 64, 64, 2, 256, 2),
    SHG_VARIANT(double, 64, 64, 1, 256, 1, false),
    SHG_SPLIT_VARIANT(double, 64, 96, 2, 576, 1),
    SHG_VARIANT(double, 64, 96, 2, 192, 1, false),
};

VariantTable variants_f64_small() { return {kTable, (int)(sizeof(kTable) / sizeof(kTable[0]))}; }

}  // namespace shg
