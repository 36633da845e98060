// ssfm_v_split64.cu — the FP64 variants beside ssfm_v_split.cu's.
#include "ssfm_launch.cuh"

namespace shg {

static const PlainVariant kTable[] = {
    SHG_SPLIT_VARIANT(double, 64, 32, 16, 64, 1),  SHG_SPLIT_VARIANT(double, 64, 48, 16, 160, 1),
    SHG_SPLIT_VARIANT(double, 64, 64, 16, 256, 1), SHG_SPLIT_VARIANT(double, 64, 128, 16, 512, 1),
    SHG_SPLIT_VARIANT(double, 64, 32, 4, 128, 4),  SHG_SPLIT_VARIANT(double, 64, 64, 4, 128, 3),
    SHG_SPLIT_VARIANT(double, 64, 96, 8, 288, 2),
};

VariantTable variants_split64() { return {kTable, (int)(sizeof(kTable) / sizeof(kTable[0]))}; }

}  // namespace shg
