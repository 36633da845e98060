// ssfm_v_split.cu — variants of the fused march for single runs and small batches: wider clusters
// than the defaults, with a thread per field and point pair (SPLIT, ssfm_plain.cuh).  Which batch
// takes which: kFew in ssfm_registry.cu.
#include "ssfm_launch.cuh"

namespace shg {

static const PlainVariant kTable[] = {
    SHG_SPLIT_VARIANT(float, 32, 32, 16, 64, 1),   SHG_SPLIT_VARIANT(float, 32, 48, 16, 96, 1),
    SHG_SPLIT_VARIANT(float, 32, 64, 16, 128, 1),  SHG_SPLIT_VARIANT(float, 32, 96, 16, 288, 1),
    SHG_SPLIT_VARIANT(float, 32, 128, 16, 256, 1), SHG_SPLIT_VARIANT(float, 32, 48, 4, 96, 6),
    SHG_SPLIT_VARIANT(float, 32, 96, 8, 288, 3),   SHG_SPLIT_VARIANT(float, 32, 96, 2, 192, 2),
    SHG_SPLIT_VARIANT(float, 32, 128, 8, 256, 3),
};

VariantTable variants_split() { return {kTable, (int)(sizeof(kTable) / sizeof(kTable[0]))}; }

}  // namespace shg
