// ssfm_v_split.cu — variants of the fused march for one run on its own: 16-CTA clusters with a
// thread per field and point pair (SPLIT, ssfm_plain.cuh).
#include "ssfm_launch.cuh"

namespace shg {

namespace {

#define SHG_SPLIT_VARIANT(T, PREC, N, NT, ROUNDS)                                                                      \
    {PREC, N, 16, NT, 1, 0, PlainCfg<T, N, 16, NT>::smem_bytes, &launch_plain<T, N, 16, NT, false, 1, true>, nullptr, \
     &plain_fit<T, N, 16, NT, false, 1, true>, ROUNDS}

const PlainVariant kTable[] = {
    SHG_SPLIT_VARIANT(float, 32, 32, 64, 1),   SHG_SPLIT_VARIANT(float, 32, 48, 96, 2),
    SHG_SPLIT_VARIANT(float, 32, 64, 128, 2),  SHG_SPLIT_VARIANT(float, 32, 96, 288, 6),
    SHG_SPLIT_VARIANT(double, 64, 32, 64, 2),  SHG_SPLIT_VARIANT(double, 64, 48, 144, 4),
    SHG_SPLIT_VARIANT(double, 64, 64, 256, 3),
};

}  // namespace

VariantTable variants_split() { return {kTable, (int)(sizeof(kTable) / sizeof(kTable[0]))}; }

}  // namespace shg
