// ssfm_wide.cu — variants and launch of the wide march (ssfm_wide.cuh).
#include <cuda_runtime.h>

#include "shg_host.h"
#include "ssfm_variants.h"
#include "ssfm_wide.cuh"

namespace shg {

namespace {

// Kernel attributes, once per device, and the instances that fit on the device at once.
template <typename T, int N, bool THERM>
cudaError_t wide_fit(int* instances) {
    using Cfg = WideCfg<T, N, THERM>;
    auto kern = ssfm_wide_kernel<T, N, THERM>;
    static PerDevice<int> state;
    return state.get(
        [&](int dev, int& res) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::smem_bytes);
            int sms = 0, per_sm = 0;
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, Cfg::NT, Cfg::smem_bytes);
            res = sms * per_sm / Cfg::G;
            return e == cudaSuccess && res < 1 ? cudaErrorCooperativeLaunchTooLarge : e;
        },
        instances);
}

template <typename T, int N, bool THERM>
cudaError_t wide_march(const InstDesc* dev_descs, const InstDesc*, int count, cudaStream_t s) {
    using Cfg = WideCfg<T, N, THERM>;
    auto kern = ssfm_wide_kernel<T, N, THERM>;
    int fit = 0;
    const cudaError_t attr_err = wide_fit<T, N, THERM>(&fit);
    if (attr_err != cudaSuccess) return attr_err;
    if (count <= 0) return cudaSuccess;
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t plane = up(sizeof(cx<T>) * (size_t)N * N);
    WideWs ws;
    ws.off_s = plane;
    ws.off_part = 2 * plane;
    ws.stride = 2 * plane + up(sizeof(double) * 2 * N);
    const BarrierLimit bl = barrier_limit();
    ws.limit_ns = bl.ns;
    ws.withheld = bl.withheld;
    const int batch = count < fit ? count : fit;
    char* buf = nullptr;
    const size_t bars = up(sizeof(unsigned) * 2 * (size_t)count);
    cudaError_t e = dev_alloc((void**)&buf, bars + ws.stride * (size_t)batch, s);
    if (e != cudaSuccess) return e;
    ws.base = buf + bars;
    e = cudaMemsetAsync(buf, 0, bars, s);
    for (int i = 0; i < count && e == cudaSuccess; i += batch) {
        ws.bar = reinterpret_cast<unsigned*>(buf) + 2 * (size_t)i;
        const InstDesc* dd = dev_descs + i;
        void* args[] = {&dd, &ws};
        e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern),
                                        dim3(Cfg::G, (unsigned)(count - i < batch ? count - i : batch)), dim3(Cfg::NT), args,
                                        Cfg::smem_bytes, s);
    }
    const cudaError_t ef = cudaFreeAsync(buf, s);
    return e != cudaSuccess ? e : ef;
}

#define SHG_WIDE_VARIANT(T, PREC, N, THERM)                                                                          \
    {PREC, N, 0, WideCfg<T, N, THERM>::NT, 1, THERM ? 1 : 0, WideCfg<T, N, THERM>::smem_bytes, nullptr, &wide_march<T, N, THERM>, \
     &wide_fit<T, N, THERM>}

const PlainVariant kTable[] = {
    SHG_WIDE_VARIANT(float, 32, 128, false),  SHG_WIDE_VARIANT(float, 32, 192, false),
    SHG_WIDE_VARIANT(float, 32, 256, false),  SHG_WIDE_VARIANT(float, 32, 512, false),
    SHG_WIDE_VARIANT(double, 64, 96, false),  SHG_WIDE_VARIANT(double, 64, 128, false),
    SHG_WIDE_VARIANT(double, 64, 192, false), SHG_WIDE_VARIANT(double, 64, 256, false),
    SHG_WIDE_VARIANT(double, 64, 512, false),
    SHG_WIDE_VARIANT(float, 32, 32, true),    SHG_WIDE_VARIANT(float, 32, 64, true),
    SHG_WIDE_VARIANT(float, 32, 128, true),   SHG_WIDE_VARIANT(float, 32, 256, true),
    SHG_WIDE_VARIANT(float, 32, 512, true),
    SHG_WIDE_VARIANT(double, 64, 32, true),   SHG_WIDE_VARIANT(double, 64, 64, true),
    SHG_WIDE_VARIANT(double, 64, 128, true),  SHG_WIDE_VARIANT(double, 64, 256, true),
    SHG_WIDE_VARIANT(double, 64, 512, true),
};

}  // namespace

VariantTable variants_wide() { return {kTable, (int)(sizeof(kTable) / sizeof(kTable[0]))}; }

// When the wide march pays for thermal passes.  It takes the whole device for `fit` instances at a
// time, so its time grows with the rounds of `fit`; the fused march's grows only when its clusters no
// longer fit side by side, the multi-pass march's slowly with the count.  Measured per step (us), wide
// against the march a batch takes (fused, or multi-pass from 128 x 128):
//   1 round   FP32: 128 x 4 10.6 / 15.6, 256 x 2 13.0 / 18.6, 512 21.4 / 29.8;
//             FP64: 128 x 4 11.7 / 17.5, 256 x 2 17.0 / 22.8, 512 33.0 / 38.0
//   2 rounds  FP32: 64 x 16 21.4 / 40.6, but 128 x 8 20.8 / 19.2, 256 x 4 25.6 / 24.5,
//             512 x 2 42.3 / 38.6; FP64: 64 x 16 23.3 / 56.8, but 128 x 8 23.1 / 22.7,
//             256 x 4 33.1 / 33.0, 512 x 2 65.4 / 57.8
const PlainVariant* wide_thermal_variant(int precision, int n, int count) {
    for (const PlainVariant& v : kTable) {
        if (v.precision != precision || v.n != n || !v.thermal) continue;
        int fit = 0;
        if (v.fit(&fit) != cudaSuccess) {
            cudaGetLastError();  // the device cannot hold the launch: the other marches can
            return nullptr;
        }
        return count <= fit * (n < 128 ? 2 : 1) ? &v : nullptr;
    }
    return nullptr;
}

}  // namespace shg
