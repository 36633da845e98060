// jacobi_resident.cu — many unchecked Jacobi sweeps of the heat equation in one cooperative
// launch, with the temperature in shared memory.
//
// Reference: the Tfield::upDate loop (src/headers/Tfield.h:350-364) around
// kernelHeatEquationTopOpen / kernelHeatEquationOvenSurrounded (Tfield.h:93-240).
//
// One launch per sweep streams T, Q and the new T through L2 and HBM: 12.4 us at 128 x 128 x 200
// FP64, the HBM rate.  That grid's T is 26 MB, and 148 SMs have 33 MB of shared memory.  Here a CTA
// keeps a tile of all x, TY rows and tz planes in shared memory for the whole window of sweeps,
// each thread a 2 x 2 (x, y) block of every plane, and updates it in place: a sweep walks the
// planes, every thread reads its lateral neighbours' old values, a CTA barrier, then the new
// values replace them (the old plane below lives on in registers).  Only Q streams, from L2 or,
// where the tile leaves room, L1.  Between sweeps the tiles' faces (rows and planes next to
// another tile) go through global memory and a grid barrier.
//
// What bounds it: the planes' chains of shared-memory reads and dependent FP64 operations, at two
// warps per scheduler (issue 36 % with one plane per barrier), then the grid barrier and the
// latency of the first face loads, about 1.7 us a sweep (32 x 32 grids are nothing else).
// Measured per sweep in windows of 4000, against the graph of one-sweep launches that ran them
// before (built in the call): 128 x 128 x 200 FP64 8.2 / 15.4 us (12.4 in a graph used 40 times),
// 256 x 256 x 100 FP32 11.3 / 21.2, 128 x 128 x 100 FP32 3.9 / 15.8, 64 x 64 x 50 FP64 2.5 / 13.8.
// Two CTAs per SM (128 registers) measured 10.0 and 3.6 for the first and third.
//
// Every voxel is jacobi_point's expression of the same operands with the same products fused,
// so the temperatures are the bits of the one-sweep kernels (thermal.cu).
#include <cuda_runtime.h>

#include <algorithm>

#include "dft.cuh"
#include "grid_barrier.cuh"
#include "jacobi_point.cuh"
#include "jacobi_tiles.h"
#include "shg_host.h"
#include "thermal.h"

namespace shg {

namespace {

template <typename R> struct pair2_t;
template <> struct pair2_t<float> { using type = float2; };
template <> struct pair2_t<double> { using type = double2; };

constexpr int kResThreads = 256;
// Planes that share a barrier, and planes of Q and of the face rows in flight.  1 / 3 / 4 / 6
// measured 13.7 / 8.3 / 8.5 / 9.5 us a sweep at 128 x 128 x 200 FP64.
constexpr int AH = 3;

// A condition known at compile time, passed like a run-time one.
template <bool B>
struct Flag {
    __device__ constexpr operator bool() const { return B; }
};

struct ResidentArgs {
    int count;       // sweeps
    int ytiles, tz;  // tiles along y, planes per tile (the last tile may have fewer)
    unsigned *bar, *err;  // arrivals at the grid barriers; set to 1 when a wait ran out
    unsigned long long limit_ns;
    unsigned withheld;  // as WideWs::withheld
};

// A voxel's class: which of its directions end at a face (1 x, 2 y, 4 z).  Every branch of
// jacobi_point is v = (X1 c1 + X2 c2 + X3 c3 + A B) sc in this order with the product X2 c2 rounded
// by itself and the others fused, X1..X3 sums of opposite neighbours (S) or the one neighbour
// of a face (g):
//   class  0: Sx Sy Sz   1: Sy gx Sz   2: Sx gy Sz   3: gy gx Sz
//          4: Sx gz Sy   5: gx gz Sy   6: gy gz Sx   7: gx gy gz
template <typename R>
struct ClassCoef {
    R c1, c2, c3, a, b, sc;
};
template <typename R>
__device__ ClassCoef<R> class_coef(int cls, const JacobiCoef<R>& k) {
    switch (cls) {
        case 0: return {k.idx2, k.idy2, k.idz2, (R)0, k.iK, k.L2};  // A = q
        case 1: return {k.ax, (R)1, k.bx, k.Bix, k.Tinf, k.fx};
        case 2: return {k.ay, (R)1, k.by, k.Biy, k.Tinf, k.fy};
        case 3: return {k.ad, k.bd, k.cd, k.td, (R)1, k.D};
        case 4: return {k.az, (R)1, k.bz, k.Biz, k.Tinf, k.fz};
        case 5: return {k.av, k.bv, k.cv, k.tv, (R)1, k.V};
        case 6: return {k.ah, k.bh, k.ch, k.th, (R)1, k.H};
        default: return {k.AV, k.BV, k.CV, k.Tinf, k.BiD, k.GV};
    }
}
template <typename R>
__device__ __forceinline__ R chain(const ClassCoef<R>& c, R x1, R x2, R x3, R a) {
    R t = fma_r(x1, c.c1, mul_r(x2, c.c2));
    t = fma_r(x3, c.c3, t);
    t = fma_r(a, c.b, t);
    return mul_r(t, c.sc);
}

// c ? a : b as one select: a branch around the chain would serialise each warp's face lane.
__device__ __forceinline__ double pick(bool c, double a, double b) {
    double r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tselp.f64 %0, %1, %2, p;\n\t}" : "=d"(r) : "d"(a), "d"(b), "r"((int)c));
    return r;
}
__device__ __forceinline__ float pick(bool c, float a, float b) {
    float r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tselp.f32 %0, %1, %2, p;\n\t}" : "=f"(r) : "f"(a), "f"(b), "r"((int)c));
    return r;
}

template <typename R, int BOUND, int N, bool HASQ>
__global__ void __launch_bounds__(kResThreads, 1)
    jacobi_resident_kernel(R* __restrict__ Ta, R* __restrict__ Tb, const R* __restrict__ Q, const JacobiCoef<R> k,
                           const ResidentArgs ra) {
    using R2 = typename pair2_t<R>::type;
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ ClassCoef<R> coef[8];
    constexpr int n = N, NXP = N / 2, TY = 2 * (kResThreads / NXP);
    const int nz = k.nz;
    R2* T = reinterpret_cast<R2*>(res_smem) + NXP;  // [tz][TY][NXP], and a row of padding on either side
    const int tid = threadIdx.x, tx = tid % NXP, ty = tid / NXP;
    const int y0 = (blockIdx.x % ra.ytiles) * TY, z0 = (blockIdx.x / ra.ytiles) * ra.tz;
    const int tzn = min(ra.tz, nz - z0);
    const int x = 2 * tx, ya = y0 + 2 * ty, yb = ya + 1;
    const bool first_row = ty == 0, last_row = 2 * ty + 2 == TY;
    constexpr size_t plane = (size_t)n * n;
    const size_t col = (size_t)z0 * plane + (size_t)ya * n + x;  // this thread's block in the first plane
    auto ldcg2 = [](const R* p) { return __ldcg(reinterpret_cast<const R2*>(p)); };
    R2 zero;
    zero.x = zero.y = (R)0;
    if (tid < 8) coef[tid] = class_coef<R>(tid, k);
    const int mine = 2 * ty * NXP + tx;  // this thread's rows in a plane of the tile: mine, mine + NXP
    for (int z = 0; z < tzn; ++z) {
        T[z * TY * NXP + mine] = ldcg2(Ta + col + z * plane);
        T[z * TY * NXP + mine + NXP] = ldcg2(Ta + col + z * plane + n);
    }
    __syncthreads();
    constexpr bool TOP = BOUND == SHG_BOUNDARY_TOP_OPEN;
    const bool fl = x == 0, fr = x + 2 == n;  // this pair holds the x = 0 / x = n - 1 face
    const bool held_a = ya == 0, held_b = !TOP && yb == n - 1;  // rows that keep their values
    const bool face_b = TOP && yb == n - 1;                     // the Robin face y = n - 1
    // factors of the block's four voxels in planes inside z
    const ClassCoef<R> cal = coef[TOP && fl ? 1 : 0], car = coef[TOP && fr ? 1 : 0];
    const ClassCoef<R> cbl = coef[(TOP && fl ? 1 : 0) | (face_b ? 2 : 0)], cbr = coef[(TOP && fr ? 1 : 0) | (face_b ? 2 : 0)];
    // one row of the block in a plane inside z: its two voxels by their classes
    auto row = [&](bool yface, const ClassCoef<R>& l, const ClassCoef<R>& r, R2 c, R xm, R xp, R2 ym, R2 yp, R2 zm, R2 zp,
                   R2 q) -> R2 {
        R2 o;
        const R sx0 = add_r(c.y, xm), sx1 = add_r(xp, c.x);
        const R sz0 = add_r(zp.x, zm.x), sz1 = add_r(zp.y, zm.y);
        if (yface) {
            o.x = chain(l, fl ? ym.x : sx0, fl ? c.y : ym.x, sz0, l.a);
            o.y = chain(r, fr ? ym.y : sx1, fr ? c.x : ym.y, sz1, r.a);
            return o;
        }
        const R sy0 = add_r(yp.x, ym.x), sy1 = add_r(yp.y, ym.y);
        if (TOP) {
            o.x = chain(l, fl ? sy0 : sx0, fl ? c.y : sy0, sz0, fl ? l.a : q.x);
            o.y = chain(r, fr ? sy1 : sx1, fr ? c.x : sy1, sz1, fr ? r.a : q.y);
        } else {  // the x faces are held
            o.x = pick(fl, c.x, chain(l, sx0, sy0, sz0, q.x));
            o.y = pick(fr, c.y, chain(r, sx1, sy1, sz1, q.y));
        }
        return o;
    };
    // one voxel of a plane at a z face
    auto any = [&](int px, int py, R c, R xm, R xp, R ym, R yp, R gz, R q) -> R {
        const bool fx = px == 0 || px == n - 1, fy = py == n - 1;
        if (py == 0 || (!TOP && (fx || fy))) return c;  // held
        const R gx = px == 0 ? xp : xm, sx = add_r(xp, xm), sy = add_r(yp, ym);
        const R x1 = fx ? gx : fy ? ym : sx;
        const R x2 = fx && fy ? ym : gz;
        const R x3 = fx && fy ? gz : fy ? sx : sy;
        const ClassCoef<R> cc = coef[4 | (fx ? 1 : 0) | (fy ? 2 : 0)];
        return chain(cc, x1, x2, x3, cc.a);
    };

    const R* qp = Q + col;
    // the rows next to the tile's; at the domain's ends a row of its own, loaded and not used
    const int off_m = ya > 0 ? -n : 0, off_p = yb + 1 < n ? 2 * n : n;
    unsigned target = ra.withheld;
    for (int s = 0; s < ra.count; ++s) {
        const R* src = ((s & 1) ? Tb : Ta) + col;  // the faces of the previous sweep (at first: the whole grid)
        R* dst = ((s & 1) ? Ta : Tb) + col;
        R2 za = zero, zb = zero, ta = zero, tb = zero;  // the planes below and above the tile
        if (z0 > 0) {
            za = ldcg2(src - plane);
            zb = ldcg2(src - plane + n);
        }
        if (z0 + tzn < nz) {
            ta = ldcg2(src + tzn * plane);
            tb = ldcg2(src + tzn * plane + n);
        }
        R2 ca = T[mine], cb = T[mine + NXP];
        // Q and the face rows of a plane (past the tile: of its last plane, unused)
        struct Ahead {
            R2 hm, hp, qa, qb;
        };
        auto fetch = [&](auto first, auto last, int z) {
            Ahead f{zero, zero, zero, zero};
            const size_t o = (size_t)min(z, tzn - 1) * plane;
            if (first) f.hm = ldcg2(src + o + off_m);
            if (last) f.hp = ldcg2(src + o + off_p);
            if (HASQ) {
                f.qa = __ldg(reinterpret_cast<const R2*>(qp + o));
                f.qb = __ldg(reinterpret_cast<const R2*>(qp + o + n));
            }
            return f;
        };
        // new values of the block in plane z (at W in shared memory), in registers
        auto step = [&](auto first, auto last, auto inner, int z, const R2* W, const Ahead& f, R2& na, R2& nb) {
            R2 ua = ta, ub = tb;
            if (inner || z + 1 < tzn) {
                ua = W[TY * NXP];
                ub = W[TY * NXP + NXP];
            }
            // (a face's missing neighbour reads a neighbouring row's voxel or the padding, unused)
            const R2 ym = first ? f.hm : W[-NXP], yp = last ? f.hp : W[2 * NXP];
            const R xma = W[-1].y, xpa = W[1].x, xmb = W[NXP - 1].y, xpb = W[NXP + 1].x;
            const int gz = z0 + z;
            if (inner || (gz > 0 && gz + 1 < nz)) {
                na = row(false, cal, car, ca, xma, xpa, ym, cb, za, ua, f.qa);
                nb = last && face_b ? row(true, cbl, cbr, cb, xmb, xpb, ca, yp, zb, ub, f.qb)
                                    : row(false, cbl, cbr, cb, xmb, xpb, ca, yp, zb, ub, f.qb);
                if (first && held_a) na = ca;
                if (last && held_b) nb = cb;
            } else {
                const R2 ga = gz == 0 ? ua : za, gb = gz == 0 ? ub : zb;
                na.x = any(x, ya, ca.x, xma, ca.y, ym.x, cb.x, ga.x, f.qa.x);
                na.y = any(x + 1, ya, ca.y, ca.x, xpa, ym.y, cb.y, ga.y, f.qa.y);
                nb.x = any(x, yb, cb.x, xmb, cb.y, ca.x, yp.x, gb.x, f.qb.x);
                nb.y = any(x + 1, yb, cb.y, cb.x, xpb, ca.y, yp.y, gb.y, f.qb.y);
            }
            // the tile's faces, for its neighbours
            const bool zface = !inner && (z == 0 || z == tzn - 1);
            if (first || zface) __stcg(reinterpret_cast<R2*>(dst + z * plane), na);
            if (last || zface) __stcg(reinterpret_cast<R2*>(dst + z * plane + n), nb);
            za = ca;
            zb = cb;
            ca = ua;
            cb = ub;
        };
        // One sweep of the tile for a warp whose rows are the tile's first, its last, or neither
        // (the row next to another tile, or the domain's end): the first plane, then AH planes at
        // a time (their lateral neighbours are read before any of them is written, so the planes'
        // chains overlap and one barrier serves all), then the last planes.
        auto sweep = [&](auto first, auto last) {
            const Flag<true> in;
            const Flag<false> edge;
            const Ahead f0 = fetch(first, last, 0);
            Ahead f[AH];
#pragma unroll
            for (int p = 0; p < AH; ++p) f[p] = fetch(first, last, 1 + p);
            R2 na[AH], nb[AH];
            step(first, last, edge, 0, T + mine, f0, na[0], nb[0]);
            __syncthreads();  // every thread has read this plane's old values
            T[mine] = na[0];
            T[mine + NXP] = nb[0];
            int zg = 1;
            for (; zg + AH < tzn; zg += AH) {
                R2* P = T + zg * TY * NXP + mine;
#pragma unroll
                for (int p = 0; p < AH; ++p) {
                    step(first, last, in, zg + p, P + p * TY * NXP, f[p], na[p], nb[p]);
                    f[p] = fetch(first, last, zg + p + AH);
                }
                __syncthreads();
#pragma unroll
                for (int p = 0; p < AH; ++p) {
                    P[p * TY * NXP] = na[p];
                    P[p * TY * NXP + NXP] = nb[p];
                }
            }
#pragma unroll
            for (int p = 0; p < AH; ++p) {
                if (zg + p >= tzn) break;
                R2* P = T + (zg + p) * TY * NXP + mine;
                step(first, last, edge, zg + p, P, f[p], na[p], nb[p]);
                __syncthreads();
                P[0] = na[p];
                P[NXP] = nb[p];
            }
        };
        using Yes = Flag<true>;
        using No = Flag<false>;
        if constexpr (N == 32) {  // a warp holds several row pairs
            sweep(first_row, last_row);
        } else {
            if (first_row) sweep(Yes(), No());
            else if (last_row) sweep(No(), Yes());
            else sweep(No(), No());
        }
        if (s + 1 < ra.count && !grid_barrier(ra.bar, target += gridDim.x, ra.limit_ns)) {
            if (tid == 0) atomicExch(ra.err, 1u);
            return;
        }
    }
    R* out = ((ra.count & 1) ? Tb : Ta) + col;
    for (int z = 0; z < tzn; ++z) {
        *reinterpret_cast<R2*>(out + z * plane) = T[z * TY * NXP + mine];
        *reinterpret_cast<R2*>(out + z * plane + n) = T[z * TY * NXP + mine + NXP];
    }
}

// The kernel's attribute, once per device, and the CTAs that a cooperative launch of it may have there.
template <typename R, int BOUND, int N, bool HASQ>
cudaError_t resident_ctas(int* ctas) {
    auto kern = jacobi_resident_kernel<R, BOUND, N, HASQ>;
    constexpr size_t smem = kResSmem + 2 * sizeof(R) * N;
    static PerDevice<int> state;
    return state.get(
        [&](int dev, int& v) {
            int sms = 0, per_sm = 0;
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kResThreads, smem);
            v = sms * per_sm;
            return e;
        },
        ctas);
}

template <typename R, int BOUND, int N, bool HASQ>
cudaError_t launch_tiles(R* Ta, R* Tb, const R* Q, const JacobiCoef<R>& k, const ResidentArgs& ra, int ctas, cudaStream_t s) {
    auto kern = jacobi_resident_kernel<R, BOUND, N, HASQ>;
    R *ta = Ta, *tb = Tb;
    const R* q = Q;
    JacobiCoef<R> kk = k;
    ResidentArgs r = ra;
    void* args[] = {&ta, &tb, &q, &kk, &r};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(ctas), dim3(kResThreads), args,
                                       sizeof(R) * (1024 * (size_t)ra.tz + 2 * N), s);
}

// f's instantiation for a grid side, boundary and source
template <typename R, int BOUND, int N, typename F>
cudaError_t with_source(bool q, F&& f) {
    return q ? f(&resident_ctas<R, BOUND, N, true>, &launch_tiles<R, BOUND, N, true>)
             : f(&resident_ctas<R, BOUND, N, false>, &launch_tiles<R, BOUND, N, false>);
}
template <typename R, int BOUND, typename F>
cudaError_t with_side(int n, bool q, F&& f) {
    switch (n) {
        case 32: return with_source<R, BOUND, 32>(q, f);
        case 64: return with_source<R, BOUND, 64>(q, f);
        case 128: return with_source<R, BOUND, 128>(q, f);
        case 256: return with_source<R, BOUND, 256>(q, f);
    }
    return cudaErrorInvalidValue;
}
template <typename R, typename F>
cudaError_t with_kernel(int boundary, int n, bool q, F&& f) {
    return boundary == SHG_BOUNDARY_OVEN_SURROUNDED ? with_side<R, SHG_BOUNDARY_OVEN_SURROUNDED>(n, q, f)
                                                    : with_side<R, SHG_BOUNDARY_TOP_OPEN>(n, q, f);
}

int sm_count() {
    static PerDevice<int> state;
    int sms = 0;
    const cudaError_t e = state.get(
        [](int dev, int& v) { return cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev); }, &sms);
    return e == cudaSuccess ? sms : 0;
}

}  // namespace

template <typename R>
bool jacobi_resident_fits(const JacobiCoef<R>& k, int boundary, bool source) {
    int ctas = 0;
    const cudaError_t e = with_kernel<R>(boundary, k.n, source, [&](auto fit, auto) { return fit(&ctas); });
    if (e != cudaSuccess) {
        cudaGetLastError();  // the one-sweep kernels can
        return false;
    }
    ResidentTiles t;
    return resident_tiles(sizeof(R), k.n, k.nz, sm_count(), ctas, &t);
}

template <typename R>
cudaError_t launch_jacobi_resident(R* Ta, R* Tb, const R* Q, const JacobiCoef<R>& k, int boundary, int count, unsigned* bar,
                                   unsigned* err, cudaStream_t s) {
    return with_kernel<R>(boundary, k.n, Q != nullptr, [&](auto fit, auto launch) {
        int ctas = 0;
        cudaError_t e = fit(&ctas);
        if (e != cudaSuccess) return e;
        ResidentTiles t;
        if (!resident_tiles(sizeof(R), k.n, k.nz, sm_count(), ctas, &t)) return cudaErrorInvalidValue;
        ResidentArgs ra;
        ra.count = count;
        ra.ytiles = t.ytiles;
        ra.tz = t.tz;
        ra.bar = bar;
        ra.err = err;
        const BarrierLimit bl = barrier_limit();
        ra.limit_ns = bl.ns;
        ra.withheld = bl.withheld;
        if ((e = cudaMemsetAsync(bar, 0, sizeof(unsigned), s)) != cudaSuccess) return e;
        return launch(Ta, Tb, Q, k, ra, t.ytiles * t.ztiles, s);
    });
}

template bool jacobi_resident_fits<float>(const JacobiCoef<float>&, int, bool);
template bool jacobi_resident_fits<double>(const JacobiCoef<double>&, int, bool);
template cudaError_t launch_jacobi_resident<float>(float*, float*, const float*, const JacobiCoef<float>&, int, int, unsigned*,
                                                   unsigned*, cudaStream_t);
template cudaError_t launch_jacobi_resident<double>(double*, double*, const double*, const JacobiCoef<double>&, int, int,
                                                    unsigned*, unsigned*, cudaStream_t);

}  // namespace shg
