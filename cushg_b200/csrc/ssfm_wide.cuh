// ssfm_wide.cuh — the SSFM march of one instance spread over the whole GPU: one cooperative
// launch of G CTAs for the z-march, for runs that have the device to themselves.
//
// The fused march (ssfm_plain.cuh) gives an instance one cluster of at most 16 SMs, which is
// the right share when a batch fills the GPU; alone, its step lasts as long as one SM's chain
// of transforms and RK4 points.  Here CTA c owns RT rows of both fields for the row phase and
// 2 RT columns of one field for the column phase, and the planes pass between the phases
// through L2 (1 MB at 256 x 256 FP32), with a grid barrier after each phase:
//
//   row phase     16-point stage from global memory, R2-point stage, RK4(z_s), RK4(z_{s+1}),
//                 R2-point stage, 16-point stage to global memory
//   column phase  R2-point stage from global memory, 16-point stage, propagator, inverse
//                 16-point stage, inverse R2-point stage to global memory
//
// Every transform stage, table entry and RK4 point is the fused march's own code on the same
// operands, so the fields are the same bits.  In global memory position p = n1 + 16 k2 of a row
// sits at n1 * R2 + k2, so that the 16-point stage's lanes (k2) touch consecutive elements.
//
// What bounds it: latency.  A step is two barriers (arrival, the slowest CTA, the poll), two
// L2 round trips and a chain of seven short transform stages and one or two RK4 points per
// thread; the SMs' arithmetic is far from busy.  RT is chosen so that G is near the SM count.
#pragma once

#include "grid_barrier.cuh"
#include "ssfm_multipass.cuh"

namespace shg {

template <typename T, int N, bool THERM>
struct WideCfg {
    static constexpr int R2 = N / 16;
    static constexpr int SW = sizeof(T) == 4 ? 16 : 8;
    static constexpr int RT = N >= 512 ? 4 : N >= 192 ? 2 : 1;  // rows per CTA
    static constexpr int G = N / RT;                            // CTAs per instance
    static constexpr int CW = 2 * RT;                           // columns (of one field) per CTA
    static constexpr int POINTS = RT * N;
    static constexpr bool PACK = !THERM && sizeof(T) == 4;     // two RK4 points per thread at once
    static constexpr int WORK = PACK ? POINTS / 2 : POINTS;
    // Threads and CTAs per SM.  At 512 x 512 one CTA fills an SM's shared memory (thermal), and
    // the 32-point FP64 stage needs 255 registers.  Below, about 170 registers (128 with 256
    // threads) leave room for several CTAs, so that a few instances march side by side.
    static constexpr bool BIG = sizeof(T) == 8 && R2 > 16;
    static constexpr int NT_MAX = N >= 512 && !BIG ? 512 : 256;
    static constexpr int NT = WORK < 64 ? 64 : WORK > NT_MAX ? NT_MAX : WORK;
    static constexpr int MINB = N >= 512 ? 1 : NT >= 192 ? 2 : THERM && NT == 128 ? 4 : 384 / NT;
    // column tile rows are padded by one every 16, so that the 16-point stage's lanes spread
    // over the banks
    static constexpr int TILE = CW * (N + N / 16);
    // Thermal: per point the running Δk prefix (FP64) and the cosines and sines of the slice's
    // three phases, computed once for the two half steps that use them; and, where it fits
    // (not at 512 x 512 FP64), two slices of the per-voxel optics staged ahead by cp.async
    static constexpr size_t THERM_BYTES = THERM ? POINTS * (sizeof(double) + 3 * sizeof(cx<T>)) : 0;
    static constexpr size_t BASE_BYTES = sizeof(mult<T>) * (2 * (size_t)N + CW) + sizeof(cx<T>) * (TILE + 12) +
                                         (PACK ? 6 * sizeof(Rk4Pack) : 0) + THERM_BYTES;
    static constexpr size_t STAGE_BYTES = THERM ? 6 * sizeof(T) * (size_t)POINTS : 0;
    static constexpr bool STAGE = THERM && BASE_BYTES + STAGE_BYTES <= 227 * 1024;
    static constexpr size_t smem_bytes = BASE_BYTES + (STAGE ? STAGE_BYTES : 0);
    static_assert(N % 16 == 0 && G % 2 == 0 && NT % 32 == 0, "bad wide split");
    static_assert(!PACK || R2 % 2 == 0, "packed points go in pairs");
};

// Workspace: barrier counters (zeroed before the launch), then per instance the two planes and
// the rows' power sums.
struct WideWs {
    unsigned* bar;  // [2 * count]: arrivals at the grid barriers, finished CTAs
    char* base;
    size_t stride, off_s, off_part;
    unsigned long long limit_ns;  // bound of each barrier wait
    unsigned withheld;            // arrivals every barrier waits for beyond those there are (self-test; else 0)
};

// SH and pump power an instance reports when one of its barrier waits ran out (powers are sums
// of squares, never negative)
constexpr double kWideTimedOut = -1.0;

// One instance per blockIdx.y, G CTAs each; every CTA of the launch is resident (cooperative).
template <typename T, int N, bool THERM>
__global__ void __launch_bounds__(WideCfg<T, N, THERM>::NT, WideCfg<T, N, THERM>::MINB)
    ssfm_wide_kernel(const InstDesc* __restrict__ descs, WideWs ws) {
    using Cfg = WideCfg<T, N, THERM>;
    constexpr int R2 = Cfg::R2, SW = Cfg::SW, RT = Cfg::RT, CW = Cfg::CW, NT = Cfg::NT, G = Cfg::G;
    constexpr bool PACK = Cfg::PACK;
    using V = cx<T>;
    using W = mult<T>;
    const InstDesc d = descs[blockIdx.y];
    const int nsteps = d.nsteps;
    char* wbase = ws.base + (size_t)blockIdx.y * ws.stride;
    V* gP = reinterpret_cast<V*>(wbase);
    V* gS = reinterpret_cast<V*>(wbase + ws.off_s);
    double* gpart = reinterpret_cast<double*>(wbase + ws.off_part);
    unsigned* bar = ws.bar + 2 * blockIdx.y;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    W* tw = reinterpret_cast<W*>(smem_raw);
    W* py = tw + N;              // y factor of this CTA's column field, by frequency
    W* px = py + N;              // x factor for its columns
    V* buf = reinterpret_cast<V*>(px + CW);  // row phase: P rows, S rows; column phase: the tile
    V* coef = buf + Cfg::TILE;   // [2][6] RK4 stage coefficients by step parity
    double* dkint = reinterpret_cast<double*>(coef + 12);  // thermal: running Δk prefix of this CTA's points
    V* cs3 = reinterpret_cast<V*>(dkint + Cfg::POINTS);   // thermal: [3][POINTS] cosine, sine of the phases
    T* stage = reinterpret_cast<T*>(cs3 + 3 * Cfg::POINTS);  // thermal: [2 slices][np, ns, dk][POINTS]
    Rk4Pack* kpk = reinterpret_cast<Rk4Pack*>(dkint);     // plain FP32: packed constants [2][3]
    V* Ps = buf;
    V* Ss = buf + RT * N;

    const int tid = threadIdx.x, c = blockIdx.x, y0 = c * RT;
    const int cf_field = c >= G / 2;                      // column phase: 0 pump, 1 SH
    const int q0 = (c - (cf_field ? G / 2 : 0)) * CW;     // first stored column
    V* gF = cf_field ? gS : gP;
    auto cj = [](V a) { return mk<T>(a.x, -a.y); };

    for (int j = tid; j < N; j += NT) {
        tw[j] = twiddle<T, N>(j);
        py[j] = prop_y<T, N>(d, cf_field ? d.a_s : d.a_p, j);
    }
    for (int j = tid; j < CW; j += NT) {
        const int q = q0 + j, p = q / R2 + 16 * (q % R2);  // logical position of stored column q
        px[j] = cf_field ? prop_x<T, N>(d, d.a_s, d.b_s, p) : prop_x<T, N>(d, d.a_p, d.b_p, p);
    }
    if (!THERM && tid < 3) {
        stage_coef<T>(d, 0, 0.0, tid, coef);
        if constexpr (PACK) stage_pack(coef, tid, kpk);
    }
    // initial fields: setPump (Efields.h:84-119), SH = 0 or given
    for (int e = tid; e < RT * N; e += NT) {
        const int lr = e / N, x = e % N;
        const size_t g = (size_t)(y0 + lr) * N + x;
        const double2 pv = pump_value(d, x, y0 + lr, d.amp_re, d.amp_im, d.den_re, d.den_im);
        const V p0 = mk<T>((T)pv.x, (T)pv.y);
        const V s0 = d.has_signal_in ? get_field<T>(d, d.signal_in, g) : mk<T>((T)0, (T)0);
        Ps[sidx<N, R2, SW>(lr, x)] = p0;
        Ss[sidx<N, R2, SW>(lr, x)] = s0;
        if (d.slices_p) put_field<T>(d, d.slices_p, g, p0);
        if (d.slices_s) put_field<T>(d, d.slices_s, g, s0);
    }
    __syncthreads();

    const T hap = (T)d.hap, has = (T)d.has, qs = (T)d.qs, dz6 = (T)(d.dz / 6.0);

    // R2-point stage of every (field, row, n1), in place
    auto row_r2 = [&](bool inv) {
        for (int j = tid; j < 2 * RT * 16; j += NT) {
            const int n1 = j & 15, lr = (j >> 4) % RT;
            V* F = j >= RT * 16 ? Ss : Ps;
            V v[R2];
#pragma unroll
            for (int k = 0; k < R2; ++k) v[k] = F[sidx<N, R2, SW>(lr, n1 + 16 * k)];
            r2_stage<T, R2>(v, tw, n1, inv);
#pragma unroll
            for (int k = 0; k < R2; ++k) F[sidx<N, R2, SW>(lr, n1 + 16 * k)] = v[k];
        }
    };
    // thermal: the per-voxel optics of a slice, into its half of the stage (asynchronous)
    const T* opt[3] = {reinterpret_cast<const T*>(d.t_np), reinterpret_cast<const T*>(d.t_ns),
                       reinterpret_cast<const T*>(d.t_dk)};
    auto stage_slice = [&](int sl) {
        if constexpr (Cfg::STAGE) {
            constexpr int PER = 16 / sizeof(T), CH = Cfg::POINTS / PER;  // 16-byte chunks: a CTA's rows are contiguous
            if (sl < nsteps) {
                for (int j = tid; j < 3 * CH; j += NT) {
                    const int a = j / CH, o = (j % CH) * PER;
                    const T* src = (a == 0 ? opt[0] : a == 1 ? opt[1] : opt[2]) + (size_t)sl * N * N + (size_t)y0 * N + o;
                    const unsigned dst = (unsigned)__cvta_generic_to_shared(stage + (size_t)((sl & 1) * 3 + a) * Cfg::POINTS + o);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    // optics a (0 np, 1 ns, 2 dk) of point e in slice sl
    auto optic = [&](int a, int sl, int e) -> T {
        if constexpr (Cfg::STAGE) return stage[((sl & 1) * 3 + a) * Cfg::POINTS + e];
        else return __ldg((a == 0 ? opt[0] : a == 1 ? opt[1] : opt[2]) + (size_t)sl * N * N + (size_t)y0 * N + e);
    };
    // the pointwise work between step s (s = -1: none) and step s + 1
    auto points = [&](int mode, int s) {
        if constexpr (THERM) {
            // boundary_point with the phases' cosines and sines kept from the first half of a
            // step for its second half
            if constexpr (Cfg::STAGE) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncthreads();
            }
            for (int e = tid; e < RT * N; e += NT) {
                const int o = sidx<N, R2, SW>(e / N, e % N);
                const size_t g = (size_t)y0 * N + e;
                V p = Ps[o], q = Ss[o], w[3], cf[6];
                T np = 0, ns = 0, np1 = 0, ns1 = 0, dk1 = 0;
                if (mode != 0) {
                    np = optic(0, s, e);
                    ns = optic(1, s, e);
                }
                if (mode != 2) {
                    np1 = optic(0, s + 1, e);
                    ns1 = optic(1, s + 1, e);
                    dk1 = optic(2, s + 1, e);
                }
                if (mode != 0) {
#pragma unroll
                    for (int j = 0; j < 3; ++j) w[j] = cs3[j * Cfg::POINTS + e];
                    thermal_cf<T>(d, np, ns, w, cf);
                    rk4_point<T>(p, q, cf, hap, has, thermal_qs<T>(d, ns), dz6);
                    if (d.t_q) reinterpret_cast<T*>(d.t_q)[(size_t)s * N * N + g] = thermal_q<T>(d, np, ns, p, q);
                    if (s + 1 < d.nslices) {
                        const size_t gs = (size_t)(s + 1) * N * N + g;
                        if (d.slices_p) put_field<T>(d, d.slices_p, gs, p);
                        if (d.slices_s) put_field<T>(d, d.slices_s, gs, q);
                    }
                    if (s + 1 == d.out_after) {
                        if (d.pump_out) put_field<T>(d, d.pump_out, g, p);
                        if (d.signal_out) put_field<T>(d, d.signal_out, g, q);
                        d.w_out[g] = weighted_abs2<T>((double)ns1, q);
                        d.w_out[(size_t)N * N + g] = weighted_abs2<T>((double)np1, p);
                    }
                }
                if (mode != 2) {
                    const double dk_run = add_r(mode == 0 ? 0.0 : dkint[e], (double)dk1);
                    dkint[e] = dk_run;
                    thermal_phase<T>(d, dk_run, s + 1, w);
#pragma unroll
                    for (int j = 0; j < 3; ++j) cs3[j * Cfg::POINTS + e] = w[j];
                    thermal_cf<T>(d, np1, ns1, w, cf);
                    rk4_point<T>(p, q, cf, hap, has, thermal_qs<T>(d, ns1), dz6);
                    Ps[o] = p;
                    Ss[o] = q;
                }
            }
            if constexpr (Cfg::STAGE) __syncthreads();  // the consumed half is refilled next
            stage_slice(s + 2);
            return;
        }
        const V* cf_prev = coef + 6 * (s & 1);
        const V* cf_next = coef + 6 * ((s + 1) & 1);
        if constexpr (PACK) {
            if (mode == 1 && s + 1 >= d.nslices) {
                const Rk4Pack* kprev = kpk + 3 * (s & 1);
                const Rk4Pack* knext = kpk + 3 * ((s + 1) & 1);
                const float2 nhap = bc2(-hap), nhas = bc2(-has), nqs = bc2(-qs), dzz = bc2(dz6);
                for (int j = tid; j < RT * 16 * (R2 / 2); j += NT) {
                    const int n1 = j & 15, kk = (j >> 4) % (R2 / 2), lr = (j >> 4) / (R2 / 2);
                    const int o0 = sidx<N, R2, SW>(lr, n1 + 32 * kk), o1 = sidx<N, R2, SW>(lr, n1 + 32 * kk + 16);
                    const V p0 = Ps[o0], q0v = Ss[o0], p1 = Ps[o1], q1 = Ss[o1];
                    Cx2 P{make_float2(p0.x, p1.x), make_float2(p0.y, p1.y)};
                    Cx2 S{make_float2(q0v.x, q1.x), make_float2(q0v.y, q1.y)};
                    rk4_pair(P, S, kprev, nhap, nhas, nqs, dzz);
                    rk4_pair(P, S, knext, nhap, nhas, nqs, dzz);
                    Ps[o0] = make_float2(P.r.x, P.i.x);
                    Ps[o1] = make_float2(P.r.y, P.i.y);
                    Ss[o0] = make_float2(S.r.x, S.i.x);
                    Ss[o1] = make_float2(S.r.y, S.i.y);
                }
                return;
            }
        }
        for (int e = tid; e < RT * N; e += NT) {
            const int lr = e / N, x = e % N, o = sidx<N, R2, SW>(lr, x);
            const size_t g = (size_t)(y0 + lr) * N + x;
            V p = Ps[o], q = Ss[o];
            const ThermPre<T> pre = thermal_pre<T, false>(d, mode, s, g, (size_t)N * N, nullptr);
            boundary_point<T, false>(d, mode, s, g, (size_t)N * N, p, q, cf_prev, cf_next, hap, has, qs, dz6, nullptr,
                                     pre);
            Ps[o] = p;
            Ss[o] = q;
        }
    };
    // forward row transform of the rows in shared memory, out to global memory
    auto rows_out = [&]() {
        __syncthreads();
        row_r2(false);
        __syncthreads();
        for (int j = tid; j < 2 * RT * R2; j += NT) {
            const int k2 = j % R2, lr = (j / R2) % RT;
            const bool f = j >= RT * R2;
            const V* F = f ? Ss : Ps;
            V* row = (f ? gS : gP) + (size_t)(y0 + lr) * N;
            V u[16];
#pragma unroll
            for (int n = 0; n < 16; ++n) u[n] = F[sidx<N, R2, SW>(lr, n + 16 * k2)];
            Dft<16, -1, T>::run(u);
#pragma unroll
            for (int n = 0; n < 16; ++n) __stcg(row + n * R2 + k2, u[n]);
        }
    };
    // inverse row transform from global memory
    auto rows_in = [&]() {
        for (int j = tid; j < 2 * RT * R2; j += NT) {
            const int k2 = j % R2, lr = (j / R2) % RT;
            const bool f = j >= RT * R2;
            V* F = f ? Ss : Ps;
            const V* row = (f ? gS : gP) + (size_t)(y0 + lr) * N;
            V u[16];
#pragma unroll
            for (int n = 0; n < 16; ++n) u[n] = cj(__ldcg(row + n * R2 + k2));
            Dft<16, -1, T>::run(u);
#pragma unroll
            for (int n = 0; n < 16; ++n) F[sidx<N, R2, SW>(lr, n + 16 * k2)] = cj(u[n]);
        }
        __syncthreads();
        row_r2(true);
        __syncthreads();
    };
    // diffraction of this CTA's columns
    auto columns = [&]() {
        for (int j = tid; j < CW * 16; j += NT) {
            const int cc = j % CW, n1 = j / CW;
            V v[R2];
#pragma unroll
            for (int k = 0; k < R2; ++k) v[k] = __ldcg(gF + (size_t)(n1 + 16 * k) * N + q0 + cc);
            r2_stage<T, R2>(v, tw, n1, false);
#pragma unroll
            for (int k = 0; k < R2; ++k) buf[(n1 + 17 * k) * CW + cc] = v[k];
        }
        __syncthreads();
        for (int j = tid; j < CW * R2; j += NT) {
            const int cc = j % CW, k2 = j / CW;
            V u[16];
#pragma unroll
            for (int n = 0; n < 16; ++n) u[n] = buf[(n + 17 * k2) * CW + cc];
#pragma unroll 1
            for (int it = 0; it < 2; ++it) {
                if (it) {
#pragma unroll
                    for (int n = 0; n < 16; ++n) u[n] = cj(u[n]);
                }
                Dft<16, -1, T>::run(u);
                if (!it) {
#pragma unroll
                    for (int k1 = 0; k1 < 16; ++k1) u[k1] = mulw(mulw(u[k1], py[k2 + R2 * k1]), px[cc]);
                } else {
#pragma unroll
                    for (int n = 0; n < 16; ++n) u[n] = cj(u[n]);
                }
            }
#pragma unroll
            for (int n = 0; n < 16; ++n) buf[(n + 17 * k2) * CW + cc] = u[n];
        }
        __syncthreads();
        for (int j = tid; j < CW * 16; j += NT) {
            const int cc = j % CW, n1 = j / CW;
            V v[R2];
#pragma unroll
            for (int k = 0; k < R2; ++k) v[k] = buf[(n1 + 17 * k) * CW + cc];
            r2_stage<T, R2>(v, tw, n1, true);
#pragma unroll
            for (int k = 0; k < R2; ++k) __stcg(gF + (size_t)(n1 + 16 * k) * N + q0 + cc, v[k]);
        }
    };

    if constexpr (THERM) stage_slice(0);
    points(0, -1);
    rows_out();
    unsigned target = ws.withheld;
    double z = 0.0;
    bool ok = true;
    for (int s = 0; s < nsteps; ++s) {
        if (!(ok = grid_barrier(bar, target += G, ws.limit_ns))) break;
        columns();
        if (!THERM && s + 1 < nsteps && tid >= NT - 3) {
            // the next step's stage coefficients, by threads of the last warp
            const int j = tid - (NT - 3);
            stage_coef<T>(d, s + 1, add_r(z, d.dz), j, coef + 6 * ((s + 1) & 1));
            if constexpr (PACK) stage_pack(coef + 6 * ((s + 1) & 1), j, kpk + 3 * ((s + 1) & 1));
        }
        if (!(ok = grid_barrier(bar, target += G, ws.limit_ns))) break;
        const bool more = s + 1 < nsteps;
        rows_in();
        points(more ? 1 : 2, s);
        if (more) rows_out();
        z = add_r(z, d.dz);
    }
    if (!ok) {
        if (tid == 0 && d.power_out) {
            d.power_out[0] = kWideTimedOut;
            d.power_out[1] = kWideTimedOut;
        }
        return;
    }
    if constexpr (THERM) return;  // its powers are summed from w_out
    // SH and pump power: this CTA's row sums, then the last CTA to finish adds the rows
    const int warp = tid >> 5, lane = tid & 31;
    __syncthreads();
    for (int r = warp; r < 2 * RT; r += NT / 32) {
        const double a = row_abs2<T, N>(r < RT ? Ss : Ps, r % RT, lane);
        if (lane == 0) __stcg(gpart + (r < RT ? 0 : N) + y0 + r % RT, a);
    }
    __shared__ unsigned s_done;
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_done = atomicAdd(bar + 1, 1u);
        __threadfence();
    }
    __syncthreads();
    if (s_done != G - 1 || warp != 0 || !d.power_out) return;
    for (int f = 0; f < 2; ++f) {
        const double a = sum_rows<N>([&](int y) { return __ldcg(gpart + f * N + y); }, lane);
        if (lane == 0) d.power_out[f] = a * (f ? d.pw_p : d.pw_s);
    }
}

}  // namespace shg
