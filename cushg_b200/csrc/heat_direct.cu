// heat_direct.cu — the steady temperature of the heat equation that the reference's Jacobi
// sweeps converge to (kernelHeatEquationTopOpen / OvenSurrounded, src/headers/Tfield.h:93-240;
// the loop Solver.h:339-355), computed directly instead of one sweep at a time.  No counterpart
// in the reference.
//
// The linear system.  Every update of Tfield.h:93-240 is one row of A T = b once the row is
// multiplied by its own scale: inner points by 1/L2 (Tfield.h:113-115), faces by 2/d^2 of their
// normal direction (Tfield.h:119-137, 229-236), edges by 4/(d_a d_b) (Tfield.h:143-177) and
// vertices by 2/(dx dy dz) (Tfield.h:181-196).  In that form every row is the sum of three
// one-dimensional parts, one per direction, each of which is
//   (2 u_i - u_{i-1} - u_{i+1}) / d^2                  inside the direction,
//   (2 (1 + Bi) u_0 - 2 u_1) / d^2  (right-hand 2 Bi T_inf / d^2)   at a Robin face,
//   and, next to a Dirichlet voxel g, the inside form with g moved to the right-hand side,
// plus Q / kappa on inner points only.  (The face, edge and vertex coefficients ax .. GV of
// the reference reduce exactly to these: e.g. the vertical edge's 0.5 (Bix + Biz) times
// 4/(dx dz) is 2 Bix / dx^2 + 2 Biz / dz^2.)  So A = Ax (+) Ay (+) Az, a Kronecker sum.
//
// The solve.  Two of the three operators are diagonalised by dense transforms (F = V^T S forward,
// G = S^{-1} V back, of the symmetric form S M S^{-1} = V diag(lambda) V^T) and the third direction
// is solved by elimination.  x is always transformed.  Of y and z the cheaper one is (axis_of):
// a direction with the same kind of end at both sides has modes of exact parity, and its
// transform folds into two of half the size, so z (Robin at both ends) costs nz / 2 products
// per point against ny for TOP_OPEN's y (Dirichlet and Robin).  With t the transformed one of the
// two and s the other:
//   1. b (FP64) from Q, the Dirichlet voxels and T_inf, folded               rhs_kernel
//   2. b <- b Fx^T (along x), then Ft b (along t)                            dgemm_kernel
//   3. for every mode (kt, kx): (As + lambda_x + lambda_t) v = b along s     thomas_kernel
//   4. v <- Gt v, then v Gx^T; unfolded                                      dgemm_kernel, unfold_kernel
//   5. T <- v, with the FP64 residual of one Jacobi sweep of v and the change  finish_kernel
// The x and y modes come from the host (implicit QL, once per operator and device), the z modes
// from their closed form on the device in every solve (z_modes_kernel, microseconds).
// Unknowns: TOP_OPEN, x 0..n-1 (Robin both ends), y 1..n-1 (y = 0 Dirichlet, Robin at n-1),
// z 0..nz-1 (Robin); OVEN_SURROUNDED, x and y 1..n-2 (Dirichlet both ends), z as above.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "jacobi_point.cuh"
#include "shg_host.h"
#include "thermal.h"

namespace shg {

namespace {

// One direction's operator: m unknowns at spacing d, each end Robin (with Biot number bi) or
// next to a Dirichlet voxel.
struct Op1D {
    int m = 0;
    double d = 0.0;
    int lo_robin = 0, hi_robin = 0;
    double bi = 0.0;
    bool operator==(const Op1D& o) const {
        return m == o.m && d == o.d && lo_robin == o.lo_robin && hi_robin == o.hi_robin && bi == o.bi;
    }
};

// Rows of the scaled operator: diagonal a, below-diagonal l (l[0] unused), above-diagonal r
// (r[m-1] unused).
void op_rows(const Op1D& op, std::vector<double>& a, std::vector<double>& l, std::vector<double>& r) {
    const int m = op.m;
    const double i2 = 1.0 / (op.d * op.d);
    a.assign(m, 2.0 * i2);
    l.assign(m, -i2);
    r.assign(m, -i2);
    l[0] = 0.0;
    r[m - 1] = 0.0;
    if (op.lo_robin) {
        a[0] = 2.0 * (1.0 + op.bi) * i2;
        if (m > 1) r[0] = -2.0 * i2;
    }
    if (op.hi_robin) {
        a[m - 1] = 2.0 * (1.0 + op.bi) * i2;
        if (m > 1) l[m - 1] = -2.0 * i2;
    }
}

// Eigenvalues and eigenvectors of the symmetric tridiagonal matrix with diagonal d[0..m) and
// off-diagonal e[0..m-1) (e[i] couples i and i+1): implicit QL iterations with Wilkinson
// shifts (Bowdler, Martin, Reinsch and Wilkinson, Numer. Math. 11, 293-306 (1968)).  On
// return d holds the eigenvalues and z (column-major: vector k is z[k*m .. k*m+m)) the
// orthonormal eigenvectors.  False if an eigenvalue took more than 64 iterations.
bool tridiag_eigen(int m, std::vector<double>& d, std::vector<double> e, std::vector<double>& z) {
    z.assign((size_t)m * m, 0.0);
    for (int k = 0; k < m; ++k) z[(size_t)k * m + k] = 1.0;
    e.resize(m);
    e[m - 1] = 0.0;
    for (int l = 0; l < m; ++l) {
        for (int iter = 0;; ++iter) {
            int j = l;
            for (; j < m - 1; ++j)  // first negligible off-diagonal at or after l
                if (std::fabs(e[j]) <= DBL_EPSILON * (std::fabs(d[j]) + std::fabs(d[j + 1]))) break;
            if (j == l) break;  // d[l] converged
            if (iter >= 64) return false;
            // shift: the eigenvalue of the leading 2x2 block nearer to d[l]
            double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
            double r = std::hypot(g, 1.0);
            g = d[j] - d[l] + e[l] / (g + std::copysign(r, g));
            double s = 1.0, c = 1.0, p = 0.0;
            bool split = false;
            for (int i = j - 1; i >= l; --i) {  // chase the bulge from the bottom of the block up
                const double f = s * e[i], b = c * e[i];
                r = std::hypot(f, g);
                e[i + 1] = r;
                if (r == 0.0) {  // the block split: restart on the smaller one
                    d[i + 1] -= p;
                    e[j] = 0.0;
                    split = true;
                    break;
                }
                s = f / r;
                c = g / r;
                g = d[i + 1] - p;
                r = (d[i] - g) * s + 2.0 * c * b;
                p = s * r;
                d[i + 1] = g + p;
                g = c * r - b;
                double* zi = &z[(size_t)i * m];
                double* zj = &z[(size_t)(i + 1) * m];
                for (int k = 0; k < m; ++k) {
                    const double t = zj[k];
                    zj[k] = s * zi[k] + c * t;
                    zi[k] = c * zi[k] - s * t;
                }
            }
            if (split) continue;
            d[l] -= p;
            e[l] = g;
            e[j] = 0.0;
        }
    }
    return true;
}

// Eigenvalues, forward transform F (row k: mode k) and inverse G (row i: point i) of one
// operator, all row-major m x m.  The operator M is similar to the symmetric B = S M S^{-1}
// with S = diag(s), s[i+1] = s[i] sqrt(r[i] / l[i+1]); B = V diag(lambda) V^T gives
// F = V^T S and G = S^{-1} V.
// An operator with the same kind of end at both sides and m even is symmetric under
// i -> m-1-i (B and S alike), and B splits into an even and an odd block of half size: for
// v = (w, +-J w) / sqrt(2) (J the reversal), B v = lambda v exactly when w is an eigenvector of
// the leading h x h block of B with its last diagonal entry d[h-1] +- e[h-1].  The modes are
// then built from the blocks' eigenvectors, even modes first (k < h), so that their parity is
// exact, which the folded transforms rely on; and the QL work is a quarter.
bool op_modes(const Op1D& op, std::vector<double>& lam, std::vector<double>& F, std::vector<double>& G) {
    const int m = op.m;
    std::vector<double> a, l, r;
    op_rows(op, a, l, r);
    std::vector<double> s(m, 1.0), e(m, 0.0);
    for (int i = 0; i + 1 < m; ++i) {
        s[i + 1] = s[i] * std::sqrt(r[i] / l[i + 1]);
        e[i] = -std::sqrt(r[i] * l[i + 1]);
    }
    std::vector<double> V;  // column-major: vector k at V[k*m .. k*m+m)
    if (op.lo_robin == op.hi_robin && m % 2 == 0 && m >= 2) {
        const int h = m / 2;
        V.assign((size_t)m * m, 0.0);
        lam.assign(m, 0.0);
        const double r2 = 1.0 / std::sqrt(2.0);
        for (int par = 0; par < 2; ++par) {  // 0: even, 1: odd
            std::vector<double> d(a.begin(), a.begin() + h), eh(e.begin(), e.begin() + h), W;
            d[h - 1] += par == 0 ? e[h - 1] : -e[h - 1];
            eh[h - 1] = 0.0;
            if (!tridiag_eigen(h, d, eh, W)) return false;
            for (int q = 0; q < h; ++q) {
                const int k = par * h + q;
                lam[k] = d[q];
                for (int i = 0; i < h; ++i) {
                    const double w = W[(size_t)q * h + i] * r2;
                    V[(size_t)k * m + i] = w;
                    V[(size_t)k * m + (m - 1 - i)] = par == 0 ? w : -w;
                }
            }
        }
    } else {
        lam = a;
        if (!tridiag_eigen(m, lam, e, V)) return false;
    }
    F.assign((size_t)m * m, 0.0);
    G.assign((size_t)m * m, 0.0);
    for (int k = 0; k < m; ++k)
        for (int i = 0; i < m; ++i) {
            const double v = V[(size_t)k * m + i];  // component i of eigenvector k
            F[(size_t)k * m + i] = v * s[i];
            G[(size_t)i * m + k] = v / s[i];
        }
    return true;
}

// Device copies of one operator's transforms: F and G row-major, their transposes, lambda.  The
// matrices' rows are ld = m rounded up to even doubles (zero-padded), so that every row starts
// on 16 bytes for the GEMM's copies.
struct OpMats {
    Op1D op;
    int dev = -1;
    int ld = 0;
    double *F = nullptr, *G = nullptr, *FT = nullptr, *GT = nullptr, *lam = nullptr;
    // Folded form, for an operator symmetric under i -> m-1-i (the same kind at both ends) with
    // m a multiple of 4: its modes are even or odd, so with s_i = b_i + b_{m-1-i} and
    // d_i = b_i - b_{m-1-i} (i < h = m/2) the even amplitudes are FeT-products of s and the odd
    // ones FoT-products of d, and back, P = GeT-products and Q = GoT-products give
    // u_i = P_i + Q_i, u_{m-1-i} = P_i - Q_i.  Half matrices h x h, row-major (ld = h, even),
    // laid out for C = A B like FT and GT; lamf the eigenvalues, even modes first.
    bool fold = false;
    double *FeT = nullptr, *FoT = nullptr, *GeT = nullptr, *GoT = nullptr, *lamf = nullptr;
    // The same halves as left factors (rows modes for F, rows points for G), for a symmetric
    // operator with m even, as the y direction of OVEN_SURROUNDED has; rows of ldl = h rounded up
    // to even doubles.
    bool fold_left = false;
    int ldl = 0;
    double *Fe = nullptr, *Fo = nullptr, *Ge = nullptr, *Go = nullptr;
};

// Process-wide cache of operator transforms, per device (an operator's eigendecomposition
// costs O(m^3) on the host: about 0.3 s at m = 512).
std::mutex g_ops_mu;
std::vector<OpMats*> g_ops;
constexpr size_t kMaxCachedOps = 64;

shg_status get_op(const Op1D& op, const OpMats** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    std::lock_guard<std::mutex> lk(g_ops_mu);
    for (const OpMats* c : g_ops)
        if (c->dev == dev && c->op == op) {
            *out = c;
            return SHG_OK;
        }
    std::vector<double> lam, F, G;
    if (!op_modes(op, lam, F, G)) return fail(SHG_ERR_NOT_CONVERGED, "heat operator eigendecomposition (m = %d)", op.m);
    const int m = op.m, ld = m + (m & 1);
    const size_t mm = (size_t)m * ld;
    std::vector<double> Fp(mm, 0.0), Gp(mm, 0.0), FT(mm, 0.0), GT(mm, 0.0);
    for (int i = 0; i < m; ++i)
        for (int k = 0; k < m; ++k) {
            Fp[(size_t)k * ld + i] = F[(size_t)k * m + i];
            Gp[(size_t)i * ld + k] = G[(size_t)i * m + k];
            FT[(size_t)i * ld + k] = F[(size_t)k * m + i];
            GT[(size_t)k * ld + i] = G[(size_t)i * m + k];
        }
    // the folded form (op_modes gives a symmetric operator's even modes first, then its odd
    // ones, each of exact parity); m a multiple of 4 keeps the half rows 16-byte aligned
    const int h = m / 2;
    const bool fold = op.lo_robin == op.hi_robin && m % 4 == 0;
    const size_t hh = fold ? (size_t)h * h : 0;
    std::vector<double> FeT(hh), FoT(hh), GeT(hh), GoT(hh), lamf(fold ? m : 0);
    for (int a = 0; fold && a < h; ++a) {
        const int ke = a, ko = h + a;
        lamf[a] = lam[ke];
        lamf[h + a] = lam[ko];
        for (int i = 0; i < h; ++i) {
            FeT[(size_t)i * h + a] = F[(size_t)ke * m + i];  // B operand: rows i, columns modes
            FoT[(size_t)i * h + a] = F[(size_t)ko * m + i];
            GeT[(size_t)a * h + i] = G[(size_t)i * m + ke];  // B operand: rows modes, columns i
            GoT[(size_t)a * h + i] = G[(size_t)i * m + ko];
        }
    }
    const bool fold_left = op.lo_robin == op.hi_robin && m % 2 == 0;
    const int ldl = h + (h & 1);
    const size_t hl = fold_left ? (size_t)h * ldl : 0;
    std::vector<double> Fe(hl, 0.0), Fo(hl, 0.0), Ge(hl, 0.0), Go(hl, 0.0);
    for (int a = 0; fold_left && a < h; ++a)
        for (int i = 0; i < h; ++i) {
            Fe[(size_t)a * ldl + i] = F[(size_t)a * m + i];
            Fo[(size_t)a * ldl + i] = F[(size_t)(h + a) * m + i];
            Ge[(size_t)i * ldl + a] = G[(size_t)i * m + a];
            Go[(size_t)i * ldl + a] = G[(size_t)i * m + h + a];
        }
    if (g_ops.size() >= kMaxCachedOps) return fail(SHG_ERR_UNSUPPORTED, "more than %d heat operators cached", (int)kMaxCachedOps);
    double* buf = nullptr;
    if ((e = cudaMalloc((void**)&buf, sizeof(double) * (4 * mm + (m + (m & 1)) + 4 * hh + lamf.size() + 4 * hl))) != cudaSuccess)
        return cuda_fail(e, "cudaMalloc");
    OpMats* c = new OpMats;
    c->op = op;
    c->dev = dev;
    c->ld = ld;
    c->F = buf;
    c->G = buf + mm;
    c->FT = buf + 2 * mm;
    c->GT = buf + 3 * mm;
    c->lam = buf + 4 * mm;
    c->fold = fold;
    double* fb = c->lam + (m + (m & 1));  // 16-byte aligned (4 mm and the padded m are even)
    if (fold) {
        c->FeT = fb;
        c->FoT = fb + hh;
        c->GeT = fb + 2 * hh;
        c->GoT = fb + 3 * hh;
        c->lamf = fb + 4 * hh;
    }
    c->fold_left = fold_left;
    c->ldl = ldl;
    if (fold_left) {
        c->Fe = fb + 4 * hh + lamf.size();  // even offsets: 4 hh, and m with the fold
        c->Fo = c->Fe + hl;
        c->Ge = c->Fe + 2 * hl;
        c->Go = c->Fe + 3 * hl;
    }
    const double* src[14] = {Fp.data(),  Gp.data(),  FT.data(),   GT.data(), lam.data(), FeT.data(), FoT.data(),
                             GeT.data(), GoT.data(), lamf.data(), Fe.data(), Fo.data(),  Ge.data(),  Go.data()};
    double* dst[14] = {c->F,   c->G,   c->FT,  c->GT, c->lam, c->FeT, c->FoT,
                       c->GeT, c->GoT, c->lamf, c->Fe, c->Fo,  c->Ge,  c->Go};
    const size_t cnt[14] = {mm, mm, mm, mm, (size_t)m, hh, hh, hh, hh, lamf.size(), hl, hl, hl, hl};
    for (int k = 0; k < 14 && e == cudaSuccess; ++k)
        if (cnt[k]) e = cudaMemcpy(dst[k], src[k], sizeof(double) * cnt[k], cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(buf);
        delete c;
        return cuda_fail(e, "heat operator upload");
    }
    g_ops.push_back(c);
    *out = c;
    return SHG_OK;
}

// The grid's three directions: unknown ranges and operators.
struct HeatGrid {
    int n = 0, nz = 0;
    int x0 = 0, y0 = 0, mx = 0, my = 0;  // first unknown and count along x and y
    Op1D ox, oy;
    double dx = 0, dy = 0, dz = 0, biz = 0;
};

HeatGrid heat_grid(const shg_params& p) {
    HeatGrid g;
    g.n = p.nx;
    g.nz = p.nz;
    g.dx = p.lx / (p.nx - 1);
    g.dy = p.ly / (p.ny - 1);
    g.dz = p.lz / (p.nz - 1);
    const double bix = p.h_conv * g.dx / p.kappa, biy = p.h_conv * g.dy / p.kappa;
    g.biz = p.h_conv * g.dz / p.kappa;
    if (p.boundary == SHG_BOUNDARY_TOP_OPEN) {
        g.x0 = 0;
        g.mx = g.n;
        g.ox = {g.mx, g.dx, 1, 1, bix};
        g.y0 = 1;
        g.my = g.n - 1;
        g.oy = {g.my, g.dy, 0, 1, biy};
    } else {
        g.x0 = g.y0 = 1;
        g.mx = g.my = g.n - 2;
        g.ox = {g.mx, g.dx, 0, 0, bix};
        g.oy = {g.my, g.dy, 0, 0, biy};
    }
    return g;
}

// What the kernels need of the grid and the model, in FP64.
struct HeatArgs {
    int n, nz, x0, y0, mx, my;
    int lo_x_robin, hi_x_robin, lo_y_robin, hi_y_robin;
    double idx2, idy2, idz2, iK, tinf, bix, biy, biz;
};

// Compact volume index c = (z * my + j) * mx + i of unknown (x0 + i, y0 + j, z).
// 1. Right-hand side of the scaled system: Q / kappa on inner points, 2 Bi T_inf / d^2 at each
//    Robin end, g / d^2 for each Dirichlet neighbour g (read from T).
template <typename R>
__device__ __forceinline__ double rhs_value(const R* __restrict__ T, const R* __restrict__ Q, const HeatArgs& a, int i,
                                            int j, int z) {
    const size_t nn = (size_t)a.n;
    const int x = a.x0 + i, y = a.y0 + j;
    const size_t v = ((size_t)z * nn + y) * nn + x;
    double s = 0.0;
    if (Q && x > 0 && x < a.n - 1 && y > 0 && y < a.n - 1 && z > 0 && z < a.nz - 1) s = (double)Q[v] * a.iK;
    if (i == 0) s += a.lo_x_robin ? 2.0 * a.bix * a.tinf * a.idx2 : (double)T[v - 1] * a.idx2;
    if (i == a.mx - 1) s += a.hi_x_robin ? 2.0 * a.bix * a.tinf * a.idx2 : (double)T[v + 1] * a.idx2;
    if (j == 0) s += a.lo_y_robin ? 2.0 * a.biy * a.tinf * a.idy2 : (double)T[v - nn] * a.idy2;
    if (j == a.my - 1) s += a.hi_y_robin ? 2.0 * a.biy * a.tinf * a.idy2 : (double)T[v + nn] * a.idy2;
    if (z == 0) s += 2.0 * a.biz * a.tinf * a.idz2;
    if (z == a.nz - 1) s += 2.0 * a.biz * a.tinf * a.idz2;
    return s;
}

// Which directions the transforms fold: fx the x direction, ft the other transformed one (0 none,
// 1 y, 2 z); wx, wy, wz the half counts along the folded directions.  A folded direction of m
// points holds the sums v_q + v_{m-1-q} (the middle point alone where m is odd) in its first
// ceil(m/2) places and the differences v_q - v_{m-1-q} in the others.
struct Fold {
    int fx, ft, wx, wy, wz;
};
struct FoldItem {
    int i, j, z;    // the item's point
    int j2, z2;     // its mirror image along the folded y or z (equal: none, or the middle)
    int jd, zd;     // where the differences go
    bool pair;
};
__device__ __forceinline__ FoldItem fold_item(const Fold& f, const HeatArgs& a, size_t c) {
    FoldItem t;
    t.i = (int)(c % f.wx);
    const size_t r = c / f.wx;
    t.j = (int)(r % f.wy);
    t.z = (int)(r / f.wy);
    t.j2 = f.ft == 1 ? a.my - 1 - t.j : t.j;
    t.z2 = f.ft == 2 ? a.nz - 1 - t.z : t.z;
    t.jd = f.ft == 1 ? f.wy + t.j : t.j;
    t.zd = f.ft == 2 ? f.wz + t.z : t.z;
    t.pair = t.j2 != t.j || t.z2 != t.z;
    return t;
}

template <typename R, bool FX>
__global__ void rhs_kernel(const R* __restrict__ T, const R* __restrict__ Q, double* __restrict__ b, const HeatArgs a,
                           const Fold f) {
    const size_t total = (size_t)f.wx * f.wy * f.wz;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < total; c += (size_t)gridDim.x * blockDim.x) {
        const FoldItem t = fold_item(f, a, c);
        auto put = [&](int j, int z, double v0, double v1) {  // a row's entries of points i and mx-1-i
            double* row = b + ((size_t)z * a.my + j) * a.mx;
            row[t.i] = FX ? v0 + v1 : v0;
            if (FX) row[f.wx + t.i] = v0 - v1;
        };
        const double e0 = rhs_value<R>(T, Q, a, t.i, t.j, t.z);
        const double e1 = FX ? rhs_value<R>(T, Q, a, a.mx - 1 - t.i, t.j, t.z) : 0.0;
        if (t.pair) {
            const double m0 = rhs_value<R>(T, Q, a, t.i, t.j2, t.z2);
            const double m1 = FX ? rhs_value<R>(T, Q, a, a.mx - 1 - t.i, t.j2, t.z2) : 0.0;
            put(t.j, t.z, e0 + m0, e1 + m1);
            put(t.jd, t.zd, e0 - m0, e1 - m1);
        } else {
            put(t.j, t.z, e0, e1);
        }
    }
}

// The modes of the z operator (m = nz points, Robin at both ends with Biot number bi), one block
// per mode.  With c = (m-1)/2 the eigenvectors are v_i = cos(theta (i-c)) (even) and
// sin(theta (i-c)) (odd), eigenvalue 4 sin^2(theta/2) / dz^2; the end rows give
//   sin(theta) tan(e) = bi,  theta c = k pi + e (even, k = 0..) or (k + 1/2) pi + e (odd),
// with 0 <= e < pi/2, except for the mode with theta = pi at bi = 0, which becomes
// v_i = (-1)^i cosh(eta (i-c)), sinh(eta) tanh(eta c) = bi, eigenvalue 4 cosh^2(eta/2) / dz^2.
// The phase k pi (i-c)/c is reduced in integers, so the entries are good to rounding.  In the
// weights s_i^2 = 1, 2, .., 2, 1 of the symmetric form, F[k][i] = s_i^2 v_i / |v| and
// G[i][k] = v_i / |v| with |v|^2 = sum s_i^2 v_i^2.  Even modes first; halves as in OpMats.
__global__ void __launch_bounds__(128) z_modes_kernel(int m, double bi, double idz2, double* __restrict__ lam,
                                                      double* __restrict__ Fe, double* __restrict__ Fo,
                                                      double* __restrict__ Ge, double* __restrict__ Go, int lde, int ldo) {
    const int he = (m + 1) / 2, mode = blockIdx.x, odd = mode >= he, k = odd ? mode - he : mode;
    const int h = odd ? m / 2 : he;                  // points of the half
    const bool top = mode == (m & 1 ? he - 1 : m - 1);  // the last mode of the parity that holds (-1)^i
    const double c = 0.5 * (m - 1), half_pi = 1.57079632679489661923, pi = 3.14159265358979323846;
    // root of an increasing function on (lo, hi) by Newton steps kept inside the bracket
    double root, lo = 0.0, hi;
    if (top) {
        hi = 2.0 * (asinh(bi) + sqrt(bi / c));  // above the root
        root = bi > 0.0 ? fmin(hi, fmax(asinh(bi), sqrt(bi / c))) : 0.0;
    } else {
        hi = half_pi;
        const double th0 = (k + 0.5 * odd) * pi / c;
        root = th0 > 0.0 ? atan(bi / sin(th0)) : fmin(sqrt(bi * c), 1.5);
    }
    for (int it = 0; it < 80 && bi > 0.0; ++it) {
        double g, dg;
        if (top) {
            const double t = tanh(root * c);
            g = sinh(root) * t - bi;
            dg = cosh(root) * t + sinh(root) * c * (1.0 - t * t);
        } else {
            double sn, cs, se, ce;
            sincos(((k + 0.5 * odd) * pi + root) / c, &sn, &cs);
            sincos(root, &se, &ce);
            g = sn * se - bi * ce;
            dg = cs * se / c + sn * ce + bi * se;
        }
        if (g > 0.0) hi = root;
        else lo = root;
        double next = dg > 0.0 ? root - g / dg : 0.5 * (lo + hi);
        if (!(next >= lo && next <= hi)) next = 0.5 * (lo + hi);
        const double step = fabs(next - root);
        root = next;
        if (step <= 2e-16 * root) break;
    }
    const int n1 = m - 1;
    auto value = [&](int i) -> double {  // v_i
        const int r = 2 * i - n1;        // (i - c) / c = r / n1
        if (top) {
            const double x = fabs(0.5 * r) * root;  // eta |i - c|; cosh over cosh(eta c), no overflow
            const double v = exp(x - root * c) * (1.0 + exp(-2.0 * x)) / (1.0 + exp(-2.0 * root * c));
            return (i & 1) ? -v : v;
        }
        const long long q = ((long long)(2 * k + odd) * r) % (4ll * n1);  // phase = pi q / (2 n1) + e r / n1
        const double ph = (double)q / (2.0 * n1) + root / pi * ((double)r / n1);
        return odd ? sinpi(ph) : cospi(ph);
    };
    double sum = 0.0;
    for (int i = threadIdx.x; i < m; i += 128) {
        const double v = value(i);
        sum += (i == 0 || i == n1 ? 1.0 : 2.0) * v * v;
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    __shared__ double part[4];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    const double nrm = 1.0 / sqrt(part[0] + part[1] + part[2] + part[3]);
    double* F = odd ? Fo : Fe;
    double* G = odd ? Go : Ge;
    const int ld = odd ? ldo : lde;
    for (int i = threadIdx.x; i < ld; i += 128) {
        const double v = i < h ? value(i) * nrm : 0.0;  // zero in the row's padding
        F[(size_t)k * ld + i] = (i == 0 || i == n1 ? 1.0 : 2.0) * v;
        if (i < h) G[(size_t)i * ld + k] = v;
    }
    if (k == h - 1 && ld > h)  // and the padding column of G
        for (int i = threadIdx.x; i < h; i += 128) G[(size_t)i * ld + h] = 0.0;
    if (threadIdx.x == 0) {
        const double q = top ? cosh(0.5 * root) : sin(0.5 * ((k + 0.5 * odd) * pi + root) / c);
        lam[mode] = 4.0 * q * q * idz2;
    }
}

// A block computes a BM x BN tile of C with WR x WC warps, each a 16 MI x 8 NJ part of it as
// MI x NJ FP64 tensor-core products (mma.sync m16n8k4); k runs in 32-wide slices through a
// three-stage ring of cp.async copies.  Row pitches: A slices 36 doubles, B slices BN + 4, so
// that the fragment reads of a half-warp (4 rows x 4 columns of A, 4 rows x 4 columns of B)
// fall in 16 different 8-byte bank pairs; every row starts on 16 bytes.
//   128 x 128 (eight 64 x 32 warps) has the fewest shared-memory reads per product and runs the
// FP64 pipe at 82-85 % of its peak, but leaves the device idle where it cuts a product into few
// tiles: 96 x 96 x 37 has 28, of 25 k cycles each.  32 x 32 (four 16 x 16 warps) and 64 x 64 (four
// 32 x 32 warps) are for those (gemm picks).
template <int MI_, int NJ_, int WR_, int WC_, int MINB_>
struct GemmCfg {
    static constexpr int MI = MI_, NJ = NJ_, WR = WR_, WC = WC_, MINB = MINB_;
    static constexpr int BM = 16 * MI * WR, BN = 8 * NJ * WC, BK = 32, THREADS = 32 * WR * WC, STAGES = 3;
    static constexpr int ALD = BK + 4, BLD = BN + 4;
    static constexpr int STAGE = BM * ALD + BK * BLD;  // doubles
    static constexpr size_t SMEM = sizeof(double) * STAGE * STAGES;
};
using GemmBig = GemmCfg<4, 4, 2, 4, 1>;    // 128 x 128, 207 KB
using GemmMid = GemmCfg<2, 4, 2, 2, 2>;    // 64 x 64, 107 KB
using GemmSmall = GemmCfg<1, 2, 2, 2, 4>;  // 32 x 32, 54 KB

// 16 bytes from global to shared memory, asynchronously; the bytes past `valid` (0..16) are
// zero-filled and not read.
__device__ __forceinline__ void cp_async16(double* dst, const double* src, int valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid) : "memory");
}

// c += A B for one 16 x 8 x 4 FP64 product held in the fragments of mma.sync m16n8k4: with
// g = lane / 4 and t = lane % 4, a0 = A[g][t], a1 = A[g + 8][t], b = B[t][g], and c = C[g][2t],
// C[g][2t + 1], C[g + 8][2t], C[g + 8][2t + 1].
__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a0), "d"(a1), "d"(b));
}

// 2, 4. C[b] = A[b] B[b] in FP64 for row-major A (M x K, lda), B (K x N, ldb) and C (M x N, ldc),
// batch b = blockIdx.z at element strides sA, sB, sC.  lda, ldb, ldc, the strides and the three
// base addresses are even (16-byte rows).  Copies past M, N and K are zero-filled.
template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::MINB)
    dgemm_kernel(const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ C, int M, int N, int K,
                 int lda, int ldb, int ldc, long long sA, long long sB, long long sC) {
    constexpr int MI = Cfg::MI, NJ = Cfg::NJ, BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, STAGES = Cfg::STAGES;
    constexpr int ALD = Cfg::ALD, BLD = Cfg::BLD;
    extern __shared__ __align__(16) double gsm[];
    A += blockIdx.z * sA;
    B += blockIdx.z * sB;
    C += blockIdx.z * sC;
    // the few tiles of the short side run side by side and share the long operand's slices in L2
    const int m0 = (M < N ? blockIdx.x : blockIdx.y) * BM, n0 = (M < N ? blockIdx.y : blockIdx.x) * BN;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = (warp % Cfg::WR) * 16 * MI, wn = (warp / Cfg::WR) * 8 * NJ;  // this warp's part of the tile
    // k slice `tile` into stage st, in chunks of 16 bytes
    auto load = [&](int tile, int st) {
        double* As = gsm + st * Cfg::STAGE;
        double* Bs = As + BM * ALD;
        const int k0 = tile * BK;
#pragma unroll
        for (int j = 0; j < BM * BK / 2 / Cfg::THREADS; ++j) {
            const int c = tid + j * Cfg::THREADS;
            const int row = c / (BK / 2), col = (c % (BK / 2)) * 2;
            const int gr = m0 + row, gc = k0 + col;
            const int valid = gr < M ? 8 * max(0, min(2, K - gc)) : 0;
            cp_async16(As + row * ALD + col, valid ? A + (size_t)gr * lda + gc : A, valid);
        }
#pragma unroll
        for (int j = 0; j < BK * BN / 2 / Cfg::THREADS; ++j) {
            const int c = tid + j * Cfg::THREADS;
            const int row = c / (BN / 2), col = (c % (BN / 2)) * 2;
            const int gr = k0 + row, gc = n0 + col;
            const int valid = gr < K ? 8 * max(0, min(2, N - gc)) : 0;
            cp_async16(Bs + row * BLD + col, valid ? B + (size_t)gr * ldb + gc : B, valid);
        }
    };
    double acc[MI][NJ][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;
    const int tiles = (K + BK - 1) / BK;
#pragma unroll
    for (int st = 0; st < STAGES - 1; ++st) {
        if (st < tiles) load(st, st);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int tl = 0; tl < tiles; ++tl) {
        // this thread's copies of slice tl have landed; the barrier makes everyone's visible and
        // ends every read of the stage the next load overwrites (slice tl - 1's)
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        if (tl + STAGES - 1 < tiles) load(tl + STAGES - 1, (tl + STAGES - 1) % STAGES);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double* As = gsm + (tl % STAGES) * Cfg::STAGE;
        const double* Bs = As + BM * ALD;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            double a[MI][2], b[NJ];
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                a[i][0] = As[(wm + 16 * i + g) * ALD + kk + t];
                a[i][1] = As[(wm + 16 * i + g + 8) * ALD + kk + t];
            }
#pragma unroll
            for (int j = 0; j < NJ; ++j) b[j] = Bs[(kk + t) * BLD + wn + 8 * j + g];
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) mma_f64(acc[i][j], a[i][0], a[i][1], b[j]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = m0 + wm + 16 * i + g + 8 * h;
            if (row >= M) continue;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int col = n0 + wn + 8 * j + 2 * t;  // even: 16-byte aligned in C
                double* out = C + (size_t)row * ldc + col;
                if (col + 1 < N) *reinterpret_cast<double2*>(out) = make_double2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
                else if (col < N) out[0] = acc[i][j][2 * h];
            }
        }
}

// 3. For every pair of modes (a, b), a = kx: (As + la[a] + lb[b]) u = f along s, Thomas elimination
// (diagonally dominant: the eigenvalues' sum is positive whenever a transformed direction has a
// Dirichlet end or a Robin end with Bi > 0; along the eliminated one the rows are dominant by
// themselves).  Line (a, b) starts at b * stride_b + a and has `len` points `stride` apart; each
// end is next to a Dirichlet voxel or a Robin face.  f and then u in v; the eliminated upper
// diagonal in cp.  Both sweeps load kThomasChunk points ahead of the dependent recurrence, so
// each thread keeps that many loads in flight.
constexpr int kThomasChunk = 8;

struct ThomasArgs {
    int na, nb, len, lo_robin, hi_robin;
    size_t stride_b, stride;
    double id2, bi;
};

__global__ void thomas_kernel(double* __restrict__ v, double* __restrict__ cp, const double* __restrict__ la,
                              const double* __restrict__ lb, const ThomasArgs p) {
    const size_t lines = (size_t)p.na * p.nb;
    const int len = p.len;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < lines; t += (size_t)gridDim.x * blockDim.x) {
        const int a = (int)(t % p.na), b = (int)(t / p.na);
        const double lam = la[a] + lb[b];
        const double a_in = 2.0 * p.id2 + lam, a_rob = 2.0 * (1.0 + p.bi) * p.id2 + lam;
        const size_t base = (size_t)b * p.stride_b + a;
        double c = 0.0, d = 0.0;
        for (int z0 = 0; z0 < len; z0 += kThomasChunk) {
            double f[kThomasChunk];
#pragma unroll
            for (int q = 0; q < kThomasChunk; ++q)
                if (z0 + q < len) f[q] = v[base + (size_t)(z0 + q) * p.stride];
#pragma unroll
            for (int q = 0; q < kThomasChunk; ++q) {
                const int z = z0 + q;
                if (z >= len) break;
                const bool first = z == 0, last = z == len - 1;
                const bool rob = (first && p.lo_robin) || (last && p.hi_robin);
                const double lo = first ? 0.0 : (last && p.hi_robin ? -2.0 * p.id2 : -p.id2);
                const double up = last ? 0.0 : (first && p.lo_robin ? -2.0 * p.id2 : -p.id2);
                const double r = 1.0 / ((rob ? a_rob : a_in) - lo * c);
                c = up * r;
                d = (f[q] - lo * d) * r;
                const size_t o = base + (size_t)z * p.stride;
                cp[o] = c;
                v[o] = d;
            }
        }
        double u = d;  // u at the last point
        for (int z1 = len - 1; z1 > 0; z1 -= kThomasChunk) {  // points z1 - 1 down to z1 - kThomasChunk
            double dv[kThomasChunk], cv[kThomasChunk];
#pragma unroll
            for (int q = 0; q < kThomasChunk; ++q) {
                const int z = z1 - 1 - q;
                if (z >= 0) {
                    dv[q] = v[base + (size_t)z * p.stride];
                    cv[q] = cp[base + (size_t)z * p.stride];
                }
            }
#pragma unroll
            for (int q = 0; q < kThomasChunk; ++q) {
                const int z = z1 - 1 - q;
                if (z < 0) break;
                u = dv[q] - cv[q] * u;
                v[base + (size_t)z * p.stride] = u;
            }
        }
    }
}

__device__ __forceinline__ double nan_max(double a, double b) { return (b > a || b != b) ? b : a; }

// 4'. From the folded transforms' output (a folded direction holds its even part P in the places
// of the sums and its odd part Q in those of the differences: u_q = P + Q, u_{m-1-q} = P - Q) to
// the solution, in one streaming pass into the other volume, so that the finishing pass reads
// one value per neighbour.
template <bool FX>
__global__ void unfold_kernel(const double* __restrict__ pq, double* __restrict__ u, const HeatArgs a, const Fold f) {
    const size_t total = (size_t)f.wx * f.wy * f.wz;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < total; c += (size_t)gridDim.x * blockDim.x) {
        const FoldItem t = fold_item(f, a, c);
        auto at = [&](int j, int z) { return ((size_t)z * a.my + j) * a.mx; };
        auto put = [&](int j, int z, double p, double q) {
            double* row = u + at(j, z);
            row[t.i] = FX ? p + q : p;
            if (FX) row[a.mx - 1 - t.i] = p - q;
        };
        const size_t re = at(t.j, t.z);
        const double pe = pq[re + t.i], qe = FX ? pq[re + f.wx + t.i] : 0.0;
        if (t.pair) {
            const size_t rd = at(t.jd, t.zd);
            const double pd = pq[rd + t.i], qd = FX ? pq[rd + f.wx + t.i] : 0.0;
            put(t.j, t.z, pe + pd, qe + qd);
            put(t.j2, t.z2, pe - pd, qe - qd);
        } else {
            put(t.j, t.z, pe, qe);
        }
    }
}

// 5. T <- u (rounded to R) for every unknown, with four sums into out: [0] max |J(u) - u| and
// [1] sum (J(u) - u)^2 for one FP64 Jacobi sweep J of u (jacobi_point, coefficients in FP64),
// [2] max |u - T_before| and [3] sum (u - T_before)^2.  Maxima are kept as the bits of
// non-negative doubles (ordered like unsigned integers; a NaN wins).  A thread walks
// zc planes (finish_planes) of one (x, y) column with u's z neighbours in registers, so every load of a
// plane is independent of the arithmetic; neighbours outside the unknowns are Dirichlet
// voxels of T, which nothing writes.
constexpr int kFinishZ = 16;

// Planes per thread: 16, or fewer (at least 2) where that would leave SMs without three blocks.
int finish_planes(size_t plane, int nz) {
    int zc = kFinishZ;
    while (zc > 2 && plane * ((nz + zc - 1) / zc) < (size_t)148 * 3 * 256) zc /= 2;
    return zc;
}

template <typename R, int BOUND>
__global__ void __launch_bounds__(256, 3) finish_kernel(R* __restrict__ T, const R* __restrict__ Q, const double* __restrict__ u,
                                                     const HeatArgs a, const JacobiCoef<double> k, int zc, double* __restrict__ out) {
    auto U = [&](size_t rowbase, int col) -> double { return u[rowbase + col]; };  // the solution
    const size_t plane = (size_t)a.mx * a.my, nn = (size_t)a.n, tplane = nn * nn;
    const int chunks = (a.nz + zc - 1) / zc;
    const size_t items = plane * chunks;
    double rmax = 0.0, rsum = 0.0, cmax = 0.0, csum = 0.0;
    for (size_t it = blockIdx.x * (size_t)blockDim.x + threadIdx.x; it < items; it += (size_t)gridDim.x * blockDim.x) {
        const size_t t = it % plane;
        const int z0 = (int)(it / plane) * zc, z1 = min(a.nz, z0 + zc);
        const int i = (int)(t % a.mx), j = (int)(t / a.mx);
        const int x = a.x0 + i, y = a.y0 + j;
        const bool uxm = i > 0, uxp = i + 1 < a.mx, uym = j > 0, uyp = j + 1 < a.my;
        const bool gxm = x > 0, gxp = x + 1 < a.n, gym = y > 0, gyp = y + 1 < a.n;
        size_t rb = (size_t)z0 * plane + (size_t)j * a.mx;  // this column's row in plane z
        size_t v = (size_t)z0 * tplane + (size_t)y * nn + x;
        double below = z0 > 0 ? U(rb - plane, i) : 0.0;
        double cur = U(rb, i);
#pragma unroll 2
        for (int z = z0; z < z1; ++z, rb += plane, v += tplane) {
            const double above = z + 1 < a.nz ? U(rb + plane, i) : 0.0;
            const double xm = uxm ? U(rb, i - 1) : (gxm ? (double)T[v - 1] : 0.0);
            const double xp = uxp ? U(rb, i + 1) : (gxp ? (double)T[v + 1] : 0.0);
            const double ym = uym ? U(rb - a.mx, i) : (gym ? (double)T[v - nn] : 0.0);
            const double yp = uyp ? U(rb + a.mx, i) : (gyp ? (double)T[v + nn] : 0.0);
            const double q = Q ? (double)Q[v] : 0.0;
            const double before = (double)T[v];
            auto get = [&](int dx, int dy, int dz) -> double {
                if (dz) return dz > 0 ? above : below;
                if (dy) return dy > 0 ? yp : ym;
                return dx > 0 ? xp : xm;
            };
            double w = cur;
            jacobi_point<double, BOUND>(x, y, z, k, q, get, &w);
            const double r = fabs(w - cur), dc = fabs(cur - before);
            rmax = nan_max(rmax, r);
            rsum += r * r;
            cmax = nan_max(cmax, dc);
            csum += dc * dc;
            T[v] = (R)cur;
            below = cur;
            cur = above;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        rmax = nan_max(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
        rsum += __shfl_xor_sync(0xffffffffu, rsum, o);
        cmax = nan_max(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
        csum += __shfl_xor_sync(0xffffffffu, csum, o);
    }
    __shared__ double red[4][8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        red[0][wid] = rmax;
        red[1][wid] = rsum;
        red[2][wid] = cmax;
        red[3][wid] = csum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w2 = 1; w2 < (int)(blockDim.x >> 5); ++w2) {
            rmax = nan_max(rmax, red[0][w2]);
            rsum += red[1][w2];
            cmax = nan_max(cmax, red[2][w2]);
            csum += red[3][w2];
        }
        atomicMax(reinterpret_cast<unsigned long long*>(out), (unsigned long long)__double_as_longlong(rmax));
        atomicAdd(out + 1, rsum);
        atomicMax(reinterpret_cast<unsigned long long*>(out + 2), (unsigned long long)__double_as_longlong(cmax));
        atomicAdd(out + 3, csum);
    }
}

// C = A B over `batch` matrices (see dgemm_kernel); the longer side is split into launches of at
// most 65535 tiles.
template <class Cfg>
cudaError_t gemm_tiles(const double* A, const double* B, double* C, int M, int N, int K, int lda, int ldb, int ldc,
                       int batch, long long sA, long long sB, long long sC, cudaStream_t s) {
    auto kern = dgemm_kernel<Cfg>;
    static PerDevice<int> attr;  // the kernel's dynamic shared memory, once per device
    const cudaError_t ae = attr.get([&](int, int&) {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM);
    });
    if (ae != cudaSuccess) return ae;
    const bool wide = M < N;
    const int span = 65535 * (wide ? Cfg::BN : Cfg::BM), total = wide ? N : M;
    for (int o = 0; o < total; o += span) {
        const int part = std::min(total - o, span), m = wide ? M : part, n = wide ? part : N;
        const unsigned mt = (unsigned)((m + Cfg::BM - 1) / Cfg::BM), nt = (unsigned)((n + Cfg::BN - 1) / Cfg::BN);
        const dim3 grid(wide ? mt : nt, wide ? nt : mt, (unsigned)batch);
        kern<<<grid, Cfg::THREADS, Cfg::SMEM, s>>>(A + (wide ? 0 : (size_t)o * lda), B + (wide ? o : 0),
                                                   C + (wide ? o : (size_t)o * ldc), m, n, K, lda, ldb, ldc, sA, sB, sC);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Which tile: the one whose busiest SM has the least to do, counting its tiles' products (padding
// included) at the share of the FP64 pipe the tile reaches.
cudaError_t gemm(const double* A, const double* B, double* C, int M, int N, int K, int lda, int ldb, int ldc, int batch,
                 long long sA, long long sB, long long sC, cudaStream_t s) {
    auto cost = [&](int bm, int bn, double share) {
        const double tiles = (double)((M + bm - 1) / bm) * ((N + bn - 1) / bn) * batch;
        return std::ceil(tiles / 148.0) * bm * bn / share;
    };
    const double big = cost(GemmBig::BM, GemmBig::BN, 0.84), mid = cost(GemmMid::BM, GemmMid::BN, 0.7),
                 small = cost(GemmSmall::BM, GemmSmall::BN, 0.5);
    if (big <= mid && big <= small) return gemm_tiles<GemmBig>(A, B, C, M, N, K, lda, ldb, ldc, batch, sA, sB, sC, s);
    if (mid <= small) return gemm_tiles<GemmMid>(A, B, C, M, N, K, lda, ldb, ldc, batch, sA, sB, sC, s);
    return gemm_tiles<GemmSmall>(A, B, C, M, N, K, lda, ldb, ldc, batch, sA, sB, sC, s);
}

// Microseconds that `products` products per point (4 flops each, there and back) take at the
// 28 TFLOP/s the large tiles reach.
double transform_us(double vol, double products) { return 4.0 * vol * products / 28e6; }

// Whether y's transform is folded (a symmetric operator): half the products, but two launches for
// one and smaller tiles, so only where the products saved take 50 us.  126x126x200 measured 301 us
// whole, 313 us folded (29 us of products saved), 94x94x37 92 / 103 us.
bool folds_y(const HeatGrid& g) {
    return g.oy.lo_robin == g.oy.hi_robin && g.my % 2 == 0 &&
           transform_us((double)g.mx * g.my * g.nz, 0.5 * g.my) >= 50.0;
}

// The direction transformed beside x: 1 y, 2 z, by modelled time: the transform's products, and the
// elimination's dependent rows along the other direction, about 0.25 us each however many
// lines run side by side; z where that takes less than 0.7 of it.  Measured solves, y against z
// transformed: 512x512x501 16.5 / 12.7 ms, 512x512x64 2145 / 1289 us, 256x256x60 401 / 327 us,
// and where y is kept 192x192x60 217 / 212 us, 128x128x100 156 / 159 us, 126x126x200 301 / 317 us.
int axis_of(const HeatGrid& g) {
    const double vol = (double)g.mx * g.my * g.nz;
    const double ty = transform_us(vol, folds_y(g) ? 0.5 * g.my : g.my) + 0.25 * g.nz;
    const double tz = transform_us(vol, 0.5 * g.nz) + 0.25 * g.my;
    return tz < 0.7 * ty ? 2 : 1;
}

int grid_for(size_t work, int threads) {
    return (int)std::max<size_t>(1, std::min<size_t>((work + threads - 1) / threads, (size_t)148 * 16));
}

}  // namespace

HeatDirect::~HeatDirect() {
    if (ws_) cudaFree(ws_);  // synchronous: nothing queued may still use it
}

void HeatDirect::release(cudaStream_t s) {
    if (ws_) cudaFreeAsync(ws_, s);
    ws_ = nullptr;
    cap_ = size_ = 0;
}

template <typename R>
shg_status HeatDirect::solve(const shg_params& p, R* T, const R* Q, double t_inf, cudaStream_t s) {
    const HeatGrid g = heat_grid(p);
    if (g.nz > 65535) return fail(SHG_ERR_UNSUPPORTED, "direct heat solve: nz = %d above 65535", g.nz);
    const int axis = axis_of(g);
    const OpMats *ox = nullptr, *oy = nullptr;
    shg_status rc;
    if ((rc = get_op(g.ox, &ox)) != SHG_OK || (axis == 1 && (rc = get_op(g.oy, &oy)) != SHG_OK)) return rc;
    const size_t vol = (size_t)g.mx * g.my * g.nz;
    // z modes: even and odd halves of F and G, eigenvalues
    const int he = (g.nz + 1) / 2, ho = g.nz / 2, lde = he + (he & 1), ldo = ho + (ho & 1);
    const size_t zmodes = axis == 2 ? 2 * ((size_t)he * lde + (size_t)ho * ldo) + g.nz : 0;
    const size_t need = 2 * (vol + (vol & 1)) + 4 + zmodes;
    cudaError_t e;
    if (need > size_) {
        release(s);
        if ((e = dev_alloc((void**)&ws_, sizeof(double) * need, s)) != cudaSuccess) {
            ws_ = nullptr;
            return cuda_fail(e, "cudaMallocAsync");
        }
        size_ = need;
    }
    cap_ = vol + (vol & 1);
    nt_ = (size_t)g.n * g.n * g.nz;
    double* X = ws_;
    double* Y = ws_ + cap_;
    double* out = ws_ + 2 * cap_;
    HeatArgs a;
    a.n = g.n;
    a.nz = g.nz;
    a.x0 = g.x0;
    a.y0 = g.y0;
    a.mx = g.mx;
    a.my = g.my;
    a.lo_x_robin = g.ox.lo_robin;
    a.hi_x_robin = g.ox.hi_robin;
    a.lo_y_robin = g.oy.lo_robin;
    a.hi_y_robin = g.oy.hi_robin;
    a.idx2 = 1.0 / (g.dx * g.dx);
    a.idy2 = 1.0 / (g.dy * g.dy);
    a.idz2 = 1.0 / (g.dz * g.dz);
    a.iK = 1.0 / p.kappa;
    a.tinf = t_inf;
    a.bix = g.ox.bi;
    a.biy = g.oy.bi;
    a.biz = g.biz;
    shg_params pk = p;
    pk.t_inf = t_inf;
    const JacobiCoef<double> k = make_jacobi_coef<double>(pk);
    const int mx = g.mx, my = g.my, nz = g.nz;
    const long long pl = (long long)mx * my;
    if ((e = cudaMemsetAsync(out, 0, 4 * sizeof(double), s)) != cudaSuccess) return cuda_fail(e, "memset");
    const bool fx = ox->fold;
    const int h = mx / 2;
    Fold f;
    f.fx = fx;
    f.ft = axis == 2 ? 2 : folds_y(g) ? 1 : 0;
    f.wx = fx ? h : mx;
    f.wy = f.ft == 1 ? my / 2 : my;
    f.wz = f.ft == 2 ? he : nz;
    const size_t fitems = (size_t)f.wx * f.wy * f.wz;
    if (fx) rhs_kernel<R, true><<<grid_for(fitems, 256), 256, 0, s>>>(T, Q, X, a, f);
    else rhs_kernel<R, false><<<grid_for(fitems, 256), 256, 0, s>>>(T, Q, X, a, f);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "heat right-hand side");
    double *zFe = out + 4, *zFo = zFe + (size_t)he * lde, *zGe = zFo + (size_t)ho * ldo, *zGo = zGe + (size_t)he * lde,
           *zlam = zGo + (size_t)ho * ldo;
    if (axis == 2) {
        z_modes_kernel<<<nz, 128, 0, s>>>(nz, a.biz, a.idz2, zlam, zFe, zFo, zGe, zGo, lde, ldo);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "heat z modes");
    }
    // the transforms: along x from rows, folded as a batch of two halves (FoT = FeT + h*h); along y
    // one product per z plane, along z one over all columns, each half by itself when folded
    const long long hh = (long long)h * h;
    auto along_x = [&](const double* eT, const double* full, const double* from, double* to) {
        return fx ? gemm(from, eT, to, nz * my, h, h, mx, h, mx, 2, h, hh, h, s)
                  : gemm(from, full, to, nz * my, mx, mx, mx, ox->ld, mx, 1, 0, 0, 0, s);
    };
    auto along_t = [&](const double* full, const double* even, const double* odd, const double* from, double* to) {
        if (axis == 2) {
            if (he == ho)
                return gemm(even, from, to, he, (int)pl, he, lde, (int)pl, (int)pl, 2, odd - even, he * pl, he * pl, s);
            const cudaError_t e1 = gemm(even, from, to, he, (int)pl, he, lde, (int)pl, (int)pl, 1, 0, 0, 0, s);
            return e1 != cudaSuccess ? e1
                                     : gemm(odd, from + he * pl, to + he * pl, ho, (int)pl, ho, ldo, (int)pl, (int)pl, 1, 0, 0, 0, s);
        }
        if (f.ft == 0) return gemm(full, from, to, my, mx, my, oy->ld, mx, mx, nz, 0, pl, pl, s);
        const int w = my / 2;
        const size_t off = (size_t)w * mx;
        const cudaError_t e1 = gemm(even, from, to, w, mx, w, oy->ldl, mx, mx, nz, 0, pl, pl, s);
        return e1 != cudaSuccess ? e1 : gemm(odd, from + off, to + off, w, mx, w, oy->ldl, mx, mx, nz, 0, pl, pl, s);
    };
    if ((e = along_x(ox->FeT, ox->FT, X, Y)) != cudaSuccess ||
        (e = axis == 2 ? along_t(nullptr, zFe, zFo, Y, X) : along_t(oy->F, oy->Fe, oy->Fo, Y, X)) != cudaSuccess)
        return cuda_fail(e, "heat transform");
    ThomasArgs ta;
    ta.na = mx;
    ta.nb = axis == 2 ? nz : my;
    ta.len = axis == 2 ? my : nz;
    ta.stride_b = axis == 2 ? (size_t)pl : (size_t)mx;
    ta.stride = axis == 2 ? (size_t)mx : (size_t)pl;
    ta.lo_robin = axis == 2 ? g.oy.lo_robin : 1;
    ta.hi_robin = axis == 2 ? g.oy.hi_robin : 1;
    ta.id2 = axis == 2 ? a.idy2 : a.idz2;
    ta.bi = axis == 2 ? a.biy : a.biz;
    thomas_kernel<<<grid_for((size_t)ta.na * ta.nb, 128), 128, 0, s>>>(X, Y, fx ? ox->lamf : ox->lam,
                                                                        axis == 2 ? zlam : oy->lam, ta);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "heat tridiagonal solve");
    if ((e = axis == 2 ? along_t(nullptr, zGe, zGo, X, Y) : along_t(oy->G, oy->Ge, oy->Go, X, Y)) != cudaSuccess ||
        (e = along_x(ox->GeT, ox->GT, Y, X)) != cudaSuccess)
        return cuda_fail(e, "heat transform");
    const double* u = X;
    if (fx || f.ft) {
        if (fx) unfold_kernel<true><<<grid_for(fitems, 256), 256, 0, s>>>(X, Y, a, f);
        else unfold_kernel<false><<<grid_for(fitems, 256), 256, 0, s>>>(X, Y, a, f);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "heat solution");
        u = Y;
    }
    const int zc = finish_planes((size_t)pl, nz);
    const int fb = grid_for((size_t)pl * ((nz + zc - 1) / zc), 256);
    if (p.boundary == SHG_BOUNDARY_TOP_OPEN)
        finish_kernel<R, SHG_BOUNDARY_TOP_OPEN><<<fb, 256, 0, s>>>(T, Q, u, a, k, zc, out);
    else
        finish_kernel<R, SHG_BOUNDARY_OVEN_SURROUNDED><<<fb, 256, 0, s>>>(T, Q, u, a, k, zc, out);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "heat solution");
    return SHG_OK;
}

shg_status HeatDirect::result(int rule, double* residual, double* change, cudaStream_t s) {
    if (!ws_) return fail(SHG_ERR_INVALID, "no heat solve to read");
    double h[4] = {0, 0, 0, 0};
    cudaError_t e;
    if ((e = cudaMemcpyAsync(h, ws_ + 2 * cap_, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return cuda_fail(e, "heat solve result");
    const double nt = (double)nt_;
    if (residual) *residual = rule == SHG_CONV_REFERENCE ? std::sqrt(h[1]) / nt : h[0];
    if (change) *change = rule == SHG_CONV_REFERENCE ? std::sqrt(h[3]) / nt : h[2];
    return SHG_OK;
}

template shg_status HeatDirect::solve<float>(const shg_params&, float*, const float*, double, cudaStream_t);
template shg_status HeatDirect::solve<double>(const shg_params&, double*, const double*, double, cudaStream_t);

shg_status heat_steady_device(const shg_params& p, void* temperature, const void* q, double* residual,
                              cudaStream_t s) {
    HeatDirect h;
    shg_status rc = p.precision == 32
                        ? h.solve<float>(p, reinterpret_cast<float*>(temperature), reinterpret_cast<const float*>(q), p.t_inf, s)
                        : h.solve<double>(p, reinterpret_cast<double*>(temperature), reinterpret_cast<const double*>(q),
                                          p.t_inf, s);
    double r = 0.0;
    if (rc == SHG_OK) rc = h.result(SHG_CONV_MAXABS, &r, nullptr, s);
    h.release(s);
    const cudaError_t e = cudaStreamSynchronize(s);
    if (rc == SHG_OK && e != cudaSuccess) rc = cuda_fail(e, "heat steady solve");
    if (rc == SHG_OK && !std::isfinite(r)) rc = fail(SHG_ERR_NONFINITE, "heat steady solve: residual %g", r);
    if (residual) *residual = r;
    return rc;
}

}  // namespace shg

extern "C" shg_status shg_heat_operator_modes(int32_t m, double d, int32_t lo_robin, int32_t hi_robin, double bi,
                                              double* lambda_out, double* forward_out, double* inverse_out) {
    using namespace shg;
    clear_error();
    if (m < 1 || m > 65536) return fail(SHG_ERR_INVALID, "m = %d must be in 1..65536", m);
    if (!(d > 0) || !std::isfinite(d) || !(bi >= 0) || !std::isfinite(bi))
        return fail(SHG_ERR_INVALID, "spacing must be > 0 and the Biot number >= 0, both finite");
    if (!lambda_out || !forward_out || !inverse_out) return fail(SHG_ERR_INVALID, "output pointer is NULL");
    Op1D op;
    op.m = m;
    op.d = d;
    op.lo_robin = lo_robin ? 1 : 0;
    op.hi_robin = hi_robin ? 1 : 0;
    op.bi = bi;
    std::vector<double> lam, F, G;
    if (!op_modes(op, lam, F, G)) return fail(SHG_ERR_NOT_CONVERGED, "heat operator eigendecomposition (m = %d)", m);
    std::memcpy(lambda_out, lam.data(), sizeof(double) * m);
    std::memcpy(forward_out, F.data(), sizeof(double) * F.size());
    std::memcpy(inverse_out, G.data(), sizeof(double) * G.size());
    return SHG_OK;
}
