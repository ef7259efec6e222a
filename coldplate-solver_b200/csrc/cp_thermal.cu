// B200 3-D conjugate-heat-transfer solve (C ABI in include/cp_thermal.h).
//
// The reference (ThermalSolver/thermal_solver.cpp) assembles a 7-point
// finite-volume system on Nx x Ny x Nz cells into CSR on the host and solves
// it with AMGCL's IDR(s) preconditioned by smoothed-aggregation AMG
// (thermal_solver.cpp:417-553).  Here:
//   k_th_assemble   one thread per cell computes the reference's row in FP64
//                   (same formulas and summation order, thermal_solver.cpp:
//                   420-520) into seven coefficient arrays and b;
//   k_th_coarsen    Galerkin coarse operators P^T A P of a hierarchy that
//                   aggregates 2 x 2 columns (all z-layers kept) down to one
//                   column; P piecewise constant, so every level keeps the
//                   7-point form and the levels of A^T are the transposes;
//   k_th_lu         Thomas factors of every column's tridiagonal z-block, per
//                   level;
//   k_th_matrix     the V-cycle from the first level with at most kThApply
//                   cells down, as a matrix: one column a CTA, the unit vector
//                   cycled in shared memory;
//   k_th_bicgstab   persistent cooperative BiCGStab right-preconditioned by
//                   one V-cycle: damped z-line Jacobi smoothing (one sweep
//                   down, one up), each direction of a level one pass over
//                   tiles of whole columns (residual or restriction a thread a
//                   cell, the z-solve from shared memory), the small levels one
//                   matrix product.  Bounded grid barriers with the dot
//                   products on them, deterministic sums, AMGCL's stop test
//                   ||r|| <= rtol ||b||.  The same kernel solves A^T x = rhs
//                   for the p-norm adjoint;
//   k_th_sens       dJ/dgamma from the adjoint field, one thread per column.
// Layout: every array is indexed k Nx Ny + j Nx + i (i contiguous), so the
// stencil loads of a warp are coalesced.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/cp_thermal.h"
#include "cp_device.cuh"
#include "cp_pool.cuh"

// error string of the library (cp_solver.cu)
cp_status cp_internal_set_error(cp_status s, const char* msg);

namespace {

cp_status tfail(cp_status s, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    return cp_internal_set_error(s, buf);
}

#define TCK(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return tfail(CP_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_),      \
                         __FILE__, __LINE__);                                                      \
    } while (0)

constexpr int kThThreads = 256;           // element-wise kernels
constexpr int kThMaxNz = 16;              // most layers (a tile holds whole columns: at least 16 of them)
constexpr int kThMaxLevels = 16;          // 2 x 2 aggregation from up to 2^15 columns per side
constexpr long long kThLarge = 1 << 20;   // cells from which the solver runs 1024 threads an SM instead of 512
constexpr long long kThApply = 1024;      // levels of at most this many cells: their V-cycle is a matrix
constexpr int kThMatThreads = 128;
// three vectors of every level from kThApply cells down: halving in one
// direction only (a level one column wide) they sum to less than twice the
// first, plus up to one layer stack a level
constexpr size_t kThMatSmemMax = 3 * sizeof(double) * (size_t)(2 * kThApply + kThMaxLevels * kThMaxNz);
constexpr double kThOmega = 0.8;          // z-line Jacobi damping
constexpr double kThScale0 = 1.4;         // coarse-correction factor into level 0
constexpr double kThScale = 1.4;          // ... into the deeper levels (1.2 / 1.1: 95 / more iterations
                                          // at 1024 x 512 x 12, against 84)
constexpr int kThRefineRounds = 4;        // mixed precision: BiCGStab launches per solve at most

}  // namespace

namespace cp {

struct ThK {
    int Nx, Ny, Nz, nzS, nzF, mode;
    long long n, ncol;
    double dx, dy, dzS, dzF, Ht, kS, kF, rhoCp, Tin, qk;
};

// The seven coefficient arrays of a 7-point system and its right-hand side
// (T = double: the assembled system and its Galerkin levels; T = float: the
// preconditioner's copies in the mixed-precision solve)
template <typename T>
struct ThSysT {
    T *aP, *aW, *aE, *aS, *aN, *aB, *aT, *b;
};
using ThSys = ThSysT<double>;

struct ThStatus {
    int iterations, converged, err, pad;
    double residual;
};

__device__ __forceinline__ double th_dz(const ThK& k, int kk) { return kk < k.nzS ? k.dzS : k.dzF; }

// thermal_solver.cpp:271-305 (gamma clamped to [0, 1]); k_s in the base plate
__device__ __forceinline__ double th_kval(const ThK& k, const double* gamma, int i, int j, int kk) {
    if (kk < k.nzS) return k.kS;
    double g = gamma[(size_t)j * k.Nx + i];
    g = fmax(0.0, fmin(1.0, g));
    if (k.mode == 1) {
        const double num = 1.0 - g;
        const double den = 1.0 + __dmul_rn(k.qk, g);
        return k.kF + (k.kS - k.kF) * num / den;
    }
    if (k.mode == 2) return k.kS * k.kF / (__dmul_rn(1.0 - g, k.kF) + __dmul_rn(g, k.kS) + 1e-30);
    return __dmul_rn(k.kS, 1.0 - g) + __dmul_rn(k.kF, g);
}

// 1 = fluid: above the base plate with gamma > 0.01 (thermal_solver.cpp:240-244)
__device__ __forceinline__ bool th_fluid(const ThK& k, const double* gamma, int i, int j, int kk) {
    if (kk < k.nzS) return false;
    return gamma[(size_t)j * k.Nx + i] > 0.01;
}

// Poiseuille factor of a fluid layer (thermal_solver.cpp:323-327)
__device__ __forceinline__ double th_pois(const ThK& k, int kk) {
    if (kk < k.nzS) return 0.0;
    const double z = (kk - k.nzS + 0.5) * k.dzF / k.Ht;
    return 4.0 * z * (1 - z);
}

__device__ __forceinline__ double th_harm(double a, double b) { return 2 * a * b / (a + b + 1e-30); }

// One row of the reference's system, in its summation order
// (thermal_solver.cpp:420-520).  Every product that feeds a sum is rounded
// on its own (__dmul_rn) so that no multiply-add is fused and the row has the
// reference's bits.  Off-diagonal entries are the matrix values (negative);
// the reference's two entries for one neighbour (diffusion and upwind
// advection) are summed like its CSR conversion sums them.
__global__ void k_th_assemble(ThK k, const double* gamma, const double* u_xy, const double* v_xy, const double* q0,
                              ThSys S) {
    const int Nx = k.Nx, Ny = k.Ny, Nz = k.Nz;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < k.n;
         t += (long long)gridDim.x * blockDim.x) {
        const int kk = (int)(t / ((long long)Nx * Ny));
        const int rem = (int)(t - (long long)kk * Nx * Ny);
        const int j = rem / Nx, i = rem % Nx;
        const double dx = k.dx, dy = k.dy, rhoCp = k.rhoCp, T_in = k.Tin;
        const double dz_k = th_dz(k, kk), Ax = dy * dz_k, Ay = dx * dz_k, Az_cell = dx * dy;
        double diag = 0, bb = 0;
        const double kP = th_kval(k, gamma, i, j, kk), po = th_pois(k, kk);
        double g = (kk < k.nzS) ? 0.0 : gamma[(size_t)j * Nx + i];
        g = fmax(0.0, fmin(1.0, g));
        const double uP = (g > 0.01) ? __dmul_rn(u_xy[(size_t)j * Nx + i], po) : 0.0;
        const double vP = (g > 0.01) ? __dmul_rn(v_xy[(size_t)j * Nx + i], po) : 0.0;
        const bool regP = th_fluid(k, gamma, i, j, kk);
        double aW = 0, aE = 0, aS = 0, aN = 0, aB = 0, aT = 0;
        // x faces
        if (i > 0) {
            const double kf = th_harm(kP, th_kval(k, gamma, i - 1, j, kk)), D = kf * Ax / dx;
            diag += D;
            aW = -D;
            if (regP && th_fluid(k, gamma, i - 1, j, kk)) {
                const double uW = __dmul_rn(u_xy[(size_t)j * Nx + i - 1], po), F = rhoCp * 0.5 * (uP + uW) * Ax;
                diag += fmax(-F, 0.0);
                aW = aW + (-fmax(F, 0.0));
            }
        } else if (regP) {
            const double D_bc = 2.0 * kP * Ax / dx, F_bc = __dmul_rn(rhoCp * uP, Ax);
            diag += D_bc;
            bb += __dmul_rn(D_bc, T_in);
            if (F_bc > 0) bb += __dmul_rn(F_bc, T_in);
            else diag += -F_bc;
        }
        if (i < Nx - 1) {
            const double kf = th_harm(kP, th_kval(k, gamma, i + 1, j, kk)), D = kf * Ax / dx;
            diag += D;
            aE = -D;
            if (regP && th_fluid(k, gamma, i + 1, j, kk)) {
                const double uE = __dmul_rn(u_xy[(size_t)j * Nx + i + 1], po), F = rhoCp * 0.5 * (uP + uE) * Ax;
                diag += fmax(F, 0.0);
                aE = aE + (-fmax(-F, 0.0));
            }
        } else if (regP && uP > 0) {
            diag += __dmul_rn(rhoCp * uP, Ax);
        }
        // y faces
        if (j > 0) {
            const double kf = th_harm(kP, th_kval(k, gamma, i, j - 1, kk)), D = kf * Ay / dy;
            diag += D;
            aS = -D;
            if (regP && th_fluid(k, gamma, i, j - 1, kk)) {
                const double vS = __dmul_rn(v_xy[(size_t)(j - 1) * Nx + i], po), F = rhoCp * 0.5 * (vP + vS) * Ay;
                diag += fmax(-F, 0.0);
                aS = aS + (-fmax(F, 0.0));
            }
        }
        if (j < Ny - 1) {
            const double kf = th_harm(kP, th_kval(k, gamma, i, j + 1, kk)), D = kf * Ay / dy;
            diag += D;
            aN = -D;
            if (regP && th_fluid(k, gamma, i, j + 1, kk)) {
                const double vN = __dmul_rn(v_xy[(size_t)(j + 1) * Nx + i], po), F = rhoCp * 0.5 * (vP + vN) * Ay;
                diag += fmax(F, 0.0);
                aN = aN + (-fmax(-F, 0.0));
            }
        } else if (regP && vP > 0) {
            diag += __dmul_rn(rhoCp * vP, Ay);
        }
        // z faces (diffusion only)
        if (kk > 0) {
            const double kN = th_kval(k, gamma, i, j, kk - 1), dz_P = dz_k, dz_N = th_dz(k, kk - 1);
            const double kf = (dz_P + dz_N) / (dz_P / kP + dz_N / kN);
            const double D = kf * Az_cell / (0.5 * (dz_P + dz_N));
            diag += D;
            aB = -D;
        } else {
            bb += __dmul_rn(q0[(size_t)j * Nx + i], Az_cell);
        }
        if (kk < Nz - 1) {
            const double kN = th_kval(k, gamma, i, j, kk + 1), dz_P = dz_k, dz_N = th_dz(k, kk + 1);
            const double kf = (dz_P + dz_N) / (dz_P / kP + dz_N / kN);
            const double D = kf * Az_cell / (0.5 * (dz_P + dz_N));
            diag += D;
            aT = -D;
        }
        S.aP[t] = diag + 1e-12;
        S.aW[t] = aW; S.aE[t] = aE; S.aS[t] = aS; S.aN[t] = aN; S.aB[t] = aB; S.aT[t] = aT;
        S.b[t] = bb;
    }
}

// One level of the hierarchy (level 0: the assembled system).  x holds the
// pre-smoothed iterate, b the restricted residual and y the post-smoothed
// iterate of a coarse level.
template <typename T>
struct ThLevelT {
    int nx, ny;
    long long ncol, n;
    ThSysT<T> S;
    T *lc, *linv;
    T *b, *x, *y;
};
using ThLevel = ThLevelT<double>;

// Entry of row q of A (Tr = false) or of A^T (Tr = true) towards the lower and
// upper neighbour.  Row q of A^T holds column q of A.
template <bool Tr, typename T>
__device__ __forceinline__ T th_sub(const ThSysT<T>& S, long long q, long long L) {
    return __ldg(Tr ? S.aT + (q - L) : S.aB + q);
}
template <bool Tr, typename T>
__device__ __forceinline__ T th_sup(const ThSysT<T>& S, long long q, long long L) {
    return __ldg(Tr ? S.aB + (q + L) : S.aT + q);
}

// Row q of the operator and its neighbours' indices.  A neighbour outside the
// level is the cell itself with a zero entry, so that no load waits for a
// branch: with a branch a neighbour, a cell of a small level took seven load
// latencies one after the other.
template <typename T>
struct ThRow {
    T p, w, e, s, n, b, t;
    unsigned qw, qe, qs, qn, qb, qt;
};

template <bool Tr, typename T>
__device__ __forceinline__ ThRow<T> th_row(const ThLevelT<T>& F, int Nz, unsigned q, int i, int j, int kk) {
    const unsigned L = (unsigned)F.ncol, nx = (unsigned)F.nx;
    const bool hw = i > 0, he = i < F.nx - 1, hs = j > 0, hn = j < F.ny - 1, hb = kk > 0, ht = kk < Nz - 1;
    ThRow<T> r;
    r.qw = hw ? q - 1 : q;
    r.qe = he ? q + 1 : q;
    r.qs = hs ? q - nx : q;
    r.qn = hn ? q + nx : q;
    r.qb = hb ? q - L : q;
    r.qt = ht ? q + L : q;
    r.p = __ldg(F.S.aP + q);
    r.w = __ldg(Tr ? F.S.aE + r.qw : F.S.aW + q);
    r.e = __ldg(Tr ? F.S.aW + r.qe : F.S.aE + q);
    r.s = __ldg(Tr ? F.S.aN + r.qs : F.S.aS + q);
    r.n = __ldg(Tr ? F.S.aS + r.qn : F.S.aN + q);
    r.b = __ldg(Tr ? F.S.aT + r.qb : F.S.aB + q);
    r.t = __ldg(Tr ? F.S.aB + r.qt : F.S.aT + q);
    if (Tr) {
        r.w = hw ? r.w : T(0);
        r.e = he ? r.e : T(0);
        r.s = hs ? r.s : T(0);
        r.n = hn ? r.n : T(0);
        r.b = hb ? r.b : T(0);
        r.t = ht ? r.t : T(0);
    }
    return r;
}

// (op x)_q on a level, op = A or A^T, in the level's arithmetic T (x may be
// stored narrower: the FP64 matvec of a float preconditioner output)
template <bool Tr, typename T, typename X>
__device__ __forceinline__ T th_ax(const ThLevelT<T>& F, int Nz, const X* x, unsigned q, int i, int j, int kk) {
    const ThRow<T> r = th_row<Tr>(F, Nz, q, i, j, kk);
    const T xp = T(x[q]), xw = T(x[r.qw]), xe = T(x[r.qe]), xs = T(x[r.qs]), xn = T(x[r.qn]), xb = T(x[r.qb]), xt = T(x[r.qt]);
    T s = r.p * xp;
    s += r.w * xw;
    s += r.e * xe;
    s += r.s * xs;
    s += r.n * xn;
    s += r.b * xb;
    s += r.t * xt;
    return s;
}

// Galerkin coarse operator P^T A P of 2 x 2 column aggregates, P piecewise
// constant: couplings inside an aggregate fold into the diagonal, couplings
// across an aggregate edge add up into the coarse neighbour's entry.
__global__ void k_th_coarsen(int Nz, ThLevel F, ThLevel C) {
    for (long long qc = (long long)blockIdx.x * blockDim.x + threadIdx.x; qc < C.n;
         qc += (long long)gridDim.x * blockDim.x) {
        const int kk = (int)(qc / C.ncol);
        const long long rem = qc - kk * C.ncol;
        const int I = (int)(rem % C.nx), J = (int)(rem / C.nx);
        double aP = 0, aW = 0, aE = 0, aS = 0, aN = 0, aB = 0, aT = 0;
        for (int dj = 0; dj < 2; ++dj) {
            const int j = 2 * J + dj;
            if (j >= F.ny) break;
            for (int di = 0; di < 2; ++di) {
                const int i = 2 * I + di;
                if (i >= F.nx) break;
                const long long q = kk * F.ncol + (long long)j * F.nx + i;
                aP += F.S.aP[q];
                aB += F.S.aB[q];
                aT += F.S.aT[q];
                if (di == 1) aP += F.S.aW[q]; else aW += F.S.aW[q];
                if (di == 0 && i + 1 < F.nx) aP += F.S.aE[q]; else aE += F.S.aE[q];
                if (dj == 1) aP += F.S.aS[q]; else aS += F.S.aS[q];
                if (dj == 0 && j + 1 < F.ny) aP += F.S.aN[q]; else aN += F.S.aN[q];
            }
        }
        C.S.aP[qc] = aP; C.S.aW[qc] = aW; C.S.aE[qc] = aE; C.S.aS[qc] = aS; C.S.aN[qc] = aN;
        C.S.aB[qc] = aB; C.S.aT[qc] = aT;
    }
}

// float copy of a level array (the mixed-precision preconditioner's levels)
__global__ void k_th_narrow(const double* __restrict__ src, float* __restrict__ dst, long long n) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = (float)src[q];
}

// Thomas factors of each column's tridiagonal z-block of a level:
// inv_k = 1 / (d_k - sub_k c_{k-1}), c_k = sup_k inv_k
template <bool Tr>
__global__ void k_th_lu(int Nz, ThLevel F) {
    const long long L = F.ncol;
    for (long long col = (long long)blockIdx.x * blockDim.x + threadIdx.x; col < F.ncol;
         col += (long long)gridDim.x * blockDim.x) {
        double cprev = 0.0;
        for (int kk = 0; kk < Nz; ++kk) {
            const long long q = kk * L + col;
            const double den = F.S.aP[q] - (kk > 0 ? th_sub<Tr>(F.S, q, L) * cprev : 0.0);
            const double inv = 1.0 / den;
            const double c = (kk < Nz - 1 ? th_sup<Tr>(F.S, q, L) : 0.0) * inv;
            F.linv[q] = inv;
            F.lc[q] = c;
            cprev = c;
        }
    }
}

// A tile: W = blockDim / Nz whole columns of a level (in column order, so a
// tile may span rows), a thread a cell: layer kk, tile column c.  The z-solve
// of a tile runs from shared memory, a thread a column: in double the cell threads
// store f = r inv and g = sub inv and lc, so that a step of either sweep is one
// multiply-add, y = f - g y and x = y - lc x.  In float, where sub inv would be a
// third rounding a step, f = r and g = sub, with inv in x: y = (f - g y) inv.
template <typename T>
struct ThTile {
    T *f, *g, *lc, *x;      // [Nz][W] each
    int W, kk, c;
    bool on;                // the thread has a cell (kk < Nz)
    __device__ __forceinline__ int at() const { return kk * W + c; }
    // one cell's share of the z-block M x = r
    __device__ __forceinline__ void put(T r, T inv, T sub, T l) const {
        if constexpr (sizeof(T) == 4) {
            f[at()] = r;
            g[at()] = sub;
            x[at()] = inv;
        } else {
            f[at()] = r * inv;
            g[at()] = sub * inv;
        }
        lc[at()] = l;
    }
    // after it x holds M^-1 r; the caller may put the next tile's cells at
    // once: a thread reads and puts its own cell alone, and the next solve's
    // first barrier comes before the columns' threads read them
    __device__ __forceinline__ void solve(int Nz) const {
        __syncthreads();
        if (threadIdx.x < W) {
            const T* __restrict__ F = f + threadIdx.x;
            const T* __restrict__ G = g + threadIdx.x;
            const T* __restrict__ C = lc + threadIdx.x;
            T* __restrict__ X = x + threadIdx.x;
            T v = T(0);
#pragma unroll 4
            for (int k = 0; k < Nz; ++k) {
                v = F[k * W] - G[k * W] * v;
                if constexpr (sizeof(T) == 4) v *= X[k * W];
                X[k * W] = v;
            }
            v = T(0);
#pragma unroll 4
            for (int k = Nz - 1; k >= 0; --k) {
                v = X[k * W] - C[k * W] * v;
                X[k * W] = v;
            }
        }
        __syncthreads();
    }
};

// Entry below of the z-block and the Thomas factors of a cell
template <bool Tr, typename T>
__device__ __forceinline__ void th_zrow(const ThLevelT<T>& F, unsigned q, int kk, T& inv, T& sub, T& l) {
    const unsigned L = (unsigned)F.ncol, qb = kk > 0 ? q - L : q;
    inv = __ldg(F.linv + q);
    l = __ldg(F.lc + q);
    sub = __ldg(Tr ? F.S.aT + qb : F.S.aB + q);
    if (kk == 0) sub = T(0);
}

// Pre-smoothing from zero on level 0, with the vector update that makes its
// right-hand side: b = A0 + c1 A1 + c2 A2 (A2 optional; stored to bout),
// x = omega Mz^-1 b.
template <bool Tr, typename T>
__device__ __forceinline__ void th_presmooth(const ThLevelT<T>& F, int Nz, const double* A0, const double* A1, double c1,
                                             const double* A2, double c2, double* bout, double omega, const ThTile<T>& t) {
    const unsigned L = (unsigned)F.ncol;
    for (unsigned c0 = blockIdx.x * t.W; c0 < L; c0 += gridDim.x * t.W) {
        const unsigned col = c0 + t.c, q = t.kk * L + col;
        const bool on = t.on && col < L;
        if (on) {
            T inv, sub, l;
            th_zrow<Tr>(F, q, t.kk, inv, sub, l);
            double b = A0[q];
            const double a1 = A1[q], a2 = A2 ? A2[q] : 0.0;
            b += c1 * a1;
            if (A2) b += c2 * a2;
            bout[q] = b;
            t.put(T(b), inv, sub, l);
        }
        t.solve(Nz);
        if (on) F.x[q] = T(omega) * t.x[t.at()];
    }
}

// Descent from level F to C: b_C = the sum over the 2 x 2 aggregate of
// b - op x, and the pre-smoothing of C, x_C = omega Mz^-1 b_C (unless C is
// solved by its matrix, `last`).  A thread a coarse cell, its four fine
// residuals' loads in flight two by two.
template <bool Tr, typename T, typename B>
__device__ __forceinline__ void th_down(const ThLevelT<T>& F, const ThLevelT<T>& C, int Nz, const B* bF, double omega,
                                        bool last, const ThTile<T>& t) {
    const unsigned LF = (unsigned)F.ncol, LC = (unsigned)C.ncol, cnx = (unsigned)C.nx;
    for (unsigned c0 = blockIdx.x * t.W; c0 < LC; c0 += gridDim.x * t.W) {
        const unsigned col = c0 + t.c, qc = t.kk * LC + col;
        const bool on = t.on && col < LC;
        if (on) {
            const unsigned J = col / cnx, I = col - J * cnx;
            T inv = T(0), sub = T(0), l = T(0);
            if (!last) th_zrow<Tr>(C, qc, t.kk, inv, sub, l);
            T b = T(0);
#pragma unroll 1
            for (int d = 0; d < 4; ++d) {
                const int i = 2 * (int)I + (d & 1), j = 2 * (int)J + (d >> 1);
                // an odd edge's missing cell is read inside and dropped
                const int ii = min(i, F.nx - 1), jj = min(j, F.ny - 1);
                const unsigned q = t.kk * LF + (unsigned)jj * F.nx + ii;
                const T v = T(bF[q]) - th_ax<Tr>(F, Nz, F.x, q, ii, jj, t.kk);
                b += (i < F.nx && j < F.ny) ? v : T(0);
            }
            C.b[qc] = b;
            if (!last) t.put(b, inv, sub, l);
        }
        if (last) continue;
        t.solve(Nz);
        if (on) C.x[qc] = T(omega) * t.x[t.at()];
    }
}

// Ascent from level C to F with the post-smoothing: xp = x + scale P xC formed
// at every stencil point, out = xp + omega Mz^-1 (b - op xp).
template <bool Tr, typename T, typename B>
__device__ __forceinline__ void th_up(const ThLevelT<T>& F, const ThLevelT<T>& C, int Nz, const B* bF, const T* xC,
                                      double scale, double omega, T* out, const ThTile<T>& t) {
    const unsigned L = (unsigned)F.ncol, LC = (unsigned)C.ncol, nx = (unsigned)F.nx, cnx = (unsigned)C.nx;
    const T sc = T(scale);
    const T* xF = F.x;
    for (unsigned c0 = blockIdx.x * t.W; c0 < L; c0 += gridDim.x * t.W) {
        const unsigned col = c0 + t.c, q = t.kk * L + col;
        const bool on = t.on && col < L;
        T xp = T(0);
        if (on) {
            const unsigned ju = col / nx, iu = col - ju * nx;
            const int i = (int)iu, j = (int)ju;
            const ThRow<T> r = th_row<Tr>(F, Nz, q, i, j, t.kk);
            T inv, sub, l;
            th_zrow<Tr>(F, q, t.kk, inv, sub, l);
            // the parents: a neighbour's is the cell's own or the one across
            const unsigned kc = t.kk * LC, I = iu >> 1, J = ju >> 1;
            const unsigned Iw = i > 0 ? (iu - 1) >> 1 : I, Ie = i < F.nx - 1 ? (iu + 1) >> 1 : I;
            const unsigned Js = j > 0 ? (ju - 1) >> 1 : J, Jn = j < F.ny - 1 ? (ju + 1) >> 1 : J;
            const unsigned kb = t.kk > 0 ? kc - LC : kc, kt = t.kk < Nz - 1 ? kc + LC : kc;
            const T cp = xC[kc + J * cnx + I], cw = xC[kc + J * cnx + Iw], ce = xC[kc + J * cnx + Ie],
                    cs = xC[kc + Js * cnx + I], cn = xC[kc + Jn * cnx + I], cb = xC[kb + J * cnx + I],
                    ct = xC[kt + J * cnx + I];
            const T fp = xF[q], fw = xF[r.qw], fe = xF[r.qe], fs = xF[r.qs], fn = xF[r.qn], fb = xF[r.qb], ft = xF[r.qt];
            const T bq = T(bF[q]);
            xp = fp + sc * cp;
            T ax = r.p * xp;
            ax += r.w * (fw + sc * cw);
            ax += r.e * (fe + sc * ce);
            ax += r.s * (fs + sc * cs);
            ax += r.n * (fn + sc * cn);
            ax += r.b * (fb + sc * cb);
            ax += r.t * (ft + sc * ct);
            t.put(bq - ax, inv, sub, l);
        }
        t.solve(Nz);
        if (on) out[q] = xp + T(omega) * t.x[t.at()];
    }
}

// y = B b on the level that is solved by its matrix, a warp a row.  Summed in
// double in either form: the rows of a nearly singular level are long sums of
// nearly cancelling terms, and sums in float cost mixed adjoints of small plates 5
// to 10 % more iterations, and two of 500 their convergence.
template <typename T>
__device__ __forceinline__ void th_apply(const ThLevelT<T>& F, const T* __restrict__ bm) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = gridDim.x * (blockDim.x >> 5), n = (int)F.n;
    for (int i = wid * gridDim.x + blockIdx.x; i < n; i += nw) {
        const T* row = bm + (size_t)i * n;
        double s = 0.0;
#pragma unroll 16
        for (int q = lane; q < n; q += 32) s += (double)row[q] * (double)F.b[q];
        s = warp_sum(s);
        if (lane == 0) F.y[i] = T(s);
    }
}

// out = w Mz^-1 r of a level's columns, from and to shared memory (in place
// allowed), a thread a column
template <bool Tr>
__device__ __forceinline__ void th_mat_zsolve(const ThLevel& F, int Nz, const double* r, double w, double* out) {
    const int L = (int)F.ncol;
    for (int c = threadIdx.x; c < L; c += blockDim.x) {
        double y = 0.0;
        for (int k = 0; k < Nz; ++k) {
            const int q = k * L + c;
            y = (r[q] - (k > 0 ? th_sub<Tr>(F.S, q, L) : 0.0) * y) * F.linv[q];
            out[q] = y;
        }
        double x = 0.0;
        for (int k = Nz - 1; k >= 0; --k) {
            const int q = k * L + c;
            x = out[q] - (k < Nz - 1 ? F.lc[q] * x : 0.0);
            out[q] = w * x;
        }
    }
    __syncthreads();
}

// Column q of the V-cycle's matrix on levels [m, L): the cycle of the unit
// vector e_q in shared memory (b, x, y of every level), a CTA a column.
template <bool Tr, typename T>
__global__ void __launch_bounds__(kThMatThreads) k_th_matrix(int Nz, const ThLevel* __restrict__ lv, int m, int L,
                                                             double omega, double scale, T* bm) {
    extern __shared__ double sh[];
    __shared__ double* at[kThMaxLevels];
    const int n = (int)lv[m].n;
    if (threadIdx.x == 0) {
        double* p = sh;
        for (int l = m; l < L; ++l) {
            at[l] = p;
            p += 3 * lv[l].n;
        }
    }
    __syncthreads();
    for (int q0 = blockIdx.x; q0 < n; q0 += gridDim.x) {
        for (int q = threadIdx.x; q < n; q += blockDim.x) at[m][q] = q == q0 ? 1.0 : 0.0;
        __syncthreads();
        for (int l = m;; ++l) {
            const ThLevel F = lv[l];
            double *b = at[l], *x = b + F.n;
            th_mat_zsolve<Tr>(F, Nz, b, l + 1 == L ? 1.0 : omega, x);
            if (l + 1 == L) break;
            const ThLevel C = lv[l + 1];
            for (int qc = threadIdx.x; qc < (int)C.n; qc += blockDim.x) {
                const int kk = qc / (int)C.ncol, rem = qc - kk * (int)C.ncol, J = rem / C.nx, I = rem - J * C.nx;
                double r = 0.0;
                for (int d = 0; d < 4; ++d) {
                    const int i = 2 * I + (d & 1), j = 2 * J + (d >> 1);
                    if (i >= F.nx || j >= F.ny) continue;
                    const unsigned q = (unsigned)(kk * (int)F.ncol + j * F.nx + i);
                    r += b[q] - th_ax<Tr>(F, Nz, x, q, i, j, kk);
                }
                at[l + 1][qc] = r;
            }
            __syncthreads();
        }
        for (int l = L - 2; l >= m; --l) {
            const ThLevel F = lv[l], C = lv[l + 1];
            double *b = at[l], *x = b + F.n, *y = x + F.n;
            const double* xc = at[l + 1] + (l + 2 == L ? 1 : 2) * C.n;
            for (int q = threadIdx.x; q < (int)F.n; q += blockDim.x) {
                const int kk = q / (int)F.ncol, rem = q - kk * (int)F.ncol, j = rem / F.nx, i = rem - j * F.nx;
                x[q] += scale * xc[kk * (int)C.ncol + (j >> 1) * C.nx + (i >> 1)];
            }
            __syncthreads();
            for (int q = threadIdx.x; q < (int)F.n; q += blockDim.x) {
                const int kk = q / (int)F.ncol, rem = q - kk * (int)F.ncol, j = rem / F.nx, i = rem - j * F.nx;
                y[q] = b[q] - th_ax<Tr>(F, Nz, x, (unsigned)q, i, j, kk);
            }
            __syncthreads();
            th_mat_zsolve<Tr>(F, Nz, y, omega, y);
            for (int q = threadIdx.x; q < (int)F.n; q += blockDim.x) y[q] += x[q];
            __syncthreads();
        }
        const double* out = at[m] + (m + 1 == L ? 1 : 2) * n;
        for (int i = threadIdx.x; i < n; i += blockDim.x) bm[(size_t)i * n + q0] = (T)out[i];
        __syncthreads();
    }
}

// The preconditioner's hierarchy in type T (level 0's arrays: copies of the
// assembled system when T is float)
template <typename T>
struct ThHierT {
    int L, m;               // levels; the V-cycle from level m (>= 1) down is the matrix bm
    double omega, scale0, scale;   // coarse-correction factor into level 0, into the deeper levels
    const ThLevelT<T>* lv;  // device array of L levels
    T* bm;                  // n x n for the n cells of level m
    unsigned long long* prof;  // per-phase nanoseconds (CP_TH_PROFILE), or null
};
using ThHier = ThHierT<double>;

// phase slots of the profile: the BiCGStab phases, then 16 slots per
// V-cycle direction indexed by level
enum ThProfSlot {
    TH_P_INIT = 0, TH_P_PRE_P = 1, TH_P_MATVEC_V = 2, TH_P_PRE_S = 3, TH_P_MATVEC_T = 4, TH_P_UPDATE = 5,
    TH_P_APPLY = 6, TH_P_DOWN = 16, TH_P_UP = 32, TH_P_COUNT = 48
};

// BiCGStab's vectors, FP64; the preconditioned directions ph = M^-1 p and
// sh = M^-1 s are stored in the preconditioner's type T
template <typename T>
struct ThVecsT {
    double *x, *r, *rh, *p, *v, *s, *t;
    T *ph, *sh;
};
using ThVecs = ThVecsT<double>;

// BiCGStab (van der Vorst), right-preconditioned by one V-cycle, for
// A x = rhs (Tr = false) or A^T x = rhs (Tr = true), from the x in V.x.
// F0 is the FP64 system (matvecs, residuals, dot products); the V-cycle runs
// on H in type T (T = float: the mixed-precision form; T = double: H.lv[0]
// is F0).
// Two V-cycles, two matvecs and an update an iteration: 2 (2 m + 3) + 3
// barriers, 27 at 151 x 97 x 9 and 37 at 1024 x 512 x 12.  At the small end
// these are the cost; an iteration takes 94 us there instead of 310.  At
// 1024 x 512 x 12 the passes over level 0 are, bound by their loads (the seven
// coefficient arrays first): 1.20 ms instead of 1.85.
// NT threads a CTA, two CTAs an SM: 256 (128 registers, no spills) where the
// barriers are the cost, 512 from kThLarge
// cells on, where more warps in flight are worth more (1.20 against 1.46 ms an
// iteration at 1024 x 512 x 12; 94 against 113 us at 151 x 97 x 9).
template <bool Tr, typename T, int NT>
__global__ void __launch_bounds__(NT, 2) k_th_bicgstab(ThK k, ThLevel F0, ThHierT<T> H, const double* rhs,
                                                              ThVecsT<T> V, double* part, unsigned* bar, ThStatus* st,
                                                              int maxiter, double rtol) {
    __shared__ double sm[kReduceSm];
    __shared__ ThLevelT<T> lv[kThMaxLevels];
    __shared__ T tile[4][NT];
    const int Nz = k.Nz;
    const unsigned tid = blockIdx.x * NT + threadIdx.x, nth = gridDim.x * NT;
    const Team team = grid_team(bar, &st->err);
    unsigned target = 0;
    for (int l = threadIdx.x; l < H.L; l += NT) lv[l] = H.lv[l];
    ThTile<T> tl;
    tl.f = tile[0]; tl.g = tile[1]; tl.lc = tile[2]; tl.x = tile[3];
    tl.W = NT / Nz;
    tl.kk = threadIdx.x / tl.W;
    tl.c = threadIdx.x - tl.kk * tl.W;
    tl.on = tl.kk < Nz;
    __syncthreads();
    unsigned long long tprev = (H.prof && team.lead()) ? globaltimer_ns() : 0ull;
    // with the profile on, block 0 books the time since the previous barrier
    // to the phase slot
    auto tick = [&](int slot) {
        if (H.prof && team.lead()) {
            const unsigned long long t = globaltimer_ns();
            H.prof[slot] += t - tprev;
            tprev = t;
        }
    };
    auto sync = [&](int slot) -> bool {
        const bool ok = team_sync(team, target);
        tick(slot);
        return ok;
    };
    auto reduce = [&](int slot, double (&v)[2]) -> bool {
        const bool ok = team_reduce(team, target, v, part, sm);
        tick(slot);
        return ok;
    };
    // Two cells a thread per step: compute(q, i, j, kk) only loads and
    // computes (its loads for both cells in flight together), commit(q, v)
    // stores and accumulates; 32-bit index math.
    auto cells2 = [&](auto&& compute, auto&& commit) {
        const unsigned n = (unsigned)k.n, L = (unsigned)k.ncol, nx = (unsigned)k.Nx;
        auto at = [&](unsigned q) {
            const unsigned kk = q / L, rem = q - kk * L, j = rem / nx;
            return compute(q, (int)(rem - j * nx), (int)j, (int)kk);
        };
        unsigned q = tid;
        for (; q < n && n - q > nth; q += 2 * nth) {
            const auto a = at(q);
            const auto b = at(q + nth);
            commit(q, a);
            commit(q + nth, b);
        }
        if (q < n) commit(q, at(q));
    };
    // The V-cycle after the level-0 pre-smoothing (lv[0].x = omega Mz^-1 b0):
    // out0 = M^-1 b0.  Ends with a grid barrier.
    auto vcycle = [&](const double* b0, T* out0) __attribute__((always_inline)) -> bool {
        for (int l = 0; l < H.m; ++l) {
            if (l == 0) th_down<Tr>(lv[0], lv[1], Nz, b0, H.omega, H.m == 1, tl);
            else th_down<Tr>(lv[l], lv[l + 1], Nz, (const T*)lv[l].b, H.omega, l + 1 == H.m, tl);
            if (!sync(TH_P_DOWN + l)) return false;
        }
        th_apply(lv[H.m], H.bm);
        if (!sync(TH_P_APPLY)) return false;
        for (int l = H.m - 1; l >= 0; --l) {
            if (l == 0) th_up<Tr>(lv[0], lv[1], Nz, b0, lv[1].y, H.scale0, H.omega, out0, tl);
            else th_up<Tr>(lv[l], lv[l + 1], Nz, (const T*)lv[l].b, lv[l + 1].y, H.scale, H.omega, lv[l].y, tl);
            if (!sync(TH_P_UP + l)) return false;
        }
        return true;
    };
    // ---- r = rhs - op x, rh = r, p = v = 0; ||rhs||^2, ||r||^2
    double acc[2] = {0.0, 0.0};
    cells2([&](unsigned q, int i, int j, int kk) {
        const double b = rhs[q];
        return make_double2(b, b - th_ax<Tr>(F0, Nz, V.x, q, i, j, kk));
    }, [&](unsigned q, double2 a) {
        V.r[q] = a.y;
        V.rh[q] = a.y;
        V.p[q] = 0.0;
        V.v[q] = 0.0;
        acc[0] += a.x * a.x;
        acc[1] += a.y * a.y;
    });
    if (!reduce(TH_P_INIT, acc)) return;
    const double bnorm = sqrt(acc[0]) > 0.0 ? sqrt(acc[0]) : 1.0;
    double res = sqrt(acc[1]) / bnorm;
    double rho = 1.0, alpha = 1.0, omega = 1.0, rho1 = acc[1];
    int it = 0;
    bool conv = res <= rtol;
    for (; it < maxiter && !conv; ++it) {
        if (rho1 == 0.0) break;
        const double beta = (rho1 / rho) * (alpha / omega);
        // ---- p = r + beta p - beta omega v, fused with the level-0 pre-smoothing; ph = M^-1 p
        th_presmooth<Tr>(lv[0], Nz, V.r, V.p, beta, V.v, -beta * omega, V.p, H.omega, tl);
        if (!sync(TH_P_PRE_P)) return;
        if (!vcycle(V.p, V.ph)) return;
        // ---- v = op ph; (rh, v)
        acc[0] = acc[1] = 0.0;
        cells2([&](unsigned q, int i, int j, int kk) {
            return make_double2(th_ax<Tr>(F0, Nz, V.ph, q, i, j, kk), V.rh[q]);
        }, [&](unsigned q, double2 a) {
            V.v[q] = a.x;
            acc[0] += a.y * a.x;
        });
        if (!reduce(TH_P_MATVEC_V, acc)) return;
        if (acc[0] == 0.0) break;
        alpha = rho1 / acc[0];
        // ---- s = r - alpha v, fused with the level-0 pre-smoothing; sh = M^-1 s
        th_presmooth<Tr>(lv[0], Nz, V.r, V.v, -alpha, (const double*)nullptr, 0.0, V.s, H.omega, tl);
        if (!sync(TH_P_PRE_S)) return;
        if (!vcycle(V.s, V.sh)) return;
        // ---- t = op sh; (t, s), (t, t)
        acc[0] = acc[1] = 0.0;
        cells2([&](unsigned q, int i, int j, int kk) {
            return make_double2(th_ax<Tr>(F0, Nz, V.sh, q, i, j, kk), V.s[q]);
        }, [&](unsigned q, double2 a) {
            V.t[q] = a.x;
            acc[0] += a.x * a.y;
            acc[1] += a.x * a.x;
        });
        if (!reduce(TH_P_MATVEC_T, acc)) return;
        omega = acc[1] > 0.0 ? acc[0] / acc[1] : 0.0;
        // ---- x += alpha ph + omega sh; r = s - omega t; (r, r), (rh, r)
        acc[0] = acc[1] = 0.0;
        cells2([&](unsigned q, int, int, int) {
            return make_double3(V.x[q] + alpha * double(V.ph[q]) + omega * double(V.sh[q]), V.s[q] - omega * V.t[q],
                                V.rh[q]);
        }, [&](unsigned q, double3 a) {
            V.x[q] = a.x;
            V.r[q] = a.y;
            acc[0] += a.y * a.y;
            acc[1] += a.z * a.y;
        });
        if (!reduce(TH_P_UPDATE, acc)) return;
        res = sqrt(acc[0]) / bnorm;
        rho = rho1;
        rho1 = acc[1];
        if (!(res == res)) {
            if (team.lead()) atomicCAS(&st->err, 0, (int)CP_ERR_NONFINITE);
            return;
        }
        if (res <= rtol) { conv = true; ++it; break; }
        if (omega == 0.0) { ++it; break; }
    }
    if (team.lead()) {
        st->iterations = it;
        st->converged = conv ? 1 : 0;
        st->residual = res;
    }
}

// bottom layer: partials of max T and sum T^p
__global__ void k_th_pnorm(ThK k, const double* T, double pexp, double* part) {
    __shared__ double sm[64];
    __shared__ double smx[32];
    double mx = -1e300, s[1] = {0.0};
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < k.ncol;
         q += (long long)gridDim.x * blockDim.x) {
        const double t = T[q];
        mx = fmax(mx, t);
        s[0] += pow(t, pexp);
    }
    block_sum<1>(s, sm);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) smx[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = -1e300;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, smx[w]);
        part[2 * blockIdx.x] = m;
        part[2 * blockIdx.x + 1] = s[0];
    }
}

__global__ void k_th_fill(double* x, long long n, double v) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        x[q] = v;
}

// dJ/dT of J = (mean over the bottom layer of T^p)^(1/p):
// (T / J)^(p-1) / (Nx Ny) on k = 0, zero above
__global__ void k_th_adj_rhs(ThK k, const double* T, double J, double pexp, double* rhs) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < k.n;
         q += (long long)gridDim.x * blockDim.x)
        rhs[q] = q < k.ncol ? pow(T[q] / J, pexp - 1.0) / (double)k.ncol : 0.0;
}

// dk/dgamma of a cell above the base plate at the clamped gamma; for RAMP
// the reference's dk_dgamma (thermal_solver.cpp:317-321)
__device__ __forceinline__ double th_dkdg(const ThK& k, double g) {
    g = fmax(0.0, fmin(1.0, g));
    if (k.mode == 1) {
        const double den = 1.0 + k.qk * g;
        return (k.kS - k.kF) * (-(1.0 + k.qk)) / (den * den);
    }
    if (k.mode == 2) {
        const double den = (1.0 - g) * k.kF + g * k.kS + 1e-30;
        return -k.kS * k.kF * (k.kS - k.kF) / (den * den);
    }
    return k.kF - k.kS;
}

// d harm(a, b) / da for harm = 2ab / (a + b + 1e-30)
__device__ __forceinline__ double th_dharm(double a, double b) {
    const double s = a + b + 1e-30;
    return 2.0 * b * (b + 1e-30) / (s * s);
}

// dJ/dgamma(i, j) = -lambda^T dR/dgamma(i, j) for R = A(gamma) T - b(gamma),
// one thread per column.  gamma(i, j) sets k of every cell of the column
// above the base plate, which enters the x/y face conductances (harmonic
// means), the inlet conductance 2 k Ax / dx and the z conductances
// (thickness-weighted); the velocities and the fluid/solid masks are held
// fixed (the mask is a step at gamma = 0.01 without a derivative).  A face
// of conductance D between P and N contributes (l_P - l_N)(T_P - T_N) dD.
__global__ void k_th_sens(ThK k, const double* gamma, const double* T, const double* lam, double* grad) {
    const long long L = (long long)k.Nx * k.Ny;
    const double dx = k.dx, dy = k.dy;
    for (long long col = (long long)blockIdx.x * blockDim.x + threadIdx.x; col < k.ncol;
         col += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(col % k.Nx), j = (int)(col / k.Nx);
        double acc = 0.0;
        for (int kk = k.nzS; kk < k.Nz; ++kk) {
            const long long q = kk * L + col;
            const double kP = th_kval(k, gamma, i, j, kk), dz = th_dz(k, kk);
            const double Ax = dy * dz, Ay = dx * dz, lP = lam[q], TP = T[q];
            if (i > 0)
                acc += (lP - lam[q - 1]) * (TP - T[q - 1]) * th_dharm(kP, th_kval(k, gamma, i - 1, j, kk)) * Ax / dx;
            if (i < k.Nx - 1)
                acc += (lP - lam[q + 1]) * (TP - T[q + 1]) * th_dharm(kP, th_kval(k, gamma, i + 1, j, kk)) * Ax / dx;
            if (j > 0)
                acc += (lP - lam[q - k.Nx]) * (TP - T[q - k.Nx]) * th_dharm(kP, th_kval(k, gamma, i, j - 1, kk)) *
                       Ay / dy;
            if (j < k.Ny - 1)
                acc += (lP - lam[q + k.Nx]) * (TP - T[q + k.Nx]) * th_dharm(kP, th_kval(k, gamma, i, j + 1, kk)) *
                       Ay / dy;
            if (i == 0 && th_fluid(k, gamma, i, j, kk)) acc += lP * (TP - k.Tin) * 2.0 * Ax / dx;
        }
        // z faces (kk, kk + 1) with a cell above the base plate
        for (int kk = k.nzS - 1; kk < k.Nz - 1; ++kk) {
            const long long q = kk * L + col;
            const double kL = th_kval(k, gamma, i, j, kk), kU = th_kval(k, gamma, i, j, kk + 1);
            const double dL = th_dz(k, kk), dU = th_dz(k, kk + 1), den = dL / kL + dU / kU;
            double dkf = (dL + dU) * (dU / (kU * kU)) / (den * den);
            if (kk >= k.nzS) dkf += (dL + dU) * (dL / (kL * kL)) / (den * den);
            acc += (lam[q] - lam[q + L]) * (T[q] - T[q + L]) * dkf * (dx * dy) / (0.5 * (dL + dU));
        }
        grad[col] = -th_dkdg(k, gamma[col]) * acc;
    }
}

}  // namespace cp

using namespace cp;

struct cp_thermal {
    cp_thermal_params prm{};
    ThK k{};
    int dev = 0, numSMs = 0, grid = 0, gElem = 0, threads = 256;   // grid, threads: the solver kernel's
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    double *gamma = nullptr, *u = nullptr, *v = nullptr, *q0 = nullptr;
    ThSys S{};
    double *lc = nullptr, *linv = nullptr, *z0 = nullptr, *lam = nullptr, *rhs = nullptr, *grad = nullptr;
    ThVecs V{};
    std::vector<ThLevel> lv;          // the hierarchy (level 0: S, lc, linv, z0)
    ThLevel* dlv = nullptr;           // its device copy
    ThHier H{};
    // CP_PREC_MIXED: float copies of the levels that the V-cycle passes over,
    // and the preconditioned directions in float
    bool mixed = false;
    size_t matSmem = 0;               // k_th_matrix's dynamic shared memory (bytes)
    std::vector<ThLevelT<float>> lvf;
    ThLevelT<float>* dlvf = nullptr;
    ThHierT<float> Hf{};
    float *phf = nullptr, *shf = nullptr;
    double* part = nullptr;
    unsigned* bar = nullptr;
    ThStatus* st = nullptr;
    bool hasInputs = false, solved = false;
    Arena mem;                        // every device array
};

namespace {

template <typename T>
cp_status th_alloc(cp_thermal* t, T** p, size_t n) {
    void* q = nullptr;
    TCK(t->mem.take(n * sizeof(T), &q));
    TCK(cudaMemsetAsync(q, 0, std::max<size_t>(n, 1) * sizeof(T), t->stream));
    *p = static_cast<T*>(q);
    return CP_OK;
}

// the solver kernel of a context's size and precision
template <bool Tr>
const void* th_kernel(const cp_thermal* t) {
    if (t->mixed)
        return t->threads == 512 ? (const void*)k_th_bicgstab<Tr, float, 512> : (const void*)k_th_bicgstab<Tr, float, 256>;
    return t->threads == 512 ? (const void*)k_th_bicgstab<Tr, double, 512> : (const void*)k_th_bicgstab<Tr, double, 256>;
}

// float copy of a level array (mixed precision)
cp_status th_narrow(cp_thermal* t, const double* src, float* dst, long long n) {
    const int g = (int)std::min<long long>(t->gElem, (n + kThThreads - 1) / kThThreads);
    k_th_narrow<<<std::max(g, 1), kThThreads, 0, t->stream>>>(src, dst, n);
    TCK(cudaGetLastError());
    return CP_OK;
}

// The float levels of the mixed-precision V-cycle, shaped like the FP64
// hierarchy.  Level 0 needs no b (its right-hand side is a Krylov vector)
// and no y (its output is ph or sh); level m, which is solved by its matrix,
// needs nothing else, and the levels behind it nothing at all.
cp_status th_build_float_hierarchy(cp_thermal* t) {
    const int L = (int)t->lv.size(), m = t->H.m;
    t->lvf.assign(L, ThLevelT<float>{});
    for (int l = 0; l <= m; ++l) {
        const ThLevel& F = t->lv[l];
        ThLevelT<float>& G = t->lvf[l];
        G.nx = F.nx;
        G.ny = F.ny;
        G.ncol = F.ncol;
        G.n = F.n;
        std::vector<float**> arr;
        if (l < m) arr = {&G.S.aP, &G.S.aW, &G.S.aE, &G.S.aS, &G.S.aN, &G.S.aB, &G.S.aT, &G.lc, &G.linv, &G.x};
        if (l > 0) {
            arr.push_back(&G.b);
            arr.push_back(&G.y);
        }
        for (float** q : arr) {
            cp_status s = th_alloc(t, q, (size_t)G.n);
            if (s != CP_OK) return s;
        }
    }
    void* q = nullptr;
    TCK(t->mem.take(sizeof(ThLevelT<float>) * L, &q));
    t->dlvf = static_cast<ThLevelT<float>*>(q);
    TCK(cudaMemcpyAsync(t->dlvf, t->lvf.data(), sizeof(ThLevelT<float>) * L, cudaMemcpyHostToDevice, t->stream));
    t->Hf.L = t->H.L;
    t->Hf.m = m;
    t->Hf.omega = t->H.omega;
    t->Hf.scale0 = t->H.scale0;
    t->Hf.scale = t->H.scale;
    t->Hf.lv = t->dlvf;
    t->Hf.prof = t->H.prof;
    const size_t nm = (size_t)t->lv[m].n;
    cp_status s = th_alloc(t, &t->Hf.bm, nm * nm);
    if (s == CP_OK) s = th_alloc(t, &t->phf, (size_t)t->k.n);
    if (s != CP_OK) return s;
    return th_alloc(t, &t->shf, (size_t)t->k.n);
}

// Levels of 2 x 2 column aggregates down to a single column, all z-layers
// kept; level 0 is the assembled system.  From the first coarse level with at
// most kThApply cells on the V-cycle is a matrix.  CP_TH_OMEGA, CP_TH_SCALE0
// and CP_TH_SCALE override the smoothing weight and the coarse-correction
// factors into level 0 and into the deeper levels.
cp_status th_build_hierarchy(cp_thermal* t) {
    const ThK& k = t->k;
    ThLevel f0{};
    f0.nx = k.Nx;
    f0.ny = k.Ny;
    f0.ncol = k.ncol;
    f0.n = k.n;
    f0.S = t->S;
    f0.lc = t->lc;
    f0.linv = t->linv;
    f0.x = t->z0;
    t->lv.assign(1, f0);
    while (t->lv.back().nx > 1 || t->lv.back().ny > 1) {
        if ((int)t->lv.size() == kThMaxLevels)
            return tfail(CP_ERR_BAD_PARAM, "grid %d x %d needs more than %d levels", k.Nx, k.Ny, kThMaxLevels);
        const ThLevel& F = t->lv.back();
        ThLevel C{};
        C.nx = (F.nx + 1) / 2;
        C.ny = (F.ny + 1) / 2;
        C.ncol = (long long)C.nx * C.ny;
        C.n = C.ncol * k.Nz;
        double** arr[] = {&C.S.aP, &C.S.aW, &C.S.aE, &C.S.aS, &C.S.aN, &C.S.aB, &C.S.aT,
                          &C.lc,   &C.linv, &C.b,    &C.x,    &C.y};
        for (double** q : arr) {
            cp_status s = th_alloc(t, q, (size_t)C.n);
            if (s != CP_OK) return s;
        }
        t->lv.push_back(C);
    }
    const int L = (int)t->lv.size();
    int m = 1;
    while (t->lv[m].n > kThApply) ++m;    // the last level is one column: Nz <= 16 cells
    void* q = nullptr;
    TCK(t->mem.take(sizeof(ThLevel) * L, &q));
    t->dlv = static_cast<ThLevel*>(q);
    TCK(cudaMemcpyAsync(t->dlv, t->lv.data(), sizeof(ThLevel) * L, cudaMemcpyHostToDevice, t->stream));
    t->H.L = L;
    t->H.m = m;
    t->H.omega = kThOmega;
    t->H.scale0 = kThScale0;
    t->H.scale = kThScale;
    if (const char* e = getenv("CP_TH_OMEGA")) t->H.omega = atof(e);
    if (const char* e = getenv("CP_TH_SCALE0")) t->H.scale0 = atof(e);
    if (const char* e = getenv("CP_TH_SCALE")) t->H.scale = atof(e);
    t->H.lv = t->dlv;
    t->H.prof = nullptr;
    t->H.bm = nullptr;
    t->matSmem = 0;
    for (int l = m; l < L; ++l) t->matSmem += 3 * sizeof(double) * (size_t)t->lv[l].n;
    if (!t->mixed) {
        cp_status s = th_alloc(t, &t->H.bm, (size_t)t->lv[m].n * t->lv[m].n);
        if (s != CP_OK) return s;
    }
    if (getenv("CP_TH_PROFILE")) {
        TCK(t->mem.take(sizeof(unsigned long long) * TH_P_COUNT, &q));
        t->H.prof = static_cast<unsigned long long*>(q);
    }
    return CP_OK;
}

// CP_TH_PROFILE: the phase times of the last solve, to stderr
void th_print_profile(cp_thermal* t, bool Tr, int iters) {
    unsigned long long h[TH_P_COUNT];
    if (cudaMemcpy(h, t->H.prof, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return;
    const double it = iters > 0 ? iters : 1;
    fprintf(stderr, "thermal %s profile, us per iteration (%d iterations):\n", Tr ? "adjoint" : "forward", iters);
    const char* top[] = {"init(total)", "update p + presmooth 0", "matvec v", "update s + presmooth 0", "matvec t",
                         "update x, r", "matrix level"};
    for (int i = 0; i <= TH_P_APPLY; ++i)
        if (h[i]) fprintf(stderr, "  %-26s %9.1f\n", top[i], h[i] * 1e-3 / (i == TH_P_INIT ? 1.0 : it));
    const char* kind[] = {"down from", "up into"};
    for (int kd = 0; kd < 2; ++kd)
        for (int l = 0; l < 16; ++l) {
            const unsigned long long v = h[TH_P_DOWN + 16 * kd + l];
            if (v) fprintf(stderr, "  %-10s level %2d %9.1f\n", kind[kd], l, v * 1e-3 / it);
        }
}

cp_status th_objective(cp_thermal* t, double p, double* Tb_max, double* Tb_pnorm) {
    k_th_pnorm<<<t->gElem, kThThreads, 0, t->stream>>>(t->k, t->V.x, p, t->part);
    TCK(cudaGetLastError());
    std::vector<double> h((size_t)2 * t->gElem);
    TCK(cudaMemcpyAsync(h.data(), t->part, h.size() * 8, cudaMemcpyDeviceToHost, t->stream));
    TCK(cudaStreamSynchronize(t->stream));
    double mx = -1e300, s = 0.0;
    for (int b = 0; b < t->gElem; ++b) {
        mx = std::max(mx, h[2 * b]);
        s += h[2 * b + 1];
    }
    if (Tb_max) *Tb_max = mx;
    if (Tb_pnorm) *Tb_pnorm = std::pow(s / (double)t->k.ncol, 1.0 / p);
    return CP_OK;
}

// Column factorisation and the persistent BiCGStab for op x = rhs, op = A or
// A^T, from V.x; records ev1 after the solve and reads the status back.
// Mixed precision: the factors are narrowed to the float levels above the
// matrix, and the
// solve is restarted from its iterate while the FP64 residual it computes
// on entry (b - op x, not the recursive one) is above rtol, for at most
// kThRefineRounds launches in all; the iterations add up.
template <bool Tr>
cp_status th_krylov(cp_thermal* t, const double* rhs, const ThVecs& V, ThStatus* hs) {
    const ThK& k = t->k;
    for (size_t l = 0; l < t->lv.size(); ++l) {
        const ThLevel& F = t->lv[l];
        const int g = (int)std::min<long long>(t->gElem, (F.ncol + kThThreads - 1) / kThThreads);
        k_th_lu<Tr><<<g, kThThreads, 0, t->stream>>>(k.Nz, F);
        TCK(cudaGetLastError());
        if (t->mixed && (int)l < t->H.m) {
            cp_status s = th_narrow(t, F.lc, t->lvf[l].lc, F.n);
            if (s == CP_OK) s = th_narrow(t, F.linv, t->lvf[l].linv, F.n);
            if (s != CP_OK) return s;
        }
    }
    // the matrix of the small levels, from the FP64 levels in either precision
    {
        const int g = (int)t->lv[t->H.m].n;
        if (t->mixed)
            k_th_matrix<Tr, float><<<g, kThMatThreads, t->matSmem, t->stream>>>(k.Nz, t->dlv, t->H.m, t->H.L, t->H.omega,
                                                                               t->H.scale, t->Hf.bm);
        else
            k_th_matrix<Tr, double><<<g, kThMatThreads, t->matSmem, t->stream>>>(k.Nz, t->dlv, t->H.m, t->H.L,
                                                                                t->H.omega, t->H.scale, t->H.bm);
        TCK(cudaGetLastError());
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(t->grid);
    cfg.blockDim = dim3(t->threads);
    cfg.stream = t->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.dynamicSmemBytes = 0;
    const ThVecsT<float> Vf{V.x, V.r, V.rh, V.p, V.v, V.s, V.t, t->phf, t->shf};
    const int rounds = t->mixed ? kThRefineRounds : 1;
    int total = 0;
    for (int round = 0; round < rounds; ++round) {
        TCK(cudaMemsetAsync(t->bar, 0, sizeof(unsigned), t->stream));
        TCK(cudaMemsetAsync(t->st, 0, sizeof(ThStatus), t->stream));
        if (t->H.prof) TCK(cudaMemsetAsync(t->H.prof, 0, sizeof(unsigned long long) * TH_P_COUNT, t->stream));
        const int left = std::max(t->prm.maxiter - total, 0);
        if (t->mixed)
            TCK(cudaLaunchKernelEx(&cfg, t->threads == 512 ? k_th_bicgstab<Tr, float, 512> : k_th_bicgstab<Tr, float, 256>,
                                   k, t->lv[0], t->Hf, rhs, Vf, t->part, t->bar, t->st, left, t->prm.rtol));
        else
            TCK(cudaLaunchKernelEx(&cfg, t->threads == 512 ? k_th_bicgstab<Tr, double, 512> : k_th_bicgstab<Tr, double, 256>,
                                   k, t->lv[0], t->H, rhs, V, t->part, t->bar, t->st, left, t->prm.rtol));
        TCK(cudaEventRecord(t->ev1, t->stream));
        TCK(cudaMemcpyAsync(hs, t->st, sizeof *hs, cudaMemcpyDeviceToHost, t->stream));
        TCK(cudaStreamSynchronize(t->stream));
        if (hs->err)
            return tfail((cp_status)hs->err, "device reported %s in the thermal %s solve",
                         cp_status_string((cp_status)hs->err), Tr ? "adjoint" : "forward");
        if (t->H.prof) th_print_profile(t, Tr, hs->iterations);
        total += hs->iterations;
        // stop once a launch found the true residual at rtol on entry, or did not converge
        if (!hs->converged || hs->iterations == 0) break;
    }
    hs->iterations = total;
    return CP_OK;
}

void th_report(cp_thermal* t, const ThStatus& hs, cp_thermal_report* rep) {
    if (!rep) return;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, t->ev0, t->ev1);
    rep->iterations = hs.iterations;
    rep->converged = hs.converged;
    rep->residual = hs.residual;
    rep->device_ms = ms;
}

}  // namespace

extern "C" {

void cp_thermal_params_default(cp_thermal_params* p) {
    if (!p) return;
    memset(p, 0, sizeof(*p));
    p->nz_solid = 2;
    p->nz_fluid = 7;
    p->H_b = 0.0005;
    p->H_t = 0.004;
    p->k_s = 400.0;
    p->k_f = 0.6;
    p->rho = 998.0;
    p->Cp = 4180.0;
    p->T_inlet = 30.0;
    p->rtol = 1e-6;
    p->maxiter = 1000;
    p->k_interp_mode = 1;
    p->qk = 1.0;
    p->precision = CP_PREC_FP64;
}

cp_status cp_thermal_create(const cp_thermal_params* p, cp_thermal** out) {
    if (!p || !out) return tfail(CP_ERR_BAD_PARAM, "NULL argument");
    *out = nullptr;
    if (p->Nx < 2 || p->Ny < 2 || p->nz_solid < 1 || p->nz_fluid < 1 || p->nz_solid + p->nz_fluid > kThMaxNz)
        return tfail(CP_ERR_BAD_PARAM, "grid %d x %d x (%d + %d): need Nx, Ny >= 2, nz_solid, nz_fluid >= 1 "
                     "and Nz <= %d", p->Nx, p->Ny, p->nz_solid, p->nz_fluid, kThMaxNz);
    const double pos[] = {p->dx, p->dy, p->H_b, p->H_t, p->k_s, p->k_f, p->rho, p->Cp};
    for (double x : pos)
        if (!(x > 0.0) || !std::isfinite(x)) return tfail(CP_ERR_BAD_PARAM, "dx, dy, H_b, H_t, k, rho, Cp must be > 0");
    if (!std::isfinite(p->T_inlet) || !(p->rtol >= 0.0) || p->maxiter < 0 || p->k_interp_mode < 0 ||
        p->k_interp_mode > 2 || !std::isfinite(p->qk) ||
        (p->precision != CP_PREC_FP64 && p->precision != CP_PREC_MIXED))
        return tfail(CP_ERR_BAD_PARAM, "T_inlet, rtol, maxiter, k_interp_mode, qk or precision out of range");
    cp_thermal* t = new cp_thermal();
    t->prm = *p;
    auto bail = [&](cp_status s) {
        cp_thermal_destroy(t);
        return s;
    };
    if (cudaGetDevice(&t->dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&t->numSMs, cudaDevAttrMultiProcessorCount, t->dev) != cudaSuccess) {
        cudaGetLastError();
        delete t;
        return tfail(CP_ERR_CUDA, "no CUDA device");
    }
    if (cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&t->ev0) != cudaSuccess || cudaEventCreate(&t->ev1) != cudaSuccess)
        return bail(tfail(CP_ERR_CUDA, "stream / events"));
    ThK& k = t->k;
    k.Nx = p->Nx; k.Ny = p->Ny; k.nzS = p->nz_solid; k.nzF = p->nz_fluid; k.Nz = k.nzS + k.nzF;
    k.mode = p->k_interp_mode;
    k.ncol = (long long)k.Nx * k.Ny;
    k.n = k.ncol * k.Nz;
    // the reference keeps the domain length and divides it again (thermal_solver.cpp:186-187, 729)
    k.dx = (k.Nx * p->dx) / k.Nx;
    k.dy = (k.Ny * p->dy) / k.Ny;
    k.dzS = p->H_b / p->nz_solid;
    k.dzF = p->H_t / p->nz_fluid;
    k.Ht = p->H_t; k.kS = p->k_s; k.kF = p->k_f; k.rhoCp = p->rho * p->Cp; k.Tin = p->T_inlet; k.qk = p->qk;
    if (k.n >= (1LL << 31))
        return bail(tfail(CP_ERR_BAD_PARAM, "%lld cells: the solver indexes fewer than 2^31", k.n));
    const size_t n = (size_t)k.n, nc = (size_t)k.ncol;
    cp_status s;
    double** planes[] = {&t->gamma, &t->u, &t->v, &t->q0, &t->grad};
    for (double** q : planes)
        if ((s = th_alloc(t, q, nc)) != CP_OK) return bail(s);
    double** vols[] = {&t->S.aP, &t->S.aW, &t->S.aE, &t->S.aS, &t->S.aN, &t->S.aB, &t->S.aT, &t->S.b,
                       &t->lc,   &t->linv, &t->V.x,  &t->V.r,  &t->V.rh, &t->V.p,  &t->V.v,  &t->V.s,
                       &t->V.t,  &t->V.ph, &t->V.sh, &t->lam,  &t->rhs, &t->z0};
    for (double** q : vols)
        if ((s = th_alloc(t, q, n)) != CP_OK) return bail(s);
    // the forward and the adjoint kernel run on the same grid: every block resident
    // (the forward and adjoint kernels of the solve's precision)
    t->mixed = p->precision == CP_PREC_MIXED;
    t->threads = k.n >= kThLarge ? 512 : 256;
    const void* kern[2] = {th_kernel<false>(t), th_kernel<true>(t)};
    int nb = 1 << 30;
    for (const void* f : kern) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, t->threads, 0);
        nb = std::min(nb, b);
    }
    if (nb < 1) return bail(tfail(CP_ERR_CUDA, "the thermal solver kernel does not fit on an SM"));
    t->grid = t->numSMs * std::min(nb, 2);
    const void* mat[4] = {(const void*)k_th_matrix<false, double>, (const void*)k_th_matrix<true, double>,
                          (const void*)k_th_matrix<false, float>, (const void*)k_th_matrix<true, float>};
    for (const void* f : mat)
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kThMatSmemMax) != cudaSuccess)
            return bail(tfail(CP_ERR_CUDA, "the thermal matrix kernel's shared memory (%zu bytes)", kThMatSmemMax));
    if ((s = th_build_hierarchy(t)) != CP_OK) return bail(s);
    if (t->mixed && (s = th_build_float_hierarchy(t)) != CP_OK) return bail(s);
    t->gElem = t->numSMs * 4;
    if ((s = th_alloc(t, &t->part, (size_t)6 * kMaxBlocks)) != CP_OK) return bail(s);
    void* q = nullptr;
    if (t->mem.take(64, &q) != cudaSuccess) return bail(tfail(CP_ERR_CUDA, "cudaMalloc"));
    t->bar = static_cast<unsigned*>(q);
    if (t->mem.take(sizeof(ThStatus), &q) != cudaSuccess) return bail(tfail(CP_ERR_CUDA, "cudaMalloc"));
    t->st = static_cast<ThStatus*>(q);
    if (cudaStreamSynchronize(t->stream) != cudaSuccess) return bail(tfail(CP_ERR_CUDA, "stream"));
    *out = t;
    return CP_OK;
}

cp_status cp_thermal_destroy(cp_thermal* t) {
    if (!t) return CP_OK;
    if (t->stream) cudaStreamSynchronize(t->stream);
    t->mem.give_back();
    if (t->ev0) cudaEventDestroy(t->ev0);
    if (t->ev1) cudaEventDestroy(t->ev1);
    if (t->stream) cudaStreamDestroy(t->stream);
    delete t;
    return CP_OK;
}

cp_status cp_thermal_set_inputs(cp_thermal* t, const double* gamma, const double* u, const double* v,
                                const double* q0) {
    if (!t || !gamma || !u || !v || !q0) return tfail(CP_ERR_BAD_PARAM, "NULL argument");
    const size_t nc = (size_t)t->k.ncol;
    const double* src[] = {gamma, u, v, q0};
    for (const double* a : src)
        for (size_t q = 0; q < nc; ++q)
            if (!std::isfinite(a[q])) return tfail(CP_ERR_NONFINITE, "non-finite input at %zu", q);
    TCK(cudaMemcpyAsync(t->gamma, gamma, nc * 8, cudaMemcpyHostToDevice, t->stream));
    TCK(cudaMemcpyAsync(t->u, u, nc * 8, cudaMemcpyHostToDevice, t->stream));
    TCK(cudaMemcpyAsync(t->v, v, nc * 8, cudaMemcpyHostToDevice, t->stream));
    TCK(cudaMemcpyAsync(t->q0, q0, nc * 8, cudaMemcpyHostToDevice, t->stream));
    TCK(cudaStreamSynchronize(t->stream));
    t->hasInputs = true;
    t->solved = false;
    return CP_OK;
}

cp_status cp_thermal_solve(cp_thermal* t, cp_thermal_report* rep) {
    if (!t) return tfail(CP_ERR_BAD_PARAM, "NULL argument");
    if (!t->hasInputs) return tfail(CP_ERR_STATE, "cp_thermal_set_inputs first");
    const ThK& k = t->k;
    t->solved = false;
    TCK(cudaEventRecord(t->ev0, t->stream));
    k_th_assemble<<<t->gElem, kThThreads, 0, t->stream>>>(k, t->gamma, t->u, t->v, t->q0, t->S);
    TCK(cudaGetLastError());
    // initial guess T = T_inlet
    k_th_fill<<<t->gElem, kThThreads, 0, t->stream>>>(t->V.x, k.n, t->prm.T_inlet);
    TCK(cudaGetLastError());
    for (size_t l = 0; l + 1 < t->lv.size(); ++l) {
        const ThLevel& C = t->lv[l + 1];
        const int g = (int)std::min<long long>(t->gElem, (C.n + kThThreads - 1) / kThThreads);
        k_th_coarsen<<<g, kThThreads, 0, t->stream>>>(k.Nz, t->lv[l], C);
        TCK(cudaGetLastError());
    }
    // mixed precision: the V-cycle's float copies of the operators that it applies
    if (t->mixed)
        for (int l = 0; l < t->H.m; ++l) {
            const ThSys& A = t->lv[l].S;
            const ThSysT<float>& B = t->lvf[l].S;
            const double* src[7] = {A.aP, A.aW, A.aE, A.aS, A.aN, A.aB, A.aT};
            float* dst[7] = {B.aP, B.aW, B.aE, B.aS, B.aN, B.aB, B.aT};
            for (int a = 0; a < 7; ++a) {
                cp_status s = th_narrow(t, src[a], dst[a], t->lv[l].n);
                if (s != CP_OK) return s;
            }
        }
    ThStatus hs;
    cp_status s = th_krylov<false>(t, t->S.b, t->V, &hs);
    if (s != CP_OK) return s;
    t->solved = true;
    th_report(t, hs, rep);
    return CP_OK;
}

cp_status cp_thermal_get_T(cp_thermal* t, double* T) {
    if (!t || !T) return tfail(CP_ERR_BAD_PARAM, "NULL argument");
    if (!t->solved) return tfail(CP_ERR_STATE, "no solution yet (cp_thermal_solve)");
    TCK(cudaMemcpyAsync(T, t->V.x, (size_t)t->k.n * 8, cudaMemcpyDeviceToHost, t->stream));
    TCK(cudaStreamSynchronize(t->stream));
    return CP_OK;
}

cp_status cp_thermal_objective(cp_thermal* t, double p, double* Tb_max, double* Tb_pnorm) {
    if (!t) return tfail(CP_ERR_BAD_PARAM, "NULL argument");
    if (!t->solved) return tfail(CP_ERR_STATE, "no solution yet (cp_thermal_solve)");
    if (!(p > 0.0) || !std::isfinite(p)) return tfail(CP_ERR_BAD_PARAM, "p must be > 0");
    return th_objective(t, p, Tb_max, Tb_pnorm);
}

cp_status cp_thermal_pnorm_gradient(cp_thermal* t, double p, double* J, double* dJ_dgamma, cp_thermal_report* rep) {
    if (!t || !dJ_dgamma) return tfail(CP_ERR_BAD_PARAM, "NULL argument");
    if (!t->solved) return tfail(CP_ERR_STATE, "no solution yet (cp_thermal_solve)");
    if (!(p >= 1.0) || !std::isfinite(p)) return tfail(CP_ERR_BAD_PARAM, "p must be >= 1");
    const ThK& k = t->k;
    double Jv = 0.0;
    cp_status s = th_objective(t, p, nullptr, &Jv);
    if (s != CP_OK) return s;
    if (!(Jv > 0.0) || !std::isfinite(Jv))
        return tfail(CP_ERR_NONFINITE, "the p-norm of the bottom temperatures is %g", Jv);
    TCK(cudaEventRecord(t->ev0, t->stream));
    k_th_adj_rhs<<<t->gElem, kThThreads, 0, t->stream>>>(k, t->V.x, Jv, p, t->rhs);
    TCK(cudaGetLastError());
    TCK(cudaMemsetAsync(t->lam, 0, (size_t)k.n * 8, t->stream));
    ThVecs W = t->V;
    W.x = t->lam;
    ThStatus hs;
    s = th_krylov<true>(t, t->rhs, W, &hs);
    if (s != CP_OK) return s;
    k_th_sens<<<t->gElem, kThThreads, 0, t->stream>>>(k, t->gamma, t->V.x, t->lam, t->grad);
    TCK(cudaGetLastError());
    TCK(cudaEventRecord(t->ev1, t->stream));
    TCK(cudaMemcpyAsync(dJ_dgamma, t->grad, (size_t)k.ncol * 8, cudaMemcpyDeviceToHost, t->stream));
    TCK(cudaStreamSynchronize(t->stream));
    if (J) *J = Jv;
    th_report(t, hs, rep);
    return CP_OK;
}

}  // extern "C"
