// Jacobi-preconditioned CG on the pressure correction (pressureSolverType 1,
// pressure_solver.cpp:121-184):
//   unknowns (i, j) in [1, M-1] x [1, N-2]; p'(:, N-1) = 0;
//   aE = rho dE(i,j) hy, aW = rho dE(i,j-1) hy (j > 1), aN = rho dN(i,j) hx
//   (i < M-1), aS = rho dN(i-1,j) hx (i > 1); aP = aE+aW+aN+aS (1 if < 1e-20).
// Matrix-free on a zero frame: fE(i,j) holds the east-face coefficient (zero
// at j = 0; the outlet's, with no unknown behind it, is in d only) and fN(i,j)
// the north-face one (zero at rows 0 and M-1).
//
// Two passes and two grid barriers an iteration, which is what CG needs:
//   p = z + beta p_old, Ap, p.Ap, and the x += alpha p_old that waited for
//   this read of p_old (sa0_matvec: one element a lane where one row a warp
//   covers the grid, marches of 16 bytes otherwise);
//   r -= alpha Ap, z = r / d, r.r and r.z.
// z is stored (in the rhs array, which the solve consumes first): recomputing
// it at five points cost five divisions a point.  The sums ride on the
// barriers.  An iteration takes 7.1 us instead of 12.0 at 256 x 64, 14.3
// instead of 28.5 at 1024 x 512 and 37 instead of 70 at 1700 x 900 (double).
// The reference's early exits are kept: |p.Ap| < 1e-20 and sqrt(r.r) < pTol,
// and the returned count is the loop index at exit (maxPressureIter if none).
#pragma once

#include "cp_sa.cuh"

namespace cp {

constexpr int kPcgThreads = 512;

// The CG update on the unknowns; returns the shares of r.r and r.z.
template <typename TV>
__device__ __forceinline__ void pcg_update(const Team& T, const Sa0<TV>& A, TV al, TV* __restrict__ r,
                                           const TV* __restrict__ Ap, TV* __restrict__ z, bool vec, double (&acc)[2]) {
    if (vec) {
        constexpr int V = Vec16<TV>::n;
        row_segments<TV>(T, A.nI, A.nJ, [&](int i, int j0, bool act, int) {
            if (!act) return;
            const size_t q = (size_t)i * A.P + j0;
            Vec16<TV> rr = ld16(r + q), zz;
            const Vec16<TV> aa = ld16(Ap + q), dd = ld16(A.d + q);
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const bool in = j0 + k >= 1 && j0 + k <= A.nJ;
                rr.v[k] = rr.v[k] - al * aa.v[k];
                zz.v[k] = in ? rr.v[k] / dd.v[k] : (TV)0;
                acc[0] += (double)rr.v[k] * (double)rr.v[k];
                acc[1] += (double)rr.v[k] * (double)zz.v[k];
            }
            st16(r + q, rr);
            st16(z + q, zz);
        });
    } else {
        sa_cells(SaSplit{T.tid(), T.nth()}, A.nI, A.nJ, [&](int i, int j) {
            const size_t q = (size_t)i * A.P + j;
            const TV rr = r[q] - al * Ap[q], zz = rr / A.d[q];
            r[q] = rr;
            z[q] = zz;
            acc[0] += (double)rr * (double)rr;
            acc[1] += (double)rr * (double)zz;
        });
    }
}

template <typename TV>
__global__ void __launch_bounds__(kPcgThreads, 1) k_pcg(KParams k, Status* st, const double* dE, const double* dN,
                                                        PcgBufs<TV> B, double* pStar, double* part, unsigned* bar) {
    if (st->done) return;
    __shared__ double sm[kReduceSm];
    const Dims d = k.d;
    const int M = d.M, N = d.N, w = N - 2;
    const Team T = grid_team(bar, &st->err);
    const SaSplit all{T.tid(), T.nth()};
    unsigned target = 0;
    // 16-byte accesses need the contexts' layout (rows of a multiple of 32
    // elements from an aligned base); a caller's pitch may be anything
    const bool vec = (d.P & 31) == 0 && (reinterpret_cast<size_t>(B.r) & 15) == 0 && (reinterpret_cast<size_t>(B.fE) & 15) == 0;
    const Sa0<TV> A{B.fE, B.fN, B.d, nullptr, M - 1, w, d.P, (TV)0, (TV)0};
    TV* const z = B.rhs;
    // init: faces, diagonal, r = b (A 0 = 0), z = r / d, r.z
    double acc[2] = {0.0, 0.0};
    sa_cells(all, M - 1, w, [&](int i, int j) {
        const size_t c = at(d, i, j);
        const double aE = k.rho * dE[c] * k.hy;
        const double aW = (j > 1) ? k.rho * dE[c - 1] * k.hy : 0.0;
        const double aN = (i < M - 1) ? k.rho * dN[c] * k.hx : 0.0;
        const double aS = (i > 1) ? k.rho * dN[c - d.P] * k.hx : 0.0;
        double aP = aE + aW + aN + aS;
        if (aP < 1e-20) aP = 1.0;
        B.fE[c] = j < w ? (TV)aE : (TV)0;
        B.fN[c] = (TV)aN;
        B.d[c] = (TV)aP;
        const TV r = z[c], zz = r / (TV)aP;
        B.r[c] = r;
        z[c] = zz;
        acc[1] += (double)r * (double)zz;
    });
    if (!team_reduce(T, target, acc, part, sm)) return;
    double rz = acc[1], beta = 0.0;
    TV al = (TV)0;          // step of the newest direction, not yet in x
    bool pend = false, haveX = false;
    const TV* p = B.pa;
    int it = 0;
    for (; it < k.maxP; ++it) {
        TV* pnew = (it & 1) ? B.pb : B.pa;
        const SaMat<TV> m{z, (it & 1) ? B.pa : B.pb, B.x, pnew, B.Ap, (TV)beta, al, min(it, 2)};
        double v[1] = {vec ? sa0_matvec(T, A, m) : sa0_mat_step<1>(T, A, m)};
        haveX = pend;
        pend = false;
        if (!team_reduce(T, target, v, part, sm)) return;
        if (fabs(v[0]) < 1e-20) break;
        al = (TV)(rz / v[0]);
        p = pnew;
        pend = true;
        acc[0] = acc[1] = 0.0;
        pcg_update(T, A, al, B.r, B.Ap, z, vec, acc);
        if (!team_reduce(T, target, acc, part, sm)) return;
        if (sqrt(acc[0]) < k.pTol) break;
        beta = acc[1] / rz;
        rz = acc[1];
    }
    // p' = x + alpha p (the last step); p'(:, N-1) = 0 (pressure_solver.cpp:814)
    sa_cells(all, M - 1, w, [&](int i, int j) {
        const size_t c = at(d, i, j);
        TV x = haveX ? B.x[c] : (TV)0;
        if (pend) x = x + al * p[c];
        pStar[c] = (double)x;
        if (j == w) pStar[c + 1] = 0.0;
    });
    if (T.lead()) st->itersP = it;
}

}  // namespace cp
