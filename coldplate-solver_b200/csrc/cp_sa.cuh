// Smoothed-aggregation multigrid as the CG preconditioner of the pressure
// correction (pressureSolverType 4).
//
// The reference runs type 4 with AMGCL's AMG-CG: smoothed aggregation
// (amgcl::coarsening::smoothed_aggregation) with SPAI0/Jacobi relaxation as
// the preconditioner of CG (pressure_solver.cu:81-163, cuda_common.cuh:44-53).
// AMGCL is not vendored with the reference and its version is not pinned, so
// this follows the published method on the structured pressure grid, with
// geometric aggregates:
//   * aggregates of 3 x 3 unknowns; tentative prolongation P0 piecewise
//     constant; smoothed prolongation P = (I - w D^-1 A) P0; restriction P^T;
//   * Galerkin coarse operators A_c = P^T A P.  The smoothed support of an
//     aggregate is 5 x 5 fine unknowns, so A_c is a 9-point stencil on the
//     coarse grid;
//   * w = 4 / (3 lambda) with lambda the largest eigenvalue of D^-1 A: 2/3 on
//     the fine 5-point level (lambda near 2) and 0.8 on the 9-point coarse
//     levels (lambda 1.6-1.8 there); on the density workload these fixed
//     weights give the CG counts of power-iteration estimates (12 at
//     512 x 256, 14 at 1024 x 512, emulated in double);
//   * V(1,1) cycle with damped Jacobi (omega 0.9) before and after the
//     coarse correction, a dense inverse on the coarsest level (<= 64
//     unknowns).  The cycle is symmetric, so CG applies.
// A row of P has at most four entries: the unknown's own aggregate and the
// aggregates across its horizontal, vertical and diagonal neighbours (none
// diagonal on the 5-point level 0), so the restriction P^T t is a weighted sum
// over the 5 x 5 support and the prolongation four multiply-adds per unknown.
//
// One CG iteration is a chain of dependent passes over levels that fit the
// L2, so it is bound by the number of grid barriers and by the load latency
// behind each of them (about 1.5 us + 1 us), not by bytes.  Hence:
//   * every pass is a march: a warp owns a strip of columns and a run of
//     rows, reads each row once with the next row's loads in flight, keeps
//     the neighbour rows in registers and gets the horizontal neighbours by
//     shuffles (the outer lanes only supply halo columns).  A smoothing step
//     and the transfer next to it then need no barrier between them: level
//     0's CG update, pre-smoothing, residual and restriction are one pass,
//     prolongation and post-smoothing another, and so is each direction of a
//     coarse level;
//   * level 0's prolongation weights are recomputed from the face
//     coefficients a pass reads anyway, the pre-smoothed iterate from the
//     residual, and x += alpha p waits for the next matvec, which reads p:
//     20 words an unknown and CG iteration on level 0 against 33 with each
//     of them stored;
//   * the V-cycle from the first level with at most kSaApply unknowns down
//     (fewer on a team of CTAs, sa_apply_team) is one symmetric matrix, formed
//     whenever the coarse operators are rebuilt and applied by the whole grid,
//     one warp a row;
//   * block sums ride on the barrier that follows them (team_reduce).
// Barriers a CG iteration: 4 + 2 (grid-wide coarse levels), 10 at
// 2048 x 1024 and 6 at 253 x 127, against 14 and 10 with a barrier between
// every two steps and the small levels on one CTA.  Measured a pressure solve,
// the mean of a density field's first 20 outer iterations (17.1, 17.1, 17.2, 15.6
// CG iterations), before and after: 2048 x 1024 float 2.52 and 1.56 ms, double 3.66
// and 2.11 ms; 811 x 389 float 1.06 and 0.64 ms; 253 x 127 double 0.70 and 0.37 ms.
// The coarse operators are rebuilt every `reuse` outer iterations; the CG
// matvec and level 0's smoother and prolongation always use the current
// operator.  The CG recurrences, the |p.Ap| < 1e-20 exit and AMGCL's
// relative stop rule ||r|| <= pTol ||b|| are those of k_pcg_mg.
#pragma once

#include "cp_mg.cuh"

namespace cp {

constexpr int kSaMaxLevels = 12;
constexpr int kSaDense = 64;         // coarsest level size, inverted by elimination
constexpr int kSaApply = 1024;       // levels at or below this size: their V-cycle is a stored matrix
// The same on a team of CTAs (batches).  A few SMs read the matrix at their own
// rate and form it a column a CTA, so it is the marches over one more level that
// are faster.  us an outer iteration, with that level by its matrix and by marches:
// 24 fields of 90 x 90 (900 unknowns, double), teams of 2 2705 / 961, of 4 1623 /
// 709, of 8 1702 / 1074, of 16 1648 / 1468, of 32 2471 / 2724; 16 of 247 x 130 (420),
// of 2 2516 / 2182, of 4 1497 / 1354, of 8 1048 / 1002, of 16 1441 / 1557; 32 of
// 80 x 40 (378), of 2 781 / 515, of 4 504 / 424, of 8 688 / 711.
inline int sa_apply_team(int ctas) { return ctas < 4 ? 128 * ctas : ctas < 32 ? 512 : kSaApply; }
// dynamic shared memory of the solve: the matrix set-up's iterate with its
// frame (at most 3 x 1026) and coarse correction (at most 342), which the
// restriction's column buffers (1 KB a warp) share
constexpr size_t kSaSmem = sizeof(double) * (3 * (kSaApply + 2) + (kSaApply + 2) / 3 + 64);

// A level: unknowns i in [1, nI], j in [1, nJ] with a zero frame, row pitch P.
// Level 0 keeps its 5-point operator as face coefficients (fE, fN, d of the
// PCG buffers); levels >= 1 hold a 9-point stencil c[k], k = (di+1)*3 + (dj+1),
// c[4] the diagonal, entries towards unknowns outside the level zero.
// pw[0..3]: the prolongation weights of each unknown towards its own,
// horizontal, vertical and diagonal aggregate (every level that has a coarser
// one; zero on the frame; level 0's only for the Galerkin product).
template <typename TV>
struct SaLevel {
    int nI, nJ, P, Pb;      // Pb: pitch of b, P but on the level that is solved by its matrix
    TV* c[9];
    TV *x, *y, *b;          // pre-smoothed iterate, corrected iterate, rhs
    TV* pw[4];
};

// Entries of a stored row of n unknowns.  Rows laid out with the level's pitch (at
// least 32) would be up to 32 times as long on a grid a few columns wide, and every
// CG iteration reads them: 268 MB of 8.4 at 4 x 3070 in double, where an outer
// iteration took 1003 us with them and takes 274 (4 x 2000: 722 and 225).
template <typename TV>
__host__ __device__ __forceinline__ int sa_row(int n) {
    constexpr int V = 16 / (int)sizeof(TV);
    return (n + V - 1) / V * V;
}

template <typename TV>
struct SaHier {
    int L, Ld;              // levels; levels [0, Ld) run grid-wide, level Ld is solved by bm[Ld]
    SaLevel<TV> lv[kSaMaxLevels];
    TV* dinv0;              // level-0 inverse diagonal
    // V-cycle matrices of levels [Ld, L): row q (unknown q, row-major) holds the
    // level's nI nJ entries, without its frame, and zeros up to a whole 16 bytes
    // (sa_row).  Level Ld's right-hand side is stored the same way: b there is
    // nJ + 1 elements ahead of it and Pb = nJ, so that unknown (i, j) is at i Pb + j.
    TV* bm[kSaMaxLevels];
    double omega, w0, wc;   // Jacobi damping, prolongator smoothing weights
    TV* r2;                 // second CG residual buffer (the residual ping-pongs)
    int reuse;              // rebuild the coarse operators every `reuse` outer iterations (0: only when
                            // the stored ones are stale)
    int* built;             // device word: the Ld that the stored hierarchy was built for, 0 when it is stale
    unsigned long long* prof;  // optional per-phase device time (ns, block 0's view), or null
};

// profile slots: set-up, coarse operators, CG matvec, CG update with the
// restriction out of level 0, the stored V-cycle, then the restriction out of
// level l at SA_P_DOWN + l and the prolongation into level l at SA_P_UP + l
enum SaPhase { SA_P_SETUP = 0, SA_P_GALERKIN, SA_P_MATVEC, SA_P_UPDATE, SA_P_DENSE, SA_P_DOWN, SA_P_UP = SA_P_DOWN + kSaMaxLevels,
               SA_P_COUNT = SA_P_UP + kSaMaxLevels };

__host__ __device__ __forceinline__ int sa_coarse(int n) { return (n + 2) / 3; }

struct SaSplit {
    int t0, nt;
};

// cells t0, t0 + nt, ... of a level in row-major order, (i, j) stepped
// without a division per cell
template <typename F>
__device__ __forceinline__ void sa_cells(SaSplit s, int nI, int nJ, F&& fn) {
    const int n = nI * nJ;
    if (s.t0 >= n) return;
    int i = 1 + s.t0 / nJ, j = 1 + s.t0 % nJ;
    const int di = s.nt / nJ, dj = s.nt % nJ;
    for (int t = s.t0; t < n; t += s.nt) {
        fn(i, j);
        i += di;
        j += dj;
        if (j > nJ) {
            j -= nJ;
            ++i;
        }
    }
}

// First task of a warp that takes tasks w, w + nw, ... of n: with fewer tasks
// than warps they are spread over the CTAs (an SM's load queue, not its warps,
// is what a short pass waits for); otherwise neighbouring warps take
// neighbouring tasks, which share rows in the SM's L1.
__device__ __forceinline__ int sa_task(const Team& T, int n, int nw) {
    const int wid = threadIdx.x >> 5;
    return n < nw ? wid * T.size + T.rank : T.rank * (int)(blockDim.x >> 5) + wid;
}

// A march's work: S strips of columns times runs of R rows, as many runs as
// there are warps where the level is large enough; run c covers strip c % S
// (neighbouring warps read neighbouring columns of the same rows).
struct SaRuns {
    int S, R, n;
    __device__ __forceinline__ SaRuns(int strips, int rows, int nw) {
        S = strips;
        R = (rows * strips + nw - 1) / nw;
        n = strips * ((rows + R - 1) / R);
    }
};

// Offset (-1, 0 or +1) of the aggregate across an unknown's horizontal
// (vertical) neighbours when it sits on the first or last column (row) of its
// aggregate; 0 in the middle one.
__device__ __forceinline__ int sa_side(int i) {
    const int r = (i - 1) % 3;
    return r == 0 ? -1 : (r == 2 ? 1 : 0);
}

// ---------------------------------------------------------------- coarse operators
// Row (i, j) of P = (I - w D^-1 A) P0 on a 9-point level: pw[0] towards the
// own aggregate, pw[1] / pw[2] / pw[3] towards the horizontal / vertical /
// diagonal one.
template <typename TV>
__device__ __forceinline__ void sa_pweights(const SaLevel<TV>& f, double w, int i, int j) {
    const int ri = (i - 1) % 3, rj = (j - 1) % 3;
    const size_t q = (size_t)i * f.P + j;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int di = k / 3 - 1, dj = k % 3 - 1;
        const bool oi = ri + di < 0 || ri + di > 2, oj = rj + dj < 0 || rj + dj > 2;
        const double a = (double)f.c[k][q];
#pragma unroll
        for (int m = 0; m < 4; ++m) s[m] += ((oi ? 2 : 0) + (oj ? 1 : 0) == m) ? a : 0.0;
    }
    const double sc = w / (double)f.c[4][q];
    f.pw[0][q] = (TV)(1.0 - sc * s[0]);
    f.pw[1][q] = (TV)(-sc * s[1]);
    f.pw[2][q] = (TV)(-sc * s[2]);
    f.pw[3][q] = (TV)(-sc * s[3]);
}

// Coarse row (I, J) of A_c = P^T A P: the sum over the 5 x 5 support of the
// aggregate of P(m, (I, J)) times row m of A P, whose entries fall on the
// nine coarse neighbours.  Five: level 0 (faces fE, fN, diagonal d; no
// diagonal weight).  Column offsets are compile-time; per fine row the row
// products are gathered per neighbour row and then added to the coarse rows
// they fall on.
template <typename TV, bool Five>
__device__ __forceinline__ void sa_galerkin(const SaLevel<TV>& f, const TV* fE, const TV* fN, const TV* d,
                                            const SaLevel<TV>& C, int I, int J) {
    double ac[3][3];
#pragma unroll
    for (int a = 0; a < 9; ++a) ac[a / 3][a % 3] = 0.0;
    const int j0 = 3 * J - 3;
#pragma unroll 1
    for (int a = 0; a < 5; ++a) {
        const int ii = 3 * I - 3 + a;
        if (ii < 1 || ii > f.nI) continue;
        const bool ra = a == 0 || a == 4;
        // own[di][oj]: towards the aggregate row of fine row ii + di; ver: towards the one across it
        double own[3][3], ver[3][3];
#pragma unroll
        for (int e = 0; e < 9; ++e) own[e / 3][e % 3] = ver[e / 3][e % 3] = 0.0;
#pragma unroll
        for (int b = 0; b < 5; ++b) {
            constexpr int kOff[7] = {-1, -1, 0, 0, 0, 1, 1};     // aggregate column of column j0 + rel, rel + 1
            constexpr int kSide[7] = {0, 1, -1, 0, 1, -1, 0};
            const bool rb = b == 0 || b == 4;
            const int jj = j0 + b;
            if (jj < 1 || jj > f.nJ || (Five && ra && rb)) continue;
            const size_t q = (size_t)ii * f.P + jj;
            const double p = (double)f.pw[(ra ? 2 : 0) + (rb ? 1 : 0)][q];
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const int di = k / 3 - 1, dj = k % 3 - 1;
                if (Five && di != 0 && dj != 0) continue;
                const int ni = ii + di, nj = jj + dj;
                if (ni < 1 || ni > f.nI || nj < 1 || nj > f.nJ) continue;
                double A;
                if (Five)
                    A = k == 4 ? (double)d[q]
                               : -(double)(k == 5 ? fE[q] : k == 3 ? fE[q - 1] : k == 7 ? fN[q] : fN[q - f.P]);
                else A = (double)f.c[k][q];
                const double v = p * A;
                const size_t m = (size_t)ni * f.P + nj;
                const int o = kOff[b + dj + 1] + 1, s = kSide[b + dj + 1];
                own[di + 1][o] += v * (double)f.pw[0][m];
                ver[di + 1][o] += v * (double)f.pw[2][m];
                if (s != 0) {
                    own[di + 1][o + s] += v * (double)f.pw[1][m];
                    if (!Five) ver[di + 1][o + s] += v * (double)f.pw[3][m];
                }
            }
        }
#pragma unroll
        for (int di = -1; di <= 1; ++di) {
            const int rel = a + di;                                  // -1 .. 5; own rows 1 .. 3
            const int o = rel < 1 ? 0 : (rel > 3 ? 2 : 1);
            const int r = (rel + 2) % 3;                             // place in its aggregate
            const int v = o + (r == 0 ? -1 : (r == 2 ? 1 : 0));
#pragma unroll
            for (int e = 0; e < 3; ++e)
#pragma unroll
                for (int c = 0; c < 3; ++c) ac[e][c] += (e == o ? own[di + 1][c] : 0.0) + (e == v && r != 1 ? ver[di + 1][c] : 0.0);
        }
    }
    const size_t qc = (size_t)I * C.P + J;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int di = k / 3 - 1, dj = k % 3 - 1;
        const bool in = I + di >= 1 && I + di <= C.nI && J + dj >= 1 && J + dj <= C.nJ;
        double v = in ? ac[k / 3][k % 3] : 0.0;
        if (k == 4 && !(v > 0.0)) v = 1.0;   // guard: an isolated coarse unknown
        C.c[k][qc] = (TV)v;
    }
}

// Inverse of the coarsest operator (SPD, at most 64 unknowns) by in-place
// Gauss-Jordan on one CTA of 512 threads, eight elements a thread in
// registers, the pivot row and column through double-buffered shared memory
// (one CTA barrier a step); written as the level's V-cycle matrix.
template <typename TV>
__device__ void sa_invert(const SaLevel<TV>& l, TV* bm, double* work /* 4 x 64 */) {
    constexpr int W = kSaDense, K = W * W / 512;
    const int n = l.nI * l.nJ, c = threadIdx.x % W, r0 = threadIdx.x / W;
    double a[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int r = r0 + k * (512 / W);
        a[k] = 0.0;
        if (r < n && c < n) {
            const int i = 1 + r / l.nJ, j = 1 + r % l.nJ, di = 1 + c / l.nJ - i, dj = 1 + c % l.nJ - j;
            if (di >= -1 && di <= 1 && dj >= -1 && dj <= 1) a[k] = (double)l.c[(di + 1) * 3 + dj + 1][(size_t)i * l.P + j];
        }
    }
    for (int s = 0; s < n; ++s) {
        double* row = work + (s & 1) * 2 * W;
        double* col = row + W;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int r = r0 + k * (512 / W);
            if (r == s) row[c] = a[k];
            if (c == s) col[r] = a[k];
        }
        __syncthreads();
        const double ip = 1.0 / row[s], rc = row[c] * ip;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int r = r0 + k * (512 / W);
            if (r == s) a[k] = c == s ? ip : rc;
            else a[k] = c == s ? -a[k] * ip : a[k] - col[r] * rc;
        }
    }
    const int len = sa_row<TV>(n);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int r = r0 + k * (512 / W);
        if (r < n && c < n) bm[(size_t)r * len + c] = (TV)a[k];
    }
    __syncthreads();
}

// The V-cycle matrix B of level f from the one of the next level C: column q
// is the V-cycle of the unit vector e_q, and B is symmetric, so it is stored
// as row q.  One CTA a column:
//   r = e_q - A x with x = omega e_q / d_q has at most nine entries; P^T r at
//   most nine, on the coarse neighbours of q's aggregate; e = B_C P^T r;
//   t = x + P e; y = t + omega (e_q - A t) / d.
template <typename TV>
__device__ __forceinline__ void sa_matrix(const Team& T, const SaLevel<TV>& f, const SaLevel<TV>& C, const TV* bc, TV* bm,
                          double om, double* work) {
    const int n = f.nI * f.nJ, nc = C.nI * C.nJ, Pt = f.nJ + 2;
    double* t = work;                        // (nI + 2) x (nJ + 2), zero frame
    double* e = t + (f.nI + 2) * Pt;         // coarse correction
    double* rr = e + nc;                     // nine residual entries, then P^T r
    const int len = sa_row<TV>(n), lenc = sa_row<TV>(nc), tx = threadIdx.x;
    for (int q = tx; q < (f.nI + 2) * Pt; q += blockDim.x) t[q] = 0.0;
    __syncthreads();
    for (int q = T.rank; q < n; q += T.size) {
        const int i = 1 + q / f.nJ, j = 1 + q % f.nJ;
        const int Ia = (i - 1) / 3 + 1, Ja = (j - 1) / 3 + 1;
        const double xq = om / (double)f.c[4][(size_t)i * f.P + j];
        if (tx < 9) {
            const int ii = i + tx / 3 - 1, jj = j + tx % 3 - 1;
            double r = 0.0;
            if (ii >= 1 && ii <= f.nI && jj >= 1 && jj <= f.nJ)
                r = (tx == 4 ? 1.0 : 0.0) - (double)f.c[8 - tx][(size_t)ii * f.P + jj] * xq;
            rr[tx] = r;
        }
        __syncthreads();
        if (tx < 9) {
            const int I = Ia + tx / 3 - 1, J = Ja + tx % 3 - 1;
            double s = 0.0;
            for (int k = 0; k < 9; ++k) {
                const int ii = i + k / 3 - 1, jj = j + k % 3 - 1;
                if (ii < 1 || ii > f.nI || jj < 1 || jj > f.nJ) continue;
                const int Io = (ii - 1) / 3 + 1, Jo = (jj - 1) / 3 + 1, sv = sa_side(ii), sh = sa_side(jj);
                const bool ov = I == Io, oh = J == Jo, av = sv != 0 && I == Io + sv, ah = sh != 0 && J == Jo + sh;
                if ((ov || av) && (oh || ah)) s += (double)f.pw[(av ? 2 : 0) + (ah ? 1 : 0)][(size_t)ii * f.P + jj] * rr[k];
            }
            rr[16 + tx] = (I >= 1 && I <= C.nI && J >= 1 && J <= C.nJ) ? s : 0.0;
        }
        __syncthreads();
        for (int c = tx; c < nc; c += blockDim.x) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const int I = Ia + k / 3 - 1, J = Ja + k % 3 - 1;
                if (I >= 1 && I <= C.nI && J >= 1 && J <= C.nJ)
                    s += (double)bc[(size_t)((I - 1) * C.nJ + J - 1) * lenc + c] * rr[16 + k];
            }
            e[c] = s;
        }
        __syncthreads();
        for (int c = tx; c < n; c += blockDim.x) {
            const int ii = 1 + c / f.nJ, jj = 1 + c % f.nJ;
            const size_t m = (size_t)ii * f.P + jj;
            const int Io = (ii - 1) / 3, Jo = (jj - 1) / 3, sv = sa_side(ii), sh = sa_side(jj);
            const bool iv = Io + sv >= 0 && Io + sv < C.nI, ih = Jo + sh >= 0 && Jo + sh < C.nJ;
            double s = (c == q ? xq : 0.0) + (double)f.pw[0][m] * e[Io * C.nJ + Jo];
            if (sh != 0 && ih) s += (double)f.pw[1][m] * e[Io * C.nJ + Jo + sh];
            if (sv != 0 && iv) s += (double)f.pw[2][m] * e[(Io + sv) * C.nJ + Jo];
            if (sv != 0 && sh != 0 && iv && ih) s += (double)f.pw[3][m] * e[(Io + sv) * C.nJ + Jo + sh];
            t[ii * Pt + jj] = s;
        }
        __syncthreads();
        for (int c = tx; c < n; c += blockDim.x) {
            const int ii = 1 + c / f.nJ, jj = 1 + c % f.nJ;
            const size_t m = (size_t)ii * f.P + jj;
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < 9; ++k) s += (double)f.c[k][m] * t[(ii + k / 3 - 1) * Pt + jj + k % 3 - 1];
            bm[(size_t)q * len + c] =
                (TV)(t[ii * Pt + jj] + om * ((c == q ? 1.0 : 0.0) - s) / (double)f.c[4][m]);
        }
    }
    __syncthreads();
}

// y = B b on the stored level, one warp a row, 16-byte loads
template <typename TV>
__device__ __forceinline__ void sa_apply(const Team& T, const SaLevel<TV>& f, const TV* __restrict__ bm) {
    constexpr int V = Vec16<TV>::n;
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int n = f.nI * f.nJ, len = sa_row<TV>(n);
    const TV* b = f.b + (f.nJ + 1);
    for (int q = sa_task(T, n, nw); q < n; q += nw) {
        const TV* row = bm + (size_t)q * len;
        double s = 0.0;
        // several loads in flight whatever the row's length: a loop of single ones
        // waited for each on rows shorter than four trips (0.6 and 1.1 us a CG
        // iteration at 1200 x 600 and 20000 x 100); in double four of m and b at
        // once cost the other passes registers (2048 x 1024: 1836 and 1814 us a
        // solve, float the other way round)
        constexpr int U = sizeof(TV) == 4 ? 4 : 2;
#pragma unroll 2
        for (int e = lane * V; e < len; e += 32 * U * V) {
            Vec16<TV> m[U], v[U];
#pragma unroll
            for (int h = 0; h < U; ++h) {
                const bool on = e + 32 * V * h < len;
                m[h] = on ? ld16(row + e + 32 * V * h) : zero16<TV>();
                v[h] = on ? ld16(b + e + 32 * V * h) : zero16<TV>();
            }
#pragma unroll
            for (int h = 0; h < U; ++h) {
                TV u = m[h].v[0] * v[h].v[0];
#pragma unroll
                for (int k = 1; k < V; ++k) u += m[h].v[k] * v[h].v[k];
                s += (double)u;
            }
        }
        s = warp_sum(s);
        if (lane == 0) f.y[(size_t)(1 + q / f.nJ) * f.P + 1 + q % f.nJ] = (TV)s;
    }
}

// ---------------------------------------------------------------- grid-wide coarse levels
template <int N>
struct SaInt {
    static constexpr int value = N;
};

// Three horizontal neighbours of one row
template <typename TV>
struct SaTriple {
    TV w, c, e;
};
template <typename TV>
__device__ __forceinline__ SaTriple<TV> sa_triple(TV v) { return {from_west(v), v, from_east(v)}; }

// a . x over the nine neighbours, x row by row
template <typename TV, typename X>
__device__ __forceinline__ double sa_dot9(const TV (&a)[9], const SaTriple<X>& s, const SaTriple<X>& c, const SaTriple<X>& n) {
    double v = (double)a[0] * (double)s.w + (double)a[1] * (double)s.c + (double)a[2] * (double)s.e;
    v += (double)a[3] * (double)c.w + (double)a[4] * (double)c.c + (double)a[5] * (double)c.e;
    v += (double)a[6] * (double)n.w + (double)a[7] * (double)n.c + (double)a[8] * (double)n.e;
    return v;
}

// Restriction out of a coarse level, one row of aggregates of one strip a
// warp and step, every load issued before the first use: t = b - A x (x the
// pre-smoothed iterate) on the support's five rows, b_c = P^T t,
// x_c = omega b_c / d_c (unless C is solved by its matrix).  Lane L of strip s
// holds column 27 s - 1 + L; t is complete on lanes 1 .. 30, which covers the
// supports of the strip's nine aggregates.
template <typename TV>
__device__ __forceinline__ void sa_down(const Team& T, const SaLevel<TV>& f, const SaLevel<TV>& C, double om, bool last) {
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int S = (C.nJ + 8) / 9, n = S * C.nI;
    for (int c = sa_task(T, n, nw); c < n; c += nw) {
        const int s = c % S, I = 1 + c / S;
        const int col = 27 * s - 1 + lane, r0 = 3 * I - 3;
        const bool act = col >= 1 && col <= f.nJ;
        const int J = 9 * s + 1 + lane;
        const bool out = lane < 9 && J <= C.nJ;
        const size_t qc = (size_t)I * C.Pb + J;
        TV x[7];
#pragma unroll
        for (int r = 0; r < 7; ++r) {
            const int i = r0 - 1 + r;
            x[r] = act && i >= 1 && i <= f.nI ? f.x[(size_t)i * f.P + col] : (TV)0;
        }
        const TV d = out && !last ? C.c[4][qc] : (TV)1;
        double vO = 0.0, vH = 0.0;
        // the aggregates' own rows, then the two ring rows: all five at once
        // do not fit the registers, and what spills comes back from the L2,
        // since every barrier empties the L1
        auto rows = [&](auto first, auto count, auto stride) {
            constexpr int r1 = decltype(first)::value, n = decltype(count)::value, st = decltype(stride)::value;
            TV a[n][9], b[n], p[n][2];
#pragma unroll
            for (int h = 0; h < n; ++h) {
                const int r = r1 + h * st, i = r0 + r, m = (r == 0 || r == 4) ? 2 : 0;
                const bool in = act && i >= 1 && i <= f.nI;
                const size_t q = (size_t)i * f.P + col;
#pragma unroll
                for (int k = 0; k < 9; ++k) a[h][k] = in ? f.c[k][q] : (TV)0;
                b[h] = in ? f.b[q] : (TV)0;
                p[h][0] = in ? f.pw[m][q] : (TV)0;
                p[h][1] = in ? f.pw[m + 1][q] : (TV)0;
            }
#pragma unroll
            for (int h = 0; h < n; ++h) {
                const int r = r1 + h * st;
                const double t = (double)b[h] - sa_dot9(a[h], sa_triple(x[r]), sa_triple(x[r + 1]), sa_triple(x[r + 2]));
                vO += (double)p[h][0] * t;
                vH += (double)p[h][1] * t;
            }
        };
        rows(SaInt<1>{}, SaInt<3>{}, SaInt<1>{});
        rows(SaInt<0>{}, SaInt<2>{}, SaInt<4>{});
        const double h0 = __shfl_sync(0xffffffffu, vH, 3 * lane + 1), o1 = __shfl_sync(0xffffffffu, vO, 3 * lane + 2),
                     o2 = __shfl_sync(0xffffffffu, vO, 3 * lane + 3), o3 = __shfl_sync(0xffffffffu, vO, 3 * lane + 4),
                     h4 = __shfl_sync(0xffffffffu, vH, 3 * lane + 5);
        if (out) {
            const double v = ((h0 + o1) + (o2 + o3)) + h4;
            C.b[qc] = (TV)v;
            if (!last) C.x[qc] = (TV)(om * v / (double)d);
        }
    }
}

// Prolongation into a coarse level and its post-smoothing, one row of one
// strip a warp and step: t = x + P e on the row and its two neighbours,
// y = t + omega (b - A t) / d.  Lane L of strip s holds column 30 s + L and
// writes on lanes 1 .. 30.
template <typename TV>
__device__ __forceinline__ void sa_up(const Team& T, const SaLevel<TV>& f, const SaLevel<TV>& C, double om) {
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int S = (f.nJ + 29) / 30, n = S * f.nI;
    const TV* e = C.y;
    for (int c = sa_task(T, n, nw); c < n; c += nw) {
        const int s = c % S, i = 1 + c / S;
        const int col = 30 * s + lane;
        const bool act = col >= 1 && col <= f.nJ, own = act && lane >= 1 && lane <= 30;
        const int J = act ? (col - 1) / 3 + 1 : 0, Jh = act ? J + sa_side(col) : 0;
        const size_t qy = (size_t)i * f.P + col;
        TV x[3], p[3][4], g[3][4], a[9], b;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int ii = i - 1 + r;
            const bool in = act && ii >= 1 && ii <= f.nI;
            const size_t q = (size_t)ii * f.P + col;
            // frame entries of e are zero, so an unknown outside reads those
            const int I = in ? (ii - 1) / 3 + 1 : 0, Iv = in ? I + sa_side(ii) : 0;
            x[r] = in ? f.x[q] : (TV)0;
#pragma unroll
            for (int k = 0; k < 4; ++k) p[r][k] = in ? f.pw[k][q] : (TV)0;
            g[r][0] = e[(size_t)I * C.P + J];
            g[r][1] = e[(size_t)I * C.P + Jh];
            g[r][2] = e[(size_t)Iv * C.P + J];
            g[r][3] = e[(size_t)Iv * C.P + Jh];
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) a[k] = own ? f.c[k][qy] : (TV)1;
        b = own ? f.b[qy] : (TV)0;
        SaTriple<double> t[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double v = (double)x[r];
#pragma unroll
            for (int k = 0; k < 4; ++k) v += (double)p[r][k] * (double)g[r][k];
            t[r] = sa_triple(v);
        }
        if (own) f.y[qy] = (TV)(t[1].c + om * ((double)b - sa_dot9(a, t[0], t[1], t[2])) / (double)a[4]);
    }
}

// The two transfers as marches over rows, for teams of a few CTAs (batches),
// whose warps each have many rows of a level: t of a row is formed once instead
// of 5/3 times and three times, and what a team is short of is instructions, not
// loads in flight.  24 batched fields, 20 iterations: 156 ms with the steps
// above, 140 with these.  On the whole grid the steps are the faster ones
// (level 1 of 2048 x 1024 excepted, and there the registers of both forms
// together cost more in the passes over level 0 than the march saves).
template <typename TV>
__device__ __forceinline__ void sa_down_march(const Team& T, const SaLevel<TV>& f, const SaLevel<TV>& C, double om, bool last) {
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const SaRuns W((C.nJ + 8) / 9, C.nI, nw);
    for (int c = sa_task(T, W.n, nw); c < W.n; c += nw) {
        const int s = c % W.S, I0 = 1 + (c / W.S) * W.R, I1 = min(C.nI, I0 + W.R - 1);
        const int col = 27 * s - 1 + lane;
        const bool act = col >= 1 && col <= f.nJ;
        const int J = 9 * s + 1 + lane;
        const bool out = lane < 9 && J <= C.nJ;
        auto ldx = [&](int r) -> TV { return act && r >= 1 && r <= f.nI ? f.x[(size_t)r * f.P + col] : (TV)0; };
        const int rb = 3 * I0 - 3, re = 3 * I1 + 1;
        SaTriple<TV> xs = sa_triple(ldx(rb - 1)), xc = sa_triple(ldx(rb));
        // the ring row above waits for the emission, where its terms come after
        // the own rows' as in sa_down: the same sums to the last bit
        double vO = 0.0, vH = 0.0, tA = 0.0, tR = 0.0;
        TV pA[2] = {(TV)0, (TV)0}, pR[2] = {(TV)0, (TV)0};
        int role = 2, I = I0 - 1;
        for (int r = rb; r <= re; ++r) {
            const bool in = act && r >= 1 && r <= f.nI;
            const size_t q = (size_t)r * f.P + col;
            TV a[9], b = (TV)0, p[4];
#pragma unroll
            for (int k = 0; k < 9; ++k) a[k] = in ? f.c[k][q] : (TV)0;
#pragma unroll
            for (int k = 0; k < 4; ++k) p[k] = in ? f.pw[k][q] : (TV)0;
            if (in) b = f.b[q];
            TV d = (TV)1;
            if (role == 0 && out && !last && I >= I0) d = C.c[4][(size_t)I * C.P + J];
            const SaTriple<TV> xn = sa_triple(ldx(r + 1));
            const double t = (double)b - sa_dot9(a, xs, xc, xn);
            xs = xc;
            xc = xn;
            if (role == 0) {
                // the ring row below the previous aggregate completes it
                vO += (double)pR[0] * tR;
                vH += (double)pR[1] * tR;
                vO += (double)p[2] * t;
                vH += (double)p[3] * t;
                const double h0 = __shfl_sync(0xffffffffu, vH, 3 * lane + 1), o1 = __shfl_sync(0xffffffffu, vO, 3 * lane + 2),
                             o2 = __shfl_sync(0xffffffffu, vO, 3 * lane + 3), o3 = __shfl_sync(0xffffffffu, vO, 3 * lane + 4),
                             h4 = __shfl_sync(0xffffffffu, vH, 3 * lane + 5);
                if (I >= I0 && out) {
                    const double v = ((h0 + o1) + (o2 + o3)) + h4;
                    const size_t qc = (size_t)I * C.Pb + J;
                    C.b[qc] = (TV)v;
                    if (!last) C.x[qc] = (TV)(om * v / (double)d);
                }
                ++I;
                vO = vH = 0.0;
                tR = tA;
                pR[0] = pA[0];
                pR[1] = pA[1];
            }
            vO += (double)p[0] * t;
            vH += (double)p[1] * t;
            tA = t;
            pA[0] = p[2];
            pA[1] = p[3];
            role = role == 2 ? 0 : role + 1;
        }
    }
}

template <typename TV>
__device__ __forceinline__ void sa_up_march(const Team& T, const SaLevel<TV>& f, const SaLevel<TV>& C, double om) {
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const SaRuns W((f.nJ + 29) / 30, f.nI, nw);
    const TV* e = C.y;
    for (int c = sa_task(T, W.n, nw); c < W.n; c += nw) {
        const int s = c % W.S, i0 = 1 + (c / W.S) * W.R, i1 = min(f.nI, i0 + W.R - 1);
        const int col = 30 * s + lane;
        const bool act = col >= 1 && col <= f.nJ, own = act && lane >= 1 && lane <= 30;
        const int J = act ? (col - 1) / 3 + 1 : 0, Jh = act ? J + sa_side(col) : 0;
        auto ldO = [&](int I) -> TV { return e[(size_t)I * C.P + J]; };
        auto ldH = [&](int I) -> TV { return e[(size_t)I * C.P + Jh]; };
        const int rb = max(i0 - 1, 1), re = i1 + 1;
        int I = (rb - 1) / 3 + 1, role = (rb - 1) % 3;
        TV oP = ldO(I - 1), hP = ldH(I - 1), oC = ldO(I), hC = ldH(I), oN = ldO(I + 1), hN = ldH(I + 1);
        SaTriple<double> ts = {0.0, 0.0, 0.0}, tc = ts;
        for (int r = rb; r <= re; ++r) {
            // y of row r - 1 needs its operator row; loaded with row r's weights
            const int ry = r - 1;
            const bool yr = own && ry >= i0;
            const size_t q = (size_t)r * f.P + col, qy = q - f.P;
            const bool in = act && r <= f.nI;
            TV a[9], b = (TV)0, p[4], x = (TV)0;
#pragma unroll
            for (int k = 0; k < 9; ++k) a[k] = yr ? f.c[k][qy] : (TV)0;
#pragma unroll
            for (int k = 0; k < 4; ++k) p[k] = in ? f.pw[k][q] : (TV)0;
            if (yr) b = f.b[qy];
            if (in) x = f.x[q];
            const TV oV = role == 0 ? oP : oN, hV = role == 0 ? hP : hN;
            double t = (double)x;
            t += (double)p[0] * (double)oC;
            t += (double)p[1] * (double)hC;
            if (role != 1) {
                t += (double)p[2] * (double)oV;
                t += (double)p[3] * (double)hV;
            }
            const SaTriple<double> tn = sa_triple(t);
            if (yr) {
                f.y[qy] = (TV)(tc.c + om * ((double)b - sa_dot9(a, ts, tc, tn)) / (double)a[4]);
            }
            ts = tc;
            tc = tn;
            if (++role == 3) {
                role = 0;
                ++I;
                oP = oC; hP = hC;
                oC = oN; hC = hN;
                if (r < re && I + 1 <= C.nI + 1) { oN = ldO(I + 1); hN = ldH(I + 1); }
            }
        }
    }
}

// ---------------------------------------------------------------- level 0
// Level 0's operator: face coefficients fE (east), fN (north), the diagonal
// d and its inverse.  The passes form the weights of P in TV from them; the
// Galerkin product has them from the double set-up, so in float the two P differ by
// roundings (the CG counts over 60 outer iterations are those of weights rounded
// once: 751, 781, 825, 841 and 883 from 120 x 60 to 2048 x 1024).  Every level-0 array is zero on the frame (only the
// unknowns are ever written) and fE / fN are zero on the frame rows and
// columns, so the passes read neighbours without range checks.  The outlet
// face (east of the last column, with no unknown behind it) is in d only: with
// a zero in fE the frame column behind it needs no mask either.  Arithmetic in
// TV.
//
// Each pass has two forms.  A march (sa0_*_march) takes 16 bytes a lane and a
// run of rows a warp, with the next row's loads in flight.  A step
// (sa0_*_step) takes one row (one row of aggregates) a warp with V elements a
// lane and issues every load before the first use; V is the smallest with
// which the grid covers the level in one step.  Below that size a pass is one
// load latency long, and a march would wait for one at every row.
template <typename TV>
struct Sa0 {
    const TV *fE, *fN, *d, *dinv;
    int nI, nJ, P;
    TV om, w0;
};

// Per-lane constants of the prolongation weights of a vector of columns:
// whether the west face of column k stays inside the aggregate (in[k % 3], 0
// or 1; the east face's is in[(k + 1) % 3])
template <typename TV>
struct SaCols {
    TV in[3];
    __device__ __forceinline__ explicit SaCols(int j0) {
        const int c = (j0 + 2 + 3 * 1024) % 3;   // column j0's place in its aggregate (j0 >= -4)
        in[0] = c != 0 ? (TV)1 : (TV)0;
        in[1] = c != 2 ? (TV)1 : (TV)0;
        in[2] = c != 1 ? (TV)1 : (TV)0;
    }
};

// Row i's weights of P times wd = w / d from its faces: own 1 - w + wd * same,
// horizontal wd * fh, vertical wd * (fs on an aggregate's first row, fn on its
// last one)
template <typename TV, int V>
__device__ __forceinline__ void sa0_faces(const SaCols<TV>& K, const VecN<TV, V>& fe, TV fw, const VecN<TV, V>& fn,
                                          const VecN<TV, V>& fs, int role, TV (&same)[V], TV (&fh)[V]) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const TV FW = k ? fe.v[k ? k - 1 : 0] : fw, wI = K.in[k % 3] * FW, eI = K.in[(k + 1) % 3] * fe.v[k];
        TV s = wI + eI;
        if (role != 2) s += fn.v[k];
        if (role != 0) s += fs.v[k];
        same[k] = s;
        fh[k] = (FW - wI) + (fe.v[k] - eI);
    }
}

// (A p) on one row from p on it and its neighbour rows; returns p.Ap
template <typename TV, int V>
__device__ __forceinline__ double sa0_row_ap(bool own, const VecN<TV, V>& ps, const VecN<TV, V>& pc,
                                             const VecN<TV, V>& pn, const VecN<TV, V>& d, const VecN<TV, V>& fe,
                                             const VecN<TV, V>& fn, const VecN<TV, V>& fs, VecN<TV, V>& ap) {
    const TV pw = from_west(pc.v[V - 1]), pe = from_east(pc.v[0]), fw = from_west(fe.v[V - 1]);
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const TV W = k ? pc.v[k ? k - 1 : 0] : pw, E = k < V - 1 ? pc.v[k < V - 1 ? k + 1 : 0] : pe, FW = k ? fe.v[k ? k - 1 : 0] : fw;
        TV a = d.v[k] * pc.v[k] - fe.v[k] * E - FW * W - fn.v[k] * pn.v[k] - fs.v[k] * ps.v[k];
        ap.v[k] = a;
        if (own) acc += (double)pc.v[k] * (double)a;
    }
    return acc;
}

// CG matvec on p = z + beta p_old, and the x += alpha_old p_old that the last
// update left: lane L of strip s holds columns [(30 s - 1 + L) V, + V) and
// writes on lanes 1 .. 30.  mode 0: the first matvec (p = z); 1: the second
// (x = alpha p_old); 2: later ones.  Returns the lane's share of p.Ap.
template <typename TV>
struct SaMat {
    const TV *z, *pold;
    TV *x, *pnew, *Ap;
    TV bt, al;
    int mode;
};

template <int V, typename TV>
__device__ __forceinline__ VecN<TV, V> sa0_dir(const SaMat<TV>& m, const VecN<TV, V>& z, const VecN<TV, V>& o) {
    if (m.mode == 0) return z;
    VecN<TV, V> p;
#pragma unroll
    for (int k = 0; k < V; ++k) p.v[k] = (TV)(z.v[k] + m.bt * o.v[k]);
    return p;
}

template <int V, typename TV>
__device__ __forceinline__ double sa0_mat_step(const Team& T, const Sa0<TV>& A, const SaMat<TV>& m) {
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int P = A.P, Ga = A.nJ / V + 1, S = (Ga + 29) / 30, n = S * A.nI;
    double acc = 0.0;
    for (int c = sa_task(T, n, nw); c < n; c += nw) {
        const int s = c % S, i = 1 + c / S, g = 30 * s - 1 + lane, j0 = g * V;
        const bool act = g >= 0 && g < Ga, own = act && lane >= 1 && lane <= 30;
        const size_t q = (size_t)i * P + j0;
        VecN<TV, V> z[3], o[3], d = zerov<TV, V>(), fe = d, fn = d, fs = d, xx = d, ap;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            z[r] = act ? ldv<V>(m.z + (q - P + (size_t)r * P)) : zerov<TV, V>();
            o[r] = act && m.mode ? ldv<V>(m.pold + (q - P + (size_t)r * P)) : zerov<TV, V>();
        }
        if (act) {
            d = ldv<V>(A.d + q);
            fe = ldv<V>(A.fE + q);
            fn = ldv<V>(A.fN + q);
            fs = ldv<V>(A.fN + (q - P));
            if (m.mode == 2 && own) xx = ldv<V>(m.x + q);
        }
        const VecN<TV, V> ps = sa0_dir<V>(m, z[0], o[0]), pc = sa0_dir<V>(m, z[1], o[1]), pn = sa0_dir<V>(m, z[2], o[2]);
        acc += sa0_row_ap(own, ps, pc, pn, d, fe, fn, fs, ap);
        if (own) {
            stv(m.pnew + q, pc);
            stv(m.Ap + q, ap);
            if (m.mode) {
#pragma unroll
                for (int k = 0; k < V; ++k) xx.v[k] = xx.v[k] + m.al * o[1].v[k];
                stv(m.x + q, xx);
            }
        }
    }
    return acc;
}

template <typename TV>
__device__ __forceinline__ double sa0_mat_march(const Team& T, const Sa0<TV>& A, const SaMat<TV>& m) {
    constexpr int V = Vec16<TV>::n;
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int P = A.P, Ga = A.nJ / V + 1;
    const SaRuns W((Ga + 29) / 30, A.nI, nw);
    double acc = 0.0;
    for (int c = sa_task(T, W.n, nw); c < W.n; c += nw) {
        const int s = c % W.S, i0 = 1 + (c / W.S) * W.R, i1 = min(A.nI, i0 + W.R - 1);
        const int g = 30 * s - 1 + lane, j0 = g * V;
        const bool act = g >= 0 && g < Ga, own = act && lane >= 1 && lane <= 30;
        auto ld = [&](const TV* f, int r, bool on) { return on ? ldv<V>(f + (size_t)r * P + j0) : zerov<TV, V>(); };
        const bool ao = act && m.mode, ox = own && m.mode == 2;
        // row i's d, faces and x, and the directions of rows i .. i + 1, are in registers when its turn comes
        VecN<TV, V> zS = ld(m.z, i0 - 1, act), zC = ld(m.z, i0, act), zN = ld(m.z, i0 + 1, act);
        VecN<TV, V> oS = ld(m.pold, i0 - 1, ao), oC = ld(m.pold, i0, ao), oN = ld(m.pold, i0 + 1, ao);
        VecN<TV, V> fs = ld(A.fN, i0 - 1, act), d = ld(A.d, i0, act), fe = ld(A.fE, i0, act), fn = ld(A.fN, i0, act),
                    xx = ld(m.x, i0, ox);
        VecN<TV, V> ps = sa0_dir<V>(m, zS, oS), pc = sa0_dir<V>(m, zC, oC);
#pragma unroll 3
        for (int i = i0; i <= i1; ++i) {
            const size_t q = (size_t)i * P + j0;
            const bool more = i < i1;
            const VecN<TV, V> zF = ld(m.z, i + 2, act && more), oF = ld(m.pold, i + 2, ao && more),
                              dF = ld(A.d, i + 1, act && more), feF = ld(A.fE, i + 1, act && more),
                              fnF = ld(A.fN, i + 1, act && more), xF = ld(m.x, i + 1, ox && more);
            const VecN<TV, V> pn = sa0_dir<V>(m, zN, oN);
            VecN<TV, V> ap;
            acc += sa0_row_ap(own, ps, pc, pn, d, fe, fn, fs, ap);
            if (own) {
                stv(m.pnew + q, pc);
                stv(m.Ap + q, ap);
                if (m.mode) {
#pragma unroll
                    for (int k = 0; k < V; ++k) xx.v[k] = xx.v[k] + m.al * oC.v[k];
                    stv(m.x + q, xx);
                }
            }
            ps = pc; pc = pn;
            fs = fn; fn = fnF; fe = feF; d = dF; xx = xF;
            oC = oN; oN = oF; zN = zF;
        }
    }
    return acc;
}

// steps of one element (or two floats) a lane where one step a warp covers the level
template <typename TV>
__device__ __forceinline__ double sa0_matvec(const Team& T, const Sa0<TV>& A, const SaMat<TV>& m) {
    const int nw = T.nth() >> 5;
    if ((A.nJ + 30) / 30 * A.nI <= nw) return sa0_mat_step<1>(T, A, m);
    if constexpr (sizeof(TV) == 4)
        if ((A.nJ / 2 + 30) / 30 * A.nI <= nw) return sa0_mat_step<2>(T, A, m);
    return sa0_mat_march(T, A, m);
}

// CG update and the descent out of level 0 in one pass: r' = r - alpha Ap
// (into rn; first: r' = r, nothing written), the pre-smoothed iterate
// x0 = omega r' / d, its residual t = r' - A x0 = (1 - omega) r' + sum over
// the faces of f x0(neighbour), b_c = P^T t and x_c = omega b_c / d_c.  Lane L
// of strip s holds columns [(27 s - 1 + L) V, + V); r' is written on lanes
// 1 .. 27, t is complete on lanes 1 .. 30, and the strip's 9 V aggregates
// have their supports inside those.  buf: 64 vectors of shared memory a warp.
// Returns the lane's share of |r'|^2.
template <typename TV>
struct SaDown {
    const TV *r, *Ap;
    TV* rn;
    TV al;
    bool first, last;
    double omC;
    TV* buf;
};

// t of one row and its contributions to the aggregates: O to the own one, H to
// the horizontal one, X (an aggregate's first and last row) to the one across
template <typename TV, int V>
__device__ __forceinline__ void sa0_row_down(const Sa0<TV>& A, const SaCols<TV>& K, bool in, int role,
                                             const VecN<TV, V>& r, const VecN<TV, V>& di, const VecN<TV, V>& xs,
                                             const VecN<TV, V>& xc, const VecN<TV, V>& xn, const VecN<TV, V>& fe,
                                             const VecN<TV, V>& fn, const VecN<TV, V>& fs, VecN<TV, V>& qO,
                                             VecN<TV, V>& qH, VecN<TV, V>& qX) {
    const TV xw = from_west(xc.v[V - 1]), xe = from_east(xc.v[0]), fw = from_west(fe.v[V - 1]);
    TV same[V], fh[V];
    sa0_faces(K, fe, fw, fn, fs, role, same, fh);
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const TV W = k ? xc.v[k ? k - 1 : 0] : xw, E = k < V - 1 ? xc.v[k < V - 1 ? k + 1 : 0] : xe, FW = k ? fe.v[k ? k - 1 : 0] : fw;
        TV t = ((TV)1 - A.om) * r.v[k] + fe.v[k] * E + FW * W + fn.v[k] * xn.v[k] + fs.v[k] * xs.v[k];
        if (!in) t = (TV)0;
        const TV wd = A.w0 * di.v[k] * t;
        qO.v[k] = ((TV)1 - A.w0) * t + wd * same[k];
        qH.v[k] = wd * fh[k];
        qX.v[k] = role == 0 ? wd * fs.v[k] : (role == 2 ? wd * fn.v[k] : (TV)0);
    }
}

// one strip's row of coarse values from the column sums: aggregate J has the
// own sums of columns 3J - 2 .. 3J and the horizontal ones of 3J - 3, 3J + 1
template <typename TV, int V>
__device__ __forceinline__ void sa0_gather(const SaLevel<TV>& C, int s, int I, const VecN<TV, V>& vO, const VecN<TV, V>& vH,
                                           double omC, bool last, TV* buf) {
    const int lane = threadIdx.x & 31;
    TV* bO = buf + (threadIdx.x >> 5) * 64 * Vec16<TV>::n;
    TV* bH = bO + 32 * Vec16<TV>::n;
    stv(bO + lane * V, vO);
    stv(bH + lane * V, vH);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < (9 * V + 31) / 32; ++h) {
        const int m = lane + 32 * h, J = 9 * V * s + 1 + m, e = V + 3 * m;
        if (m < 9 * V && J <= C.nJ) {
            const size_t qc = (size_t)I * C.Pb + J;
            const double d = last ? 1.0 : (double)C.c[4][qc];
            const double v = (double)bO[e + 1] + (double)bO[e + 2] + (double)bO[e + 3] + (double)bH[e] + (double)bH[e + 4];
            C.b[qc] = (TV)v;
            if (!last) C.x[qc] = (TV)(omC * v / d);
        }
    }
    __syncwarp();
}

template <int V, typename TV>
__device__ __forceinline__ double sa0_down_step(const Team& T, const Sa0<TV>& A, const SaDown<TV>& D, const SaLevel<TV>& C) {
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int P = A.P, Ga = A.nJ / V + 1, S = (Ga + 26) / 27, n = S * C.nI;
    double acc = 0.0;
    for (int c = sa_task(T, n, nw); c < n; c += nw) {
        const int s = c % S, I = 1 + c / S, g = 27 * s - 1 + lane, j0 = g * V, r0 = 3 * I - 3;
        const bool act = g >= 0 && g < Ga, own = act && lane >= 1 && lane <= 27;
        VecN<TV, V> r[7], a[7], di[7], fe[5], fn[6];
#pragma unroll
        for (int h = 0; h < 7; ++h) {
            const int i = r0 - 1 + h;
            const bool in = act && i >= 1 && i <= A.nI;
            const size_t q = (size_t)i * P + j0;
            r[h] = in ? ldv<V>(D.r + q) : zerov<TV, V>();
            a[h] = in && !D.first ? ldv<V>(D.Ap + q) : zerov<TV, V>();
            di[h] = in ? ldv<V>(A.dinv + q) : zerov<TV, V>();
            if (h < 6) fn[h] = in ? ldv<V>(A.fN + q) : zerov<TV, V>();
            if (h >= 1 && h < 6) fe[h - 1] = in ? ldv<V>(A.fE + q) : zerov<TV, V>();
        }
        const SaCols<TV> K(j0);
        VecN<TV, V> x[7], vO = zerov<TV, V>(), vH = vO;
#pragma unroll
        for (int h = 0; h < 7; ++h)
#pragma unroll
            for (int k = 0; k < V; ++k) {
                r[h].v[k] = r[h].v[k] - D.al * a[h].v[k];
                x[h].v[k] = A.om * r[h].v[k] * di[h].v[k];
            }
#pragma unroll
        for (int h = 0; h < 5; ++h) {
            const int i = r0 + h;
            VecN<TV, V> qO, qH, qX;
            sa0_row_down(A, K, i >= 1 && i <= A.nI, (h + 2) % 3, r[h + 1], di[h + 1], x[h], x[h + 1], x[h + 2], fe[h],
                         fn[h + 1], fn[h], qO, qH, qX);
            const bool ring = h == 0 || h == 4;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                vO.v[k] += ring ? qX.v[k] : qO.v[k];
                if (!ring) vH.v[k] += qH.v[k];
            }
            if (!ring && own && i <= A.nI) {
#pragma unroll
                for (int k = 0; k < V; ++k) acc += (double)r[h + 1].v[k] * (double)r[h + 1].v[k];
                if (!D.first) stv(D.rn + ((size_t)i * P + j0), r[h + 1]);
            }
        }
        sa0_gather(C, s, I, vO, vH, D.omC, D.last, D.buf);
    }
    return acc;
}

template <typename TV>
__device__ __forceinline__ double sa0_down_march(const Team& T, const Sa0<TV>& A, const SaDown<TV>& D, const SaLevel<TV>& C) {
    constexpr int V = Vec16<TV>::n;
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int P = A.P, Ga = A.nJ / V + 1;
    const SaRuns W((Ga + 26) / 27, C.nI, nw);
    double acc = 0.0;
    for (int c = sa_task(T, W.n, nw); c < W.n; c += nw) {
        const int s = c % W.S, I0 = 1 + (c / W.S) * W.R, I1 = min(C.nI, I0 + W.R - 1);
        const int g = 27 * s - 1 + lane, j0 = g * V;
        const bool act = g >= 0 && g < Ga, own = act && lane >= 1 && lane <= 27;
        const SaCols<TV> K(j0);
        struct Row {
            VecN<TV, V> r, a, di;
        };
        auto ld = [&](const TV* f, int i, bool on) {
            return on && i >= 1 && i <= A.nI ? ldv<V>(f + (size_t)i * P + j0) : zerov<TV, V>();
        };
        auto ldr = [&](int i, bool on) { return Row{ld(D.r, i, on), ld(D.Ap, i, on && !D.first), ld(A.dinv, i, on)}; };
        auto resid = [&](Row& o, VecN<TV, V>& x0) {
#pragma unroll
            for (int k = 0; k < V; ++k) {
                o.r.v[k] = o.r.v[k] - D.al * o.a.v[k];
                x0.v[k] = A.om * o.r.v[k] * o.di.v[k];
            }
        };
        const int rb = 3 * I0 - 3, re = 3 * I1 + 1;
        VecN<TV, V> xs, xc, xn, vO = zerov<TV, V>(), vH = vO, nO = vO;
        Row low = ldr(rb - 1, act), cur = ldr(rb, act), nxt = ldr(rb + 1, act);
        VecN<TV, V> fe = ld(A.fE, rb, act), fn = ld(A.fN, rb, act), fs = ld(A.fN, rb - 1, act);
        resid(low, xs);
        resid(cur, xc);
        int role = 2, I = I0 - 1;
#pragma unroll 3
        for (int i = rb; i <= re; ++i) {
            const bool more = act && i < re;
            const Row far = ldr(i + 2, more);
            const VecN<TV, V> feN = ld(A.fE, i + 1, more), fnN = ld(A.fN, i + 1, more);
            resid(nxt, xn);
            if (i >= 3 * I0 - 2 && i <= 3 * I1 && i <= A.nI && own) {
#pragma unroll
                for (int k = 0; k < V; ++k) acc += (double)cur.r.v[k] * (double)cur.r.v[k];
                if (!D.first) stv(D.rn + ((size_t)i * P + j0), cur.r);
            }
            VecN<TV, V> qO, qH, qX;
            sa0_row_down(A, K, i >= 1 && i <= A.nI, role, cur.r, cur.di, xs, xc, xn, fe, fn, fs, qO, qH, qX);
            if (role == 0) {
                // the ring row below completes the previous row of aggregates
#pragma unroll
                for (int k = 0; k < V; ++k) vO.v[k] += qX.v[k];
                if (I >= I0) sa0_gather(C, s, I, vO, vH, D.omC, D.last, D.buf);
                ++I;
                vO = nO;
                vH = zerov<TV, V>();
            }
#pragma unroll
            for (int k = 0; k < V; ++k) {
                vO.v[k] += qO.v[k];
                vH.v[k] += qH.v[k];
            }
            nO = qX;
            role = role == 2 ? 0 : role + 1;
            xs = xc; xc = xn;
            fs = fn; fe = feN; fn = fnN;
            cur = nxt;
            nxt = far;
        }
    }
    return acc;
}

template <typename TV>
__device__ __forceinline__ double sa0_down(const Team& T, const Sa0<TV>& A, const SaDown<TV>& D, const SaLevel<TV>& C) {
    const int nw = T.nth() >> 5;
    if ((A.nJ + 27) / 27 * C.nI <= nw) return sa0_down_step<1>(T, A, D, C);
    if constexpr (sizeof(TV) == 4)
        if ((A.nJ / 2 + 27) / 27 * C.nI <= nw) return sa0_down_step<2>(T, A, D, C);
    return sa0_down_march(T, A, D, C);
}

// The ascent into level 0 in one pass: t = x0 + P e with x0 = omega b / d,
// then y = t + omega (b - A t) / d = (1 - omega) t + omega (b + sum f t(nb)) / d.
// Lanes as in the matvec.  Returns the lane's share of b.y.
template <typename TV, int V>
__device__ __forceinline__ void sa0_row_t(const Sa0<TV>& A, const SaCols<TV>& K, bool in, int role,
                                          const VecN<TV, V>& b, const VecN<TV, V>& di, const VecN<TV, V>& fe, TV fw,
                                          const VecN<TV, V>& fn, const VecN<TV, V>& fs, const TV (&eO)[V],
                                          const TV (&eH)[V], const TV (&eX)[V], VecN<TV, V>& t) {
    TV same[V], fh[V];
    sa0_faces(K, fe, fw, fn, fs, role, same, fh);
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const TV wd = A.w0 * di.v[k];
        TV v = A.om * b.v[k] * di.v[k] + (((TV)1 - A.w0) + wd * same[k]) * eO[k] + wd * fh[k] * eH[k];
        if (role != 1) v += wd * (role == 0 ? fs.v[k] : fn.v[k]) * eX[k];
        t.v[k] = in ? v : (TV)0;
    }
}

template <typename TV, int V>
__device__ __forceinline__ double sa0_row_y(const Sa0<TV>& A, bool own, const VecN<TV, V>& b, const VecN<TV, V>& di,
                                            const VecN<TV, V>& fe, TV fw, const VecN<TV, V>& fn, const VecN<TV, V>& fs,
                                            const VecN<TV, V>& ts, const VecN<TV, V>& tc, const VecN<TV, V>& tn,
                                            VecN<TV, V>& y) {
    const TV tw = from_west(tc.v[V - 1]), te = from_east(tc.v[0]);
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const TV W = k ? tc.v[k ? k - 1 : 0] : tw, E = k < V - 1 ? tc.v[k < V - 1 ? k + 1 : 0] : te, FW = k ? fe.v[k ? k - 1 : 0] : fw;
        TV v = ((TV)1 - A.om) * tc.v[k] +
               A.om * di.v[k] * (b.v[k] + fe.v[k] * E + FW * W + fn.v[k] * tn.v[k] + fs.v[k] * ts.v[k]);
        y.v[k] = v;
        if (own) acc += (double)b.v[k] * (double)v;
    }
    return acc;
}

// a lane's columns of the coarse correction: the own aggregate's and the
// horizontal one's (0, a frame entry, outside the unknowns)
template <int V>
struct SaE {
    int o[V], h[V];
    __device__ __forceinline__ SaE(int j0, int nJ, bool act) {
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const int jj = j0 + k;
            const bool in = act && jj >= 1 && jj <= nJ;
            o[k] = in ? (jj - 1) / 3 + 1 : 0;
            h[k] = in ? o[k] + sa_side(jj) : 0;
        }
    }
    template <typename TV>
    static __device__ __forceinline__ void ld(const TV* row, const int (&at)[V], TV (&v)[V]) {
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = row[at[k]];
    }
};

template <int V, typename TV>
__device__ __forceinline__ double sa0_up_step(const Team& T, const Sa0<TV>& A, const TV* b, const SaLevel<TV>& C, TV* y) {
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int P = A.P, Ga = A.nJ / V + 1, S = (Ga + 29) / 30, n = S * A.nI;
    double acc = 0.0;
    for (int c = sa_task(T, n, nw); c < n; c += nw) {
        const int s = c % S, i = 1 + c / S, g = 30 * s - 1 + lane, j0 = g * V;
        const bool act = g >= 0 && g < Ga, own = act && lane >= 1 && lane <= 30;
        const SaE<V> E(j0, A.nJ, act);
        VecN<TV, V> bb[3], di[3], fe[3], fn[4], t[3], yv;
        // with one column a lane, lane 0's weights need the face west of it
        TV eO[3][V], eH[3][V], eX[3][V], fw0[3] = {(TV)0, (TV)0, (TV)0};
        fn[0] = act && i >= 2 ? ldv<V>(A.fN + ((size_t)(i - 2) * P + j0)) : zerov<TV, V>();
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            const int ii = i - 1 + h;
            const bool row = ii >= 1 && ii <= A.nI, in = act && row;
            const size_t q = (size_t)ii * P + j0;
            bb[h] = in ? ldv<V>(b + q) : zerov<TV, V>();
            di[h] = in ? ldv<V>(A.dinv + q) : zerov<TV, V>();
            fe[h] = in ? ldv<V>(A.fE + q) : zerov<TV, V>();
            if (V == 1 && lane == 0 && in && j0 > 0) fw0[h] = A.fE[q - 1];
            fn[h + 1] = in ? ldv<V>(A.fN + q) : zerov<TV, V>();
            const int I = row ? (ii - 1) / 3 + 1 : 0, Ix = row ? I + sa_side(ii) : 0;
            E.ld(C.y + (size_t)I * C.P, E.o, eO[h]);
            E.ld(C.y + (size_t)I * C.P, E.h, eH[h]);
            E.ld(C.y + (size_t)Ix * C.P, E.o, eX[h]);
        }
        const SaCols<TV> K(j0);
        TV fwc = (TV)0;
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            const int ii = i - 1 + h;
            TV fw = from_west(fe[h].v[V - 1]);
            if (V == 1 && lane == 0) fw = fw0[h];
            if (h == 1) fwc = fw;
            sa0_row_t(A, K, ii >= 1 && ii <= A.nI, (ii + 2) % 3, bb[h], di[h], fe[h], fw, fn[h + 1], fn[h], eO[h], eH[h],
                      eX[h], t[h]);
        }
        acc += sa0_row_y(A, own, bb[1], di[1], fe[1], fwc, fn[2], fn[1], t[0], t[1], t[2], yv);
        if (own) stv(y + ((size_t)i * P + j0), yv);
    }
    return acc;
}

template <typename TV>
__device__ __forceinline__ double sa0_up_march(const Team& T, const Sa0<TV>& A, const TV* b, const SaLevel<TV>& C, TV* y) {
    constexpr int V = Vec16<TV>::n;
    const int lane = threadIdx.x & 31, nw = T.nth() >> 5;
    const int P = A.P, Ga = A.nJ / V + 1;
    const SaRuns W((Ga + 29) / 30, A.nI, nw);
    double acc = 0.0;
    for (int c = sa_task(T, W.n, nw); c < W.n; c += nw) {
        const int s = c % W.S, i0 = 1 + (c / W.S) * W.R, i1 = min(A.nI, i0 + W.R - 1);
        const int g = 30 * s - 1 + lane, j0 = g * V;
        const bool act = g >= 0 && g < Ga, own = act && lane >= 1 && lane <= 30;
        const SaCols<TV> K(j0);
        const SaE<V> E(j0, A.nJ, act);
        struct Row {
            VecN<TV, V> b, di, fe, fn;
        };
        auto ld = [&](const TV* f, int i, bool on) {
            return on && i <= A.nI ? ldv<V>(f + (size_t)i * P + j0) : zerov<TV, V>();
        };
        auto ldr = [&](int i, bool on) { return Row{ld(b, i, on), ld(A.dinv, i, on), ld(A.fE, i, on), ld(A.fN, i, on)}; };
        const int rb = max(i0 - 1, 1), re = i1 + 1;
        int I = (rb - 1) / 3 + 1, role = (rb - 1) % 3;
        TV eP[V], eC[V], hC[V], eN[V], hN[V];
        const TV* er = C.y + (size_t)I * C.P;
        Row nxt = ldr(rb, act);
        VecN<TV, V> fs = ld(A.fN, rb - 1, act);
        E.ld(er - C.P, E.o, eP);
        E.ld(er, E.o, eC);
        E.ld(er, E.h, hC);
        E.ld(er + C.P, E.o, eN);
        E.ld(er + C.P, E.h, hN);
        VecN<TV, V> ts = zerov<TV, V>(), tc = ts, fss = ts;
        Row cur{ts, ts, ts, ts};
        TV fwC = (TV)0;
#pragma unroll 1   // unrolled it spills: 36 against 31 us a CG iteration at 2048 x 1024 in float
        for (int i = rb; i <= re; ++i) {
            const Row far = ldr(i + 1, act && i < re);
            const TV fw = from_west(nxt.fe.v[V - 1]);
            VecN<TV, V> tn, yv;
            if (role == 0) sa0_row_t(A, K, i <= A.nI, 0, nxt.b, nxt.di, nxt.fe, fw, nxt.fn, fs, eC, hC, eP, tn);
            else sa0_row_t(A, K, i <= A.nI, role, nxt.b, nxt.di, nxt.fe, fw, nxt.fn, fs, eC, hC, eN, tn);
            if (i > i0) {
                acc += sa0_row_y(A, own, cur.b, cur.di, cur.fe, fwC, cur.fn, fss, ts, tc, tn, yv);
                if (own) stv(y + ((size_t)(i - 1) * P + j0), yv);
            }
            ts = tc; tc = tn;
            fss = fs; fs = nxt.fn;
            fwC = fw;
            cur = nxt;
            nxt = far;
            if (++role == 3) {
                role = 0;
                ++I;
                er += C.P;
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    eP[k] = eC[k];
                    eC[k] = eN[k];
                    hC[k] = hN[k];
                }
                if (i < re && I <= C.nI) {
                    E.ld(er + C.P, E.o, eN);
                    E.ld(er + C.P, E.h, hN);
                }
            }
        }
    }
    return acc;
}

template <typename TV>
__device__ __forceinline__ double sa0_up(const Team& T, const Sa0<TV>& A, const TV* b, const SaLevel<TV>& C, TV* y) {
    const int nw = T.nth() >> 5;
    if ((A.nJ + 30) / 30 * A.nI <= nw) return sa0_up_step<1>(T, A, b, C, y);
    if constexpr (sizeof(TV) == 4)
        if ((A.nJ / 2 + 30) / 30 * A.nI <= nw) return sa0_up_step<2>(T, A, b, C, y);
    return sa0_up_march(T, A, b, C, y);
}

// Called for every unknown of the residual when a solve starts: clears the frame
// columns that share a 16-byte vector with the row's ends.  The passes update and
// store r in whole vectors, so a solve whose step overflowed leaves NaN there, and
// nothing else would ever take it out of the sums of the context's later solves.
template <typename TV>
__device__ __forceinline__ void clear_row_ends(TV* r, size_t c, int j, int w) {
    if (j == 1) r[c - 1] = (TV)0;
    if (j == w)
        for (int q = 1; q <= (w | (Vec16<TV>::n - 1)) - w; ++q) r[c + q] = (TV)0;
}

// ---------------------------------------------------------------- the solver
// The PCG of one pressure-correction solve on a team of CTAs (the whole grid
// in k_pcg_sa; Few: a group of CTAs in the batched kernel); returns false if a
// barrier gave up.  Ends without a barrier after writing p'.  part: at least
// 4 doubles a CTA.
template <typename TV, bool Few>
__device__ __forceinline__ bool pcg_sa(const Team& T, unsigned& target, const KParams& k, Status* st,
                                       const double* dE, const double* dN, const PcgBufs<TV>& B,
                                       const SaHier<TV>& H, double* pStar, double* part) {
    extern __shared__ __align__(128) double dsm[];
    __shared__ double sm[kReduceSm];
    const Dims d = k.d;
    const int M = d.M, N = d.N, w = N - 2;
    const int tid = T.tid(), nth = T.nth();
    const SaSplit all{tid, nth};
    const double rho = k.rho, hx = k.hx, hy = k.hy, om = H.omega;
    TV* const buf = reinterpret_cast<TV*>(dsm);
    // the coarse operators are rebuilt every H.reuse outer iterations (they
    // only precondition: the CG matvec and level 0's smoother and
    // prolongation always use the current operator), after a solve that
    // reached the iteration cap with them (early in a run the operator moves
    // fast), and whenever the stored ones are stale (the operator changed
    // from the host, another solve such as the adjoint's stored its own, or a
    // batch built its matrices for another level)
    const bool rebuild = *(volatile int*)H.built != H.Ld ||
                         (H.reuse > 0 && (H.reuse == 1 || (st->iter % H.reuse) == 0 || st->itersP >= k.maxP));

    const SaLevel<TV> L0 = H.lv[0];
    const SaLevel<TV>& C1 = H.lv[1];
    const Sa0<TV> A0{B.fE, B.fN, B.d, H.dinv0, M - 1, w, d.P, (TV)om, (TV)H.w0};
    unsigned long long tp = (H.prof && T.lead()) ? globaltimer_ns() : 0ull;
    auto tick = [&](int ph) {
        if (H.prof && T.lead()) {
            const unsigned long long t = globaltimer_ns();
            atomicAdd(H.prof + ph, t - tp);
            tp = t;
        }
    };

    // ---- set-up: level-0 operator (the reference's formulas), its inverse
    // diagonal, the prolongation weights where the coarse operators are to be
    // rebuilt, r = b
    double bb[1] = {0.0};
    sa_cells(all, M - 1, w, [&](int i, int j) {
        const int c = i * d.P + j;
        const double aE = rho * dE[c] * hy;
        const double aW = (j > 1) ? rho * dE[c - 1] * hy : 0.0;
        const double aN = (i < M - 1) ? rho * dN[c] * hx : 0.0;
        const double aS = (i > 1) ? rho * dN[c - d.P] * hx : 0.0;
        double aP = aE + aW + aN + aS;
        if (aP < 1e-20) aP = 1.0;
        B.fE[c] = j < w ? (TV)aE : (TV)0;
        B.fN[c] = (TV)aN;
        B.d[c] = (TV)aP;
        const double inv = 1.0 / aP;
        H.dinv0[c] = (TV)inv;
        if (rebuild) {
            // faces towards unknowns of the own aggregate, and towards the
            // horizontal / vertical neighbour aggregate (the east face of the
            // last column is the Dirichlet outlet, with no unknown behind it)
            const int ri = (i - 1) % 3, rj = (j - 1) % 3;
            const double eIn = (j < w) ? aE : 0.0;
            const double same = (rj != 2 ? eIn : 0.0) + (rj != 0 ? aW : 0.0) + (ri != 2 ? aN : 0.0) + (ri != 0 ? aS : 0.0);
            const double fh = rj == 0 ? aW : (rj == 2 ? eIn : 0.0);
            const double fv = ri == 0 ? aS : (ri == 2 ? aN : 0.0);
            const double sc = H.w0 * inv;
            L0.pw[0][c] = (TV)(1.0 - sc * (aP - same));
            L0.pw[1][c] = (TV)(sc * fh);
            L0.pw[2][c] = (TV)(sc * fv);
        }
        const TV rt = B.rhs[c];
        B.r[c] = rt;
        clear_row_ends(B.r, c, j, w);
        bb[0] += (double)rt * (double)rt;
    });
    // the right-hand side that the matrix is applied to, up to whole 16 bytes
    if (T.lead()) {
        const SaLevel<TV>& D = H.lv[H.Ld];
        for (int q = D.nI * D.nJ; q < sa_row<TV>(D.nI * D.nJ); ++q) D.b[D.nJ + 1 + q] = (TV)0;
    }
    if (!team_reduce(T, target, bb, part, sm)) return false;
    const double rTol = k.pTol * sqrt(bb[0]);
    tick(SA_P_SETUP);

    // ---- set-up: coarse operators and V-cycle matrices (when rebuilt)
    if (rebuild) {
        for (int l = 0; l < H.L - 1; ++l) {
            const SaLevel<TV>& f = H.lv[l];
            const SaLevel<TV>& C = H.lv[l + 1];
            if (l > 0) {
                sa_cells(all, f.nI, f.nJ, [&](int i, int j) { sa_pweights(f, H.wc, i, j); });
                if (!team_sync(T, target)) return false;
                sa_cells(all, C.nI, C.nJ, [&](int I, int J) {
                    sa_galerkin<TV, false>(f, (const TV*)nullptr, (const TV*)nullptr, (const TV*)nullptr, C, I, J);
                });
            } else {
                sa_cells(all, C.nI, C.nJ, [&](int I, int J) { sa_galerkin<TV, true>(f, B.fE, B.fN, B.d, C, I, J); });
            }
            if (!team_sync(T, target)) return false;
        }
        if (T.rank == 0) sa_invert(H.lv[H.L - 1], H.bm[H.L - 1], dsm);
        if (!team_sync(T, target)) return false;
        for (int l = H.L - 2; l >= H.Ld; --l) {
            sa_matrix(T, H.lv[l], H.lv[l + 1], H.bm[l + 1], H.bm[l], om, dsm);
            if (!team_sync(T, target)) return false;
        }
    }
    tick(SA_P_GALERKIN);

    // ---- the V-cycle below level 0 and the ascent into it: z = M b
    auto vcycle = [&](const TV* b, double& rz) __attribute__((always_inline)) -> bool {
        for (int l = 1; l < H.Ld; ++l) {
            if constexpr (Few) sa_down_march(T, H.lv[l], H.lv[l + 1], om, l + 1 == H.Ld);
            else sa_down(T, H.lv[l], H.lv[l + 1], om, l + 1 == H.Ld);
            if (!team_sync(T, target)) return false;
            tick(SA_P_DOWN + l);
        }
        sa_apply(T, H.lv[H.Ld], H.bm[H.Ld]);
        if (!team_sync(T, target)) return false;
        tick(SA_P_DENSE);
        for (int l = H.Ld - 1; l >= 1; --l) {
            if constexpr (Few) sa_up_march(T, H.lv[l], H.lv[l + 1], om);
            else sa_up(T, H.lv[l], H.lv[l + 1], om);
            if (!team_sync(T, target)) return false;
            tick(SA_P_UP + l);
        }
        double v[1] = {sa0_up(T, A0, b, C1, L0.y)};
        if (!team_reduce(T, target, v, part, sm)) return false;
        rz = v[0];
        tick(SA_P_UP);
        return true;
    };

    double rz = 0.0;
    sa0_down(T, A0, SaDown<TV>{B.r, B.r, B.r, (TV)0, true, H.Ld == 1, om, buf}, C1);
    if (!team_sync(T, target)) return false;
    tick(SA_P_UPDATE);
    if (!vcycle(B.r, rz)) return false;
    double beta = 0.0;
    TV al = (TV)0;          // step of the newest direction, not yet in x
    bool pend = false, haveX = false;
    int it = 0;
    const TV* p = B.pa;
    while (it < k.maxP) {
        TV* pnew = (it & 1) ? B.pb : B.pa;
        double v[1] = {sa0_matvec(T, A0, SaMat<TV>{L0.y, (it & 1) ? B.pa : B.pb, B.x, pnew, B.Ap, (TV)beta, al, min(it, 2)})};
        haveX = pend;
        pend = false;
        if (!team_reduce(T, target, v, part, sm)) return false;
        tick(SA_P_MATVEC);
        if (fabs(v[0]) < 1e-20) break;
        al = (TV)(rz / v[0]);
        p = pnew;
        pend = true;
        const TV* rold = (it & 1) ? H.r2 : B.r;
        TV* rnew = (it & 1) ? B.r : H.r2;
        ++it;
        if (it == k.maxP) break;   // the residual and the next direction are not needed
        v[0] = sa0_down(T, A0, SaDown<TV>{rold, B.Ap, rnew, al, false, H.Ld == 1, om, buf}, C1);
        if (!team_reduce(T, target, v, part, sm)) return false;
        tick(SA_P_UPDATE);
        if (sqrt(v[0]) <= rTol) break;
        double rzn = 0.0;
        if (!vcycle(rnew, rzn)) return false;
        beta = rzn / rz;
        rz = rzn;
    }
    // ---- p' = x + alpha p (the last step)
    sa_cells(all, M - 1, w, [&](int i, int j) {
        const int c = i * d.P + j;
        TV x = haveX ? B.x[c] : (TV)0;
        if (pend) x = x + al * p[c];
        pStar[c] = (double)x;
        if (j == w) pStar[c + 1] = 0.0;
    });
    if (T.lead()) {
        st->itersP = it;
        if (rebuild) *H.built = H.Ld;
    }
    return true;
}

template <typename TV>
__global__ void __launch_bounds__(512, 1) k_pcg_sa(KParams k, Status* st, const double* dE, const double* dN,
                                                PcgBufs<TV> B, SaHier<TV> H, double* pStar, double* part,
                                                unsigned* bar) {
    if (st->done) return;
    unsigned target = 0;
    pcg_sa<TV, false>(grid_team(bar, &st->err), target, k, st, dE, dN, B, H, pStar, part);
}

}  // namespace cp
