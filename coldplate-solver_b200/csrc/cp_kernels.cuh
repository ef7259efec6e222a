// SIMPLE outer-iteration kernels for sm_100a.
//
// One outer iteration (SIMPLE::calculateStep, iterations.cpp:82-659, with
// momentumSolverType 1) runs as:
//   k_bc        velocity + pressure boundary conditions;     boundaries.cpp:50-146
//               clears the counters of the kernels behind it
//   k_assemble  U and V momentum coefficients, fused:        momentum_solver.cpp:197-314
//               FOU upwinding, half-cell walls, Brinkman,    boundaries.cpp:148-206
//               2.5-D sink, relaxation, SOU correction,      convection.cpp:53-186
//               dE/dN, boundary neighbours folded into b
//   k_jacobi    persistent: Jacobi sweeps of U and V, stop   jacobi_solver.cpp:44-67
//               rule per component, then
//               scatter/clamp/max-change and BCs on u*, v*   momentum_solver.cpp:335-351
//               (small grids: k_jacobi_cluster)
//   k_mass      RMS of u*-u, v*-v; mass imbalance; PCG rhs   iterations.cpp:499-533,
//                                                            pressure_solver.cpp:471-488,733-742
//   the pressure solve on p', by type and size: k_pcg or     pressure_solver.cpp:121-184,
//               k_pcg_cluster (cp_pcg.cuh), k_pcg_sa         747-766
//               (cp_sa.cuh), k_pcg_mg (cp_mg.cuh)
//   k_correct   p += pAlpha p'; u, v corrections + clamps,   iterations.cpp:556-599
//               with the boundary conditions that copy them
//   k_finalize  pressure-drop sampling, residual reporting,  postprocessing.cpp:103-327,
//               history row and the stop rules              SIMPLE.cpp:378-491
//
// All kernels return immediately once Status::done is set, so a captured
// graph of one iteration can be replayed past convergence at no cost.
//
// Precision: fields (u, v, p, u*, v*, p', dE, dN) are double.  The inner
// systems are stored in TC (double for the FP64 form, float for the mixed
// form).  In the mixed form the momentum sweeps solve for a correction
// delta of the current velocity, A delta = b - A u, whose right-hand side is
// formed in double, and the PCG runs in float on the double mass imbalance;
// all global sums are double.
#pragma once

#include "cp_device.cuh"

namespace cp {

constexpr int kJacThreads = 512;      // sweeps of both components: one CTA an SM
constexpr int kJacSegThreads = 256;   // one component after the other: up to three CTAs an SM

// ------------------------------------------------------------------ systems
template <typename TC>
struct MomSys {
    TC *aP, *aE, *aW, *aN, *aS, *b;   // b: rhs (FP64 form) or b - A u (mixed form)
};

template <typename TC>
struct PcgBufs {
    TC *fE, *fN, *d;      // face coefficients rho*dE*hy (E face), rho*dN*hx (N face); diagonal
    TC *x, *r, *pa, *pb, *Ap;
    TC* rhs;              // mass imbalance per unknown (written by k_mass)
};

// ------------------------------------------------------------------ k_bc
// Velocity BCs (boundaries.cpp:50-118) on (u, v) and, when p != nullptr,
// pressure BCs (boundaries.cpp:123-146).  Every write reads only interior
// values, so the reference's sequential order is reproduced in parallel.
__device__ __forceinline__ bool inlet_fluid(const KParams& k, const double* gamma, int uRow) {
    const int M = k.d.M;
    int cellRow = uRow <= 0 ? 0 : (uRow >= M ? (M - 2 > 0 ? M - 2 : 0) : uRow - 1);
    cellRow = cellRow < 0 ? 0 : (cellRow > M - 1 ? M - 1 : cellRow);
    return gamma[at(k.d, cellRow, 0)] > 0.5;
}

__device__ __forceinline__ void apply_bc(const KParams& k, int iter, double* u, double* v, double* p,
                                         const double* gamma, int t0, int stride) {
    const Dims d = k.d;
    const int M = d.M, N = d.N;
    const double Uin = inlet_velocity(k, iter);
    const int L = (M > N ? M : N) + 1;
    for (int t = t0; t < L; t += stride) {
        if (t <= M) u[at(d, t, 0)] = inlet_fluid(k, gamma, t) ? Uin : 0.0;
        if (t >= 1 && t <= N - 1) { u[at(d, 0, t)] = 0.0; u[at(d, M, t)] = 0.0; }
        if (t >= 1 && t <= M - 1) u[at(d, t, N - 1)] = u[at(d, t, N - 2)];
        if (t <= N) { v[at(d, 0, t)] = 0.0; v[at(d, M - 1, t)] = 0.0; }
        if (t >= 1 && t <= M - 2) { v[at(d, t, 0)] = 0.0; v[at(d, t, N)] = v[at(d, t, N - 1)]; }
        if (p) {
            if (t >= 1 && t <= N - 1) { p[at(d, 0, t)] = p[at(d, 1, t)]; p[at(d, M, t)] = p[at(d, M - 1, t)]; }
            if (t >= 1 && t <= M - 1) { p[at(d, t, 0)] = p[at(d, t, 1)]; p[at(d, t, N)] = 0.0; }
        }
    }
}

// The velocity BCs that do not copy an interior value (inlet, walls).  The rest
// (the outlet's u and v, the pressure frame) follow an interior value each, and
// the passes that write that value write them with it.
__device__ __forceinline__ void apply_bc_const(const KParams& k, int iter, double* u, double* v, const double* gamma,
                                               int t0, int stride) {
    const Dims d = k.d;
    const int M = d.M, N = d.N;
    const double Uin = inlet_velocity(k, iter);
    const int L = (M > N ? M : N) + 1;
    for (int t = t0; t < L; t += stride) {
        if (t <= M) u[at(d, t, 0)] = inlet_fluid(k, gamma, t) ? Uin : 0.0;
        if (t >= 1 && t <= N - 1) { u[at(d, 0, t)] = 0.0; u[at(d, M, t)] = 0.0; }
        if (t <= N) { v[at(d, 0, t)] = 0.0; v[at(d, M - 1, t)] = 0.0; }
        if (t >= 1 && t <= M - 2) v[at(d, t, 0)] = 0.0;
    }
}

// The BCs before an iteration; block 0 also clears the iteration's max-change
// counters and the barrier counters of the persistent kernels behind it
__global__ void k_bc(KParams k, Status* st, double* u, double* v, double* p, const double* gamma, unsigned* barJ,
                     unsigned* barP) {
    if (st->done) return;
    const int iter = st->iter;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->maxDU = 0ull;
        st->maxDV = 0ull;
        *barJ = 0u;
        *barP = 0u;
    }
    apply_bc(k, iter, u, v, p, gamma, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ------------------------------------------------------------------ assembly
// Face averages of cell fields (SIMPLE.h:642-686, 740-778); the callers only
// pass unknowns, for which the reference's range checks always pass.
struct Fields {
    const double *u, *v, *p, *alpha, *gamma;
};

template <bool IsU>
struct AssembledRow {
    double aP0, aP, aE, aW, aN, aS, Sp;
};

// Coefficients of one momentum unknown; see momentum_solver.cpp:204-313.
template <bool IsU>
__device__ __forceinline__ void assemble_row(const KParams& k, const Fields& f, int i, int j, double maxVel,
                                             AssembledRow<IsU>& out) {
    const Dims d = k.d;
    const int M = d.M, N = d.N;
    const double* u = f.u;
    const double* v = f.v;
    const double hx = k.hx, hy = k.hy, vol = hx * hy, rho = k.rho, eta = k.eta;
    double alphaLocal, gammaFace, ue, uw, vn, vs;
    if (IsU) {
        alphaLocal = 0.5 * (f.alpha[at(d, i - 1, j - 1)] + f.alpha[at(d, i - 1, j)]);
        gammaFace = 0.5 * (f.gamma[at(d, i - 1, j - 1)] + f.gamma[at(d, i - 1, j)]);
        ue = dclamp(0.5 * (u[at(d, i, j)] + u[at(d, i, j + 1)]), -maxVel, maxVel);
        uw = dclamp(0.5 * (u[at(d, i, j - 1)] + u[at(d, i, j)]), -maxVel, maxVel);
        vn = dclamp(0.5 * (v[at(d, i, j)] + v[at(d, i, j + 1)]), -maxVel, maxVel);
        vs = dclamp(0.5 * (v[at(d, i - 1, j)] + v[at(d, i - 1, j + 1)]), -maxVel, maxVel);
    } else {
        alphaLocal = 0.5 * (f.alpha[at(d, i - 1, j - 1)] + f.alpha[at(d, i, j - 1)]);
        gammaFace = 0.5 * (f.gamma[at(d, i - 1, j - 1)] + f.gamma[at(d, i, j - 1)]);
        ue = dclamp(0.5 * (u[at(d, i, j)] + u[at(d, i + 1, j)]), -maxVel, maxVel);
        uw = dclamp(0.5 * (u[at(d, i, j - 1)] + u[at(d, i + 1, j - 1)]), -maxVel, maxVel);
        vn = dclamp(0.5 * (v[at(d, i, j)] + v[at(d, i + 1, j)]), -maxVel, maxVel);
        vs = dclamp(0.5 * (v[at(d, i - 1, j)] + v[at(d, i, j)]), -maxVel, maxVel);
    }
    const double cs = k.convScale;
    const double Fe = cs * rho * hy * ue, Fw = cs * rho * hy * uw;
    const double Fn = cs * rho * hx * vn, Fs = cs * rho * hx * vs;
    const double De = eta * (hy / hx), Dn = eta * (hx / hy);
    double aE = De + dmax(0.0, -Fe);
    double aW = De + dmax(0.0, Fw);
    double aN = Dn + dmax(0.0, -Fn);
    double aS = Dn + dmax(0.0, Fs);
    // face-local half-cell diffusion next to external no-slip walls
    const double vt = 1e-8;
    if (gammaFace >= 0.999) {
        if (IsU) {
            if (i == 1 && fabs(u[at(d, 0, j)]) <= vt && fabs(v[at(d, 0, j)]) <= vt && fabs(v[at(d, 0, j + 1)]) <= vt)
                aS += Dn;
            if (i == M - 1 && fabs(u[at(d, M, j)]) <= vt && fabs(v[at(d, M - 1, j)]) <= vt &&
                fabs(v[at(d, M - 1, j + 1)]) <= vt)
                aN += Dn;
        } else {
            if (j == 1 && !(fabs(k.targetVel) > vt) && fabs(v[at(d, i, 0)]) <= vt && fabs(u[at(d, i, 0)]) <= vt &&
                fabs(u[at(d, i + 1, 0)]) <= vt)
                aW += De;
            if (j == N - 1 && !(fabs(f.p[at(d, i, N)]) <= 1e-8) && fabs(v[at(d, i, N)]) <= vt &&
                fabs(u[at(d, i, N - 1)]) <= vt && fabs(u[at(d, i + 1, N - 1)]) <= vt)
                aE += De;
        }
    }
    const double sumA = aE + aW + aN + aS;
    double aP0 = sumA + (Fe - Fw + Fn - Fs) + k.sinkDiag + alphaLocal * vol;
    aP0 = dmax(aP0, 1e-10);
    double Sp;
    const double* w = IsU ? u : v;
    if (IsU) Sp = (f.p[at(d, i, j)] - f.p[at(d, i, j + 1)]) * hy;
    else Sp = (f.p[at(d, i, j)] - f.p[at(d, i + 1, j)]) * hx;
    Sp += (1.0 - k.uvAlpha) / k.uvAlpha * aP0 * w[at(d, i, j)];
    if (k.sou) {
        // deferred correction S = sum over faces of -/+ F (phi_SOU - phi_FOU)
        // with the reference's stencil-availability guards
        const int iMaxE = IsU ? N : N + 1;   // column count of this component
        const int iMaxR = IsU ? M + 1 : M;   // row count of this component
        double S = 0.0;
#define W_(a, b) w[at(d, (a), (b))]
        if (Fe >= 0.0) { if (j >= 2) S -= Fe * ((1.5 * W_(i, j) - 0.5 * W_(i, j - 1)) - W_(i, j)); }
        else { if (j + 2 < iMaxE) S -= Fe * ((1.5 * W_(i, j + 1) - 0.5 * W_(i, j + 2)) - W_(i, j + 1)); }
        if (Fw >= 0.0) { if (j >= 2) S += Fw * ((1.5 * W_(i, j - 1) - 0.5 * W_(i, j - 2)) - W_(i, j - 1)); }
        else { if (j + 1 < iMaxE) S += Fw * ((1.5 * W_(i, j) - 0.5 * W_(i, j + 1)) - W_(i, j)); }
        if (Fn >= 0.0) { if (i >= 1) S -= Fn * ((1.5 * W_(i, j) - 0.5 * W_(i - 1, j)) - W_(i, j)); }
        else { if (i + 2 < iMaxR) S -= Fn * ((1.5 * W_(i + 1, j) - 0.5 * W_(i + 2, j)) - W_(i + 1, j)); }
        if (Fs >= 0.0) { if (i >= 2) S += Fs * ((1.5 * W_(i - 1, j) - 0.5 * W_(i - 2, j)) - W_(i - 1, j)); }
        else { if (i + 1 < iMaxR) S += Fs * ((1.5 * W_(i, j) - 0.5 * W_(i + 1, j)) - W_(i, j)); }
#undef W_
        Sp += S;
    }
    out.aP0 = aP0;
    out.aP = aP0 / k.uvAlpha;
    out.aE = aE; out.aW = aW; out.aN = aN; out.aS = aS;
    out.Sp = Sp;
}

// Range of unknowns of one component: U i in [1, M-1], j in [1, N-2];
// V i in [1, M-2], j in [1, N-1] (momentum_solver.cpp:52-72).
template <bool IsU>
__host__ __device__ __forceinline__ void mom_range(const Dims& d, int& i1, int& j1) {
    i1 = IsU ? d.M - 1 : d.M - 2;
    j1 = IsU ? d.N - 2 : d.N - 1;
}

template <typename TC, bool Mixed, bool IsU>
__device__ __forceinline__ void assemble_one(const KParams& k, const Fields& f, MomSys<TC> sys, double* dEN,
                                             int i, int j, double maxVel) {
    const Dims d = k.d;
    int i1, j1;
    mom_range<IsU>(d, i1, j1);
    AssembledRow<IsU> a;
    assemble_row<IsU>(k, f, i, j, maxVel, a);
    const double* w = IsU ? f.u : f.v;
    const size_t c = at(d, i, j);
    // boundary neighbours go to the rhs with their current value, in the
    // order E, W, N, S (momentum_solver.cpp:300-303)
    const bool eIn = j + 1 <= j1, wIn = j >= 2, nIn = i + 1 <= i1, sIn = i >= 2;
    double Sp = a.Sp;
    if (!eIn) Sp += a.aE * w[c + 1];
    if (!wIn) Sp += a.aW * w[c - 1];
    if (!nIn) Sp += a.aN * w[c + d.P];
    if (!sIn) Sp += a.aS * w[c - d.P];
    const double cE = eIn ? a.aE : 0.0, cW = wIn ? a.aW : 0.0, cN = nIn ? a.aN : 0.0, cS = sIn ? a.aS : 0.0;
    dEN[c] = (IsU ? k.hy : k.hx) / a.aP0;
    sys.aP[c] = (TC)a.aP;
    sys.aE[c] = (TC)cE;
    sys.aW[c] = (TC)cW;
    sys.aN[c] = (TC)cN;
    sys.aS[c] = (TC)cS;
    if (Mixed) {
        // right-hand side of the correction: b - A u, formed in double
        double Au = a.aP * w[c];
        if (sIn) Au -= cS * w[c - d.P];
        if (wIn) Au -= cW * w[c - 1];
        if (eIn) Au -= cE * w[c + 1];
        if (nIn) Au -= cN * w[c + d.P];
        sys.b[c] = (TC)(Sp - Au);
    } else {
        sys.b[c] = (TC)Sp;
    }
}

template <typename TC, bool Mixed>
__global__ void __launch_bounds__(256, 4) k_assemble(KParams k, const Status* st, Fields f, MomSys<TC> U, MomSys<TC> V, double* dE,
                           double* dN, int doU, int doV) {
    if (st->done) return;
    const double maxVel = max_vel(inlet_velocity(k, st->iter));
    const Dims d = k.d;
    const int nU = doU ? k.nU : 0, nV = doV ? k.nV : 0;
    const int wU = d.N - 2, wV = d.N - 1;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nU + nV; t += gridDim.x * blockDim.x) {
        if (t < nU) {
            const int i = 1 + t / wU, j = 1 + t % wU;
            assemble_one<TC, Mixed, true>(k, f, U, dE, i, j, maxVel);
        } else {
            const int s = t - nU;
            const int i = 1 + s / wV, j = 1 + s % wV;
            assemble_one<TC, Mixed, false>(k, f, V, dN, i, j, maxVel);
        }
    }
}

// ------------------------------------------------------------------ Jacobi
// Jacobi sweeps x+ = x + (b - A x) / aP of the U and the V system (they are
// independent: V assembles from u, v, not from u*).  Each component stops
// after the first sweep whose pre-update sum of r^2 is below tol^2 n, or after
// maxMomentumIter sweeps (jacobi_solver.cpp:44-67).
//
// A sweep is short (8 words an unknown from the L2), so the barrier and the
// sum behind it count: both components sweep between the same two barriers
// while both run, and the sums ride on the barrier (team_reduce).  The sweeps
// of an outer iteration took 103 us one after the other and take 72 together
// at 253 x 127 (double, 21 sweeps of one component), 163 and 131 at 811 x 389
// (float, 30).  Larger systems: jacobi_component.
// A warp takes a run of rows of a strip of 30 V columns: the next row's
// coefficients are in flight while it works on one, the iterate's rows stay in
// registers and its horizontal neighbours come by shuffles (lanes 0 and 31
// only supply them).  V = 16 bytes where the grid has more rows of strips than
// warps; otherwise the smallest that gives every warp at most one row, which
// puts all of a sweep's loads in flight at once.
template <typename TC, bool Mixed, int V>
__device__ __forceinline__ double jacobi_run(const Dims& d, const MomSys<TC>& S, const double* field, const TC* xc,
                                             TC* __restrict__ xn, int j1, int s, int i0, int i1) {
    const int lane = threadIdx.x & 31;
    const int g = 30 * s - 1 + lane, j0 = g * V;
    const bool act = g >= 0 && g < j1 / V + 1, own = act && lane >= 1 && lane <= 30;
    struct Row {
        VecN<TC, V> aP, aE, aW, aN, aS, b;
    };
    auto ldr = [&](int i, bool on) {
        Row r;
        if (on) {
            const size_t q = at(d, i, j0);
            r = Row{ldv<V>(S.aP + q), ldv<V>(S.aE + q), ldv<V>(S.aW + q), ldv<V>(S.aN + q), ldv<V>(S.aS + q), ldv<V>(S.b + q)};
        } else {
            r = Row{zerov<TC, V>(), zerov<TC, V>(), zerov<TC, V>(), zerov<TC, V>(), zerov<TC, V>(), zerov<TC, V>()};
        }
        return r;
    };
    // the iterate (the current field, or zero in the mixed form, before the
    // first sweep); couplings to anything outside the unknowns are zero
    auto ldx = [&](int i, bool on) -> VecN<TC, V> {
        if (!on) return zerov<TC, V>();
        if (xc) return ldv<V>(xc + at(d, i, j0));
        if constexpr (Mixed) return zerov<TC, V>();
        else return ldv<V>(field + at(d, i, j0));
    };
    VecN<TC, V> xS = ldx(i0 - 1, own), xP = ldx(i0, act), xN = ldx(i0 + 1, act);
    Row cur = ldr(i0, own);
    double acc = 0.0;
#pragma unroll 1
    for (int i = i0; i <= i1; ++i) {
        const bool more = i < i1;
        const VecN<TC, V> xF = ldx(i + 2, act && more);
        const Row nxt = ldr(i + 1, own && more);
        const TC xw = from_west(xP.v[V - 1]), xe = from_east(xP.v[0]);
        VecN<TC, V> o;
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const int j = j0 + q;
            const bool in = own && j >= 1 && j <= j1;
            const TC W = q ? xP.v[q ? q - 1 : 0] : xw, E = q < V - 1 ? xP.v[q < V - 1 ? q + 1 : 0] : xe;
            // S, W, P, E, N order of the reference's CSR rows
            TC Ax = (TC)0;
            Ax += (-cur.aS.v[q]) * xS.v[q];
            Ax += (-cur.aW.v[q]) * W;
            Ax += cur.aP.v[q] * xP.v[q];
            Ax += (-cur.aE.v[q]) * E;
            Ax += (-cur.aN.v[q]) * xN.v[q];
            const TC r = cur.b.v[q] - Ax;
            const TC dg = in ? cur.aP.v[q] : (TC)1;
            o.v[q] = in ? (TC)(xP.v[q] + r / dg) : (TC)0;
            if (in) acc += (double)r * (double)r;
        }
        if (own) stv(xn + at(d, i, j0), o);
        xS = xP;
        xP = xN;
        xN = xF;
        cur = nxt;
    }
    return acc;
}

// One component of a sweep: its strips and rows, and the runs they are cut into
struct JacSplit {
    int S, R, n;
    __device__ __forceinline__ JacSplit(int V, int i1, int j1, int nw, int both) {
        S = (j1 / V + 30) / 30;
        R = max(1, (i1 * S * both + nw - 1) / nw);
        n = S * ((i1 + R - 1) / R);
    }
};

template <typename TC, bool Mixed, int V>
__device__ __forceinline__ void jacobi_pass(const KParams& k, const MomSys<TC>& U, const MomSys<TC>& W, const double* u,
                                            const double* v, const TC* xUc, TC* xUn, const TC* xVc, TC* xVn,
                                            bool doU, bool doV, const Team& T, double (&acc)[2]) {
    const int nw = T.nth() >> 5, wid = threadIdx.x >> 5;
    int iU, jU, iV, jV;
    mom_range<true>(k.d, iU, jU);
    mom_range<false>(k.d, iV, jV);
    const int both = doU && doV ? 2 : 1;
    const JacSplit sU(V, iU, jU, nw, both), sV(V, iV, jV, nw, both);
    const int nU = doU ? sU.n : 0, n = nU + (doV ? sV.n : 0);
    // with fewer runs than warps, spread over the CTAs
    for (int c = n < nw ? wid * T.size + T.rank : T.rank * (int)(blockDim.x >> 5) + wid; c < n; c += nw) {
        if (c < nU) {
            const int i0 = 1 + c / sU.S * sU.R;
            acc[0] += jacobi_run<TC, Mixed, V>(k.d, U, u, xUc, xUn, jU, c % sU.S, i0, min(iU, i0 + sU.R - 1));
        } else {
            const int e = c - nU, i0 = 1 + e / sV.S * sV.R;
            acc[1] += jacobi_run<TC, Mixed, V>(k.d, W, v, xVc, xVn, jV, e % sV.S, i0, min(iV, i0 + sV.R - 1));
        }
    }
}

// Elements a lane of a march over `rows` rows of strips on nw warps: 1, 2 (floats)
// or 16 bytes
inline __host__ __device__ int jacobi_width(int N, int rows, int nw, int es) {
    return (N + 30) / 30 * rows <= nw ? 1 : es == 4 && (N / 2 + 30) / 30 * rows <= nw ? 2 : 16 / es;
}

// The sweeps of both components (or of one); cur: the buffer that holds the
// result (-1: the initial iterate), its: the sweeps.  part: 4 doubles a CTA.
// Returns false if a barrier gave up.
template <typename TC, bool Mixed>
__device__ __forceinline__ bool jacobi_sweeps(const KParams& k, const MomSys<TC>& U, const MomSys<TC>& W, const double* u,
                                              const double* v, TC* xU0, TC* xU1, TC* xV0, TC* xV1, bool doU, bool doV,
                                              double* part, const Team& T, unsigned& target, int& curU, int& curV,
                                              int& itU, int& itV) {
    __shared__ double sm[kReduceSm];
    const int nw = T.nth() >> 5;
    const double lim = k.momTol * k.momTol, limU = lim * (double)k.nU, limV = lim * (double)k.nV;
    curU = curV = -1;
    itU = itV = 0;
    bool onU = doU && k.maxMom > 0, onV = doV && k.maxMom > 0;
    while (onU || onV) {
        const TC* xUc = curU < 0 ? nullptr : (curU ? xU1 : xU0);
        const TC* xVc = curV < 0 ? nullptr : (curV ? xV1 : xV0);
        TC* xUn = curU == 0 ? xU1 : xU0;
        TC* xVn = curV == 0 ? xV1 : xV0;
        double acc[2] = {0.0, 0.0};
        // rows of the components that still sweep
        const int V = jacobi_width(k.d.N, (onU ? k.d.M - 1 : 0) + (onV ? k.d.M - 2 : 0), nw, (int)sizeof(TC));
        if (V == 1)
            jacobi_pass<TC, Mixed, 1>(k, U, W, u, v, xUc, xUn, xVc, xVn, onU, onV, T, acc);
        else if (sizeof(TC) == 4 && V == 2)
            jacobi_pass<TC, Mixed, sizeof(TC) == 4 ? 2 : 1>(k, U, W, u, v, xUc, xUn, xVc, xVn, onU, onV, T, acc);
        else
            jacobi_pass<TC, Mixed, Vec16<TC>::n>(k, U, W, u, v, xUc, xUn, xVc, xVn, onU, onV, T, acc);
        if (!team_reduce(T, target, acc, part, sm)) return false;
        if (onU) {
            curU = curU == 0 ? 1 : 0;
            onU = ++itU < k.maxMom && !(acc[0] < limU);
        }
        if (onV) {
            curV = curV == 0 ? 1 : 0;
            onV = ++itV < k.maxMom && !(acc[1] < limV);
        }
    }
    return true;
}

// The sweeps of one component on row segments (32 lane groups of 16 bytes),
// one segment a warp and trip.  Used where both components' systems do not stay
// in the L2 or one is swept alone (host: jacobi_sequential), and in the batched
// kernel, whose fields share the L2: there the sweeps of U and then V beat
// those of both at once (34 sweeps at 2048 x 1024 in float: 0.42 against
// 0.58 ms; 24 batched fields: 155 against 172 ms), and more warps with fewer
// registers beat the prefetch (0.42 against 0.49 ms).
template <typename TC, bool Mixed, bool IsU, int Loads = kReduceLoads>
__device__ __forceinline__ bool jacobi_component(const KParams& k, const MomSys<TC>& S, const double* field,
                                                 TC* x0, TC* x1, double* part, const Team& T, unsigned& target,
                                                 int& cur, int& its) {
    __shared__ double sm[kReduceSm];
    const Dims d = k.d;
    int i1, j1;
    mom_range<IsU>(d, i1, j1);
    const int n = i1 * j1;
    const double lim = k.momTol * k.momTol * (double)n;
    TC* xs[2] = {x0, x1};
    cur = -1;
    its = 0;
    for (int s = 0; s < k.maxMom; ++s) {
        const int nxt = cur < 0 ? 0 : 1 - cur;
        const TC* xc = cur < 0 ? nullptr : xs[cur];
        TC* __restrict__ xn = xs[nxt];
        const bool first = cur < 0;
        double acc[1] = {0.0};
        // row segments: a lane takes 16 bytes of a row (4 floats or 2
        // doubles); horizontal neighbours from the adjacent lanes
        constexpr int V = Vec16<TC>::n;
        row_segments<TC>(T, i1, j1, [&](int i, int j0, bool act, int lane) {
            const size_t c = at(d, i, j0);
            auto Xv = [&](size_t q) -> Vec16<TC> {
                if (first) {
                    if constexpr (Mixed) return zero16<TC>();
                    else return ld16(field + q);
                }
                return ld16(xc + q);
            };
            auto Xs = [&](size_t q) -> TC {
                if (first) return Mixed ? (TC)0 : (TC)field[q];
                return xc[q];
            };
            Vec16<TC> aP = zero16<TC>(), aE = aP, aW = aP, aN = aP, aS = aP, b = aP, xP = aP, xN = aP, xS = aP;
            if (act) {
                aP = ld16(S.aP + c);
                aE = ld16(S.aE + c);
                aW = ld16(S.aW + c);
                aN = ld16(S.aN + c);
                aS = ld16(S.aS + c);
                b = ld16(S.b + c);
                xP = Xv(c);
                if (i > 1) xS = Xv(c - d.P);
                if (i < i1) xN = Xv(c + d.P);
            }
            TC xw = from_west(xP.v[V - 1]), xe = from_east(xP.v[0]);
            if (lane == 0) xw = (act && j0 > 0) ? Xs(c - 1) : (TC)0;
            if (lane == 31) xe = act ? Xs(c + V) : (TC)0;
            Vec16<TC> o;
#pragma unroll
            for (int q = 0; q < V; ++q) {
                const int j = j0 + q;
                const bool in = act && j >= 1 && j <= j1;
                const TC W = (j > 1) ? (q ? xP.v[q - 1] : xw) : (TC)0;
                const TC E = (j < j1) ? (q < V - 1 ? xP.v[q + 1] : xe) : (TC)0;
                // S, W, P, E, N order of the reference's CSR rows
                TC Ax = (TC)0;
                Ax += (-aS.v[q]) * xS.v[q];
                Ax += (-aW.v[q]) * W;
                Ax += aP.v[q] * xP.v[q];
                Ax += (-aE.v[q]) * E;
                Ax += (-aN.v[q]) * xN.v[q];
                const TC r = b.v[q] - Ax;
                o.v[q] = in ? (TC)(xP.v[q] + r / aP.v[q]) : (TC)0;
                if (in) acc[0] += (double)r * (double)r;
            }
            if (act) st16(xn + c, o);
        });
        if (!team_reduce<1, Loads>(T, target, acc, part, sm)) return false;
        cur = nxt;
        its = s + 1;
        if (acc[0] < lim) break;
    }
    return true;
}

// scatter with clamp and max |u* - u| (momentum_solver.cpp:335-351); with
// outlet, the outlet column (boundaries.cpp:50-118) as a copy of the last one
template <typename TC, bool Mixed, bool IsU>
__device__ __forceinline__ double jacobi_scatter(const KParams& k, const double* field, const TC* xr,
                                                 double* out, double maxVel, bool outlet, int tid, int nth) {
    const Dims d = k.d;
    int i1, j1;
    mom_range<IsU>(d, i1, j1);
    const int w = j1, n = i1 * j1;
    double m = 0.0;
    for (int t = tid; t < n; t += nth) {
        const int i = 1 + t / w, j = 1 + t % w;
        const size_t c = at(d, i, j);
        double xv = xr ? (double)xr[c] : (Mixed ? 0.0 : field[c]);
        if (Mixed) xv += field[c];
        const double nv = dclamp(xv, -maxVel, maxVel);
        m = dmax(m, fabs(nv - field[c]));
        out[c] = nv;
        if (outlet && j == j1) out[c + 1] = nv;
    }
    return m;
}

struct JacobiOut {
    double *uStar, *vStar;
};

// The sweeps (Seq: one component after the other), then the scatter with
// clamps and the BCs on u*, v*
template <typename TC, bool Mixed, bool Seq>
__global__ void __launch_bounds__(Seq ? kJacSegThreads : kJacThreads, Seq ? 3 : 1) k_jacobi(KParams k, Status* st, MomSys<TC> U, MomSys<TC> V,
                                                const double* u, const double* v, TC* xU0, TC* xU1, TC* xV0,
                                                TC* xV1, JacobiOut out, const double* gamma, double* part,
                                                unsigned* bar, int doU, int doV, int applyBC) {
    if (st->done) return;
    const int G = gridDim.x;
    const int iter = st->iter;
    const double maxVel = max_vel(inlet_velocity(k, iter));
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = G * blockDim.x;
    unsigned target = 0;
    const Team T = grid_team(bar, &st->err);
    int curU = -1, curV = -1, itU = 0, itV = 0;
    if constexpr (Seq) {
        // (three CTAs an SM have 444 partials, 14 a lane)
        if (doU && !jacobi_component<TC, Mixed, true, 14>(k, U, u, xU0, xU1, part, T, target, curU, itU)) return;
        if (doV && !jacobi_component<TC, Mixed, false, 14>(k, V, v, xV0, xV1, part, T, target, curV, itV)) return;
    } else {
        if (!jacobi_sweeps<TC, Mixed>(k, U, V, u, v, xU0, xU1, xV0, xV1, doU, doV, part, T, target, curU, curV, itU, itV))
            return;
    }
    double mu = 0.0, mv = 0.0;
    if (doU) mu = jacobi_scatter<TC, Mixed, true>(k, u, curU < 0 ? nullptr : (curU ? xU1 : xU0), out.uStar, maxVel, applyBC, tid, nth);
    if (doV) mv = jacobi_scatter<TC, Mixed, false>(k, v, curV < 0 ? nullptr : (curV ? xV1 : xV0), out.vStar, maxVel, applyBC, tid, nth);
    if (applyBC) apply_bc_const(k, iter, out.uStar, out.vStar, gamma, tid, nth);
    mu = warp_max(mu);
    mv = warp_max(mv);
    if ((threadIdx.x & 31) == 0) {
        atomic_max_nonneg(&st->maxDU, mu);
        atomic_max_nonneg(&st->maxDV, mv);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (doU) st->itersU = itU;
        if (doV) st->itersV = itV;
    }
}

// The same on two clusters, one a component, for grids small enough (at most
// kClMaxK x 512 unknowns of either in a CTA's share of the rows, cluster_unknowns): the six coefficients of a thread's unknowns stay
// in registers and the iterate, with the neighbour blocks' rows beside a
// block's, in two buffers of shared memory, so that a sweep is one pass over
// them and one cluster barrier, which carries the sum too.  Per unknown the
// arithmetic is jacobi_run's, so the same number of sweeps gives the same bits of
// u* and v*; the sums that end them are added in another order.  us for the
// sweeps, here and on every SM: 15.6 and 34.0 at 40 x 17 (11.5 sweeps, double),
// 27.2 and 56.6 at 256 x 64 (19.5), 38.6 and 75.0 at 253 x 127 (26.6), 40.7 and
// 60.1 at 400 x 100 (float, 19.4), 47.6 and 61.0 there in double with K = 6.
constexpr size_t kJacClSmemMax = 2 * 3 * (kClMaxK * kClThreads + 3) * 8;   // one row a CTA, or rows of two unknowns
inline size_t jac_cl_smem(const Dims& d, size_t es) { return (size_t)2 * (cluster_rows(d.M - 1) + 2) * (d.N + 1) * es; }
inline int jac_cl_k(const Dims& d) {
    const int U = cluster_unknowns(d.M - 1, d.N - 2), V = cluster_unknowns(d.M - 2, d.N - 1);
    return U && V ? (U > V ? U : V) : 0;
}

template <typename TC, bool Mixed, bool IsU, int K>
__device__ __forceinline__ void jacobi_cluster(const KParams& k, Status* st, const MomSys<TC>& S, const double* field,
                                               double* out, double maxVel, bool outlet, TC* buf, ClusterSums& sm) {
    const Dims d = k.d;
    int i1, j1;
    mom_range<IsU>(d, i1, j1);
    const int rank = blockIdx.x % kClCtas, tid = threadIdx.x, W = d.N + 1;
    const int R = cluster_rows(i1), i0 = 1 + rank * R, rows = max(0, min(R, i1 + 1 - i0));
    const int len = (R + 2) * W;    // a buffer: row l of the block at (l + 1) W, column j at j
    for (int t = tid; t < 2 * len; t += kClThreads) buf[t] = (TC)0;
    __syncthreads();
    TC aP[K], aE[K], aW[K], aN[K], aS[K], b[K];
    int at0[K];     // place in a buffer, 0 past the block's unknowns
#pragma unroll
    for (int m = 0; m < K; ++m) {
        const int q = tid + m * kClThreads, l = q / j1, j = 1 + q - l * j1;
        at0[m] = 0;
        aP[m] = aE[m] = aW[m] = aN[m] = aS[m] = b[m] = (TC)0;
        if (l >= rows) continue;
        const size_t c = at(d, i0 + l, j);
        at0[m] = (l + 1) * W + j;
        aP[m] = S.aP[c];
        aE[m] = S.aE[c];
        aW[m] = S.aW[c];
        aN[m] = S.aN[c];
        aS[m] = S.aS[c];
        b[m] = S.b[c];
        // the current field, or zero in the mixed form
        if constexpr (!Mixed) {
            buf[at0[m]] = field[c];
            if (l == 0 && rank > 0) buf[j] = field[c - d.P];
            if (l == rows - 1 && i0 + l < i1) buf[at0[m] + W] = field[c + d.P];
        }
    }
    // the neighbour blocks' rows beside this block's: north of rank - 1, south of rank + 1
    const bool hasS = rank > 0 && rows > 0, hasN = rows > 0 && i0 + rows <= i1;
    const unsigned toS = cluster_addr(buf + (R + 1) * W, hasS ? rank - 1 : rank),
                   toN = cluster_addr(buf, hasN ? rank + 1 : rank);
    const double lim = k.momTol * k.momTol * (double)(IsU ? k.nU : k.nV);
    int flip = 0, its = 0;
    bool on = k.maxMom > 0;
    const TC* x = buf;
    cluster_barrier();   // every block's shared memory is there, and loaded
    while (on) {
        const int nx = its & 1 ? 0 : len;
        TC* const xn = buf + nx;
        double acc[1] = {0.0};
#pragma unroll
        for (int m = 0; m < K; ++m) {
            const int o = at0[m];
            if (!o) continue;
            const TC xP = x[o];
            // S, W, P, E, N order of the reference's CSR rows
            TC Ax = (TC)0;
            Ax += (-aS[m]) * x[o - W];
            Ax += (-aW[m]) * x[o - 1];
            Ax += aP[m] * xP;
            Ax += (-aE[m]) * x[o + 1];
            Ax += (-aN[m]) * x[o + W];
            const TC r = b[m] - Ax;
            const TC y = (TC)(xP + r / aP[m]);
            acc[0] += (double)r * (double)r;
            xn[o] = y;
            if (hasS && o < 2 * W) cluster_store(toS + (unsigned)((nx + o - W) * sizeof(TC)), y);
            if (hasN && o >= rows * W) cluster_store(toN + (unsigned)((nx + o - rows * W) * sizeof(TC)), y);
        }
        cluster_reduce(sm, flip, rank, acc);
        x = xn;
        on = ++its < k.maxMom && !(acc[0] < lim);
    }
    double mx = 0.0;
#pragma unroll
    for (int m = 0; m < K; ++m) {
        const int q = tid + m * kClThreads, l = q / j1, j = 1 + q - l * j1;
        if (!at0[m]) continue;
        const size_t c = at(d, i0 + l, j);
        double xv = (double)x[at0[m]];
        if (Mixed) xv += field[c];
        const double nv = dclamp(xv, -maxVel, maxVel);
        mx = dmax(mx, fabs(nv - field[c]));
        out[c] = nv;
        if (outlet && j == j1) out[c + 1] = nv;
    }
    mx = warp_max(mx);
    if ((tid & 31) == 0) atomic_max_nonneg(IsU ? &st->maxDU : &st->maxDV, mx);
    if (rank == 0 && tid == 0) {
        if (IsU) st->itersU = its;
        else st->itersV = its;
    }
}

template <typename TC, bool Mixed, int K>
__global__ void __launch_bounds__(kClThreads, 1) k_jacobi_cluster(KParams k, Status* st, MomSys<TC> U, MomSys<TC> V,
                                                                  const double* u, const double* v, JacobiOut out,
                                                                  const double* gamma, int doU, int doV, int applyBC) {
    if (st->done) return;
    extern __shared__ __align__(128) double jsm[];
    __shared__ ClusterSums sm;
    const int iter = st->iter;
    const double maxVel = max_vel(inlet_velocity(k, iter));
    TC* const buf = reinterpret_cast<TC*>(jsm);
    if (blockIdx.x < kClCtas) {
        if (doU) jacobi_cluster<TC, Mixed, true, K>(k, st, U, u, out.uStar, maxVel, applyBC, buf, sm);
    } else {
        if (doV) jacobi_cluster<TC, Mixed, false, K>(k, st, V, v, out.vStar, maxVel, applyBC, buf, sm);
    }
    if (applyBC)
        apply_bc_const(k, iter, out.uStar, out.vStar, gamma, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ------------------------------------------------------------------ mass
// One pass over cells (i, j) in [1, M-1] x [1, N-1]: RMS sums of u* - u and
// v* - v over their unknowns (iterations.cpp:507-525), the mass imbalance
// max and sum of squares (pressure_solver.cpp:473-487), and the PCG rhs on
// the pressure unknowns j <= N-2 (pressure_solver.cpp:733-742).
// part[b*4 + {0,1,2,3}] = {sum du^2, sum dv^2, sum b^2, max |b|}.
template <typename TV>
__device__ __forceinline__ void mass_pass(const KParams& k, const double* u, const double* v, const double* uStar,
                                          const double* vStar, TV* rhs, int tid, int nth, double* o) {
    __shared__ double sm[128];
    const Dims d = k.d;
    const int M = d.M, N = d.N, w = N - 1;
    const double rho = k.rho, hx = k.hx, hy = k.hy;
    double acc[3] = {0.0, 0.0, 0.0};
    double mmax = 0.0;
    const int n = (M - 1) * w;
    for (int t = tid; t < n; t += nth) {
        const int i = 1 + t / w, j = 1 + t % w;
        const size_t c = at(d, i, j);
        const double massE = rho * uStar[c] * hy, massW = rho * uStar[c - 1] * hy;
        const double massN = rho * vStar[c] * hx, massS = rho * vStar[c - d.P] * hx;
        const double b = massW - massE + massS - massN;
        const double ab = fabs(b);
        mmax = dmax(mmax, ab);
        acc[2] += ab * ab;
        if (j <= N - 2) {
            const double du = uStar[c] - u[c];
            acc[0] += du * du;
            rhs[c] = (TV)b;
        }
        if (i <= M - 2) {
            const double dv = vStar[c] - v[c];
            acc[1] += dv * dv;
        }
    }
    block_sum<3>(acc, sm);
    mmax = warp_max(mmax);
    if ((threadIdx.x & 31) == 0) sm[96 + (threadIdx.x >> 5)] = mmax;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int q = 0; q < (int)((blockDim.x + 31) >> 5); ++q) m = dmax(m, sm[96 + q]);
        o[0] = acc[0]; o[1] = acc[1]; o[2] = acc[2]; o[3] = m;
    }
}

template <typename TV>
__global__ void k_mass(KParams k, const Status* st, const double* u, const double* v, const double* uStar,
                       const double* vStar, TV* rhs, double* part) {
    if (st->done) return;
    mass_pass<TV>(k, u, v, uStar, vStar, rhs, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x,
                  part + (size_t)blockIdx.x * 4);
}

// ------------------------------------------------------------------ correction
// p += pAlpha p' on [1,M-1] x [1,N-1]; u = clamp(u* + clamp(dE (p'_ij - p'_i,j+1)))
// on U unknowns and the same for v (iterations.cpp:558-597); then the boundary
// conditions (iterations.cpp:567, 599), each by the thread that owns the
// interior value it copies.  The inlet and the walls have their values from the
// start of the iteration.
__device__ __forceinline__ void correct_cells(const KParams& k, int iter, double* u, double* v, double* p,
                                              const double* uStar, const double* vStar, const double* pStar,
                                              const double* dE, const double* dN, int tid, int nth) {
    const Dims d = k.d;
    const int M = d.M, N = d.N, w = N - 1;
    const double maxVel = max_vel(inlet_velocity(k, iter));
    const int n = (M - 1) * w;
    for (int t = tid; t < n; t += nth) {
        const int i = 1 + t / w, j = 1 + t % w;
        const size_t c = at(d, i, j);
        const double ps = pStar[c];
        const double np = p[c] + k.pAlpha * ps;
        p[c] = np;
        if (i == 1) p[at(d, 0, j)] = np;
        if (i == M - 1) p[at(d, M, j)] = np;
        if (j == 1) p[at(d, i, 0)] = np;
        if (j == w) p[c + 1] = 0.0;
        if (j <= N - 2) {
            double du = dE[c] * (ps - pStar[c + 1]);
            du = dmax(-maxVel, dmin(maxVel, du));
            const double nu = dmax(-maxVel, dmin(maxVel, uStar[c] + du));
            u[c] = nu;
            if (j == N - 2) u[c + 1] = nu;
        }
        if (i <= M - 2) {
            double dv = dN[c] * (ps - pStar[c + d.P]);
            dv = dmax(-maxVel, dmin(maxVel, dv));
            const double nv = dmax(-maxVel, dmin(maxVel, vStar[c] + dv));
            v[c] = nv;
            if (j == w) v[c + 1] = nv;
        }
    }
}

__global__ void k_correct(KParams k, const Status* st, double* u, double* v, double* p, const double* uStar,
                          const double* vStar, const double* pStar, const double* dE, const double* dN) {
    if (st->done) return;
    correct_cells(k, st->iter, u, v, p, uStar, vStar, pStar, dE, dN, blockIdx.x * blockDim.x + threadIdx.x,
                  gridDim.x * blockDim.x);
}

// ------------------------------------------------------------------ finalize
// Pressure sampling (postprocessing.cpp:103-327): metrics m[5] =
// {flowArea, massFlux, avgStatic, avgDynamic, avgTotal}.  Sums are double
// block reductions (the reference adds floats sequentially).
__device__ void finish_metrics(double area, double fs, double st, double dy, double tw, double* m) {
    double aS = 0.0, aD = 0.0, aT = 0.0;
    if (area > 0.0) { aS = st / area; aD = dy / area; }
    if (fs > 0.0) aT = tw / fs;
    else if (area > 0.0) aT = aS + aD;
    m[0] = area; m[1] = fs; m[2] = aS; m[3] = aD; m[4] = aT;
}

// kind 0: plane at x (interpolated), 1: inlet patch, 2: outlet patch
// one thread's share of the sample, rows 1 + t, 1 + t + nt, ...: acc[5] = {area,
// flux, static, dynamic, flux-weighted total}
__device__ __forceinline__ void sample_rows(const KParams& k, const double* u, const double* v, const double* p,
                                            const double* gamma, int kind, double x, int t, int nt, double (&acc)[5]) {
    const Dims d = k.d;
    const int M = d.M, N = d.N, NC = N - 1;
    const double hx = k.hx, hy = k.hy, rho = k.rho;
    int cl = 0, cr = 0;
    double wt = 0.0;
    if (kind == 0 && NC > 1) {
        const double xMin = 0.5 * hx, xMax = ((double)NC - 0.5) * hx;
        const double xc = dmax(xMin, dmin(x, xMax));
        cl = (int)floor(xc / hx - 0.5);
        if (cl > NC - 2) cl = NC - 2;
        if (cl < 0) cl = 0;
        cr = cl + 1;
        const double xl = ((double)cl + 0.5) * hx, xr = ((double)cr + 0.5) * hx;
        wt = (fabs(xr - xl) < 1e-12) ? 0.0 : (xc - xl) / (xr - xl);
        wt = dmax(0.0, dmin(1.0, wt));
    }
    for (int i = 1 + t; i < M; i += nt) {
        const int row = i - 1;
        const int vt = (i - 1 < M - 1) ? i - 1 : M - 1, vb = (i < M - 1) ? i : M - 1;
        double staticP, un, vtan;
        if (kind == 0) {
            if (cl < 0 || cl >= NC || cr < 0 || cr >= NC) continue;
            if (gamma[at(d, row, cl)] < 1.0 - 1e-6 || gamma[at(d, row, cr)] < 1.0 - 1e-6) continue;
            const int pl = cl + 1 < N ? cl + 1 : N, pr = cr + 1 < N ? cr + 1 : N;
            staticP = (1.0 - wt) * p[at(d, i, pl)] + wt * p[at(d, i, pr)];
            const int ul = cl < N - 1 ? cl : N - 1, ur = cr < N - 1 ? cr : N - 1;
            un = (1.0 - wt) * u[at(d, i, ul)] + wt * u[at(d, i, ur)];
            const int vl = cl < N ? cl : N, vr = cr < N ? cr : N;
            const double vTop = (1.0 - wt) * v[at(d, vt, vl)] + wt * v[at(d, vt, vr)];
            const double vBot = (1.0 - wt) * v[at(d, vb, vl)] + wt * v[at(d, vb, vr)];
            vtan = 0.5 * (vTop + vBot);
        } else {
            const bool inlet = (kind == 1);
            const int adj = inlet ? 0 : NC - 1;
            if (adj < 0 || adj >= NC) continue;
            if (gamma[at(d, row, adj)] < 1.0 - 1e-6) continue;
            const int uCol = inlet ? 0 : N - 1, pCol = inlet ? 0 : N, vCol = inlet ? 0 : N;
            staticP = p[at(d, i, pCol)];
            un = u[at(d, i, uCol)];
            vtan = 0.5 * (v[at(d, vt, vCol)] + v[at(d, vb, vCol)]);
        }
        const double vm = sqrt(un * un + vtan * vtan);
        const double dynP = 0.5 * rho * vm * vm;
        const double tot = staticP + dynP;
        acc[0] += hy;
        acc[2] += staticP * hy;
        acc[3] += dynP * hy;
        const double fa = fabs(rho * un * hy);
        if (fa > 0.0) { acc[1] += fa; acc[4] += tot * fa; }
    }
}

struct FinalizeArgs {
    const double *u, *v, *p, *gamma;
    const double* partM;   // k_mass partials
    int nbM;
    double* hist;          // [cap][kHistCols]
    int histCap;
    double* dpWin;         // [dpWindow]
};

// One block: residual norms from the k_mass partials, the four pressure
// samples, the history row and the stop rules of one field.  Everything it
// reads is in flight at once (a quarter of the block a sample) and summed
// behind one block barrier; a sample after the other took 21 us at 253 x 127
// and 29 us at 2048 x 1024, launch included, now 13 and 19.  At least 128 threads, a multiple of 128.
__device__ __forceinline__ void finalize_block(const KParams& k, Status* st, const FinalizeArgs& a) {
    __shared__ double sm[32][9];
    __shared__ double met[4][5];
    __shared__ double sums[4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    {
        // {sum du^2, sum dv^2, sum b^2, max |b|} and the warp's sample
        double r[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int b = threadIdx.x; b < a.nbM; b += blockDim.x) {
            r[0] += a.partM[b * 4 + 0];
            r[1] += a.partM[b * 4 + 1];
            r[2] += a.partM[b * 4 + 2];
            r[3] = dmax(r[3], a.partM[b * 4 + 3]);
        }
        const int nt = blockDim.x >> 2, q = threadIdx.x / nt;
        double acc[5] = {0, 0, 0, 0, 0};
        sample_rows(k, a.u, a.v, a.p, a.gamma, q < 2 ? 0 : q - 1, q == 0 ? k.xCoreIn : k.xCoreOut, threadIdx.x - q * nt, nt, acc);
#pragma unroll
        for (int e = 0; e < 5; ++e) r[4 + e] = acc[e];
#pragma unroll
        for (int e = 0; e < 9; ++e) {
            r[e] = e == 3 ? warp_max(r[e]) : warp_sum(r[e]);
            if (lane == 0) sm[wid][e] = r[e];
        }
        __syncthreads();
        if (threadIdx.x < 4) {
            double t = 0.0;
            for (int w = 0; w < nw; ++w) t = threadIdx.x == 3 ? dmax(t, sm[w][3]) : t + sm[w][threadIdx.x];
            sums[threadIdx.x] = t;
        } else if (threadIdx.x >= 32 && threadIdx.x < 36) {
            const int s = threadIdx.x - 32, w0 = s * (nw >> 2);
            double t[5] = {0, 0, 0, 0, 0};
            for (int w = w0; w < w0 + (nw >> 2); ++w)
#pragma unroll
                for (int e = 0; e < 5; ++e) t[e] += sm[w][4 + e];
            double m[5];
            finish_metrics(t[0], t[1], t[2], t[3], t[4], m);
            for (int e = 0; e < 5; ++e) met[s][e] = m[e];
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;

    const int iter = st->iter;
    const double nU = (double)k.nU, nV = (double)k.nV, nM = (double)((k.d.M - 1) * (k.d.N - 1));
    const double rmsU = nU > 0 ? sqrt(sums[0] / nU) : 0.0;
    const double rmsV = nV > 0 ? sqrt(sums[1] / nV) : 0.0;
    const double rmsM = nM > 0 ? sqrt(sums[2] / nM) : 0.0;
    const double maxM = sums[3];
    const double maxU = __longlong_as_double((long long)st->maxDU);
    const double maxV = __longlong_as_double((long long)st->maxDV);
    // residual normalisation bookkeeping (iterations.cpp:628-656)
    const double velFloor = dmax(k.velFloor, 1e-30), massFloor = dmax(k.massFloor, 1e-30);
    if (!st->rms0Uset && rmsU > velFloor) { st->rms0U = rmsU; st->rms0Uset = 1; }
    if (!st->rms0Vset && rmsV > velFloor) { st->rms0V = rmsV; st->rms0Vset = 1; }
    if (!st->rms0Mset && rmsM > massFloor) { st->rms0M = rmsM; st->rms0Mset = 1; }
    if (!st->rms0Uset) st->rms0U = velFloor;
    if (!st->rms0Vset) st->rms0V = velFloor;
    if (!st->rms0Mset) st->rms0M = massFloor;
    double rU = rmsU, rV = rmsV, rM = rmsM;
    if (k.normalized) { rU = rmsU / st->rms0U; rV = rmsV / st->rms0V; rM = rmsM / st->rms0M; }
    const double error = dmax(dmax(rU, rV), rM);
    const double coreTotal = met[0][4] - met[1][4], fullTotal = met[2][4] - met[3][4];
    const double coreStatic = met[0][2] - met[1][2], fullStatic = met[2][2] - met[3][2];
    if (iter < a.histCap) {
        double* h = a.hist + (size_t)iter * kHistCols;
        h[H_ITER] = iter; h[H_ERROR] = error; h[H_RMS_U] = rmsU; h[H_RMS_V] = rmsV; h[H_RMS_MASS] = rmsM;
        h[H_MAX_U] = maxU; h[H_MAX_V] = maxV; h[H_MAX_MASS] = maxM; h[H_ITERS_P] = st->itersP;
        h[H_CORE_TOTAL] = coreTotal; h[H_FULL_TOTAL] = fullTotal; h[H_CORE_STATIC] = coreStatic;
        h[H_FULL_STATIC] = fullStatic; h[H_IN_FLUX] = met[2][1]; h[H_OUT_FLUX] = met[3][1];
        h[H_ITERS_U] = st->itersU; h[H_ITERS_V] = st->itersV; h[H_RES_U] = rU; h[H_RES_V] = rV; h[H_RES_MASS] = rM;
    }
    st->lastError = error;
    // stop rules of the outer loop (SIMPLE.cpp:378, 449-491)
    int done = 0, reason = CP_RUNNING;
    if (!(error == error) || isinf(error) || !(coreTotal == coreTotal) || !(fullTotal == fullTotal)) {
        done = 1; reason = CP_STOP_ERROR;
        atomicCAS(&st->err, 0, (int)CP_ERR_NONFINITE);
    }
    if (st->err != 0) { done = 1; reason = CP_STOP_ERROR; }
    if (!done && k.dpConv && iter >= k.dpRampSteps && k.dpWindow > 0) {
        a.dpWin[st->dpIdx] = coreTotal;
        st->dpIdx = (st->dpIdx + 1) % k.dpWindow;
        if (st->dpIdx == 0) st->dpFilled = 1;
        if (st->dpFilled) {
            double sum = 0.0;
            for (int q = 0; q < k.dpWindow; ++q) sum += a.dpWin[q];
            const double mean = sum / (double)k.dpWindow;
            double var = 0.0;
            for (int q = 0; q < k.dpWindow; ++q) { const double df = a.dpWin[q] - mean; var += df * df; }
            const double sd = sqrt(var / (double)k.dpWindow);
            const double denom = dmax(fabs(mean), 1.0);
            const double stdPct = sd / denom * 100.0;
            const int last = (st->dpIdx - 1 + k.dpWindow) % k.dpWindow;
            const double latestPct = fabs(a.dpWin[last] - mean) / denom * 100.0;
            if (stdPct < k.dpPercent && latestPct < k.dpPercent) { done = 1; reason = CP_STOP_DP_WINDOW; }
        }
    }
    if (!done && !(error > k.eps)) { done = 1; reason = CP_STOP_RESIDUAL; }
    if (!done && iter + 1 >= k.maxIterations) { done = 1; reason = CP_STOP_MAX_ITER; }
    st->iter = iter + 1;
    if (done) { st->reason = reason; __threadfence(); st->done = 1; }
}

__global__ void __launch_bounds__(1024) k_finalize(KParams k, Status* st, FinalizeArgs a) {
    if (st->done) return;
    finalize_block(k, st, a);
}

}  // namespace cp
