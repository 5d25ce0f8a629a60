// Differentiated FP64 step: tangent-linear (forward mode, Dual numbers) and
// hand-written adjoint (reverse mode) of the reference-pipeline step
// (ref_pipeline.cu, i.e. fvDVM::evolution, src/fvDVM/fvDVM/fvDVM.C:1086-1108),
// with respect to the wall temperatures T_w (per wall face) and the viscosity
// scale mu_ref (tau = mu_ref (T/Tref)^omega / (rho R T), fvDVM::updateTau,
// fvDVM.C:808-817).  Objective: sum over a window of steps of
//   sum_w S_w . qWall_w  (one patch)  +  sum_w |S_w| stressWall_w,xy  (one patch),
// with qWall / stressWall as fvDVM::updateMacroSurf forms them (fvDVM.C:535-576).
//
// The tangent-linear step runs the passes of ref_kernels.cuh on Dual scalars
// (value, derivative along one parameter direction): 32^2 quads x 28^2, 6 steps
// 14.3 -> 3.5 ms against kernels that formed the equilibrium, its divisions and
// exponentials per velocity.
// Adjoint kernels (r_*) run the passes in reverse:
//   r_cell_mom  P9  cell macros        <- g~n+1
//   r_cell_flux P8  g~n+1 = -g~/3 + 4/3 gbar+ - dt/V sum (xi.S) g_f
//   r_face      P7  face relaxation, P6 face macros (+ objective seeds)
//   r_wall      P5  incoming rho_w M_w, P4 rho_w = outgoing / |inComingByRho(T_w)|
//   r_recon     P3  upwind reconstruction (+ lagged wall gradient output)
//   r_grad      P2  least-squares gradient (+ lagged wall gradient input)
//   r_barp      P1  cell relaxation toward the Shakhov equilibrium
// Local Jacobians are analytic (Shakhov and Maxwellian in (rho, U, T, q)).
#include "device_common.cuh"
#include "dual.cuh"
#include "fused.h"
#include "gradient.h"
#include "ref_kernels.cuh"

namespace dugks {
namespace {

constexpr int kT = 256;
constexpr int kRT = 128;

int grid(long long n, int threads, int sms) {
    long long b = (n + threads - 1) / threads;
    long long cap = (long long)sms * 32;
    return (int)(b < cap ? (b > 0 ? b : 1) : cap);
}

// ------------------------------------------------------------ shared forms
template <class R>
__device__ __forceinline__ R maxwellT(double Ux, double Uy, double Uz, R T, double xx, double xy, double xz,
                                      double Rg, int D) {
    double ax = Ux - xx, ay = Uy - xy, az = Uz - xz;
    R s = sqrt(2.0 * kPi * Rg * T);
    R pw = (D == 2) ? s * s : (D == 3 ? s * s * s : s);
    return 1.0 / pw * exp(-(ax * ax + ay * ay + az * az) / (2.0 * Rg * T));
}

template <class R>
__device__ __forceinline__ R tauT(R T, R rho, R muRef, double omega, double Tref, double Rg) {
    return muRef * exp(omega * log(T / Tref)) / rho / T / Rg;
}

// ============================================================ tangent-linear
struct TArgs {
    StepArgs a;
    Dual *rho, *U, *T, *q, *tau;
    Dual *rhoF, *UF, *TF, *qF, *tauF;
    Dual *rhoW, *qWall, *stressWall;
    const Dual* Tw;
    Dual* incAbs;
    Dual muRef;
};

__global__ void t_incabs(TArgs t) {
    __shared__ double red[32 * 2];
    const StepArgs& a = t.a;
    const int wf = blockIdx.x, Vp = a.Vp;
    const double* S = a.Sf + 3 * (a.nI + wf);
    const double* Uw = a.Uw + 3 * wf;
    double acc[2] = {0.0, 0.0};
    for (int v = threadIdx.x; v < a.nV; v += blockDim.x) {
        double x0 = a.xi[v], x1 = a.xi[Vp + v], x2 = a.xi[2 * Vp + v];
        double xs = x0 * S[0] + x1 * S[1] + x2 * S[2];
        if (xs < 0) {
            Dual M = maxwellT<Dual>(Uw[0], Uw[1], Uw[2], t.Tw[wf], x0, x1, x2, a.R, a.D);
            Dual r = -a.w[v] * xs * M;
            acc[0] += r.v;
            acc[1] += r.d;
        }
    }
    block_sum<2>(acc, red);
    if (threadIdx.x == 0) t.incAbs[wf] = fabs(Dual{acc[0], acc[1]});
}

__global__ void t_init(TArgs t, const double* rho0, const double* U0, const double* T0) {
    const StepArgs& a = t.a;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.nC) return;
    t.rho[c] = dual(rho0[c]);
    for (int k = 0; k < 3; ++k) { t.U[3 * c + k] = dual(U0[3 * c + k]); t.q[3 * c + k] = dual(0.0); }
    t.T[c] = dual(T0[c]);
    t.tau[c] = tauT<Dual>(dual(T0[c]), dual(rho0[c]), t.muRef, a.omega, a.Tref, a.R);
}

// J += scale * (sum_w wq_w . qWall_w + ws_w stressWall_w,xy), one block, fixed order.
template <class R>
__global__ void k_objective(int nW, const double* wq, const double* ws, const R* qWall, const R* stressWall,
                            double scale, R* J) {
    __shared__ double red[32 * 2];
    double acc[2] = {0.0, 0.0};
    for (int w = threadIdx.x; w < nW; w += blockDim.x) {
        R s = wq[3 * w] * qWall[3 * w] + wq[3 * w + 1] * qWall[3 * w + 1] + wq[3 * w + 2] * qWall[3 * w + 2] +
              ws[w] * stressWall[9 * w + 1];
        if constexpr (sizeof(R) == sizeof(double)) {
            acc[0] += (double)s;
        } else {
            acc[0] += reinterpret_cast<const Dual&>(s).v;
            acc[1] += reinterpret_cast<const Dual&>(s).d;
        }
    }
    block_sum<2>(acc, red);
    if (threadIdx.x == 0) {
        if constexpr (sizeof(R) == sizeof(double)) {
            J[0] = (double)J[0] + scale * acc[0];
        } else {
            Dual& j = reinterpret_cast<Dual&>(J[0]);
            j.v += scale * acc[0];
            j.d += scale * acc[1];
        }
    }
}

// ============================================================ adjoint
// Per-cell adjoint of the macro tuple m = (rho, Ux, Uy, Uz, T, qx, qy, qz, tau)
// (9 doubles per cell; P1 of the next step reads all nine).
constexpr int kM = 9;

struct AArgs {
    StepArgs a;
    const double* Tw;   // wall temperatures (forward values)
    double muRef;
};

// The reverse passes run one warp per cell or face, like the forward ones, and
// are bound by the FP64 pipe as they are: what depends on the entity alone is
// formed by one lane per entity of the block, what depends on one direction of
// the tensor-product grid once per abscissa, into per-warp tables.
//
// Reverse of the Shakhov equilibrium (gE, hE)(rho, U, T, q) for one velocity's
// adjoints (lg, lh).  theta = R T, c = xi - U, a = |c|^2/theta, A = a - D - 2,
// G0 = (2 pi theta)^(-D/2) exp(-a/2), p = (1-Pr)/(5 theta^2) c.q, k3 = K+3-D,
// ck = 2 - 2K/k3:
//   gE = rho G0 + p G0 A,   hE = theta k3 (gE + ck p G0).
// With l3 = theta k3 lh, L = lg + l3, W = G0 L, V = G0 (A L + ck l3):
//   F = gE lg + hE lh = rho W + p V
//   dF/drho = W,  dF/dq_k = kap c_k V,  dF/dU_k = c_k (F - 2 p W)/theta - kap q_k V,
//   theta dF/dtheta = F (A+2)/2 - 2 p V - (A+D+2) p W + l3 G0 (rho + p (A + ck))
// (kap = (1-Pr)/(5 theta^2)), so a velocity costs 30 FP64 operations in 2D; the
// sums below are combined per entity (finish).  It was ~70 with every partial
// derivative formed per velocity.
template <int D, bool H, bool SEC>
struct Rev {
    static constexpr int U = 1, V = U + D, Q = V + 1, FA = Q + D, EV = FA + 1, AE = EV + 1, E = AE + 1, H2 = E + 1,
                         R = H2 + 1, S = R + 1;
    static constexpr int N2 = D * (D + 1) / 2;         // second moments sum w c_i c_j g (SEC)
    static constexpr int N = S + (SEC ? N2 : 0);
    static constexpr int NS = N <= 16 ? 16 : 32;
    static __device__ __forceinline__ void add(double* acc, double G0, double A, double p, const double* c, double g,
                                               double h, double lg, double lh, double rho, double tk3, double ck) {
        const double l3 = H ? tk3 * lh : 0.0, L = H ? lg + l3 : lg;
        const double AL = A * L, V0 = H ? fma(ck, l3, AL) : AL;
        const double W = G0 * L, v = G0 * V0, ev = p * v, F = fma(rho, W, ev), eL = p * W, t1 = fma(-2.0, eL, F);
        acc[0] += W;
        acc[V] += v;
        acc[EV] += ev;
        acc[E] += eL;
        acc[FA] = fma(F, A, acc[FA]);
        acc[AE] = fma(A, eL, acc[AE]);
        acc[R] = fma(g, lg, acc[R]);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            acc[U + k] = fma(c[k], t1, acc[U + k]);
            acc[Q + k] = fma(c[k], v, acc[Q + k]);
        }
        if (H) {
            acc[H2] = fma(l3 * G0, fma(p, A + ck, rho), acc[H2]);
            acc[R] = fma(h, lh, acc[R]);
        }
    }
    static __device__ __forceinline__ void add2(double* acc, double wg, const double* c) {  // N2 sums
        int n = 0;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const double t = wg * c[i];
#pragma unroll
            for (int j = i; j < D; ++j, ++n) acc[n] = fma(t, c[j], acc[n]);
        }
    }
    // Adjoint of (rho, U, T, q, tau) from the totals; w the relaxation weight, dw its tau derivative.
    static __device__ __forceinline__ void finish(const double* t, const double* m, double w, double dw, double Rg,
                                                  double Pr, double* lm) {
        const double ith = 1.0 / (Rg * m[4]), kap = (1.0 - Pr) / 5.0 * ith * ith;
        const double F = m[0] * t[0] + t[EV];
        lm[0] = w * t[0];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lm[1 + k] = k < D ? w * (ith * t[U + (k < D ? k : 0)] - m[5 + k] * kap * t[V]) : 0.0;
            lm[5 + k] = k < D ? w * kap * t[Q + (k < D ? k : 0)] : 0.0;
        }
        const double th = 0.5 * t[FA] + F - 2.0 * t[EV] - t[AE] - (D + 2.0) * t[E] + (H ? t[H2] : 0.0);
        lm[4] = w * Rg * th * ith;
        lm[8] = dw * (F - t[R]);
    }
};
__host__ __device__ constexpr int sidx(int D, int i, int j) {  // upper triangle, row-major
    return i <= j ? i * D - i * (i - 1) / 2 + (j - i) : j * D - j * (j - 1) / 2 + (i - j);
}

// Per-entity scalars of the equilibrium tables, one lane per entity.
struct EqScal {
    double U[3], kq[3], ith, N, rho, tk3;
};
template <int D>
__device__ __forceinline__ void eq_scal(EqScal& s, const double* m, const StepArgs& a) {
    const double th = a.R * m[4], ith = 1.0 / th, s2 = 2.0 * kPi * th, kap = (1.0 - a.Pr) / 5.0 * ith * ith;
    s.rho = m[0];
    s.ith = ith;
    s.N = D == 2 ? 1.0 / s2 : 1.0 / (s2 * sqrt(s2));
    s.tk3 = th * (a.K + 3.0 - D);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s.U[k] = m[1 + k];
        s.kq[k] = kap * m[5 + k];
    }
}
// Tables of one entity, [4][D][M]: G0 factors, A terms, p terms, c.
template <int D>
__device__ __forceinline__ void eq_tables(const StepArgs& a, const EqScal& s, double* tb, int lane) {
    const int DM = D * a.M;
    for (int t = lane; t < DM; t += 32) {
        const int k = t / a.M;
        const double c = a.x1[t - k * a.M] - s.U[k], ci = c * c * s.ith;
        const double G = exp(-0.5 * ci);
        tb[t] = k == 0 ? s.N * G : G;
        tb[DM + t] = k == 0 ? ci - (D + 2.0) : ci;
        tb[2 * DM + t] = c * s.kq[k];
        tb[3 * DM + t] = c;
    }
    __syncwarp();
}
template <int D>
__device__ __forceinline__ void eq_lookup(const double* tb, int DM, int M, const DvIdx<D>& id, double& G0, double& A,
                                          double& p, double* c) {
    const double *x = tb + id.ix, *y = tb + M + id.iy;
    G0 = x[0] * y[0];
    A = x[DM] + y[DM];
    p = x[2 * DM] + y[2 * DM];
    c[0] = x[3 * DM];
    c[1] = y[3 * DM];
    if (D == 3) {
        const double* z = tb + 2 * M + id.iz;
        G0 *= z[0];
        A += z[DM];
        p += z[2 * DM];
        c[D - 1] = z[3 * DM];
    }
}

// Reverse of the macro evaluation of one entity (P9 for cells, P6 for faces;
// fvDVM::updateMacroVol fvDVM.C:597-728, updateMacroSurf :456-582).  Inputs:
// the forward macros m, lm = adjoint of (rho, U, T, q, tau) with q = fac(tau) Q
// and fac = 2 tau / (2 tau + facA) (cells facA = dt Pr, faces dt Pr / 2), the
// second moments S_ij = sum w c_i c_j g; sum w (|c|^2 g + h) = (K+3) R rho T and
// Q = q / fac come from the macros.  On walls lqw, lsw are the adjoints of
// qWall = fac Qw and stressWall = fs X (fs = 2 tau / (2 tau + dt/2)) and sw holds
// Qw_i = 1/2 sum w e_i (|e|^2 g + h) (e = xi - Uw), X_ij = sum w xi_i xi_j g.
// Output: coefficients so that
//   lg += w [lrho + lP.xi + hE |xi|^2 + (hQ.c) |c|^2 + (hQw.e)|e|^2 + xi.lX.xi]
//   lh += w [hE + hQ.c + hQw.e],
// and the mu_ref adjoint (tau = mu_ref (T/Tref)^omega / (rho R T)), returned.
template <int D>
struct MacroAdj {
    double lrho, hE, lP[3], hQ[3], hQw[3], lX[9], U[3];
    __device__ __forceinline__ double chain(const StepArgs& a, const double* m, const double* lm, const double* S,
                                            double facA, double muRef, bool wall, const double* lqw, const double* lsw,
                                            const double* sw) {
        const double rho = m[0], T = m[4], tau = m[8], cv = (a.K + 3) / 2.0 * a.R;
        const double den = 1.0 / (2.0 * tau + facA), fac = 2.0 * tau * den, dfac = 2.0 * facA * den * den;
        const double irho = 1.0 / rho, icv = 1.0 / cv, S0 = 2.0 * cv * rho * T, ifac = 1.0 / fac;
        double lU[D], lQ[D], uu = 0.0, lT = lm[4], ltau = lm[8];
        lrho = lm[0];
#pragma unroll
        for (int i = 0; i < D; ++i) {
            U[i] = m[1 + i];
            uu += U[i] * U[i];
            lU[i] = lm[1 + i];
            lQ[i] = lm[5 + i] * fac;
            ltau += lm[5 + i] * m[5 + i] * ifac * dfac;
        }
        if (wall) {
            const double ds = 1.0 / (2.0 * tau + 0.5 * a.dt), fs = 2.0 * tau * ds, dfs = a.dt * ds * ds;
#pragma unroll
            for (int i = 0; i < D; ++i) {
                hQw[i] = 0.5 * (lqw[i] * fac);
                ltau += lqw[i] * sw[i] * dfac;
            }
#pragma unroll
            for (int i = 0; i < D; ++i)
#pragma unroll
                for (int j = 0; j < D; ++j) {
                    ltau += lsw[3 * i + j] * sw[D + sidx(D, i, j)] * dfs;
                    lX[D * i + j] = fs * lsw[3 * i + j];
                }
        }
        lT += ltau * tau * (a.omega - 1.0) / T;
        lrho -= ltau * tau * irho;
        const double lmu = ltau * tau / muRef;
        // Q_i depends on U through c = xi - U
#pragma unroll
        for (int k = 0; k < D; ++k)
#pragma unroll
            for (int i = 0; i < D; ++i) lU[k] -= lQ[i] * ((i == k ? 0.5 * S0 : 0.0) + S[sidx(D, i, k)]);
        // T = (E - rho |U|^2 / 2) / (cv rho)
        const double lE = lT * icv * irho;
        lrho += lT * (-0.5 * uu * icv * irho - T * irho);
        // U = P / rho
#pragma unroll
        for (int k = 0; k < D; ++k) {
            lU[k] -= lT * U[k] * icv;
            lP[k] = lU[k] * irho;
            lrho -= lP[k] * U[k];
        }
        hE = 0.5 * lE;
#pragma unroll
        for (int i = 0; i < D; ++i) hQ[i] = 0.5 * lQ[i];
        return lmu;
    }
};
// Tables of the coefficients, [3][D][M]: lrho + lP.xi + hE |xi|^2 terms, hQ.c
// terms, c^2; so that dg = T + lc cc and dh = hE + lc take 5 operations in 2D.
template <int D>
__device__ __forceinline__ void adj_tables(const StepArgs& a, const MacroAdj<D>& o, double* tb, int lane) {
    const int DM = D * a.M;
    for (int t = lane; t < DM; t += 32) {
        const int k = t / a.M;
        const double x = a.x1[t - k * a.M], c = x - o.U[k];
        tb[t] = fma(fma(o.hE, x, o.lP[k]), x, k == 0 ? o.lrho : 0.0);
        tb[DM + t] = o.hQ[k] * c;
        tb[2 * DM + t] = c * c;
    }
    __syncwarp();
}
template <int D>
__device__ __forceinline__ void adj_lookup(const double* tb, int DM, int M, const DvIdx<D>& id, double hE, double& dg,
                                           double& dh) {
    const double *x = tb + id.ix, *y = tb + M + id.iy;
    double t = x[0] + y[0], lc = x[DM] + y[DM], cc = x[2 * DM] + y[2 * DM];
    if (D == 3) {
        const double* z = tb + 2 * M + id.iz;
        t += z[0];
        lc += z[DM];
        cc += z[2 * DM];
    }
    dg = fma(lc, cc, t);
    dh = hE + lc;
}

constexpr int kRE = 8;  // most entities (warps) per block of the reverse passes

template <int D>
__device__ __forceinline__ void load_xi(const StepArgs& a, int v, double* x) {
#pragma unroll
    for (int k = 0; k < D; ++k) x[k] = a.xi[k * a.Vp + v];
}

// P9 reverse fused with the cell part of P8: one warp per cell.  lgN (adjoint
// of state n+1) += J9^T lmN; then lgT(n) = -lgN/3 and lgB = 4/3 lgN.  mN holds
// the macros of state n+1 as stored (rho [nC], U [nC][3], T [nC], q [nC][3], tau [nC]).
template <int D, bool HH>
__global__ void __launch_bounds__(kRE * 32) r_cell_mom(AArgs A, const double* gT, const double* mN, double* lgN,
                                                       double* lhN, double* lgT, double* lhT, double* lgB, double* lhB,
                                                       const double* lmN, double* lmuC) {
    using RV = Rev<D, HH, true>;
    __shared__ double sS[kRE][8];
    __shared__ MacroAdj<D> sO[kRE];
    extern __shared__ double eTab[];
    const StepArgs& a = A.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nE = blockDim.x >> 5, Vp = a.Vp, nC = a.nC, M = a.M;
    const int c0 = blockIdx.x * nE, c = c0 + warp, DM = D * M;
    const long long base = (long long)c * Vp;
    double* tb = eTab + (size_t)warp * 4 * DM;
    DvIdx<D> id;
    if (c < nC) {
        double U[D], acc[8];
#pragma unroll
        for (int k = 0; k < D; ++k) U[k] = mN[nC + 3 * c + k];
        for (int t = lane; t < DM; t += 32) tb[t] = a.x1[t % M] - U[t / M];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0.0;
        id.init(lane, 32, M);
        for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
            double cv[D];
            cv[0] = tb[id.ix];
            cv[1] = tb[M + id.iy];
            if (D == 3) cv[D - 1] = tb[2 * M + id.iz];
            RV::add2(acc, a.w[v] * gT[base + v], cv);
        }
        const double r = scatter_sum<8>(acc, lane);
        if ((lane & 3) == 0) sS[warp][warp_slot<8>(lane)] = r;
    }
    __syncthreads();
    if (threadIdx.x < nE && c0 + threadIdx.x < nC) {
        const int e = c0 + threadIdx.x;
        double m[kM], lm[kM];
        m[0] = mN[e];
        m[4] = mN[4 * nC + e];
        m[8] = mN[8 * nC + e];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            m[1 + k] = mN[nC + 3 * e + k];
            m[5 + k] = mN[5 * nC + 3 * e + k];
        }
#pragma unroll
        for (int k = 0; k < kM; ++k) lm[k] = lmN[(size_t)kM * e + k];
        lmuC[e] += sO[threadIdx.x].chain(a, m, lm, sS[threadIdx.x], a.dt * a.Pr, A.muRef, false, nullptr, nullptr,
                                         nullptr);
    }
    __syncthreads();
    if (c >= nC) return;
    const MacroAdj<D>& o = sO[warp];
    adj_tables<D>(a, o, tb, lane);
    const double hE = o.hE;
    id.init(lane, 32, M);
    for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
        double dg, dh;
        adj_lookup<D>(tb, DM, M, id, hE, dg, dh);
        const double w = a.w[v], lg = fma(w, dg, lgN[base + v]);
        lgN[base + v] = lg;
        lgT[base + v] = -1.0 / 3 * lg;
        lgB[base + v] = 4.0 / 3 * lg;
        if (HH) {
            const double lh = fma(w, dh, lhN[base + v]);
            lhN[base + v] = lh;
            lhT[base + v] = -1.0 / 3 * lh;
            lhB[base + v] = 4.0 / 3 * lh;
        }
    }
}

// P8 reverse, cell part alone (the last step, where the macros of n+1 carry no
// adjoint): lgT(n) = -lgT(n+1)/3, lgB = 4/3 lgT(n+1).
__global__ void r_cell_flux(AArgs A, const double* lgN, const double* lhN, double* lgT, double* lhT, double* lgB,
                            double* lhB) {
    const StepArgs& a = A.a;
    const long long n = (long long)a.nC * a.Vp;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        lgT[i] = -1.0 / 3 * lgN[i];
        lgB[i] = 4.0 / 3 * lgN[i];
        if (a.hasH) {
            lhT[i] = -1.0 / 3 * lhN[i];
            lhB[i] = 4.0 / 3 * lhN[i];
        }
    }
}

// P8 reverse, face part: adjoint of the relaxed face values; one warp per face.
template <int D, bool HH>
__global__ void __launch_bounds__(64) r_face_flux(AArgs A, const double* lgN, const double* lhN, double* lgS,
                                                  double* lhS) {
    const StepArgs& a = A.a;
    const int lane = threadIdx.x & 31, Vp = a.Vp, f = blockIdx.x * 2 + (threadIdx.x >> 5);
    if (f >= a.nA) return;
    const long long base = (long long)f * Vp;
    const int o = a.own[f];
    const bool inner = f < a.nI;
    const int nb = inner ? a.nei[f] : o;
    const double kO = -a.dt / a.vol[o], kN = inner ? a.dt / a.vol[nb] : 0.0;
    const double *lgo = lgN + (long long)o * Vp, *lgn = lgN + (long long)nb * Vp;
    const double *lho = HH ? lhN + (long long)o * Vp : nullptr, *lhn = HH ? lhN + (long long)nb * Vp : nullptr;
    double S[D];
#pragma unroll
    for (int k = 0; k < D; ++k) S[k] = a.Sf[3 * f + k];
    for (int v = lane; v < a.nV; v += 32) {
        double x[D], xs = 0.0;
        load_xi<D>(a, v, x);
#pragma unroll
        for (int k = 0; k < D; ++k) xs += x[k] * S[k];
        lgS[base + v] = xs * fma(lgn[v], kN, lgo[v] * kO);
        if (HH) lhS[base + v] = xs * fma(lhn[v], kN, lho[v] * kO);
    }
}

// P7 + P6 reverse (+ objective seeds on walls): one warp per face.  In: lgS =
// adjoint of the relaxed values; out: lgS = adjoint of the face values before
// relaxation (incoming wall DVs keep theirs for r_wall).  mF: forward face
// macros (rho, U, T, q, tau) of the step.  One pass over the velocities forms
// the Shakhov sums and the second moments; a second pass writes the adjoints.
// 48^2 quads x 28^2: 1027 -> 412 us.
template <int D, bool HH>
__global__ void __launch_bounds__(kRE * 32) r_face(AArgs A, const double* gS, const double* hS, const double* mF,
                                                   double* lgS, double* lhS, const double* wq, const double* ws,
                                                   double objScale, double* lmuF) {
    using RV = Rev<D, HH, true>;
    __shared__ EqScal sE[kRE];
    __shared__ double sT[kRE][RV::NS], sB[kRE], sW[kRE][12];
    __shared__ MacroAdj<D> sO[kRE];
    extern __shared__ double eTab[];
    const StepArgs& a = A.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nE = blockDim.x >> 5, Vp = a.Vp, M = a.M, DM = D * M;
    const int f0 = blockIdx.x * nE, f = f0 + warp;
    const double hh = 0.5 * a.dt, ck = HH ? 2.0 - 2.0 * a.K / (a.K + 3.0 - D) : 0.0;
    double* tb = eTab + (size_t)warp * 4 * DM;
    if (threadIdx.x < nE && f0 + threadIdx.x < a.nA) {
        const double* m = mF + (size_t)kM * (f0 + threadIdx.x);
        eq_scal<D>(sE[threadIdx.x], m, a);
        sB[threadIdx.x] = hh / (2.0 * m[8] + hh);
    }
    __syncthreads();
    const bool live = f < a.nA, wall = live && f >= a.nI;
    const long long base = (long long)f * Vp;
    double S[3] = {0, 0, 0}, Uw[3] = {0, 0, 0};
    DvIdx<D> id;
    if (live) {
        if (wall)
            for (int k = 0; k < 3; ++k) {
                S[k] = a.Sf[3 * f + k];
                Uw[k] = a.Uw[3 * (f - a.nI) + k];
            }
        eq_tables<D>(a, sE[warp], tb, lane);
        const double rho = sE[warp].rho, tk3 = sE[warp].tk3;
        double acc[RV::NS];
#pragma unroll
        for (int i = 0; i < RV::NS; ++i) acc[i] = 0.0;
        id.init(lane, 32, M);
        if (!wall) {
            for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
                double G0, Ae, p, c[D];
                eq_lookup<D>(tb, DM, M, id, G0, Ae, p, c);
                const double g = gS[base + v];
                RV::add(acc, G0, Ae, p, c, g, HH ? hS[base + v] : 0.0, lgS[base + v], HH ? lhS[base + v] : 0.0, rho, tk3,
                        ck);
                RV::add2(acc + RV::S, a.w[v] * g, c);
            }
        } else {  // the Shakhov part for the outgoing velocities; wall moments
            double aw[12];
#pragma unroll
            for (int i = 0; i < 12; ++i) aw[i] = 0.0;
            for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
                double G0, Ae, p, c[D];
                eq_lookup<D>(tb, DM, M, id, G0, Ae, p, c);
                const double g = gS[base + v], h = HH ? hS[base + v] : 0.0, w = a.w[v], wg = w * g;
                if (dot_rn(a.xi + v, Vp, S) > 0)
                    RV::add(acc, G0, Ae, p, c, g, h, lgS[base + v], HH ? lhS[base + v] : 0.0, rho, tk3, ck);
                RV::add2(acc + RV::S, wg, c);
                double x[D], e[D], ee = 0.0;
                load_xi<D>(a, v, x);
#pragma unroll
                for (int k = 0; k < D; ++k) { e[k] = x[k] - Uw[k]; ee += e[k] * e[k]; }
                const double sw = 0.5 * (ee * wg + w * h);
#pragma unroll
                for (int k = 0; k < D; ++k) aw[k] = fma(sw, e[k], aw[k]);
                RV::add2(aw + D, wg, x);
            }
            warp_sum<12>(aw);
            if (lane == 0)
                for (int i = 0; i < 12; ++i) sW[warp][i] = aw[i];
        }
        const double r = scatter_sum<RV::NS>(acc, lane);
        if (RV::NS == 32) sT[warp][lane] = r;
        else if ((lane & 1) == 0) sT[warp][warp_slot<16>(lane) % RV::NS] = r;
    }
    __syncthreads();
    if (threadIdx.x < nE && f0 + threadIdx.x < a.nA) {
        const int e = f0 + threadIdx.x;
        double m[kM], lm[kM];
#pragma unroll
        for (int k = 0; k < kM; ++k) m[k] = mF[(size_t)kM * e + k];
        const double den = 2.0 * m[8] + hh;
        RV::finish(sT[threadIdx.x], m, sB[threadIdx.x], -2.0 * hh / (den * den), a.R, a.Pr, lm);
        double lqw[3] = {0.0, 0.0, 0.0}, lsw[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        const bool wl = e >= a.nI;
        if (wl) {
            for (int k = 0; k < 3; ++k) lqw[k] = objScale * wq[3 * (e - a.nI) + k];
            lsw[1] = objScale * ws[e - a.nI];
        }
        lmuF[e] += sO[threadIdx.x].chain(a, m, lm, sT[threadIdx.x] + RV::S, 0.5 * a.dt * a.Pr, A.muRef, wl, lqw, lsw,
                                         sW[threadIdx.x]);
    }
    __syncthreads();
    if (!live) return;
    const MacroAdj<D>& o = sO[warp];
    adj_tables<D>(a, o, tb, lane);
    const double hE = o.hE, om = 1.0 - sB[warp];
    id.init(lane, 32, M);
    if (!wall) {
        for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
            double dg, dh;
            adj_lookup<D>(tb, DM, M, id, hE, dg, dh);
            const double w = a.w[v];
            lgS[base + v] = fma(w, dg, om * lgS[base + v]);
            if (HH) lhS[base + v] = fma(w, dh, om * lhS[base + v]);
        }
        return;
    }
    for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
        double dg, dh, x[D], ee = 0.0, le = 0.0;
        adj_lookup<D>(tb, DM, M, id, hE, dg, dh);
        load_xi<D>(a, v, x);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const double e = x[k] - Uw[k];
            ee += e * e;
            le += o.hQw[k] * e;
        }
        dg += le * ee;
        dh += le;
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int j = 0; j < D; ++j) dg += o.lX[D * i + j] * x[i] * x[j];
        const double w = a.w[v], k = dot_rn(a.xi + v, Vp, S) > 0 ? om : 1.0;
        lgS[base + v] = fma(w, dg, k * lgS[base + v]);
        if (HH) lhS[base + v] = fma(w, dh, k * lhS[base + v]);
    }
}

// P5 + P4 reverse: one block per wall face; the wall Maxwellian from
// per-direction factors.
__global__ void r_wall(AArgs A, const double* gS, const double* rhoW, const double* incAbs, double* lgS, double* lhS,
                       double* lTw) {
    __shared__ double red[32 * 3];
    extern __shared__ double eTab[];
    const StepArgs& a = A.a;
    const int wf = blockIdx.x, f = a.nI + wf, Vp = a.Vp, D = a.D, M = a.M;
    const long long base = (long long)f * Vp;
    const double* S = a.Sf + 3 * f;
    const double* Uw = a.Uw + 3 * wf;
    const double Tw = A.Tw[wf], th = a.R * Tw, ith = 1.0 / th, k3 = a.K + 3.0 - D;
    const double rw = rhoW[wf], s2 = 2.0 * kPi * th, n0 = 1.0 / (D == 2 ? s2 : s2 * sqrt(s2));
    double off2 = 0.0;  // components outside the solution directions
    for (int k = D; k < 3; ++k) off2 += Uw[k] * Uw[k];
    for (int t = threadIdx.x; t < D * M; t += blockDim.x) {
        const int k = t / M;
        const double c = a.x1[t - k * M] - Uw[k];
        eTab[t] = (k == 0 ? n0 : 1.0) * exp(-0.5 * ith * (c * c + (k == 0 ? off2 : 0.0)));
    }
    __syncthreads();
    // incoming: gS = rw M, hS = gS R Tw k3
    double acc[3] = {0.0, 0.0, 0.0};  // lrw, lTw, d incAbs / dTw
    for (int v = threadIdx.x; v < a.nV; v += blockDim.x) {
        const double xs = dot_rn(a.xi + v, Vp, S);
        if (xs > 0) continue;
        const int r = v / M;
        double Mx = eTab[v - r * M] * eTab[M + (D == 3 ? r % M : r)];
        if (D == 3) Mx *= eTab[2 * M + r / M];
        double cc = 0.0;
        for (int k = 0; k < 3; ++k) {
            const double c = a.xi[k * Vp + v] - Uw[k];
            cc += c * c;
        }
        const double dM = a.R * Mx * (cc * ith - D) * (0.5 * ith);  // dM/dTw
        const double lg = lgS[base + v], lh = a.hasH ? lhS[base + v] : 0.0;
        acc[0] += lg * Mx + lh * Mx * th * k3;
        acc[1] += rw * (lg * dM + lh * k3 * (a.R * Mx + th * dM));
        lgS[base + v] = 0.0;
        if (a.hasH) lhS[base + v] = 0.0;
        if (xs < 0) acc[2] += -a.w[v] * xs * dM;
    }
    block_sum<3>(acc, red);
    // rw = sum_out w xs gS / incAbs; incAbs = |sum_in -w xs M|
    const double li = acc[0] / incAbs[wf];
    for (int v = threadIdx.x; v < a.nV; v += blockDim.x) {
        const double xs = dot_rn(a.xi + v, Vp, S);
        if (xs > 0) lgS[base + v] = fma(li * a.w[v], xs, lgS[base + v]);
    }
    if (threadIdx.x == 0) lTw[wf] += acc[1] - li * rw * acc[2];  // incoming sum is positive
}

// P3 reverse (+ the lagged wall gradient output G_b' = grad . n): one warp per
// cell, face by face: the velocities for which the cell is upwind (ties half)
// add lgS and lgS (d - xi dt/2).  The sign of xi.S is the forward's: FP32 where
// it is beyond FP32 rounding, FP64 in the warp iterations that hold a velocity
// near the face (see k_recon).  48^2 quads x 28^2: 246 -> 160 us.
template <int D>
struct ReconFace {
    double S[D], d[D];
    float s32[D];
    int e;
};
template <int D>
__device__ __forceinline__ ReconFace<D> recon_face(const StepArgs& a, int j) {
    ReconFace<D> r;
    r.e = a.cellFace[j];
    const int f = r.e >> 1;
    const double* d = (r.e & 1) == 0 ? a.dO + 3 * f : a.dN + 3 * f;
    int ex = 0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        r.S[k] = a.Sf[3 * f + k];
        r.d[k] = d[k];
        ex = max(ex, (__double2hiint(r.S[k]) >> 20) & 0x7ff);
    }
    const double sc = ex > 0 && ex < 2046 ? __hiloint2double((2046 - ex) << 20, 0) : 1.0;
#pragma unroll
    for (int k = 0; k < D; ++k) r.s32[k] = (float)(r.S[k] * sc);
    return r;
}

template <int D, bool HH>
__global__ void __launch_bounds__(64) r_recon(AArgs A, const double* lgS, const double* lhS, const double* lGbN,
                                              const double* lGbNh, double* lgB, double* lhB, double* lG, double* lhG) {
    __shared__ ReconFace<D> stage[2][kStage];
    const StepArgs& a = A.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Vp = a.Vp, c = blockIdx.x * 2 + warp;
    if (c >= a.nC) return;
    const int j0 = a.cellOff[c], nf = a.cellOff[c + 1] - j0;
    if (lane < min(nf, kStage)) stage[warp][lane] = recon_face<D>(a, j0 + lane);
    __syncwarp();
    const long long base = (long long)c * Vp;
    const double mh = -0.5 * a.dt;
    for (int v0 = lane; v0 - lane < a.nV; v0 += 32) {
        const bool live = v0 < a.nV;
        const int v = live ? v0 : a.nV - 1;
        double xi[D], sb = 0.0, sbh = 0.0, gk[D], hk[D];
        float x32[D];
        load_xi<D>(a, v, xi);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            gk[k] = hk[k] = 0.0;
            x32[k] = a.xi32[k * Vp + v];
        }
        bool walls = false;
        // gk collects sum lg d; the common shift -xi dt/2 sum lg is added once
        for (int j = 0; j < nf; ++j) {
            ReconFace<D> r;
            if (j < kStage) r = stage[warp][j];
            else r = recon_face<D>(a, j0 + j);
            const int f = r.e >> 1, side = r.e & 1;
            const bool inner = f < a.nI;
            walls = walls || !inner;
            float s32 = 0.f, b32 = 1e-30f;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                s32 = fmaf(x32[k], r.s32[k], s32);
                b32 = fmaf(fabsf(x32[k] * r.s32[k]), 1e-6f, b32);
            }
            float wgt = (side ? s32 < 0.f : s32 > 0.f) ? 1.f : 0.f;
            const unsigned near = __ballot_sync(0xffffffffu, !(fabsf(s32) > b32));
            for (unsigned m = near ? 1u : 0u; m; m = 0u) {  // a loop: as a branch its FP64 part is predicated
                double xs = 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const double t = __dmul_rn(xi[k], r.S[k]);
                    xs = k == 0 ? t : __dadd_rn(xs, t);
                }
                if (inner) {
                    const bool up = xs >= kVSmall, dn = xs < -kVSmall;
                    wgt = (side ? dn : up) ? 1.f : (!up && !dn ? 0.5f : 0.f);
                } else {
                    wgt = xs > 0 ? 1.f : 0.f;
                }
            }
            const long long fi = (long long)f * Vp + v;
            double lg = wgt != 0.f ? lgS[fi] : 0.0, lh = HH && wgt != 0.f ? lhS[fi] : 0.0;
            for (unsigned m = near && __any_sync(0xffffffffu, wgt == 0.5f) ? 1u : 0u; m; m = 0u) {
                const double t = wgt == 0.5f ? 0.5 : 1.0;
                lg *= t;
                lh *= t;
            }
            sb += lg;
            if (HH) sbh += lh;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                gk[k] = fma(lg, r.d[k], gk[k]);
                if (HH) hk[k] = fma(lh, r.d[k], hk[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const double sh = xi[k] * mh;
            gk[k] = fma(sb, sh, gk[k]);
            if (HH) hk[k] = fma(sbh, sh, hk[k]);
        }
        if (walls)  // G_b' = grad . n on the wall faces of this cell
            for (int j = j0; j < j0 + nf; ++j) {
                const int f = a.cellFace[j] >> 1;
                if (f < a.nI) continue;
                const int wf = f - a.nI;
                const double* nh = a.nHatW + 3 * wf;
                const double lb = lGbN[(long long)wf * Vp + v], lbh = HH ? lGbNh[(long long)wf * Vp + v] : 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    gk[k] += lb * nh[k];
                    hk[k] += lbh * nh[k];
                }
            }
        if (!live) continue;
        lgB[base + v] += sb;
        if (HH) lhB[base + v] += sbh;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            lG[((long long)c * D + k) * Vp + v] = gk[k];
            if (HH) lhG[((long long)c * D + k) * Vp + v] = hk[k];
        }
    }
}

// P2 reverse: lgB += transpose of the least-squares stencil; adjoint of the
// lagged wall gradient input.  One warp per cell; the cell's own vectors enter
// through their sum.  48^2 quads x 28^2: 239 -> 148 us.
template <int D, bool HH>
__global__ void __launch_bounds__(64) r_grad(AArgs A, const double* lG, const double* lhG, double* lgB, double* lhB,
                                             double* lGb, double* lGbh) {
    const StepArgs& a = A.a;
    const int lane = threadIdx.x & 31, Vp = a.Vp, c = blockIdx.x * 2 + (threadIdx.x >> 5);
    if (c >= a.nC) return;
    const int j0 = a.cellOff[c], j1 = a.cellOff[c + 1];
    const long long base = (long long)c * Vp;
    double Ls[D];  // sum of this cell's vectors over its internal faces (the boundary value moves with the cell's)
#pragma unroll
    for (int k = 0; k < D; ++k) Ls[k] = 0.0;
    bool walls = false;
    for (int j = j0; j < j1; ++j) {
        const int e = a.cellFace[j], f = e >> 1;
        if (f >= a.nI) { walls = true; continue; }
#pragma unroll
        for (int k = 0; k < D; ++k) Ls[k] += (e & 1 ? a.nVec : a.pVec)[3 * f + k];
    }
    for (int v = lane; v < a.nV; v += 32) {
        double sg = 0.0, sh = 0.0, gc[D], hc[D];
#pragma unroll
        for (int k = 0; k < D; ++k) {
            gc[k] = lG[((long long)c * D + k) * Vp + v];
            hc[k] = HH ? lhG[((long long)c * D + k) * Vp + v] : 0.0;
            sg = fma(-Ls[k], gc[k], sg);
            if (HH) sh = fma(-Ls[k], hc[k], sh);
        }
        for (int j = j0; j < j1; ++j) {
            const int e = a.cellFace[j], f = e >> 1, side = e & 1;
            if (f >= a.nI) continue;
            const long long ob = (long long)(side == 0 ? a.nei[f] : a.own[f]) * D * Vp + v;
            const double* Lo = side == 0 ? a.nVec + 3 * f : a.pVec + 3 * f;  // the other cell's vector
#pragma unroll
            for (int k = 0; k < D; ++k) {
                sg = fma(Lo[k], lG[ob + (long long)k * Vp], sg);
                if (HH) sh = fma(Lo[k], lhG[ob + (long long)k * Vp], sh);
            }
        }
        lgB[base + v] += sg;
        if (HH) lhB[base + v] += sh;
        if (!walls) continue;
        for (int j = j0; j < j1; ++j) {
            const int f = a.cellFace[j] >> 1;
            if (f < a.nI) continue;
            const int wf = f - a.nI;
            const double *L = a.bVec + 3 * wf, dc = a.dcW[wf];
            double lb = 0.0, lbh = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                lb += L[k] * gc[k];
                if (HH) lbh += L[k] * hc[k];
            }
            lGb[(long long)wf * Vp + v] = lb / dc;
            if (HH) lGbh[(long long)wf * Vp + v] = lbh / dc;
        }
    }
}

// P1 reverse: one warp per cell.  lgT += (1-r) lgB; lm = macro adjoint of the
// cell's relaxation (rho, U, T, q, tau).  48^2 quads x 28^2: 250 -> 135 us.
template <int D, bool HH>
__global__ void __launch_bounds__(kRE * 32) r_barp(AArgs A, const double* gT, const double* hT, const double* mC,
                                                   const double* lgB, const double* lhB, double* lgT, double* lhT,
                                                   double* lm) {
    using RV = Rev<D, HH, false>;
    __shared__ EqScal sE[kRE];
    __shared__ double sT[kRE][16], sR[kRE];
    extern __shared__ double eTab[];
    const StepArgs& a = A.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nE = blockDim.x >> 5, Vp = a.Vp, M = a.M, DM = D * M;
    const int c0 = blockIdx.x * nE, c = c0 + warp;
    const double ck = HH ? 2.0 - 2.0 * a.K / (a.K + 3.0 - D) : 0.0;
    double* tb = eTab + (size_t)warp * 4 * DM;
    if (threadIdx.x < nE && c0 + threadIdx.x < a.nC) {
        const double* m = mC + (size_t)kM * (c0 + threadIdx.x);
        eq_scal<D>(sE[threadIdx.x], m, a);
        sR[threadIdx.x] = 1.5 * a.dt / (2.0 * m[8] + a.dt);
    }
    __syncthreads();
    if (c < a.nC) {
        const long long base = (long long)c * Vp;
        eq_tables<D>(a, sE[warp], tb, lane);
        const double rho = sE[warp].rho, tk3 = sE[warp].tk3, om = 1.0 - sR[warp];
        double acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.0;
        DvIdx<D> id;
        id.init(lane, 32, M);
        for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
            double G0, Ae, p, cv[D];
            eq_lookup<D>(tb, DM, M, id, G0, Ae, p, cv);
            const double lg = lgB[base + v], lh = HH ? lhB[base + v] : 0.0;
            RV::add(acc, G0, Ae, p, cv, gT[base + v], HH ? hT[base + v] : 0.0, lg, lh, rho, tk3, ck);
            lgT[base + v] = fma(om, lg, lgT[base + v]);
            if (HH) lhT[base + v] = fma(om, lh, lhT[base + v]);
        }
        const double r = scatter_sum<16>(acc, lane);
        if ((lane & 1) == 0) sT[warp][warp_slot<16>(lane)] = r;
    }
    __syncthreads();
    if (threadIdx.x < nE && c0 + threadIdx.x < a.nC) {
        const int e = c0 + threadIdx.x;
        double m[kM], out[kM];
#pragma unroll
        for (int k = 0; k < kM; ++k) m[k] = mC[(size_t)kM * e + k];
        const double den = 2.0 * m[8] + a.dt;
        RV::finish(sT[threadIdx.x], m, sR[threadIdx.x], -3.0 * a.dt / (den * den), a.R, a.Pr, out);
#pragma unroll
        for (int k = 0; k < kM; ++k) lm[(size_t)kM * e + k] = out[k];
    }
}

// Pack cell / face macros of the forward pass as (rho, U, T, q, tau) tuples.
__global__ void k_pack_macros(int n, const double* rho, const double* U, const double* T, const double* q,
                              const double* tau, double* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double* o = out + (size_t)kM * i;
        o[0] = rho[i];
        for (int k = 0; k < 3; ++k) { o[1 + k] = U[3 * i + k]; o[5 + k] = q[3 * i + k]; }
        o[4] = T[i];
        o[8] = tau[i];
    }
}

__global__ void k_sum(int n, const double* x, double* out) {  // one block, fixed order
    __shared__ double red[32];
    double s[1] = {0.0};
    for (int i = threadIdx.x; i < n; i += blockDim.x) s[0] += x[i];
    block_sum<1>(s, red);
    if (threadIdx.x == 0) out[0] += s[0];
}

}  // namespace

// ------------------------------------------------------------ launchers
static Macros<Dual> tlm_macros(const TlmState& s) {
    return {s.rho, s.U, s.T, s.q, s.tau, s.rhoF, s.UF, s.TF, s.qF, s.tauF, s.rhoW, s.qWall, s.stressWall,
            s.Tw, s.incAbs, s.muRef};
}
void tlm_launch_incabs(const TlmState& s, cudaStream_t st) {
    TArgs t{s.a, s.rho, s.U, s.T, s.q, s.tau, s.rhoF, s.UF, s.TF, s.qF, s.tauF, s.rhoW, s.qWall, s.stressWall,
            s.Tw, s.incAbs, s.muRef};
    t_incabs<<<s.a.nW, kRT, 0, st>>>(t);
}
void tlm_launch_init(const TlmState& s, const double* rho0, const double* U0, const double* T0, int sms,
                     cudaStream_t st) {
    TArgs t{s.a, s.rho, s.U, s.T, s.q, s.tau, s.rhoF, s.UF, s.TF, s.qF, s.tauF, s.rhoW, s.qWall, s.stressWall,
            s.Tw, s.incAbs, s.muRef};
    t_init<<<(s.a.nC + 127) / 128, 128, 0, st>>>(t, rho0, U0, T0);
    const Macros<Dual> m = tlm_macros(s);
    with_pass<Dual>(s.a, [&](auto P) { P.template eq<kInit>(s.a, m, nullptr, nullptr, s.gT, s.hT, sms, st); });
    cudaMemsetAsync(s.Gbg, 0, sizeof(Dual) * (size_t)s.a.nW * s.a.Vp, st);
    if (s.a.hasH) cudaMemsetAsync(s.Gbh, 0, sizeof(Dual) * (size_t)s.a.nW * s.a.Vp, st);
}
void tlm_launch_step(const TlmState& s, bool objective, const double* wq, const double* ws, double scale, Dual* J,
                     int sms, cudaStream_t st) {
    const StepArgs& a = s.a;
    const Macros<Dual> m = tlm_macros(s);
    const Fields<Dual> f{s.gT, s.hT, s.gB, s.hB, s.gG, s.hG, s.Gbg, s.Gbh, s.gS, s.hS};
    for (int pass = 0; pass < 8; ++pass) {
        with_pass<Dual>(a, [&](auto P) { P.run(pass, a, m, f, sms, st); });
        if (pass == 4 && objective && a.nW > 0)
            k_objective<Dual><<<1, kT, 0, st>>>(a.nW, wq, ws, s.qWall, s.stressWall, scale, J);
    }
}

void launch_objective(const StepArgs& a, const double* wq, const double* ws, double scale, double* J, cudaStream_t st) {
    if (a.nW > 0) k_objective<double><<<1, kT, 0, st>>>(a.nW, wq, ws, a.qWall, a.stressWall, scale, J);
}

void adj_pack_macros(int n, const double* rho, const double* U, const double* T, const double* q, const double* tau,
                     double* out, int sms, cudaStream_t st) {
    k_pack_macros<<<grid(n, kT, sms), kT, 0, st>>>(n, rho, U, T, q, tau, out);
}

namespace {
// Dynamic shared memory of a kernel beyond the 48 KB every launch may ask for.
template <typename F>
void allow_smem(F* func, size_t bytes) {
    if (bytes > 32 * 1024) allow_max_dynamic_smem(func);
}

template <int D, bool HH>
void adj_step(const AdjState& s, const double* gTn, const double* hTn, const double* mTn, bool objective,
              double scale, int sms, cudaStream_t st) {
    const AArgs A{s.a, s.a.Tw, s.muRef};
    const StepArgs& a = s.a;
    const size_t tb = (size_t)4 * D * a.M * sizeof(double);  // tables of one warp
    int e = kRE;  // entities per block: fewer while the entities would not make eight blocks per SM
    while (e > 1 && (((long long)a.nC < 8LL * sms * e && e > 4) || tb * e > 160 * 1024)) e >>= 1;
    const int gC = (a.nC + e - 1) / e, gF = (a.nA + e - 1) / e, thr = 32 * e;
    allow_smem(r_cell_mom<D, HH>, tb * e);
    allow_smem(r_face<D, HH>, tb * e);
    allow_smem(r_barp<D, HH>, tb * e);
    // P9 reverse fused with the cell part of P8 (lgN += J9^T lmN; lgT, lgB from lgN)
    if (s.haveMacroAdj)
        r_cell_mom<D, HH><<<gC, thr, tb * e, st>>>(A, gTn, mTn, s.lgN, s.lhN, s.lgT, s.lhT, s.lgB, s.lhB, s.lmN, s.lmuC);
    else
        r_cell_flux<<<grid((long long)a.nC * a.Vp, kT, sms), kT, 0, st>>>(A, s.lgN, s.lhN, s.lgT, s.lhT, s.lgB,
                                                                           s.lhB);
    // P8 reverse, face part
    r_face_flux<D, HH><<<(a.nA + 1) / 2, 64, 0, st>>>(A, s.lgN, s.lhN, s.lgS, s.lhS);
    // P7 + P6 reverse
    r_face<D, HH><<<gF, thr, tb * e, st>>>(A, s.gS, s.hS, s.mF, s.lgS, s.lhS, s.wq, s.ws, objective ? scale : 0.0,
                                           s.lmuF);
    // P5 + P4 reverse
    if (a.nW > 0) {
        const size_t wb = (size_t)D * a.M * sizeof(double);
        allow_smem(r_wall, wb);
        r_wall<<<a.nW, kRT, wb, st>>>(A, s.gS, a.rhoW, a.incAbs, s.lgS, s.lhS, s.lTw);
    }
    // P3 reverse (+ G_b' = grad.n), P2 reverse
    r_recon<D, HH><<<(a.nC + 1) / 2, 64, 0, st>>>(A, s.lgS, s.lhS, s.lGbN, s.lGbNh, s.lgB, s.lhB, s.lG, s.lhG);
    r_grad<D, HH><<<(a.nC + 1) / 2, 64, 0, st>>>(A, s.lG, s.lhG, s.lgB, s.lhB, s.lGb, s.lGbh);
    // P1 reverse
    r_barp<D, HH><<<gC, thr, tb * e, st>>>(A, s.gT, s.hT, s.mC, s.lgB, s.lhB, s.lgT, s.lhT, s.lm);
}
}  // namespace

// Tables of one warp (block of one entity): the largest velocity grids the reverse takes have 48 KB.
size_t adj_table_bytes(int D, int M) { return (size_t)4 * D * M * sizeof(double); }

void adj_launch_step(const AdjState& s, const double* gTn, const double* hTn, const double* mTn, bool objective,
                     double scale, int sms, cudaStream_t st) {
    if (s.a.D == 3) {
        if (s.a.hasH) adj_step<3, true>(s, gTn, hTn, mTn, objective, scale, sms, st);
        else adj_step<3, false>(s, gTn, hTn, mTn, objective, scale, sms, st);
    } else {
        adj_step<2, true>(s, gTn, hTn, mTn, objective, scale, sms, st);
    }
}

void adj_sum(int n, const double* x, double* out, cudaStream_t st) { k_sum<<<1, kT, 0, st>>>(n, x, out); }

}  // namespace dugks
