// Reference pipeline: one FP64 kernel per pass of fvDVM::evolution()
// (src/fvDVM/fvDVM/fvDVM.C:1086-1108), with every intermediate materialised
// in HBM (DV index innermost).  It is the plain, easily checked GPU
// restatement; the fused tile sweeps (fused_pipeline.cu) are the fast path.
//
//   k_eq        P1 updateGHbarPvol             discreteVelocity.C:346-410
//   k_grad      P2 fvc::grad + fixedGradient   discreteVelocity.C:420-470
//   k_recon     P3 updateGHbarSurf             discreteVelocity.C:472-691
//   k_wall      P4+P5 MaxwellWallRho / WallIn  fvDVM.C:347-367, discreteVelocity.C:693-731
//   k_sym_*     P5b updateGHbarSurfSymmetryIn  fvDVM.C:375-454, discreteVelocity.C:733-817
//   k_mom       P6 updateMacroSurf             fvDVM.C:456-582
//   k_eq        P7 updateGHsurf                discreteVelocity.C:819-932
//   k_cell      P8 updateGHtildeVol            discreteVelocity.C:934-978
//   k_mom       P9 updateMacroVol              fvDVM.C:597-728
//   k_pressure  P10 updatePressureInOutBC      fvDVM.C:730-806
//
// Boundary faces follow the surface patch type of their rho boundary
// condition (discreteVelocity::setBCtype, discreteVelocity.C:250-300):
// diffuse walls, zeroGradient, mixed (rho fixedValue), farField (also for
// pressureIn / pressureOut) and the two symmetry types.
#include "device_common.cuh"
#include "kernels.h"

namespace dugks {
namespace {

constexpr int kRedThreads = 128;
constexpr int kMaxEnt = 16;  // most entities (warps) per block
constexpr size_t kTabMax = 44 * 1024;  // tables of a block (48 KB less the static scalars)

// Every pass but the walls runs one warp per entity (cell or face), lanes
// striding over the velocities: GB300 issues FP64 at 1/64 of the FP32 rate (a
// warp instruction holds the SM's pipe for 16 cycles however many lanes are
// active), so the passes are bound by the count of FP64 warp instructions and
// by nothing else.  What depends on the entity alone is therefore formed once
// per entity, by one lane per entity of the block (entity scalars: a block of
// 8 or 16 warps pays them once for all its entities), what depends on one
// direction of the tensor-product velocity grid once per abscissa (tables in
// shared memory), and products are fused.  The sign of xi.S is the exception:
// it is formed without FMA, as the oracle forms it, so that velocities lying
// in a face are ties here and there alike.
//   FP64 operations per cell and velocity, 2D triangles: ~620 (a square root,
//   three divisions and an exponential per velocity, two divisions per face
//   and field) -> ~100.

// Sum of NS per-lane values over the warp; the lane ends with the total of
// slot warp_slot<NS>(lane): NS - 1 + log2(32 / NS) additions instead of the
// butterfly's 5 NS.
template <int NS>
__device__ __forceinline__ double scatter_sum(double (&v)[NS], int lane) {
    int xm = 16;
#pragma unroll
    for (int half = NS / 2; half >= 1; half >>= 1, xm >>= 1) {
        const bool up = lane & xm;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, xm);
        }
    }
    double r = v[0];
#pragma unroll
    for (int o = 16 / NS; o >= 1; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}
template <int NS>
__device__ __forceinline__ int warp_slot(int lane) {  // NS = 4 or 8
    return NS == 4 ? ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1)
                   : ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}

// Relaxation toward the Shakhov equilibrium, of the cells (P1: gbar+ from g~,
// weight 1.5dt/(2tau+dt)) or of the face values in place (P7, weight
// h/(2tau+h), h = dt/2).  With c = xi - U, A = c^2/RT - D - 2 and
// P = (1-Pr) c.q / (5 rho (RT)^2):
//   gE = e (1 + P A),  hE = RT (K+3-D) (gE + (2 - 2K/(K+3-D)) e P),
// e = rho (2 pi RT)^(-D/2) exp(-c^2/2RT) a product of per-direction factors and
// A, P sums of per-direction terms (TAB: tables of the D M abscissae in shared
// memory, 9 FP64 operations per velocity in 2D with the weight folded into e;
// without room for them the exponential is taken per velocity).
// 24k triangles x 32^2: cells 5.04 -> 0.52 ms, faces 7.42 -> 0.83 ms (FP64 pipe 88 % busy).
template <int D, bool H, bool TAB, bool FACE>
__global__ void k_eq(StepArgs a, const double* gi, const double* hi, double* go, double* ho) {
    __shared__ double sc[kMaxEnt][14];
    extern __shared__ double tab[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nEnt = blockDim.x >> 5;
    const int n = FACE ? a.nA : a.nC, e0 = blockIdx.x * nEnt, M = a.M, Vp = a.Vp;
    const double K3 = a.K + 3.0 - D;
    if (threadIdx.x < nEnt && e0 + threadIdx.x < n) {
        const int i = e0 + threadIdx.x;
        const double rho = (FACE ? a.rhoF : a.rho)[i], T = (FACE ? a.TF : a.T)[i], tau = (FACE ? a.tauF : a.tau)[i];
        const double *U = (FACE ? a.UF : a.U) + 3 * i, *q = (FACE ? a.qF : a.q) + 3 * i;
        double* s = sc[threadIdx.x];
        const double RT = a.R * T, iRT = 1.0 / RT, s2 = 2.0 * kPi * RT;
        const double hh = 0.5 * a.dt;
        const double rf = FACE ? hh / (2 * tau + hh) : 1.5 * a.dt / (2.0 * tau + a.dt);
        const double k0 = (1.0 - a.Pr) * iRT * iRT / (5.0 * rho);
        s[0] = 1.0 - rf;
        s[2] = RT * K3;
        const double rr = rf * rho;  // the relaxation weight goes with the factor of e
        s[3] = D == 2 ? rr / s2 : (D == 3 ? rr / (s2 * sqrt(s2)) : rr / sqrt(s2));
        s[4] = iRT;
        double x2 = 0.0, xq = 0.0;  // components outside the solution directions: their velocity is 0
        for (int k = 0; k < 3; ++k) {
            s[5 + k] = k0 * q[k];
            s[8 + k] = U[k];
            if (k >= D) { x2 += U[k] * U[k]; xq -= U[k] * s[5 + k]; }
        }
        s[11] = x2;
        s[12] = xq;
    }
    __syncthreads();
    const int DM = D * M;
    if (TAB) {  // per entity: E [D][M] | A [D][M] | P [D][M]
        for (int t = threadIdx.x; t < nEnt * DM; t += blockDim.x) {
            const int j = t / DM, r = t - j * DM, k = r / M, i = r - k * M;
            if (e0 + j >= n) break;
            const double* s = sc[j];
            const double c = a.x1[i] - s[8 + k], c2 = c * c + (k == 0 ? s[11] : 0.0), ci = c2 * s[4];
            const double E = exp(-0.5 * ci);
            double* tb = tab + (size_t)j * 3 * DM + r;
            tb[0] = k == 0 ? E * s[3] : E;
            tb[DM] = k == 0 ? ci - (D + 2) : ci;
            tb[2 * DM] = c * s[5 + k] + (k == 0 ? s[12] : 0.0);
        }
        __syncthreads();
    }
    const int en = e0 + warp;
    if (en >= n) return;
    const double* s = sc[warp];
    const double om = s[0], hf = s[2], ck = H ? 2.0 - 2.0 * a.K / K3 : 0.0;
    const double* tb = tab + (size_t)warp * 3 * DM;
    const long long base = (long long)en * Vp;
    const bool bnd = FACE && en >= a.nI;
    DvIdx<D> id;
    id.init(lane, 32, M);
    auto equilibrium = [&](int v, double& gE, double& hE) {
        double e, A, P;
        if (TAB) {
            const double* tx = tb + id.ix;
            e = tx[0]; A = tx[DM]; P = tx[2 * DM];
            if (D > 1) {
                const double* ty = tb + M + id.iy;
                e *= ty[0]; A += ty[DM]; P += ty[2 * DM];
            }
            if (D > 2) {
                const double* tz = tb + 2 * M + id.iz;
                e *= tz[0]; A += tz[DM]; P += tz[2 * DM];
            }
        } else {
            double c2 = s[11];
            P = s[12];
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const double c = a.xi[k * Vp + v] - s[8 + k];
                c2 = fma(c, c, c2);
                P = fma(c, s[5 + k], P);
            }
            A = c2 * s[4];
            e = s[3] * exp(-0.5 * A);
            A -= D + 2;
        }
        const double ep = e * P;
        gE = fma(ep, A, e);
        hE = H ? fma(ck, ep, gE) : 0.0;
    };
    if (!bnd) {  // every velocity once
#pragma unroll 2
        for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
            double gE, hE;
            equilibrium(v, gE, hE);
            go[base + v] = fma(om, gi[base + v], gE);
            if (H) ho[base + v] = fma(hf, hE, om * hi[base + v]);
        }
        return;
    }
    // The project's surface patch types ignore the field assignment (e.g.
    // maxwellWallFvsPatchField.H:163-181), symmetryPlane takes it; then every
    // outgoing DV is relaxed once more (discreteVelocity.C:887-931); incoming
    // boundary DVs stay unrelaxed.
    const int plane = a.bKind[en - a.nI] == kBcSymmetryPlane;
    const double S[3] = {a.Sf[3 * en], a.Sf[3 * en + 1], a.Sf[3 * en + 2]};
    for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
        const int times = plane + (a.xi[v] * S[0] + a.xi[Vp + v] * S[1] + a.xi[2 * Vp + v] * S[2] > 0);
        if (times == 0) continue;
        double g = gi[base + v], h = H ? hi[base + v] : 0.0, gE, hE;
        equilibrium(v, gE, hE);
        for (int t = 0; t < times; ++t) {
            g = fma(om, g, gE);
            if (H) h = fma(hf, hE, om * h);
        }
        go[base + v] = g;
        if (H) ho[base + v] = h;
    }
}

// Faces of a cell staged per warp: vector (LS vector, or -+S dt/V), row of the
// other cell or of the face, and on boundary faces 1/deltaCoeff.  Cells with
// more faces read the rest in place.
constexpr int kStage = 8;
constexpr int kSmallBlock = 2;  // warps per block of k_grad and k_cell: even loads of the SMs on small meshes
                                // (61^2 quads with 8 warps: 466 blocks on 152 SMs, the last wave nearly empty)
struct StagedFace {
    double L[3], idc;
    int row, wall;  // wall: boundary face index, or -1
};

// Entry j of cell c's least-squares stencil (outside the velocity loop: the
// division by deltaCoeff once per boundary face).
template <int D>
__device__ __forceinline__ StagedFace grad_entry(const StepArgs& a, int j) {
    StagedFace r;
    const int e = a.cellFace[j], f = chk(e >> 1, a.nA, a.status), side = e & 1;
    if (f < a.nI) {
        r.row = chk(side ? a.own[f] : a.nei[f], a.nC, a.status);
        r.wall = -1;
        r.idc = 0.0;
#pragma unroll
        for (int k = 0; k < D; ++k) r.L[k] = (side ? a.nVec : a.pVec)[3 * f + k];
    } else {
        const int wf = f - a.nI;
        r.row = 0;
        r.wall = wf;
        // symmetryPlane is a constraint patch of gBarPvol: its scalar value is
        // the internal value, so it adds nothing
        r.idc = a.bKind[wf] == kBcSymmetryPlane ? 0.0 : 1.0 / a.dcW[wf];
#pragma unroll
        for (int k = 0; k < D; ++k) r.L[k] = a.bVec[3 * wf + k];
    }
    return r;
}

// Least-squares gradient of gBarPvol (cell-centric gather in increasing face
// order = the reference's scatter order), fixedGradient boundary value
// phi_b = phi_P + G_b/deltaCoeff_b with the lagged G_b, then G_b <- grad.n.
// VU velocities per lane share the reading of the face list.  24k triangles x
// 32^2: 1.54 -> 0.81 ms, FP64 pipe 92 % busy.
template <int D, bool H>
__global__ void __launch_bounds__(32 * kSmallBlock) k_grad(StepArgs a, const double* __restrict__ gB, const double* __restrict__ hB,
                                              double* __restrict__ gG, double* __restrict__ hG, double* Gbg,
                                              double* Gbh) {
    constexpr int VU = 2;
    __shared__ StagedFace stage[kSmallBlock][kStage];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Vp = a.Vp, nV = a.nV;
    const int c = blockIdx.x * (blockDim.x >> 5) + warp;
    if (c >= a.nC) return;
    const int j0 = a.cellOff[c], nf = a.cellOff[c + 1] - j0;
    StagedFace* st = stage[warp];
    if (lane < min(nf, kStage)) st[lane] = grad_entry<D>(a, j0 + lane);
    __syncwarp();
    const long long base = (long long)c * Vp;
    for (int v0 = lane; v0 < nV; v0 += 32 * VU) {
        int vv[VU];
        double gc[VU], hc[VU], g[VU][D], h[VU][D];
#pragma unroll
        for (int u = 0; u < VU; ++u) {
            vv[u] = min(v0 + 32 * u, nV - 1);
            gc[u] = gB[base + vv[u]];
            hc[u] = H ? hB[base + vv[u]] : 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) g[u][k] = h[u][k] = 0.0;
        }
        bool walls = false;
        for (int j = 0; j < nf; ++j) {
            StagedFace r;
            if (j < kStage) r = st[j];
            else r = grad_entry<D>(a, j0 + j);
            double dg[VU], dh[VU];
            if (r.wall < 0) {
                const long long ob = (long long)r.row * Vp;
#pragma unroll
                for (int u = 0; u < VU; ++u) {
                    dg[u] = gB[ob + vv[u]] - gc[u];
                    dh[u] = H ? hB[ob + vv[u]] - hc[u] : 0.0;
                }
            } else {
                walls = true;
#pragma unroll
                for (int u = 0; u < VU; ++u) {
                    const long long wi = (long long)r.wall * Vp + vv[u];
                    dg[u] = fma(Gbg[wi], r.idc, gc[u]) - gc[u];
                    dh[u] = H ? fma(Gbh[wi], r.idc, hc[u]) - hc[u] : 0.0;
                }
            }
#pragma unroll
            for (int u = 0; u < VU; ++u)
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    g[u][k] = fma(r.L[k], dg[u], g[u][k]);
                    if (H) h[u][k] = fma(r.L[k], dh[u], h[u][k]);
                }
        }
#pragma unroll
        for (int u = 0; u < VU; ++u) {
            const int v = v0 + 32 * u;
            if (v >= nV) break;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                gG[((long long)c * D + k) * Vp + v] = g[u][k];
                if (H) hG[((long long)c * D + k) * Vp + v] = h[u][k];
            }
            if (!walls) continue;
            for (int j = j0; j < j0 + nf; ++j) {
                const int f = chk(a.cellFace[j] >> 1, a.nA, a.status);
                if (f < a.nI) continue;
                const int wf = f - a.nI;
                const double* nh = a.nHatW + 3 * wf;
                double sg = 0.0, sh = 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) { sg += g[u][k] * nh[k]; sh += h[u][k] * nh[k]; }
                Gbg[(long long)wf * Vp + v] = sg;
                if (H) Gbh[(long long)wf * Vp + v] = sh;
            }
        }
    }
}

// gbar+ of cell c at velocity v extrapolated by dk = d - xi dt/2.
template <int D>
__device__ __forceinline__ double recon(const double* __restrict__ f, const double* __restrict__ G, int c, int v,
                                        int Vp, const double* dk) {
    double acc = 0.0;
    const double* Gc = G + (long long)c * D * Vp + v;
#pragma unroll
    for (int k = 0; k < D; ++k) acc = fma(Gc[(long long)k * Vp], dk[k], acc);
    return f[(long long)c * Vp + v] + acc;
}

// P3: face values.  On internal faces the sign of xi.S selects the upwind
// cell; it is taken in FP32 where |xi.S| is above 1e-6 sum |xi_k S_k| (FP32
// rounding of the three products and their sum stays below 5e-7 of that) and
// in FP64, without FMA, for the warp iterations that hold a velocity nearer
// to the face, so that the choice and the ties are the FP64 ones.  The shifts
// d_k - xi_k dt/2 of both sides come from per-direction tables (TAB).  FP64
// operations per velocity: 14 -> 6 (2D, g and h), 20 -> 4 (3D, g); 24k
// triangles x 32^2: 3.27 -> 0.47 ms, 15^3 hexes x 14^3: 1.65 -> 0.55 ms.
template <int D, bool H, bool TAB>
__global__ void __launch_bounds__(256) k_recon(StepArgs a, const double* __restrict__ gB, const double* __restrict__ hB,
                                               const double* __restrict__ gG, const double* __restrict__ hG,
                                               double* __restrict__ gS, double* __restrict__ hS) {
    extern __shared__ double tab[];  // per face: shift of the owner side [D][M], of the neighbour side [D][M]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Vp = a.Vp, nV = a.nV, M = a.M;
    const int f = blockIdx.x * (blockDim.x >> 5) + warp;
    if (f >= a.nA) return;
    const long long base = (long long)f * Vp;
    double dO[D], dN[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        dO[k] = a.dO[3 * f + k];
        dN[k] = f < a.nI ? a.dN[3 * f + k] : 0.0;
    }
    const double mh = -0.5 * a.dt;
    const int o = chk(a.own[f], a.nC, a.status);
    if (f < a.nI) {
        const int nb = chk(a.nei[f], a.nC, a.status), DM = D * M;
        double S[D];
        float Sf[D], Sa[D];
#pragma unroll
        for (int k = 0; k < D; ++k) {
            S[k] = a.Sf[3 * f + k];
        }
        // scaled to a largest component in [1, 2) by its exponent: no underflow in FP32
        int ex = 0;
#pragma unroll
        for (int k = 0; k < D; ++k) ex = max(ex, (__double2hiint(S[k]) >> 20) & 0x7ff);
        const double sc = ex > 0 && ex < 2046 ? __hiloint2double((2046 - ex) << 20, 0) : 1.0;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            Sf[k] = (float)(S[k] * sc);
            Sa[k] = fabsf(Sf[k]) * 1e-6f;
        }
        double* tb = tab + (size_t)warp * 2 * DM;
        if (TAB) {
            for (int t = lane; t < DM; t += 32) {
                const int k = t / M;
                const double x = a.x1[t - k * M], dok = k == 0 ? dO[0] : (k == 1 ? dO[D > 1 ? 1 : 0] : dO[D - 1]),
                             dnk = k == 0 ? dN[0] : (k == 1 ? dN[D > 1 ? 1 : 0] : dN[D - 1]);
                tb[t] = fma(x, mh, dok);
                tb[DM + t] = fma(x, mh, dnk);
            }
            __syncwarp();
        }
        DvIdx<D> id;
        id.init(lane, 32, M);
        const int nIt = (nV + 31) / 32;
        // 32 warp iterations at a time: the signs as one bit each, then the
        // velocities near the face again in FP64 (a loop of its own: as a
        // branch it was predicated and its FP64 instructions issued always),
        // the face values, and the ties
        for (int i0 = 0; i0 < nIt; i0 += 32) {
            const int n = min(32, nIt - i0);
            unsigned own = 0u, near = 0u, ties = 0u;
            for (int i = 0; i < n; ++i) {
                const int v = min(lane + 32 * (i0 + i), nV - 1);
                float s32 = 0.f, b32 = 1e-30f;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float x = a.xi32[k * Vp + v];
                    s32 = fmaf(x, Sf[k], s32);
                    b32 = fmaf(fabsf(x), Sa[k], b32);
                }
                own |= (s32 > 0.f ? 1u : 0u) << i;
                near |= (fabsf(s32) > b32 ? 0u : 1u) << i;
            }
            for (unsigned m = __reduce_or_sync(0xffffffffu, near); m; m &= m - 1) {
                const int i = __ffs(m) - 1, v = min(lane + 32 * (i0 + i), nV - 1);
                double xs = 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const double x = a.xi[k * Vp + v];
                    xs = k == 0 ? x * S[0] : xs + x * S[k];
                }
                const bool up = xs >= kVSmall, tie = !up && !(xs < -kVSmall);
                own = (own & ~(1u << i)) | ((up ? 1u : 0u) << i);
                ties |= (tie ? 1u : 0u) << i;
            }
#pragma unroll 2
            for (int i = 0; i < n; ++i, id.advance(M)) {
                const int v = lane + 32 * (i0 + i);
                if (v >= nV) break;
                const bool fromOwn = own >> i & 1u;
                double dk[D];
                if (TAB) {
                    const double* td = tb + (fromOwn ? 0 : DM);
                    dk[0] = td[id.ix];
                    if (D > 1) dk[D > 1 ? 1 : 0] = td[M + id.iy];
                    if (D > 2) dk[D > 2 ? 2 : 0] = td[2 * M + id.iz];
                } else {
#pragma unroll
                    for (int k = 0; k < D; ++k) dk[k] = fma(a.xi[k * Vp + v], mh, fromOwn ? dO[k] : dN[k]);
                }
                const int u = fromOwn ? o : nb;
                gS[base + v] = recon<D>(gB, gG, u, v, Vp, dk);
                if (H) hS[base + v] = recon<D>(hB, hG, u, v, Vp, dk);
            }
            for (unsigned m = __reduce_or_sync(0xffffffffu, ties); m; m &= m - 1) {  // averages of both sides
                const int i = __ffs(m) - 1, v = lane + 32 * (i0 + i);
                if (v >= nV || !(ties >> i & 1u)) continue;
                double dk[D], dn[D];
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    dk[k] = fma(a.xi[k * Vp + v], mh, dO[k]);
                    dn[k] = fma(a.xi[k * Vp + v], mh, dN[k]);
                }
                gS[base + v] = 0.5 * (recon<D>(gB, gG, nb, v, Vp, dn) + recon<D>(gB, gG, o, v, Vp, dk));
                if (H) hS[base + v] = 0.5 * (recon<D>(hB, hG, nb, v, Vp, dn) + recon<D>(hB, hG, o, v, Vp, dk));
            }
        }
        return;
    }
    const int wf = f - a.nI, kind = a.bKind[wf];
    const bool sym = kind == kBcSymmetryMod || kind == kBcSymmetryPlane;
    const bool far = kind == kBcFarField || kind == kBcPressureIn || kind == kBcPressureOut;
    const double sz[3] = {a.Sf[3 * f], a.Sf[3 * f + 1], a.Sf[3 * f + 2]};
    for (int v = lane; v < nV; v += 32) {
        if (kind == kBcZeroGradient) {  // gSurf == gBarPvol patchInternalField, every DV
            gS[base + v] = gB[(long long)o * Vp + v];
            if (H) hS[base + v] = hB[(long long)o * Vp + v];
            continue;
        }
        const double x[3] = {a.xi[v], a.xi[Vp + v], a.xi[2 * Vp + v]};
        const double xs = x[0] * sz[0] + x[1] * sz[1] + x[2] * sz[2];
        if (sym ? xs > -kVSmall : xs > 0) {  // outgoing (and tangential on symmetry patches)
            double dk[D];
#pragma unroll
            for (int k = 0; k < D; ++k) dk[k] = fma(x[k], mh, dO[k]);
            gS[base + v] = recon<D>(gB, gG, o, v, Vp, dk);
            if (H) hS[base + v] = recon<D>(hB, hG, o, v, Vp, dk);
        } else if (far) {
            // incoming: rho_b M(U of the owner cell, T_b) (discreteVelocity.C:570-600)
            const double Tb = a.TbM[wf];
            const double g = a.rhoB[wf] * maxwell_by_rho_ref(a.U[3 * o], a.U[3 * o + 1], a.U[3 * o + 2], Tb, x[0],
                                                             x[1], x[2], a.R, D);
            gS[base + v] = g;
            if (H) hS[base + v] = g * (a.R * Tb) * (a.K + 3 - D);
        }
    }
}

// One block per wall face: rho_w = sum_out w (xi.S) gbar / |inComingByRho|,
// then incoming DVs (xi.S <= 0) get rho_w * Maxwellian(U_w, T_w), a product of
// per-direction factors when they fit shared memory (tabBytes > 0).
__global__ void k_wall(StepArgs a, double* __restrict__ gS, double* __restrict__ hS, int useTab) {
    __shared__ double red[32];
    extern __shared__ double tab[];
    const int wf = blockIdx.x;
    if (a.bKind[wf] != kBcMaxwell) return;  // uniform over the block
    const int f = a.nI + wf;
    const int Vp = a.Vp, M = a.M, D = a.D;
    const double* S = a.Sf + 3 * f;
    const double Tw = a.Tw[wf];
    const double* Uw = a.Uw + 3 * wf;
    if (useTab) {
        const double i2 = 1.0 / (2.0 * a.R * Tw), s = sqrt(2.0 * kPi * a.R * Tw);
        for (int t = threadIdx.x; t < D * M; t += blockDim.x) {
            const int k = t / M;
            const double c = Uw[k] - a.x1[t - k * M];
            double c2 = c * c, n = 1.0;
            if (k == 0) {
                for (int q = D; q < 3; ++q) c2 += Uw[q] * Uw[q];
                n = 1.0 / (D == 2 ? s * s : (D == 3 ? s * s * s : s));
            }
            tab[t] = n * exp(-c2 * i2);
        }
    }
    double acc[1] = {0.0};
    for (int v = threadIdx.x; v < a.nV; v += blockDim.x) {
        double xs = a.xi[v] * S[0] + a.xi[Vp + v] * S[1] + a.xi[2 * Vp + v] * S[2];
        if (xs > 0) acc[0] += a.w[v] * xs * gS[(long long)f * Vp + v];
    }
    block_sum<1>(acc, red);  // its barriers also release the table
    const double rw = acc[0] / a.incAbs[wf];
    if (threadIdx.x == 0) a.rhoW[wf] = rw;
    const double hk = (a.R * Tw) * (a.K + 3 - D);
    for (int v = threadIdx.x; v < a.nV; v += blockDim.x) {
        double x0 = a.xi[v], x1 = a.xi[Vp + v], x2 = a.xi[2 * Vp + v];
        double xs = x0 * S[0] + x1 * S[1] + x2 * S[2];
        if (xs <= 0) {
            double mx;
            if (useTab) {
                const int r = v / M;
                mx = tab[v - r * M];
                if (D == 2) mx *= tab[M + r];
                if (D == 3) mx *= tab[M + r % M] * tab[2 * M + r / M];
            } else {
                mx = maxwell_by_rho_ref(Uw[0], Uw[1], Uw[2], Tw, x0, x1, x2, a.R, D);
            }
            const double g = rw * mx;
            gS[(long long)f * Vp + v] = g;
            if (a.hasH) hS[(long long)f * Vp + v] = g * hk;
        }
    }
}

// Symmetry patches, step 1: snapshot of the face values of every velocity.
__global__ void k_sym_snap(StepArgs a, const double* __restrict__ gS, const double* __restrict__ hS,
                           double* __restrict__ gSnap, double* __restrict__ hSnap) {
    const int wf = blockIdx.x;
    if (a.symOff[wf] < 0) return;
    const long long fb = (long long)(a.nI + wf) * a.Vp, wb = (long long)wf * a.Vp;
    for (int v = threadIdx.x; v < a.nV; v += blockDim.x) {
        gSnap[wb + v] = gS[fb + v];
        if (a.hasH) hSnap[wb + v] = hS[fb + v];
    }
}

// Step 2: incoming velocities (xi.S0 <= 0, S0 the patch's first face) take
// their mirror velocity's value.  DVMsymmetry reads the snapshot; symmetryPlane
// assigns velocity by velocity in index order, so a mirror that is itself an
// earlier incoming velocity already holds its own mirror's value: the chain is
// followed back to a snapshot value (one step on grids symmetric about 0).
__global__ void k_sym_in(StepArgs a, double* __restrict__ gS, double* __restrict__ hS,
                         const double* __restrict__ gSnap, const double* __restrict__ hSnap) {
    const int wf = blockIdx.x;
    const int row = a.symOff[wf];
    if (row < 0) return;
    const int Vp = a.Vp, nV = a.nV;
    const bool plane = a.bKind[wf] == kBcSymmetryPlane;
    const double* S0 = a.bS0 + 3 * wf;
    const int* tab = a.symTab + (long long)row * nV;
    const long long fb = (long long)(a.nI + wf) * Vp, wb = (long long)wf * Vp;
    auto incoming = [&](int u) { return a.xi[u] * S0[0] + a.xi[Vp + u] * S0[1] + a.xi[2 * Vp + u] * S0[2] <= 0; };
    for (int v = threadIdx.x; v < nV; v += blockDim.x) {
        if (!incoming(v)) continue;
        int cur = v, u = tab[v];
        if (plane)
            for (int guard = 0; guard < nV && u < cur && incoming(u); ++guard) {
                cur = u;
                u = tab[u];
            }
        gS[fb + v] = gSnap[wb + u];
        if (a.hasH) hS[fb + v] = hSnap[wb + u];
    }
}

// Macros of the cells (P9) or of the active faces (P6, with qWall and
// stressWall on walls), two velocity passes as the reference: density,
// momentum and energy with the weights w, w xi, w |xi|^2/2 tabulated once
// (a.mw), then the heat flux about the velocity found, with the entity's
// c and c^2 tabulated per direction (TAB).  The square root, divisions,
// logarithm and exponential of the macros run once per block, one lane per
// entity.  24k triangles x 32^2: faces 4.74 -> 0.88 ms, cells 3.07 -> 0.46 ms.
template <int D, bool H, bool TAB, bool FACE>
__global__ void k_mom(StepArgs a, const double* __restrict__ gS, const double* __restrict__ hS) {
    constexpr int NS = D == 3 ? 8 : 4, NQ = 4;  // reduced slots: rho, momentum, energy; heat flux
    __shared__ double sm[kMaxEnt][8];           // slot totals
    __shared__ double sr[kMaxEnt][8];           // rho, U, T, tau, heat-flux factor
    extern __shared__ double tab[];             // per entity: c [D][M] | c^2 [D][M]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nEnt = blockDim.x >> 5;
    const int n = FACE ? a.nA : a.nC, e0 = blockIdx.x * nEnt, en = e0 + warp, M = a.M, Vp = a.Vp, nV = a.nV;
    const bool active = en < n;
    const long long base = (long long)en * Vp;
    if (active) {
        double m[NS], eh = 0.0;
#pragma unroll
        for (int i = 0; i < NS; ++i) m[i] = 0.0;
#pragma unroll 2
        for (int v = lane; v < nV; v += 32) {
            const double g = gS[base + v];
#pragma unroll
            for (int i = 0; i <= D; ++i) m[i] = fma(a.mw[i * Vp + v], g, m[i]);
            m[D + 1] = fma(a.mw[(D + 1) * Vp + v], g, m[D + 1]);
            if (H) eh = fma(a.mw[v], hS[base + v], eh);
        }
        if (H) m[D + 1] = fma(0.5, eh, m[D + 1]);
        const double r = scatter_sum<NS>(m, lane);
        if ((lane & (32 / NS - 1)) == 0) sm[warp][warp_slot<NS>(lane)] = r;
    }
    __syncthreads();
    if (threadIdx.x < nEnt && e0 + threadIdx.x < n) {
        const int i = e0 + threadIdx.x;
        const double* m = sm[threadIdx.x];
        double* s = sr[threadIdx.x];
        const double rho = m[0], ir = 1.0 / rho;
        double U[3] = {0, 0, 0}, uu = 0.0;
#pragma unroll
        for (int k = 0; k < D; ++k) { U[k] = m[1 + k] * ir; uu += U[k] * U[k]; }
        const double T = (m[D + 1] - 0.5 * rho * uu) * ir / ((a.K + 3) / 2.0 * a.R);
        const double tau = a.muRef * exp(a.omega * log(T / a.Tref)) / (rho * T * a.R);
        const double fac = 2.0 * tau / (2.0 * tau + (FACE ? 0.5 : 1.0) * a.dt * a.Pr);
        (FACE ? a.rhoF : a.rho)[i] = rho;
        (FACE ? a.TF : a.T)[i] = T;
        (FACE ? a.tauF : a.tau)[i] = tau;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            (FACE ? a.UF : a.U)[3 * i + k] = U[k];
            if (k >= D) (FACE ? a.qF : a.q)[3 * i + k] = 0.0;
        }
        s[0] = U[0]; s[1] = U[1]; s[2] = U[2];
        s[3] = fac;
        s[4] = tau;
        if (!FACE && (!(rho > 0.0) || !(T > 0.0) || !isfinite(uu))) atomicExch(a.status, 5);
    }
    __syncthreads();
    if (!active) return;
    const double* s = sr[warp];
    const double fac = s[3];
    double U[D], qq[NQ];
#pragma unroll
    for (int k = 0; k < D; ++k) U[k] = s[k];
#pragma unroll
    for (int i = 0; i < NQ; ++i) qq[i] = 0.0;
    const int DM = D * M;
    double* tb = tab + (size_t)warp * 2 * DM;
    if (TAB) {
        for (int t = lane; t < DM; t += 32) {
            const int k = t / M;
            const double c = a.x1[t - k * M] - s[k];
            tb[t] = c;
            tb[DM + t] = c * c;
        }
        __syncwarp();
    }
    DvIdx<D> id;
    id.init(lane, 32, M);
    for (int v = lane; v < nV; v += 32, id.advance(M)) {
        const double g = gS[base + v], h = H ? hS[base + v] : 0.0;
        double c[D], cc;
        if (TAB) {
            c[0] = tb[id.ix];
            cc = tb[DM + id.ix];
            if (D > 1) { c[D > 1 ? 1 : 0] = tb[M + id.iy]; cc += tb[DM + M + id.iy]; }
            if (D > 2) { c[D > 2 ? 2 : 0] = tb[2 * M + id.iz]; cc += tb[DM + 2 * M + id.iz]; }
        } else {
            cc = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) { c[k] = a.xi[k * Vp + v] - U[k]; cc = fma(c[k], c[k], cc); }
        }
        const double ws = a.w[v] * (H ? fma(cc, g, h) : cc * g);
#pragma unroll
        for (int k = 0; k < D; ++k) qq[k] = fma(ws, c[k], qq[k]);
    }
    const double r = 0.5 * scatter_sum<NQ>(qq, lane);
    const int slot = warp_slot<NQ>(lane);
    if ((lane & 7) == 0 && slot < D) {
        (FACE ? a.qF : a.q)[3 * en + slot] = fac * r;
        if (!FACE && !isfinite(r)) atomicExch(a.status, 5);
    }
    if (!FACE || en < a.nI || a.bKind[en - a.nI] != kBcMaxwell) return;
    // wall heat flux about U_w and wall stress
    const int wf = en - a.nI;
    const double* Uw = a.Uw + 3 * wf;
    double x12[9];  // q about U_w, then the upper triangle xx xy xz yy yz zz
#pragma unroll
    for (int i = 0; i < 9; ++i) x12[i] = 0.0;
    for (int v = lane; v < nV; v += 32) {
        const double x[3] = {a.xi[v], a.xi[Vp + v], a.xi[2 * Vp + v]}, w = a.w[v];
        const double g = gS[base + v], h = H ? hS[base + v] : 0.0;
        const double e[3] = {x[0] - Uw[0], x[1] - Uw[1], x[2] - Uw[2]};
        const double sw = 0.5 * w * ((e[0] * e[0] + e[1] * e[1] + e[2] * e[2]) * g + h), wg = w * g;
        const double wx = wg * x[0], wy = wg * x[1];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x12[k] = fma(sw, e[k], x12[k]);
            x12[3 + k] = fma(wx, x[k], x12[3 + k]);
            if (k > 0) x12[5 + k] = fma(wy, x[k], x12[5 + k]);
        }
        x12[8] = fma(wg * x[2], x[2], x12[8]);
    }
    warp_sum<9>(x12);
    if (lane == 0) {
        const double tau = s[4], fs = 2.0 * tau / (2.0 * tau + 0.5 * a.dt);
        for (int k = 0; k < 3; ++k) a.qWall[3 * wf + k] = fac * x12[k];
        const int at[9] = {3, 4, 5, 4, 6, 7, 5, 7, 8};
#pragma unroll
        for (int k = 0; k < 9; ++k) a.stressWall[9 * wf + k] = fs * x12[at[k]];
    }
}

// P8: g~ <- -g~/3 + 4/3 gbar+ - dt/V sum_f (xi.S_f) g_f, one warp per cell,
// faces in increasing order; -+S dt/V is formed once per cell (it was a
// division per face, field and velocity).  With h (2D) xi.S is shared by the
// two fields; without, sum_f S_f g_f is formed per component first: D
// operations per face and D per velocity instead of D + 1 per face.  24k
// triangles x 32^2: 3.94 -> 0.89 ms (FP64 pipe 87 % busy), 15^3 hexes x 14^3:
// 1.73 -> 0.65 ms.
template <int D, bool H>
__global__ void __launch_bounds__(32 * kSmallBlock) k_cell(StepArgs a, double* gT, double* hT, const double* __restrict__ gB,
                                              const double* __restrict__ hB, const double* __restrict__ gS,
                                              const double* __restrict__ hS) {
    constexpr int VU = 2;
    __shared__ StagedFace stage[kSmallBlock][kStage];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Vp = a.Vp, nV = a.nV;
    const int c = blockIdx.x * (blockDim.x >> 5) + warp;
    if (c >= a.nC) return;
    const int j0 = a.cellOff[c], nf = a.cellOff[c + 1] - j0;
    const long long base = (long long)c * Vp;
    const double kv = a.dt / a.vol[c];
    auto entry = [&](int j) {
        StagedFace r;
        const int e = a.cellFace[j];
        const double sk = e & 1 ? kv : -kv;
        r.row = chk(e >> 1, a.nA, a.status);
        r.wall = -1;
        r.idc = 0.0;
#pragma unroll
        for (int k = 0; k < D; ++k) r.L[k] = sk * a.Sf[3 * r.row + k];
        return r;
    };
    if (lane < min(nf, kStage)) stage[warp][lane] = entry(j0 + lane);
    __syncwarp();
    for (int v0 = lane; v0 < nV; v0 += 32 * VU) {
        int vv[VU];
        double x[VU][D], g[VU], h[VU], sg[VU][D];
#pragma unroll
        for (int u = 0; u < VU; ++u) {
            vv[u] = min(v0 + 32 * u, nV - 1);
#pragma unroll
            for (int k = 0; k < D; ++k) {
                x[u][k] = a.xi[k * Vp + vv[u]];
                sg[u][k] = 0.0;
            }
            const long long i = base + vv[u];
            g[u] = fma(4.0 / 3, gB[i], -1.0 / 3 * gT[i]);
            h[u] = H ? fma(4.0 / 3, hB[i], -1.0 / 3 * hT[i]) : 0.0;
        }
        for (int j = 0; j < nf; ++j) {
            StagedFace r;
            if (j < kStage) r = stage[warp][j];
            else r = entry(j0 + j);
            const long long fb = (long long)r.row * Vp;
#pragma unroll
            for (int u = 0; u < VU; ++u) {
                const double gf = gS[fb + vv[u]];
                if (H) {
                    double xs = x[u][0] * r.L[0];
#pragma unroll
                    for (int k = 1; k < D; ++k) xs = fma(x[u][k], r.L[k], xs);
                    g[u] = fma(xs, gf, g[u]);
                    h[u] = fma(xs, hS[fb + vv[u]], h[u]);
                } else {
#pragma unroll
                    for (int k = 0; k < D; ++k) sg[u][k] = fma(r.L[k], gf, sg[u][k]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < VU; ++u) {
            if (v0 + 32 * u >= nV) break;
            if (!H)
#pragma unroll
                for (int k = 0; k < D; ++k) g[u] = fma(x[u][k], sg[u][k], g[u]);
            gT[base + vv[u]] = g[u];
            if (H) hT[base + vv[u]] = h[u];
        }
    }
}

// P10: pressureIn / pressureOut patch values from the new cell macros of the
// owner (characteristic relations of fvDVM::updatePressureInOutBC).
__global__ void k_pressure(StepArgs a) {
    const int wf = blockIdx.x * blockDim.x + threadIdx.x;
    if (wf >= a.nW) return;
    const int kind = a.bKind[wf];
    if (kind != kBcPressureIn && kind != kBcPressureOut) return;
    const int f = a.nI + wf, P = a.own[f];
    const double* Sf = a.Sf + 3 * f;
    const double magSf = sqrt(Sf[0] * Sf[0] + Sf[1] * Sf[1] + Sf[2] * Sf[2]);
    const double n[3] = {Sf[0] / magSf, Sf[1] / magSf, Sf[2] / magSf};
    const double Ui[3] = {a.U[3 * P], a.U[3 * P + 1], a.U[3 * P + 2]};
    const double Ti = a.T[P], rhoi = a.rho[P], R = a.R, p = a.pB[wf];
    const double ai = sqrt(R * Ti * (a.K + 5) / (a.K + 3));
    const double Un = Ui[0] * n[0] + Ui[1] * n[1] + Ui[2] * n[2];
    double UnIn;
    if (kind == kBcPressureIn) {
        a.rhoB[wf] = p / R / a.TbM[wf];
        UnIn = Un + (p - rhoi * R * Ti) / rhoi / ai;
    } else {
        a.rhoB[wf] = rhoi + (p - rhoi * R * Ti) / ai / ai;
        a.TbM[wf] = p / (R * rhoi);
        UnIn = Un + (rhoi * R * Ti - p) / rhoi / ai;
    }
    for (int k = 0; k < 3; ++k) a.UbM[3 * wf + k] = UnIn * n[k] + (Ui[k] - Un * n[k]);
}

// Uvol_/Tvol_.correctBoundaryConditions() (fvDVM.C:697-699) after the cell
// macros: a zeroGradient U or T patch takes its owner cell's new value (before
// P10, which reads T_b on pressureIn patches).
__global__ void k_zero_gradient_tu(StepArgs a) {
    const int wf = blockIdx.x * blockDim.x + threadIdx.x;
    if (wf >= a.nW) return;
    const int zg = a.bZG[wf];
    if (!zg) return;
    const int P = a.own[a.nI + wf];
    if (zg & 1) a.TbM[wf] = a.T[P];
    if (zg & 2)
        for (int k = 0; k < 3; ++k) a.UbM[3 * wf + k] = a.U[3 * P + k];
}

// Initial face values of mixed patches (rho fixedValue): the Maxwellian of the
// patch rho, U, T for every DV (discreteVelocity::initBoundaryField,
// discreteVelocity.C:302-345, equilibriumMaxwell :1046-1061).
__global__ void k_mixed_init(StepArgs a, double* __restrict__ gS, double* __restrict__ hS) {
    const int wf = blockIdx.x;
    if (a.bKind[wf] != kBcFixedValue) return;
    const long long fb = (long long)(a.nI + wf) * a.Vp;
    const double rho = a.rhoB[wf], T = a.TbM[wf], R = a.R;
    const double* U = a.UbM + 3 * wf;
    const double s = sqrt(2.0 * kPi * R * T);
    const double pw = (a.D == 2) ? s * s : (a.D == 3 ? s * s * s : s);
    for (int v = threadIdx.x; v < a.nV; v += blockDim.x) {
        const double c0 = U[0] - a.xi[v], c1 = U[1] - a.xi[a.Vp + v], c2 = U[2] - a.xi[2 * a.Vp + v];
        const double g = rho / pw * exp(-(c0 * c0 + c1 * c1 + c2 * c2) / (2.0 * R * T));
        gS[fb + v] = g;
        if (a.hasH) hS[fb + v] = (a.K + 3 - a.D) * R * T * g;
    }
}

// Warps per block of the passes whose block shares its entity scalars: up to
// 16 (their FP64 chain runs once per block, ~200 instructions, against ~300 to
// 600 of an entity's velocities), down to 4 while the entities would not make
// eight blocks per SM (few blocks leave SMs idle at the end), fewer when the tables (tabEnt bytes per entity) exceed
// what a block has without asking for more.
int ents_per_block(int n, size_t tabEnt, int sms, int e = kMaxEnt) {
    while (e > 1 && (((long long)n < 8LL * sms * e && e > 4) || tabEnt * e > kTabMax)) e >>= 1;
    return e;
}

template <int D, bool H>
struct Pass {
    template <bool FACE>
    static void eq(const StepArgs& a, const double* gi, const double* hi, double* go, double* ho, int sms,
                   cudaStream_t s) {
        const int n = FACE ? a.nA : a.nC;
        const size_t tb = 3 * sizeof(double) * D * a.M;
        const bool tab = tb <= kTabMax;
        const int e = ents_per_block(n, tab ? tb : 0, sms), blocks = (n + e - 1) / e;
        if (tab) k_eq<D, H, true, FACE><<<blocks, 32 * e, tb * e, s>>>(a, gi, hi, go, ho);
        else k_eq<D, H, false, FACE><<<blocks, 32 * e, 0, s>>>(a, gi, hi, go, ho);
    }
    template <bool FACE>
    static void mom(const StepArgs& a, const double* g, const double* h, int sms, cudaStream_t s) {
        const int n = FACE ? a.nA : a.nC;
        const size_t tb = 2 * sizeof(double) * D * a.M;
        const bool tab = tb <= kTabMax;
        const int e = ents_per_block(n, tab ? tb : 0, sms), blocks = (n + e - 1) / e;
        if (tab) k_mom<D, H, true, FACE><<<blocks, 32 * e, tb * e, s>>>(a, g, h);
        else k_mom<D, H, false, FACE><<<blocks, 32 * e, 0, s>>>(a, g, h);
    }
    static void run(int pass, const StepArgs& a, const RefBuffers& b, int sms, cudaStream_t s) {
        const int wC = (a.nC + kSmallBlock - 1) / kSmallBlock, wA = (a.nA + 7) / 8;
        switch (pass) {
            case 0: eq<false>(a, b.gT, b.hT, b.gB, b.hB, sms, s); break;
            case 1: k_grad<D, H><<<wC, 32 * kSmallBlock, 0, s>>>(a, b.gB, b.hB, b.gG, b.hG, b.Gbg, b.Gbh); break;
            case 2: {
                const size_t tb = 2 * sizeof(double) * D * a.M;
                const int w = ents_per_block(a.nA, tb, sms, 4), blocks = (a.nA + w - 1) / w;
                if (tb <= kTabMax) k_recon<D, H, true><<<blocks, 32 * w, tb * w, s>>>(a, b.gB, b.hB, b.gG, b.hG, b.gS, b.hS);
                else k_recon<D, H, false><<<wA, 256, 0, s>>>(a, b.gB, b.hB, b.gG, b.hG, b.gS, b.hS);
                break;
            }
            case 4: mom<true>(a, b.gS, b.hS, sms, s); break;
            case 5: eq<true>(a, b.gS, b.hS, b.gS, b.hS, sms, s); break;
            case 6: k_cell<D, H><<<wC, 32 * kSmallBlock, 0, s>>>(a, b.gT, b.hT, b.gB, b.hB, b.gS, b.hS); break;
            case 7: mom<false>(a, b.gT, b.hT, sms, s); break;
            default: break;
        }
    }
};

}  // namespace

void launch_pressure_bc(const StepArgs& a, cudaStream_t s) {
    if (a.nW > 0) k_pressure<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
}

void launch_zero_gradient_tu(const StepArgs& a, cudaStream_t s) {
    if (a.nW > 0 && a.zgMask) k_zero_gradient_tu<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
}

void launch_ref_mixed_init(const StepArgs& a, const RefBuffers& b, cudaStream_t s) {
    if (a.nW > 0 && (a.bcMask & (1 << kBcFixedValue))) k_mixed_init<<<a.nW, kRedThreads, 0, s>>>(a, b.gS, b.hS);
}

const char* const kRefKernelNames[kRefKernels] = {"k_barp", "k_grad", "k_recon", "k_wall",
                                                  "k_face_mom", "k_relax", "k_cell", "k_cell_mom"};

void launch_ref_pass(int pass, const StepArgs& a, const RefBuffers& b, int sms, cudaStream_t s) {
    if (pass == 3) {
        const size_t tb = sizeof(double) * a.D * a.M;
        const int tab = tb <= kTabMax;
        if (a.nW > 0 && (a.bcMask & (1 << kBcMaxwell))) k_wall<<<a.nW, kRedThreads, tab ? tb : 0, s>>>(a, b.gS, b.hS, tab);
        if (a.bcMask & ((1 << kBcSymmetryMod) | (1 << kBcSymmetryPlane))) {
            k_sym_snap<<<a.nW, kRedThreads, 0, s>>>(a, b.gS, b.hS, b.gSym, b.hSym);
            k_sym_in<<<a.nW, kRedThreads, 0, s>>>(a, b.gS, b.hS, b.gSym, b.hSym);
        }
        return;
    }
    switch (2 * a.D + (a.hasH ? 1 : 0)) {
        case 2: Pass<1, false>::run(pass, a, b, sms, s); break;
        case 3: Pass<1, true>::run(pass, a, b, sms, s); break;
        case 4: Pass<2, false>::run(pass, a, b, sms, s); break;
        case 5: Pass<2, true>::run(pass, a, b, sms, s); break;
        case 6: Pass<3, false>::run(pass, a, b, sms, s); break;
        case 7: Pass<3, true>::run(pass, a, b, sms, s); break;
        default: break;
    }
    if (pass == 7) {
        if (a.zgMask) k_zero_gradient_tu<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
        if (a.bcMask & ((1 << kBcPressureIn) | (1 << kBcPressureOut)))
            k_pressure<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
    }
}

}  // namespace dugks
