// One DUGKS step in FP64, pass by pass, with every intermediate in HBM (DV
// index innermost): the kernels of the plain FP64 pipeline (R = double,
// ref_pipeline.cu) and of the tangent-linear step (R = Dual, gradient.cu).
//
//   k_eq        P1 updateGHbarPvol             discreteVelocity.C:346-410
//   k_grad      P2 fvc::grad + fixedGradient   discreteVelocity.C:420-470
//   k_recon     P3 updateGHbarSurf             discreteVelocity.C:472-691
//   k_wall      P4+P5 MaxwellWallRho / WallIn  fvDVM.C:347-367, discreteVelocity.C:693-731
//   k_mom       P6 updateMacroSurf             fvDVM.C:456-582
//   k_eq        P7 updateGHsurf                discreteVelocity.C:819-932
//   k_cell      P8 updateGHtildeVol            discreteVelocity.C:934-978
//   k_mom       P9 updateMacroVol              fvDVM.C:597-728
//
// Boundary faces follow the surface patch type of their rho boundary
// condition (discreteVelocity::setBCtype, discreteVelocity.C:250-300):
// diffuse walls, zeroGradient, mixed (rho fixedValue), farField (also for
// pressureIn / pressureOut) and the two symmetry types (their copies and the
// pressure update are in ref_pipeline.cu).
#pragma once

#include <type_traits>

#include "device_common.cuh"
#include "dual.cuh"

namespace dugks {

// Macros of cells and active faces, wall data and viscosity in scalar type R.
template <class R>
struct Macros {
    R *rho, *U, *T, *q, *tau;
    R *rhoF, *UF, *TF, *qF, *tauF;
    R *rhoW, *qWall, *stressWall;
    const R *Tw, *incAbs;
    R muRef;
};
inline Macros<double> macros_of(const StepArgs& a) {
    return {a.rho, a.U, a.T, a.q, a.tau, a.rhoF, a.UF, a.TF, a.qF, a.tauF, a.rhoW, a.qWall, a.stressWall,
            a.Tw, a.incAbs, a.muRef};
}

// Distribution buffers of one step.
template <class R>
struct Fields {
    R *gT, *hT;          // [nC][Vp]      g~, h~
    R *gB, *hB;          // [nC][Vp]      gBarPvol, hBarPvol
    R *gG, *hG;          // [nC][D][Vp]   least-squares gradients
    R *Gbg, *Gbh;        // [nW][Vp]      lagged fixedGradient gradients
    R *gS, *hS;          // [nA][Vp]      face distributions
};

template <class R>
__device__ __forceinline__ R mk(double v);
template <>
__device__ __forceinline__ double mk<double>(double v) { return v; }
template <>
__device__ __forceinline__ Dual mk<Dual>(double v) { return Dual{v, 0.0}; }
__device__ __forceinline__ double val(double x) { return x; }
__device__ __forceinline__ double val(Dual x) { return x.v; }

// xi.S of the velocity at x (components Vp apart), rounded operation by
// operation (never contracted): the oracle's value, whose sign decides the
// upwind side, ties included.
__device__ __forceinline__ double dot_rn(const double* x, int Vp, const double* S) {
    return __dadd_rn(__dadd_rn(__dmul_rn(x[0], S[0]), __dmul_rn(x[Vp], S[1])), __dmul_rn(x[2 * Vp], S[2]));
}

namespace {

constexpr int kWallThreads = 128;
constexpr int kMaxEnt = 16;  // most entities (warps) per block
constexpr size_t kSmemMax = 48 * 1024;  // shared memory of a block that asks for no more
constexpr size_t kTabMax = 44 * 1024;   // tables of a block; its static scalars have the rest (asserted per kernel)

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
//   and field) -> ~90.

// Sum of NS per-lane values over the warp; the lane ends with the total of
// slot warp_slot<NS>(lane): NS - 1 + log2(32 / NS) additions instead of the
// butterfly's 5 NS.
__device__ __forceinline__ double shfl_xor(double x, int m) { return __shfl_xor_sync(0xffffffffu, x, m); }
__device__ __forceinline__ Dual shfl_xor(Dual x, int m) { return {shfl_xor(x.v, m), shfl_xor(x.d, m)}; }
template <int NS, class R>
__device__ __forceinline__ R scatter_sum(R (&v)[NS], int lane) {
    int xm = 16;
#pragma unroll
    for (int half = NS / 2; half >= 1; half >>= 1, xm >>= 1) {
        const bool up = lane & xm;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const R send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + shfl_xor(send, xm);
        }
    }
    R r = v[0];
#pragma unroll
    for (int o = 16 / NS; o >= 1; o >>= 1) r += shfl_xor(r, o);
    return r;
}
template <int NS>
__device__ __forceinline__ int warp_slot(int lane) {  // the leading bits of the lane
    return lane / (32 / NS);
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
// 24k triangles x 32^2: cells 5.04 -> 0.48 ms, faces 7.42 -> 0.78 ms (FP64 pipe
// 90 % busy; flat 0.52 and 0.83), 15^3 hexes x 14^3: faces 0.47 ms.
// COLS (kTabCols): a lane owns columns of velocities along the last direction,
// so that the other directions' factor, A and P are held in registers and the
// last direction's {E, A, E P} are read by all lanes alike: 5 operations per
// velocity without h, 8 with (9 flat).
enum EqMode { kCells, kFaces, kInit };
enum TabMode { kTabNone, kTabFlat, kTabCols };
template <class R, int D, bool H, TabMode TM, EqMode MODE>
__global__ void k_eq(StepArgs a, Macros<R> m, const R* gi, const R* hi, R* go, R* ho) {
    constexpr bool FACE = MODE == kFaces, TAB = TM != kTabNone, COLS = TM == kTabCols;
    __shared__ R sc[kMaxEnt][14];
    static_assert(sizeof(sc) + kTabMax <= kSmemMax, "k_eq: tables and scalars of a block");
    extern __shared__ __align__(16) unsigned char smemRaw[];
    R* tab = reinterpret_cast<R*>(smemRaw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nEnt = blockDim.x >> 5;
    const int n = FACE ? a.nA : a.nC, e0 = blockIdx.x * nEnt, M = a.M, Vp = a.Vp;
    const double K3 = a.K + 3.0 - D;
    if (threadIdx.x < nEnt && e0 + threadIdx.x < n) {
        const int i = e0 + threadIdx.x;
        const R rho = (FACE ? m.rhoF : m.rho)[i], T = (FACE ? m.TF : m.T)[i], tau = (FACE ? m.tauF : m.tau)[i];
        const R *U = (FACE ? m.UF : m.U) + 3 * i, *q = (FACE ? m.qF : m.q) + 3 * i;
        R* s = sc[threadIdx.x];
        const R RT = a.R * T, iRT = 1.0 / RT, s2 = 2.0 * kPi * RT;
        const double hh = 0.5 * a.dt;
        const R rf = MODE == kInit ? mk<R>(1.0) : (FACE ? hh / (2.0 * tau + hh) : 1.5 * a.dt / (2.0 * tau + a.dt));
        const R k0 = (1.0 - a.Pr) * iRT * iRT / (5.0 * rho);
        s[0] = 1.0 - rf;
        s[2] = RT * K3;
        const R rr = rf * rho;  // the relaxation weight goes with the factor of e
        s[3] = D == 2 ? rr / s2 : (D == 3 ? rr / (s2 * sqrt(s2)) : rr / sqrt(s2));
        s[4] = iRT;
        R x2 = mk<R>(0.0), xq = mk<R>(0.0);  // components outside the solution directions: their velocity is 0
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
            const R* s = sc[j];
            const R c = a.x1[i] - s[8 + k], c2 = k == 0 ? c * c + s[11] : c * c, ci = c2 * s[4];
            const R E = exp(-0.5 * ci);
            R* tb = tab + (size_t)j * 3 * DM + r;
            tb[0] = k == 0 ? E * s[3] : E;
            tb[DM] = k == 0 ? ci - (D + 2.0) : ci;
            const R P = k == 0 ? c * s[5] + s[12] : c * s[5 + k];
            tb[2 * DM] = COLS && k == D - 1 ? E * P : P;
        }
        __syncthreads();
    }
    const int en = e0 + warp;
    if (en >= n) return;
    const R* s = sc[warp];
    const R om = s[0], hf = s[2];
    const double ck = H ? 2.0 - 2.0 * a.K / K3 : 0.0;
    const R* tb = tab + (size_t)warp * 3 * DM;
    const long long base = (long long)en * Vp;
    const bool bnd = FACE && en >= a.nI;
    DvIdx<D> id;
    id.init(lane, 32, M);
    auto equilibrium = [&](int v, R& gE, R& hE) {
        R e, A, P;
        if (TAB) {
            const R* tx = tb + id.ix;
            e = tx[0]; A = tx[DM]; P = tx[2 * DM];
            if (D > 2 || (D == 2 && !COLS)) {
                const R* ty = tb + M + id.iy;
                e = e * ty[0]; A = A + ty[DM]; P = P + ty[2 * DM];
            }
            if (D > 2 && !COLS) {
                const R* tz = tb + 2 * M + id.iz;
                e = e * tz[0]; A = A + tz[DM]; P = P + tz[2 * DM];
            }
            if (COLS) {
                const R* tl = tb + (D - 1) * M + (D == 2 ? id.iy : id.iz);
                const R ep = e * fma(P, tl[0], tl[2 * DM]);
                e = e * tl[0]; A = A + tl[DM];
                gE = fma(ep, A, e);
                hE = H ? fma(ck, ep, gE) : mk<R>(0.0);
                return;
            }
        } else {
            R c2 = s[11];
            P = s[12];
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const R c = a.xi[k * Vp + v] - s[8 + k];
                c2 = fma(c, c, c2);
                P = fma(c, s[5 + k], P);
            }
            A = c2 * s[4];
            e = s[3] * exp(-0.5 * A);
            A = A - (D + 2.0);
        }
        const R ep = e * P;
        gE = fma(ep, A, e);
        hE = H ? fma(ck, ep, gE) : mk<R>(0.0);
    };
    if (COLS && !bnd) {
        const int NP = D == 2 ? M : M * M;
        const R *tE = tb + (D - 1) * M, *tA = tE + DM, *tP = tA + DM;
        for (int col = lane; col < NP; col += 32) {
            const R* tx = tb + (D == 2 ? col : col % M);
            R e = tx[0], A = tx[DM], P = tx[2 * DM];
            if (D == 3) {
                const R* ty = tb + M + col / M;
                e = e * ty[0]; A = A + ty[DM]; P = P + ty[2 * DM];
            }
            const R eh = H ? hf * e : mk<R>(0.0);
            const long long b0 = base + col;
            // the loads of a batch first: the faces are relaxed in place, and no
            // load may pass the store before it
            auto batch = [&](auto NB, int l) {
                constexpr int nb = decltype(NB)::value;
                R g[nb], h[nb];
#pragma unroll
                for (int u = 0; u < nb; ++u) {
                    const long long i = b0 + (long long)(l + u) * NP;
                    if (MODE != kInit) g[u] = gi[i];
                    if (H && MODE != kInit) h[u] = hi[i];
                }
#pragma unroll
                for (int u = 0; u < nb; ++u) {
                    const long long i = b0 + (long long)(l + u) * NP;
                    const R E = tE[l + u], ep = fma(P, E, tP[l + u]), gE = fma(ep, A + tA[l + u], E);
                    go[i] = MODE == kInit ? e * gE : fma(e, gE, om * g[u]);
                    if (H) {
                        const R hE = fma(ck, ep, gE);
                        ho[i] = MODE == kInit ? eh * hE : fma(eh, hE, om * h[u]);
                    }
                }
            };
            int l = 0;
            for (; l + 4 <= M; l += 4) batch(std::integral_constant<int, 4>(), l);
            for (; l < M; ++l) batch(std::integral_constant<int, 1>(), l);
        }
        return;
    }
    if (!bnd) {  // every velocity once
#pragma unroll 2
        for (int v = lane; v < a.nV; v += 32, id.advance(M)) {
            R gE, hE;
            equilibrium(v, gE, hE);
            go[base + v] = MODE == kInit ? gE : fma(om, gi[base + v], gE);
            if (H) ho[base + v] = MODE == kInit ? hf * hE : fma(hf, hE, om * hi[base + v]);
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
        const int times = plane + (dot_rn(a.xi + v, Vp, S) > 0);
        if (times == 0) continue;
        R g = gi[base + v], h = H ? hi[base + v] : mk<R>(0.0), gE, hE;
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
template <class R, int D, bool H>
__global__ void __launch_bounds__(32 * kSmallBlock) k_grad(StepArgs a, const R* __restrict__ gB, const R* __restrict__ hB,
                                                           R* __restrict__ gG, R* __restrict__ hG, R* Gbg, R* Gbh) {
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
        R gc[VU], hc[VU], g[VU][D], h[VU][D];
#pragma unroll
        for (int u = 0; u < VU; ++u) {
            vv[u] = min(v0 + 32 * u, nV - 1);
            gc[u] = gB[base + vv[u]];
            hc[u] = H ? hB[base + vv[u]] : mk<R>(0.0);
#pragma unroll
            for (int k = 0; k < D; ++k) g[u][k] = h[u][k] = mk<R>(0.0);
        }
        bool walls = false;
        for (int j = 0; j < nf; ++j) {
            StagedFace r;
            if (j < kStage) r = st[j];
            else r = grad_entry<D>(a, j0 + j);
            R dg[VU], dh[VU];
            if (r.wall < 0) {
                const long long ob = (long long)r.row * Vp;
#pragma unroll
                for (int u = 0; u < VU; ++u) {
                    dg[u] = gB[ob + vv[u]] - gc[u];
                    dh[u] = H ? hB[ob + vv[u]] - hc[u] : mk<R>(0.0);
                }
            } else {
                walls = true;
#pragma unroll
                for (int u = 0; u < VU; ++u) {
                    const long long wi = (long long)r.wall * Vp + vv[u];
                    dg[u] = fma(Gbg[wi], r.idc, gc[u]) - gc[u];
                    dh[u] = H ? fma(Gbh[wi], r.idc, hc[u]) - hc[u] : mk<R>(0.0);
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
                R sg = mk<R>(0.0), sh = mk<R>(0.0);
#pragma unroll
                for (int k = 0; k < D; ++k) { sg += g[u][k] * nh[k]; sh += h[u][k] * nh[k]; }
                Gbg[(long long)wf * Vp + v] = sg;
                if (H) Gbh[(long long)wf * Vp + v] = sh;
            }
        }
    }
}

// Area vector in FP32 for the signs of xi.S, scaled to a largest component in
// [1, 2) by its exponent (no underflow), and the bound below which a sign is
// taken again in FP64: FP32 rounding of the products and their sum stays below
// 5e-7 sum |xi_k S_k|.
template <int D>
struct Sign32 {
    float S[D], b[D];
    __device__ __forceinline__ void init(const double (&s)[D]) {
        int ex = 0;
#pragma unroll
        for (int k = 0; k < D; ++k) ex = max(ex, (__double2hiint(s[k]) >> 20) & 0x7ff);
        const double sc = ex > 0 && ex < 2046 ? __hiloint2double((2046 - ex) << 20, 0) : 1.0;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            S[k] = (float)(s[k] * sc);
            b[k] = fabsf(S[k]) * 1e-6f;
        }
    }
    // bits: 1 positive, 2 too near to tell
    __device__ __forceinline__ int operator()(const float* xi32, int Vp) const {
        float s32 = 0.f, b32 = 1e-30f;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const float x = xi32[k * Vp];
            s32 = fmaf(x, S[k], s32);
            b32 = fmaf(fabsf(x), b[k], b32);
        }
        return (s32 > 0.f ? 1 : 0) | (fabsf(s32) > b32 ? 0 : 2);
    }
};

// gbar+ of cell c at velocity v extrapolated by dk = d - xi dt/2.
template <int D, class R>
__device__ __forceinline__ R recon(const R* __restrict__ f, const R* __restrict__ G, int c, int v, int Vp,
                                   const double* dk) {
    R acc = f[(long long)c * Vp + v];
    const R* Gc = G + (long long)c * D * Vp + v;
#pragma unroll
    for (int k = D - 1; k >= 0; --k) acc = fma(Gc[(long long)k * Vp], dk[k], acc);
    return acc;
}

// P3: face values.  On internal faces the sign of xi.S selects the upwind
// cell; it is taken in FP32 where |xi.S| is above 1e-6 sum |xi_k S_k| (FP32
// rounding of the three products and their sum stays below 5e-7 of that) and
// in FP64, without FMA, for the warp iterations that hold a velocity nearer
// to the face, so that the choice and the ties are the FP64 ones.  The shifts
// d_k - xi_k dt/2 of both sides come from per-direction tables (TAB).  FP64
// operations per velocity: 14 -> 4 (2D, g and h), 20 -> 3 (3D, g); 24k
// triangles x 32^2: 3.27 -> 0.37 ms, 15^3 hexes x 14^3: 1.65 -> 0.36 ms (NU
// velocities' loads ahead of their stores: 0.52 -> 0.42 of it).
template <class R, int D, bool H, bool TAB>
__global__ void __launch_bounds__(256) k_recon(StepArgs a, Macros<R> mac, const R* __restrict__ gB, const R* __restrict__ hB,
                                               const R* __restrict__ gG, const R* __restrict__ hG,
                                               R* __restrict__ gS, R* __restrict__ hS) {
    constexpr int NU = H ? 2 : 4;  // velocities per lane in flight
    extern __shared__ __align__(16) unsigned char smemRaw[];
    double* tab = reinterpret_cast<double*>(smemRaw);  // per face: shift of the owner side [D][M], of the neighbour side [D][M]
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
#pragma unroll
        for (int k = 0; k < D; ++k) S[k] = a.Sf[3 * f + k];
        Sign32<D> sign;
        sign.init(S);
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
                const int sg = sign(a.xi32 + v, Vp);
                own |= (unsigned)(sg & 1) << i;
                near |= (unsigned)(sg >> 1) << i;
            }
            for (unsigned m = __reduce_or_sync(0xffffffffu, near); m; m &= m - 1) {
                const int i = __ffs(m) - 1, v = min(lane + 32 * (i0 + i), nV - 1);
                double xs = 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const double t = __dmul_rn(a.xi[k * Vp + v], S[k]);
                    xs = k == 0 ? t : __dadd_rn(xs, t);
                }
                const bool up = xs >= kVSmall, tie = !up && !(xs < -kVSmall);
                own = (own & ~(1u << i)) | ((up ? 1u : 0u) << i);
                ties |= (tie ? 1u : 0u) << i;
            }
            auto batch = [&](auto NB, int i) {  // iterations i .. i + nb - 1, all their loads ahead of their stores
                constexpr int nu = decltype(NB)::value;
                R g[nu], h[nu];
#pragma unroll
                for (int u = 0; u < nu; ++u, id.advance(M)) {
                    const int v = min(lane + 32 * (i0 + i + u), nV - 1);
                    const bool fromOwn = own >> (i + u) & 1u;
                    double dk[D];
                    if (TAB) {
                        const double* td = tb + (fromOwn ? 0 : DM);
                        dk[0] = td[id.ix];
                        // past the last velocity the lane works on it, with some of the table's values
                        if (D > 1) dk[D > 1 ? 1 : 0] = td[M + min(id.iy, M - 1)];
                        if (D > 2) dk[D > 2 ? 2 : 0] = td[2 * M + min(id.iz, M - 1)];
                    } else {
#pragma unroll
                        for (int k = 0; k < D; ++k) dk[k] = fma(a.xi[k * Vp + v], mh, fromOwn ? dO[k] : dN[k]);
                    }
                    const int c = fromOwn ? o : nb;
                    g[u] = recon<D>(gB, gG, c, v, Vp, dk);
                    if (H) h[u] = recon<D>(hB, hG, c, v, Vp, dk);
                }
#pragma unroll
                for (int u = 0; u < nu; ++u) {
                    const int v = lane + 32 * (i0 + i + u);
                    if (v < nV) {
                        gS[base + v] = g[u];
                        if (H) hS[base + v] = h[u];
                    }
                }
            };
            int i = 0;
            for (; i + NU <= n; i += NU) batch(std::integral_constant<int, NU>(), i);
            for (; i < n; ++i) batch(std::integral_constant<int, 1>(), i);
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
        const double xs = dot_rn(a.xi + v, Vp, sz);
        if (sym ? xs > -kVSmall : xs > 0) {  // outgoing (and tangential on symmetry patches)
            double dk[D];
#pragma unroll
            for (int k = 0; k < D; ++k) dk[k] = fma(x[k], mh, dO[k]);
            gS[base + v] = recon<D>(gB, gG, o, v, Vp, dk);
            if (H) hS[base + v] = recon<D>(hB, hG, o, v, Vp, dk);
        } else if (far) {
            // incoming: rho_b M(U of the owner cell, T_b) (discreteVelocity.C:570-600)
            const double Tb = a.TbM[wf];
            const double g = a.rhoB[wf] * maxwell_by_rho_ref(val(mac.U[3 * o]), val(mac.U[3 * o + 1]), val(mac.U[3 * o + 2]), Tb,
                                                             x[0], x[1], x[2], a.R, D);
            gS[base + v] = mk<R>(g);
            if (H) hS[base + v] = mk<R>(g * (a.R * Tb) * (a.K + 3 - D));
        }
    }
}

// One block per wall face: rho_w = sum_out w (xi.S) gbar / |inComingByRho|,
// then incoming DVs (xi.S <= 0) get rho_w * Maxwellian(U_w, T_w), a product of
// per-direction factors when they fit shared memory (tabBytes > 0).  Signs of
// xi.S as in k_recon.  FP64 operations per velocity (3D): 18 -> 6; 15^3 hexes x
// 14^3: 0.141 -> 0.053 ms.
template <class R, int D, bool H>
__global__ void k_wall(StepArgs a, Macros<R> mac, R* __restrict__ gS, R* __restrict__ hS, int useTab) {
    constexpr int N = sizeof(R) / sizeof(double);
    __shared__ double red[32 * N];
    static_assert(sizeof(red) + kTabMax <= kSmemMax, "k_wall: table and sums of a block");
    extern __shared__ __align__(16) unsigned char smemRaw[];
    R* tab = reinterpret_cast<R*>(smemRaw);
    const int wf = blockIdx.x;
    if (a.bKind[wf] != kBcMaxwell) return;  // uniform over the block
    const int f = a.nI + wf, nV = a.nV;
    const int Vp = a.Vp, M = a.M;
    const double sz[3] = {a.Sf[3 * f], a.Sf[3 * f + 1], a.Sf[3 * f + 2]};
    double S[D];
#pragma unroll
    for (int k = 0; k < D; ++k) S[k] = sz[k];
    Sign32<D> sign;
    sign.init(S);
    const R Tw = mac.Tw[wf];
    const double* Uw = a.Uw + 3 * wf;
    if (useTab) {
        const R i2 = 1.0 / (2.0 * a.R * Tw), s = sqrt(2.0 * kPi * a.R * Tw);
        for (int t = threadIdx.x; t < D * M; t += blockDim.x) {
            const int k = t / M;
            const double c = Uw[k] - a.x1[t - k * M];
            double c2 = c * c;
            R n = mk<R>(1.0);
            if (k == 0) {
                for (int q = D; q < 3; ++q) c2 += Uw[q] * Uw[q];
                n = 1.0 / (D == 2 ? s * s : (D == 3 ? s * s * s : s));
            }
            tab[t] = n * exp(-(c2 * i2));
        }
    }
    // signs of the thread's velocities v0 + blockDim.x i, i < n <= 32, one bit each
    auto outgoing = [&](int v0, int n) {
        unsigned out = 0u, near = 0u;
        for (int i = 0; i < n; ++i) {
            const int sg = sign(a.xi32 + v0 + i * blockDim.x, Vp);
            out |= (unsigned)(sg & 1) << i;
            near |= (unsigned)(sg >> 1) << i;
        }
        for (; near; near &= near - 1) {
            const int i = __ffs(near) - 1;
            out = (out & ~(1u << i)) | ((dot_rn(a.xi + v0 + i * blockDim.x, Vp, sz) > 0 ? 1u : 0u) << i);
        }
        return out;
    };
    R sum = mk<R>(0.0);
    unsigned out = 0u;
    for (int v0 = threadIdx.x; v0 < nV; v0 += 32 * blockDim.x) {
        const int n = min(32, (nV - v0 + (int)blockDim.x - 1) / (int)blockDim.x);
        out = outgoing(v0, n);
        for (unsigned m = out; m; m &= m - 1) {
            const int v = v0 + (__ffs(m) - 1) * blockDim.x;
            double wx = a.mw[Vp + v] * S[0];
#pragma unroll
            for (int k = 1; k < D; ++k) wx = fma(a.mw[(1 + k) * Vp + v], S[k], wx);
            sum = fma(wx, gS[(long long)f * Vp + v], sum);
        }
    }
    block_sum<N>(reinterpret_cast<double(&)[N]>(sum), red);  // its barriers also release the table
    const R rw = sum / mac.incAbs[wf];
    if (threadIdx.x == 0) mac.rhoW[wf] = rw;
    const R hk = (a.R * Tw) * (a.K + 3.0 - D);
    if (useTab) {
        for (int t = threadIdx.x; t < M; t += blockDim.x) tab[t] = rw * tab[t];
        __syncthreads();
    }
    const bool one = nV <= 32 * (int)blockDim.x;  // the bits of the first pass are those of all velocities
    for (int v0 = threadIdx.x; v0 < nV; v0 += 32 * blockDim.x) {
        const int n = min(32, (nV - v0 + (int)blockDim.x - 1) / (int)blockDim.x);
        if (!one) out = outgoing(v0, n);
        for (unsigned m = ~out & (n == 32 ? 0xffffffffu : (1u << n) - 1u); m; m &= m - 1) {
            const int v = v0 + (__ffs(m) - 1) * blockDim.x;
            R g;
            if (useTab) {
                const int r = v / M;
                g = tab[v - r * M];
                if (D == 2) g = g * tab[M + r];
                if (D == 3) g = g * (tab[M + r % M] * tab[2 * M + r / M]);
            } else {
                double c2 = 0.0;
                for (int k = 0; k < 3; ++k) {
                    const double c = Uw[k] - a.xi[k * Vp + v];
                    c2 += c * c;
                }
                const R s = sqrt(2.0 * kPi * a.R * Tw);
                g = rw * (1.0 / (D == 2 ? s * s : (D == 3 ? s * s * s : s)) * exp(-(c2 / (2.0 * a.R * Tw))));
            }
            gS[(long long)f * Vp + v] = g;
            if (H) hS[(long long)f * Vp + v] = g * hk;
        }
    }
}

// Wall heat flux about U_w and wall stress of wall face en from its values g, h.
template <bool H, class R>
__device__ __forceinline__ void wall_stress(const StepArgs& a, const Macros<R>& mac, int en, int lane,
                                            const R* __restrict__ gf, const R* __restrict__ hf, R fac, R tau) {
    const int nV = a.nV, Vp = a.Vp;
    const int wf = en - a.nI;
    const double* Uw = a.Uw + 3 * wf;
    R x12[9];  // q about U_w, then the upper triangle xx xy xz yy yz zz
#pragma unroll
    for (int i = 0; i < 9; ++i) x12[i] = mk<R>(0.0);
    for (int v = lane; v < nV; v += 32) {
        const double x[3] = {a.xi[v], a.xi[Vp + v], a.xi[2 * Vp + v]}, w = a.w[v];
        const R g = gf[v], h = H ? hf[v] : mk<R>(0.0);
        const double e[3] = {x[0] - Uw[0], x[1] - Uw[1], x[2] - Uw[2]};
        const R sw = 0.5 * w * ((e[0] * e[0] + e[1] * e[1] + e[2] * e[2]) * g + h), wg = w * g;
        const R wx = wg * x[0], wy = wg * x[1];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x12[k] = fma(sw, e[k], x12[k]);
            x12[3 + k] = fma(wx, x[k], x12[3 + k]);
            if (k > 0) x12[5 + k] = fma(wy, x[k], x12[5 + k]);
        }
        x12[8] = fma(wg * x[2], x[2], x12[8]);
    }
    constexpr int N9 = 9 * (int)(sizeof(R) / sizeof(double));
    warp_sum<N9>(reinterpret_cast<double(&)[N9]>(x12));
    if (lane == 0) {
        const R fs = 2.0 * tau / (2.0 * tau + 0.5 * a.dt);
        for (int k = 0; k < 3; ++k) mac.qWall[3 * wf + k] = fac * x12[k];
        const int at[9] = {3, 4, 5, 4, 6, 7, 5, 7, 8};
#pragma unroll
        for (int k = 0; k < 9; ++k) mac.stressWall[9 * wf + k] = fs * x12[at[k]];
    }
}

// Macros of the cells (P9) or of the active faces (P6, with qWall and
// stressWall on walls), two velocity passes as the reference: density,
// momentum and energy with the weights w, w xi, w |xi|^2/2 tabulated once
// (a.mw), then the heat flux about the velocity found, with the entity's
// c and c^2 tabulated per direction (TAB).  The square root, divisions,
// logarithm and exponential of the macros run once per block, one lane per
// entity.  24k triangles x 32^2: faces 4.74 -> 0.88 ms, cells 3.07 -> 0.46 ms;
// k_mom_cols takes the grids whose columns fill the lanes.
template <class R, int D, bool H, bool TAB, bool FACE>
__global__ void k_mom(StepArgs a, Macros<R> mac, const R* __restrict__ gS, const R* __restrict__ hS) {
    constexpr int NS = D == 3 ? 8 : 4, NQ = 4;  // reduced slots: rho, momentum, energy; heat flux
    __shared__ R sm[kMaxEnt][8];                // slot totals
    __shared__ R sr[kMaxEnt][8];                // rho, U, T, tau, heat-flux factor
    static_assert(sizeof(sm) + sizeof(sr) + kTabMax <= kSmemMax, "k_mom: tables and scalars of a block");
    extern __shared__ __align__(16) unsigned char smemRaw[];
    R* tab = reinterpret_cast<R*>(smemRaw);  // per entity: c [D][M] | c^2 [D][M]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nEnt = blockDim.x >> 5;
    const int n = FACE ? a.nA : a.nC, e0 = blockIdx.x * nEnt, en = e0 + warp, M = a.M, Vp = a.Vp, nV = a.nV;
    const bool active = en < n;
    const long long base = (long long)en * Vp;
    if (active) {
        R m[NS], eh = mk<R>(0.0);
#pragma unroll
        for (int i = 0; i < NS; ++i) m[i] = mk<R>(0.0);
#pragma unroll 2
        for (int v = lane; v < nV; v += 32) {
            const R g = gS[base + v];
#pragma unroll
            for (int i = 0; i <= D; ++i) m[i] = fma(a.mw[i * Vp + v], g, m[i]);
            m[D + 1] = fma(a.mw[(D + 1) * Vp + v], g, m[D + 1]);
            if (H) eh = fma(a.mw[v], hS[base + v], eh);
        }
        if (H) m[D + 1] = fma(0.5, eh, m[D + 1]);
        const R r = scatter_sum<NS>(m, lane);
        if ((lane & (32 / NS - 1)) == 0) sm[warp][warp_slot<NS>(lane)] = r;
    }
    __syncthreads();
    if (threadIdx.x < nEnt && e0 + threadIdx.x < n) {
        const int i = e0 + threadIdx.x;
        const R* m = sm[threadIdx.x];
        R* s = sr[threadIdx.x];
        const R rho = m[0], ir = 1.0 / rho;
        R U[3] = {mk<R>(0.0), mk<R>(0.0), mk<R>(0.0)}, uu = mk<R>(0.0);
#pragma unroll
        for (int k = 0; k < D; ++k) { U[k] = m[1 + k] * ir; uu = uu + U[k] * U[k]; }
        const R T = (m[D + 1] - 0.5 * rho * uu) * ir / ((a.K + 3) / 2.0 * a.R);
        const R tau = mac.muRef * exp(a.omega * log(T / a.Tref)) / (rho * T * a.R);
        const R fac = 2.0 * tau / (2.0 * tau + (FACE ? 0.5 : 1.0) * a.dt * a.Pr);
        (FACE ? mac.rhoF : mac.rho)[i] = rho;
        (FACE ? mac.TF : mac.T)[i] = T;
        (FACE ? mac.tauF : mac.tau)[i] = tau;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            (FACE ? mac.UF : mac.U)[3 * i + k] = U[k];
            if (k >= D) (FACE ? mac.qF : mac.q)[3 * i + k] = mk<R>(0.0);
        }
        s[0] = U[0]; s[1] = U[1]; s[2] = U[2];
        s[3] = fac;
        s[4] = tau;
        if (!FACE && (!(val(rho) > 0.0) || !(val(T) > 0.0) || !isfinite(val(uu)))) atomicExch(a.status, 5);
    }
    __syncthreads();
    if (!active) return;
    const R* s = sr[warp];
    const R fac = s[3];
    R U[D], qq[NQ];
#pragma unroll
    for (int k = 0; k < D; ++k) U[k] = s[k];
#pragma unroll
    for (int i = 0; i < NQ; ++i) qq[i] = mk<R>(0.0);
    const int DM = D * M;
    R* tb = tab + (size_t)warp * 2 * DM;
    if (TAB) {
        for (int t = lane; t < DM; t += 32) {
            const int k = t / M;
            const R c = a.x1[t - k * M] - s[k];
            tb[t] = c;
            tb[DM + t] = c * c;
        }
        __syncwarp();
    }
    DvIdx<D> id;
    id.init(lane, 32, M);
    for (int v = lane; v < nV; v += 32, id.advance(M)) {
        const R g = gS[base + v], h = H ? hS[base + v] : mk<R>(0.0);
        R c[D], cc;
        if (TAB) {
            c[0] = tb[id.ix];
            cc = tb[DM + id.ix];
            if (D > 1) { c[D > 1 ? 1 : 0] = tb[M + id.iy]; cc = cc + tb[DM + M + id.iy]; }
            if (D > 2) { c[D > 2 ? 2 : 0] = tb[2 * M + id.iz]; cc = cc + tb[DM + 2 * M + id.iz]; }
        } else {
            cc = mk<R>(0.0);
#pragma unroll
            for (int k = 0; k < D; ++k) { c[k] = a.xi[k * Vp + v] - U[k]; cc = fma(c[k], c[k], cc); }
        }
        const R ws = a.w[v] * (H ? fma(cc, g, h) : cc * g);
#pragma unroll
        for (int k = 0; k < D; ++k) qq[k] = fma(ws, c[k], qq[k]);
    }
    const R r = 0.5 * scatter_sum<NQ>(qq, lane);
    const int slot = warp_slot<NQ>(lane);
    if ((lane & 7) == 0 && slot < D) {
        (FACE ? mac.qF : mac.q)[3 * en + slot] = fac * r;
        if (!FACE && !isfinite(val(r))) atomicExch(a.status, 5);
    }
    if (!FACE || en < a.nI || a.bKind[en - a.nI] != kBcMaxwell) return;
    wall_stress<H>(a, mac, en, lane, gS + base, H ? hS + base : nullptr, s[3], s[4]);
}

// k_mom where a lane owns columns of velocities along the last direction (2D:
// one row index each; 3D: one (x, y) pair each): with c = xi - U0, the sums
// over a column of w g {1, c, c^2, c^3} and w h {1, c} (the entity's factors of
// the last direction, read by all lanes alike) hold all that density, momentum,
// energy and heat flux take from it: 6 operations per velocity with h and 4
// without, in one pass over the values, where the two passes of k_mom take 10
// and 12.  The lane's columns are then weighted by the other directions' c and
// the moments moved from U0 to the velocity found:
//   q_i(U) = q_i - d_i E - sum_j d_j P_ij + rho d^2 d_i,  d = U - U0,
// U0 being the (owner) cell's velocity of the last step, so that d is small and
// nothing cancels; on walls the same sums give the stress and, moved to U_w, the
// wall heat flux.  24k triangles x 32^2: faces 0.88 -> 0.54 ms, cells 0.46 ->
// 0.32 ms (FP64 pipe 85 and 95 % busy); 61^2 quads x 28^2: cells 87 -> 64 us;
// 15^3 hexes x 14^3: faces 1.14 -> 0.39 ms.
constexpr int kColSlots = 16;
// Tables of a block of k_mom_cols: its slot totals in Dual leave less than kTabMax.
template <class R, int D>
__host__ __device__ constexpr size_t cols_tab_max() {
    constexpr size_t left = kSmemMax - kMaxEnt * (kColSlots * sizeof(R) + D * sizeof(double));
    return left < kTabMax ? left : kTabMax;
}
// Registers: the largest instance (Dual, 3D with h) takes 128, all that a block
// of kMaxEnt warps may have.  With the block size stated (__launch_bounds__)
// 3D FP64 instances are compiled to fewer registers and a step on hexes takes
// 1 % longer; with __maxnreg__(128) most instances take more.
template <class R, int D, bool H, bool FACE>
__global__ void k_mom_cols(StepArgs a, Macros<R> mac, const R* __restrict__ gS, const R* __restrict__ hS) {
    // slots: rho | rho d [D] | sum h | 2 q [D] | P xx, xy, (xz,) yy, ..
    constexpr int NS = kColSlots, SH = 1 + D, SQ = SH + 1, SP = SQ + D;
    __shared__ R sm[kMaxEnt][NS];
    __shared__ double su[kMaxEnt][D];
    static_assert(sizeof(sm) + sizeof(su) + cols_tab_max<R, D>() <= kSmemMax, "k_mom_cols: tables and totals of a block");
    extern __shared__ __align__(16) unsigned char smemRaw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nEnt = blockDim.x >> 5;
    const int n = FACE ? a.nA : a.nC, e0 = blockIdx.x * nEnt, en = e0 + warp, M = a.M, Vp = a.Vp;
    double2* tb = reinterpret_cast<double2*>(smemRaw) + (size_t)warp * 2 * M;  // {w, w c}, {w c^2, w c^3}
    const bool active = en < n;
    const long long base = (long long)en * Vp;
    if (active) {
        const int uc = FACE ? chk(a.own[en], a.nC, a.status) : en;
        double U0[D];
#pragma unroll
        for (int k = 0; k < D; ++k) {  // inside the velocity grid, whatever the state holds
            const double lo = fmin(a.x1[0], a.x1[M - 1]), hi = fmax(a.x1[0], a.x1[M - 1]);
            U0[k] = fmin(fmax(val(mac.U[3 * uc + k]), lo), hi);
            if (lane == 0) su[warp][k] = U0[k];
        }
        for (int l = lane; l < M; l += 32) {
            const double c = a.x1[l] - U0[D - 1], w = a.w1[l], wc = w * c, wcc = wc * c;
            tb[2 * l] = {w, wc};
            tb[2 * l + 1] = {wcc, wcc * c};
        }
        __syncwarp();
        R S[NS];
#pragma unroll
        for (int i = 0; i < NS; ++i) S[i] = mk<R>(0.0);
        const int NP = D == 2 ? M : M * M;
        for (int col = lane; col < NP; col += 32) {
            R m0 = mk<R>(0.0), m1 = m0, m2 = m0, m3 = m0, h0 = m0, h1 = m0;
            const R* g = gS + base + col;
            const R* h = H ? hS + base + col : nullptr;
#pragma unroll 4
            for (int l = 0; l < M; ++l) {
                const double2 t = tb[2 * l], u = tb[2 * l + 1];
                const R gv = g[(long long)l * NP];
                m0 = fma(t.x, gv, m0);
                m1 = fma(t.y, gv, m1);
                m2 = fma(u.x, gv, m2);
                m3 = fma(u.y, gv, m3);
                if (H) {
                    const R hv = h[(long long)l * NP];
                    h0 = fma(t.x, hv, h0);
                    h1 = fma(t.y, hv, h1);
                }
            }
            const int ix = D == 2 ? col : col % M, iy = D == 2 ? 0 : col / M;
            const double cx = a.x1[ix] - U0[0], cy = D == 2 ? 0.0 : a.x1[iy] - U0[D > 2 ? 1 : 0];
            const double w = D == 2 ? a.w1[ix] : a.w1[ix] * a.w1[iy], wx = w * cx, wxx = wx * cx;
            S[0] = fma(w, m0, S[0]);
            S[1] = fma(wx, m0, S[1]);
            S[D] = fma(w, m1, S[D]);
            if (H) S[SH] = fma(w, h0, S[SH]);
            if constexpr (D == 2) {
                const R e = H ? m2 + h0 : m2, f = H ? m3 + h1 : m3;
                S[SQ] = fma(wx, fma(cx * cx, m0, e), S[SQ]);
                S[SQ + 1] = fma(w, fma(cx * cx, m1, f), S[SQ + 1]);
                S[SP] = fma(wxx, m0, S[SP]);
                S[SP + 1] = fma(wx, m1, S[SP + 1]);
                S[SP + 2] = fma(w, m2, S[SP + 2]);
            } else {
                const double wy = w * cy, c2 = fma(cx, cx, cy * cy);
                const R e = H ? m2 + h0 : m2, f = H ? m3 + h1 : m3, ec = fma(c2, m0, e);
                S[2] = fma(wy, m0, S[2]);
                S[SQ] = fma(wx, ec, S[SQ]);
                S[SQ + 1] = fma(wy, ec, S[SQ + 1]);
                S[SQ + D - 1] = fma(w, fma(c2, m1, f), S[SQ + D - 1]);
                S[SP] = fma(wxx, m0, S[SP]);
                S[SP + 1] = fma(wx * cy, m0, S[SP + 1]);
                S[SP + 2] = fma(wx, m1, S[SP + 2]);
                S[SP + 3] = fma(wy * cy, m0, S[SP + 3]);
                S[SP + 4] = fma(wy, m1, S[SP + 4]);
                S[SP + 5] = fma(w, m2, S[SP + 5]);
            }
        }
        const R r = scatter_sum<NS>(S, lane);
        if ((lane & 1) == 0) sm[warp][warp_slot<NS>(lane)] = r;
    }
    __syncthreads();
    if (threadIdx.x < nEnt && e0 + threadIdx.x < n) {
        const int i = e0 + threadIdx.x;
        const R* m = sm[threadIdx.x];
        const double* U0 = su[threadIdx.x];
        const R rho = m[0], ir = 1.0 / rho;
        auto P = [&](int k, int j) -> R {  // sum w g c_k c_j
            const int lo = j < k ? j : k, hi = j < k ? k : j;
            return m[SP + (lo == 0 ? hi : D + (lo - 1) * (D - 1) + hi - lo)];
        };
        R d[D], dd = mk<R>(0.0), uu = mk<R>(0.0), E = H ? m[SH] : mk<R>(0.0);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            d[k] = m[1 + k] * ir;
            dd = fma(d[k], d[k], dd);
            const R U = U0[k] + d[k];
            uu = fma(U, U, uu);
            (FACE ? mac.UF : mac.U)[3 * i + k] = U;
            E = E + P(k, k);
        }
        E = 0.5 * E;
        const R rd = rho * dd;
        const R T = (E - 0.5 * rd) * ir / ((a.K + 3) / 2.0 * a.R);
        const R tau = mac.muRef * exp(a.omega * log(T / a.Tref)) / (rho * T * a.R);
        const R fac = 2.0 * tau / (2.0 * tau + (FACE ? 0.5 : 1.0) * a.dt * a.Pr);
        (FACE ? mac.rhoF : mac.rho)[i] = rho;
        (FACE ? mac.TF : mac.T)[i] = T;
        (FACE ? mac.tauF : mac.tau)[i] = tau;
        bool bad = !(val(rho) > 0.0) || !(val(T) > 0.0) || !isfinite(val(uu));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            R q = mk<R>(0.0);
            if (k < D) {
                q = fma(0.5, m[SQ + k], d[k] * (rd - E));
#pragma unroll
                for (int j = 0; j < D; ++j) q = q - d[j] * P(k, j);
                q = fac * q;
                bad = bad || !isfinite(val(q));
            } else {
                (FACE ? mac.UF : mac.U)[3 * i + k] = mk<R>(0.0);
            }
            (FACE ? mac.qF : mac.q)[3 * i + k] = q;
        }
        if (!FACE && bad) atomicExch(a.status, 5);
        if (FACE && i >= a.nI && a.bKind[i - a.nI] == kBcMaxwell) {
            // heat flux about U_w (velocities outside the solution directions are 0)
            // and stress, of the same sums
            const int wf = i - a.nI;
            const double* Uw = a.Uw + 3 * wf;
            double b[3], bb = 0.0;
            R bm = mk<R>(0.0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                b[k] = k < D ? Uw[k] - U0[k < D ? k : 0] : Uw[k];
                bb = fma(b[k], b[k], bb);
                if (k < D) bm = fma(b[k], m[1 + (k < D ? k : 0)], bm);
            }
            // 1/2 sum w (|c - b|^2 g + h)
            const R Eb = E - bm + (0.5 * bb) * rho, fs = 2.0 * tau / (2.0 * tau + 0.5 * a.dt);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                R q = -b[k] * Eb;
                if (k < D) {
                    q = q + fma(0.5, m[SQ + k], (0.5 * bb) * m[1 + k]);
#pragma unroll
                    for (int j = 0; j < D; ++j) q = q - b[j] * P(k, j);
                }
                mac.qWall[3 * wf + k] = fac * q;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    R t = mk<R>(0.0);
                    if (k < D && j < D) t = P(k, j) + U0[k] * m[1 + j] + U0[j] * (m[1 + k] + U0[k] * rho);
                    mac.stressWall[9 * wf + 3 * k + j] = fs * t;
                }
            }
        }
    }
}

// P8: g~ <- -g~/3 + 4/3 gbar+ - dt/V sum_f (xi.S_f) g_f, one warp per cell;
// -+S dt/V is formed once per cell (it was a division per face, field and
// velocity).  With h (2D) xi.S is shared by the two fields; without,
// sum_f S_f g_f is formed per component first: D operations per face and D per
// velocity instead of D + 1 per face.  The staged faces are taken axis by axis,
// those with one non-zero component of S first: one operation for xi.S (none
// but the sum's without h) in place of D.  The faces beyond the staged ones have
// a loop of their own: as a condition in one loop it was predicated, and its
// products issued for every face.  24k triangles x 32^2: 3.94 -> 0.74 ms (FP64
// pipe 88 % busy), 15^3 hexes x 14^3: 1.73 -> 0.23 ms (0.67 as one loop without
// the axes), 61^2 quads x 28^2: 0.18 -> 0.12 ms.
template <class R, int D, bool H>
__global__ void __launch_bounds__(32 * kSmallBlock) k_cell(StepArgs a, R* gT, R* hT, const R* __restrict__ gB,
                                                           const R* __restrict__ hB, const R* __restrict__ gS,
                                                           const R* __restrict__ hS) {
    constexpr int VU = 2;
    struct Face {
        double L[D];
        int row;
    };
    __shared__ Face stage[kSmallBlock][kStage];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Vp = a.Vp, nV = a.nV;
    const int c = blockIdx.x * (blockDim.x >> 5) + warp;
    if (c >= a.nC) return;
    const int j0 = a.cellOff[c], nf = a.cellOff[c + 1] - j0, ns = min(nf, kStage);
    const long long base = (long long)c * Vp;
    const double kv = a.dt / a.vol[c];
    auto entry = [&](int j) {
        Face r;
        const int e = a.cellFace[j];
        const double sk = e & 1 ? kv : -kv;
        r.row = chk(e >> 1, a.nA, a.status);
#pragma unroll
        for (int k = 0; k < D; ++k) r.L[k] = sk * a.Sf[3 * r.row + k];
        return r;
    };
    int end[D];  // staged faces along direction k: [end[k - 1], end[k]), the others from end[D - 1] on
    {
        Face r;
        int kind = D + 1;  // 0 .. D - 1: along that direction; D: any other
        if (lane < ns) {
            r = entry(j0 + lane);
            int n = 0;
            kind = D;
#pragma unroll
            for (int k = 0; k < D; ++k)
                if (r.L[k] != 0.0) { ++n; kind = k; }
            if (n != 1) kind = D;
        }
        int at = 0;
#pragma unroll
        for (int k = 0; k <= D; ++k) {
            const unsigned b = __ballot_sync(0xffffffffu, kind == k);
            if (kind == k) at += __popc(b & ((1u << lane) - 1u));
            else if (kind > k) at += __popc(b);
            if (k < D) end[k < D ? k : 0] = (k > 0 ? end[k > 0 ? k - 1 : 0] : 0) + __popc(b);
        }
        if (lane < ns) stage[warp][at] = r;
    }
    __syncwarp();
    for (int v0 = lane; v0 < nV; v0 += 32 * VU) {
        int vv[VU];
        double x[VU][D];
        R g[VU], h[VU], sg[VU][D];
#pragma unroll
        for (int u = 0; u < VU; ++u) {
            vv[u] = min(v0 + 32 * u, nV - 1);
#pragma unroll
            for (int k = 0; k < D; ++k) {
                x[u][k] = a.xi[k * Vp + vv[u]];
                sg[u][k] = mk<R>(0.0);
            }
            const long long i = base + vv[u];
            g[u] = fma(4.0 / 3, gB[i], -1.0 / 3 * gT[i]);
            h[u] = H ? fma(4.0 / 3, hB[i], -1.0 / 3 * hT[i]) : mk<R>(0.0);
        }
        // face r, whose components k0 .. k1 - 1 count
        auto add = [&](const Face& r, int k0, int k1) {
            const long long fb = (long long)r.row * Vp;
#pragma unroll
            for (int u = 0; u < VU; ++u) {
                const R gf = gS[fb + vv[u]];
                double xs = 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    if (k < k0 || k >= k1) continue;
                    if (H) xs = k == k0 ? x[u][k] * r.L[k] : fma(x[u][k], r.L[k], xs);
                    else sg[u][k] = fma(r.L[k], gf, sg[u][k]);
                }
                if (H) {
                    g[u] = fma(xs, gf, g[u]);
                    h[u] = fma(xs, hS[fb + vv[u]], h[u]);
                }
            }
        };
        int j = 0;
#pragma unroll
        for (int k = 0; k < D; ++k)
            for (; j < end[k]; ++j) add(stage[warp][j], k, k + 1);
        for (; j < ns; ++j) add(stage[warp][j], 0, D);
        for (; j < nf; ++j) add(entry(j0 + j), 0, D);
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

// Warps per block of the passes whose block shares its entity scalars: up to
// 16 (their FP64 chain runs once per block, ~200 instructions, against ~300 to
// 600 of an entity's velocities), down to 4 while the entities would not make
// eight blocks per SM (few blocks leave SMs idle at the end), fewer when the tables (tabEnt bytes per entity) exceed
// what the kernel has for them without asking for more (tabMax).
inline int ents_per_block(int n, size_t tabEnt, int sms, int e = kMaxEnt, size_t tabMax = kTabMax) {
    while (e > 1 && (((long long)n < 8LL * sms * e && e > 4) || tabEnt * e > tabMax)) e >>= 1;
    return e;
}

// Share (%) of the lanes at work when they stride over the columns along the last direction.
template <int D>
int column_lanes(int M) {
    const int n = D == 2 ? M : M * M;
    return 100 * n / ((n + 31) / 32 * 32);
}

template <class R, int D, bool H>
struct Pass {
    template <EqMode MODE>
    static void eq(const StepArgs& a, const Macros<R>& m, const R* gi, const R* hi, R* go, R* ho, int sms,
                   cudaStream_t s) {
        const int n = MODE == kFaces ? a.nA : a.nC;
        const size_t tb = 3 * sizeof(R) * D * a.M;
        const bool tab = tb <= kTabMax;
        const int e = ents_per_block(n, tab ? tb : 0, sms), blocks = (n + e - 1) / e;
        if constexpr (D > 1) {
            // columns where the lanes they leave idle cost less than the operations they save
            constexpr int kFlat = 3 * D + (H ? 3 : 0), kCols = H ? 8 : 5;
            if (tab && kFlat * column_lanes<D>(a.M) > kCols * 100) {
                k_eq<R, D, H, kTabCols, MODE><<<blocks, 32 * e, tb * e, s>>>(a, m, gi, hi, go, ho);
                return;
            }
        }
        if (tab) k_eq<R, D, H, kTabFlat, MODE><<<blocks, 32 * e, tb * e, s>>>(a, m, gi, hi, go, ho);
        else k_eq<R, D, H, kTabNone, MODE><<<blocks, 32 * e, 0, s>>>(a, m, gi, hi, go, ho);
    }
    template <bool FACE>
    static void mom(const StepArgs& a, const Macros<R>& m, const R* g, const R* h, int sms, cudaStream_t s) {
        const int n = FACE ? a.nA : a.nC;
        if constexpr (D > 1) {
            // columns from three quarters of the lanes on: per velocity 6 operations with h (4 without) and
            // about one for the sums over the columns, against 10 (2D) and 12 (3D)
            constexpr size_t tabMax = cols_tab_max<R, D>();
            const size_t tc = 4 * sizeof(double) * a.M;
            if (column_lanes<D>(a.M) >= 75 && tc <= tabMax) {
                const int e = ents_per_block(n, tc, sms, kMaxEnt, tabMax), blocks = (n + e - 1) / e;
                k_mom_cols<R, D, H, FACE><<<blocks, 32 * e, tc * e, s>>>(a, m, g, h);
                return;
            }
        }
        const size_t tb = 2 * sizeof(R) * D * a.M;
        const bool tab = tb <= kTabMax;
        const int e = ents_per_block(n, tab ? tb : 0, sms), blocks = (n + e - 1) / e;
        if (tab) k_mom<R, D, H, true, FACE><<<blocks, 32 * e, tb * e, s>>>(a, m, g, h);
        else k_mom<R, D, H, false, FACE><<<blocks, 32 * e, 0, s>>>(a, m, g, h);
    }
    static void run(int pass, const StepArgs& a, const Macros<R>& m, const Fields<R>& b, int sms, cudaStream_t s) {
        const int wC = (a.nC + kSmallBlock - 1) / kSmallBlock, wA = (a.nA + 7) / 8;
        switch (pass) {
            case 0: eq<kCells>(a, m, b.gT, b.hT, b.gB, b.hB, sms, s); break;
            case 1: k_grad<R, D, H><<<wC, 32 * kSmallBlock, 0, s>>>(a, b.gB, b.hB, b.gG, b.hG, b.Gbg, b.Gbh); break;
            case 2: {
                const size_t tb = 2 * sizeof(double) * D * a.M;
                const int w = ents_per_block(a.nA, tb, sms, 4), blocks = (a.nA + w - 1) / w;
                if (tb <= kTabMax) k_recon<R, D, H, true><<<blocks, 32 * w, tb * w, s>>>(a, m, b.gB, b.hB, b.gG, b.hG, b.gS, b.hS);
                else k_recon<R, D, H, false><<<wA, 256, 0, s>>>(a, m, b.gB, b.hB, b.gG, b.hG, b.gS, b.hS);
                break;
            }
            case 3:
                if (a.nW > 0 && (a.bcMask & (1 << kBcMaxwell))) {
                    const size_t tb = sizeof(R) * D * a.M;
                    const int tab = tb <= kTabMax;
                    k_wall<R, D, H><<<a.nW, kWallThreads, tab ? tb : 0, s>>>(a, m, b.gS, b.hS, tab);
                }
                break;
            case 4: mom<true>(a, m, b.gS, b.hS, sms, s); break;
            case 5: eq<kFaces>(a, m, b.gS, b.hS, b.gS, b.hS, sms, s); break;
            case 6: k_cell<R, D, H><<<wC, 32 * kSmallBlock, 0, s>>>(a, b.gT, b.hT, b.gB, b.hB, b.gS, b.hS); break;
            case 7: mom<false>(a, m, b.gT, b.hT, sms, s); break;
            default: break;
        }
    }
};

// f(Pass<R, D, H>()) for the case's directions and fields.
template <class R, class F>
void with_pass(const StepArgs& a, F&& f) {
    switch (2 * a.D + (a.hasH ? 1 : 0)) {
        case 2: f(Pass<R, 1, false>()); break;
        case 3: f(Pass<R, 1, true>()); break;
        case 4: f(Pass<R, 2, false>()); break;
        case 5: f(Pass<R, 2, true>()); break;
        case 6: f(Pass<R, 3, false>()); break;
        case 7: f(Pass<R, 3, true>()); break;
        default: break;
    }
}

}  // namespace
}  // namespace dugks
