// Reference pipeline: one FP64 kernel per pass of fvDVM::evolution()
// (src/fvDVM/fvDVM/fvDVM.C:1086-1108), with every intermediate materialised
// in HBM (DV index innermost): the FP64 path, and the step that is
// differentiated.  The FP32 step (fused32.cuh) is the fast path.
//
// The passes are in ref_kernels.cuh; here are what only this pipeline has:
//   k_sym_*     P5b updateGHbarSurfSymmetryIn  fvDVM.C:375-454, discreteVelocity.C:733-817
//   k_pressure  P10 updatePressureInOutBC      fvDVM.C:730-806
#include "device_common.cuh"
#include "kernels.h"
#include "ref_kernels.cuh"

namespace dugks {
namespace {

constexpr int kRedThreads = 128;

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

__global__ void k_init_tau(StepArgs a) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < a.nC) a.tau[c] = tau_ref(a.T[c], a.rho[c], a.muRef, a.omega, a.Tref, a.R);
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

}  // namespace

void launch_pressure_bc(const StepArgs& a, cudaStream_t s) {
    if (a.nW > 0) k_pressure<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
}

void launch_zero_gradient_tu(const StepArgs& a, cudaStream_t s) {
    if (a.nW > 0 && a.zgMask) k_zero_gradient_tu<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
}

void launch_ref_init(const StepArgs& a, double* g, double* h, int sms, cudaStream_t s) {
    k_init_tau<<<(a.nC + 127) / 128, 128, 0, s>>>(a);
    const Macros<double> m = macros_of(a);
    with_pass<double>(a, [&](auto P) { P.template eq<kInit>(a, m, nullptr, nullptr, g, h, sms, s); });
}

void launch_ref_mixed_init(const StepArgs& a, const RefBuffers& b, cudaStream_t s) {
    if (a.nW > 0 && (a.bcMask & (1 << kBcFixedValue))) k_mixed_init<<<a.nW, kRedThreads, 0, s>>>(a, b.gS, b.hS);
}

const char* const kRefKernelNames[kRefKernels] = {"k_barp", "k_grad", "k_recon", "k_wall",
                                                  "k_face_mom", "k_relax", "k_cell", "k_cell_mom"};

void launch_ref_pass(int pass, const StepArgs& a, const RefBuffers& b, int sms, cudaStream_t s) {
    const Macros<double> m = macros_of(a);
    const Fields<double> f{b.gT, b.hT, b.gB, b.hB, b.gG, b.hG, b.Gbg, b.Gbh, b.gS, b.hS};
    with_pass<double>(a, [&](auto P) { P.run(pass, a, m, f, sms, s); });
    if (pass == 3 && (a.bcMask & ((1 << kBcSymmetryMod) | (1 << kBcSymmetryPlane)))) {
        k_sym_snap<<<a.nW, kRedThreads, 0, s>>>(a, b.gS, b.hS, b.gSym, b.hSym);
        k_sym_in<<<a.nW, kRedThreads, 0, s>>>(a, b.gS, b.hS, b.gSym, b.hSym);
    }
    if (pass == 7) {
        if (a.zgMask) k_zero_gradient_tu<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
        if (a.bcMask & ((1 << kBcPressureIn) | (1 << kBcPressureOut)))
            k_pressure<<<(a.nW + 127) / 128, 128, 0, s>>>(a);
    }
}

}  // namespace dugks
