// FusedPipelineT<S>: owns the tile plan and the double-buffered state of the
// fused step; included once per storage type (fused_fp32.cu, fused_fp64.cu).
// FP64: two tiled sweeps (fused_kernels.cuh).  FP32: face sides on one-ring
// tiles, face macros, cell gather (fused32.cuh).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../host/solver.h"
#include "../host/tile_plan.h"
#include "fused32_kernels.h"
#include "fused_kernels.cuh"
#include "kernels.h"

namespace dugks {

template <typename S>
class FusedPipelineT final : public FusedPipeline {
public:
    using KernelFn = void (*)(FusedArgs<S>);

    ~FusedPipelineT() override {
        for (void* p : allocs_) cudaFree(p);
    }

    bool init(Solver& solver, const StepArgs& a, std::string& err) {
        const Mesh& m = solver.mesh();
        if (a.D != 2 && a.D != 3) { err = "the fused pipelines need a 2D or 3D mesh (1D runs on the plain FP64 pipeline)"; return false; }
        D_ = a.D;
        bcMask_ = a.bcMask;
        H_ = a.hasH != 0;
        if (D_ != 2 && D_ != 3) { err = "fused pipeline supports 2D and 3D meshes"; return false; }
        npl_ = fused_npl(sizeof(S) == 4 ? DUGKS_FP32_FP64MOM : DUGKS_FP64);
        fp32_ = sizeof(S) == 4;
        const int KC = 32 * npl_;
        if (a.Vp % KC != 0) { err = "padded DV count is not a multiple of the DV chunk"; return false; }
        // ---- tile plan, sized to the shared-memory budget
        int dev = 0;
        cudaGetDevice(&dev);
        int maxSmem = 0;
        cudaDeviceGetAttribute(&maxSmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        row_ = a.M % npl_ == 0;
        pick();
        const size_t budget = (size_t)maxSmem - 2048;
        const char* envT = std::getenv("DUGKS_TILE_CELLS");
        const int maxCells = fused_tile_cap() > 0 ? fused_tile_cap() : (envT ? std::max(1, std::atoi(envT)) : 4096);
        // FP32: sweep A alone is tiled (one-ring halo); FP64: both sweeps (two-ring halo)
        const SmemFn fn = [this](const TileDims& d) { return fp32_ ? smemFace(d) : std::max(smemFace(d), smemCell(d)); };
        // one tile per SM at a time: balance the waves of the FP32 face sweep,
        // unless a cap was asked for or the case's tiles share the batched
        // kernels' grid with other cases' tiles
        int nsmPlan = 0;
        cudaDeviceGetAttribute(&nsmPlan, cudaDevAttrMultiProcessorCount, dev);
        const int waveSlots = fp32_ && fused_wave_balance() && !envT ? nsmPlan : 0;
        if (!build_tile_plan(m, maxCells, fn, budget, plan_, err, fp32_ ? 1 : 2, waveSlots)) return false;
        smemA_ = smemB_ = 0;
        for (const TileHdr& h : plan_.hdr) {
            TileDims d;
            d.nT = h.nT; d.nT1 = h.nT1; d.nT2 = h.nT2; d.nFA = h.nFA; d.nFB = h.nFB; d.nEnt = h.nEnt;
            smemA_ = std::max(smemA_, smemFace(d));
            if (!fp32_) smemB_ = std::max(smemB_, smemCell(d));
        }
        // The limit is a property of the kernel function, shared by every
        // pipeline (case) that launches it: allow the device maximum, each
        // launch then asks for its own size.
        allow_max_dynamic_smem(kFace_);
        if (!fp32_) allow_max_dynamic_smem(kCell_);

        // ---- upload plan
        args_.hdr = upload(plan_.hdr);
        if (!fp32_) {  // the FP32 kernels read per-tile metadata blocks instead
            args_.cells = upload(plan_.cells);
            args_.faces = upload(plan_.faces);
            args_.colorOff = upload(plan_.colorOff);
            args_.colorPerm = upload(plan_.colorPerm);
        }
        const size_t nRec = plan_.faces.size();
        if (sizeof(S) == 4) {
            // per-tile blocks: the cell-face entries of T (LS vector and other
            // row, S out of the cell and face side, Cf - C), cells, offsets
            std::vector<int4> meta;
            std::vector<int> metaOff;
            auto ints = [&](const int32_t* v, int n) {
                for (int i = 0; i < n; i += 4)
                    meta.push_back(make_int4(v[i], i + 1 < n ? v[i + 1] : 0, i + 2 < n ? v[i + 2] : 0,
                                             i + 3 < n ? v[i + 3] : 0));
            };
            auto rec = [&](double x, double y, double z, int code) {
                const float f[3] = {(float)x, (float)y, (float)z};
                int4 r;
                std::memcpy(&r, f, 12);
                r.w = code;
                meta.push_back(r);
            };
            for (const TileHdr& h : plan_.hdr) {
                metaOff.push_back((int)meta.size());
                const int base = plan_.stOff[h.stStart];
                for (int i = 0; i < h.nT; ++i) {
                    const int c = plan_.cells[h.cellStart + i];
                    for (int e = plan_.stOff[h.stStart + i], j = m.cellOff[c]; e < plan_.stOff[h.stStart + i + 1]; ++e, ++j) {
                        const int af = m.cellFace[j], f = af < m.nI ? af : m.wallFace[af - m.nI];
                        const double sg = m.cellSide[j] == 0 ? 1.0 : -1.0;
                        const double *Sv = &m.Sf[3 * (size_t)f], *Cf = &m.Cf[3 * (size_t)f], *Cc = &m.C[3 * (size_t)c];
                        rec(plan_.stL[3 * e], plan_.stL[3 * e + 1], plan_.stL[3 * e + 2], plan_.stEnt[e]);
                        rec(sg * Sv[0], sg * Sv[1], sg * Sv[2], 2 * af + m.cellSide[j]);
                        const float iS = (float)(1.0 / std::sqrt(Sv[0] * Sv[0] + Sv[1] * Sv[1] + Sv[2] * Sv[2]));
                        int code;
                        std::memcpy(&code, &iS, 4);
                        rec(Cf[0] - Cc[0], Cf[1] - Cc[1], Cf[2] - Cc[2], code);
                    }
                }
                ints(&plan_.cells[h.cellStart], h.nT2);
                std::vector<int32_t> cst(h.nT + 1);  // T cells' entry ranges, tile-relative
                for (int i = 0; i <= h.nT; ++i) {
                    cst[i] = 2 * (plan_.stOff[h.stStart + i] - base);
                    bool inner = i < h.nT;
                    for (int e = plan_.stOff[h.stStart + i]; inner && e < plan_.stOff[h.stStart + i + 1]; ++e)
                        inner = plan_.stEnt[e] >= 0;
                    cst[i] += inner;
                }
                ints(cst.data(), h.nT + 1);
                const int n16 = (int)meta.size() - metaOff.back();
                if (n16 > tile_meta32_bound(h.nEnt, h.nT2)) { err = "tile metadata exceeds its bound"; return false; }
            }
            metaOff.push_back((int)meta.size());
            args_.meta = upload(meta);
            args_.metaOff = upload(metaOff);
            {
                // faces of each cell in global face order, S oriented out of the cell
                std::vector<int> cfOff(m.nC + 1);
                std::vector<float4> cfEnt;
                for (int c = 0; c < m.nC; ++c) {
                    cfOff[c] = (int)cfEnt.size();
                    for (int j = m.cellOff[c]; j < m.cellOff[c + 1]; ++j) {
                        const int af = m.cellFace[j];
                        const int gf = af < m.nI ? af : m.wallFace[af - m.nI];
                        const double sg = m.cellSide[j] == 0 ? 1.0 : -1.0;
                        float code;
                        std::memcpy(&code, &af, 4);
                        cfEnt.push_back(make_float4((float)(sg * m.Sf[3 * (size_t)gf]), (float)(sg * m.Sf[3 * (size_t)gf + 1]),
                                                    (float)(sg * m.Sf[3 * (size_t)gf + 2]), code));
                    }
                }
                cfOff[m.nC] = (int)cfEnt.size();
                for (int c = 0; c < m.nC; ++c) gatherMF_ = std::max(gatherMF_, cfOff[c + 1] - cfOff[c]);
                gatherMF_ = std::min(gatherMF_, 8);  // further faces of a cell are read directly
                gatherSmem_ = gather_smem(kGatherWarps, gatherMF_, KC, H_);
                allow_max_dynamic_smem(kGather_);
                int per = 0, nsm = 0;
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kGather_, kGatherWarps * 32, gatherSmem_);
                // the velocity constants in shared memory when they are small
                // (2D grids up to 1536 padded velocities: <= 24 KB per block)
                // and the blocks per SM stay as they are without them
                if (fp32_ && D_ == 2 && dv_table32_bytes(D_, a.Vp) <= 24 * 1024) {
                    int perTab = 0;
                    const size_t withTab = gatherSmem_ + dv_table32_bytes(D_, a.Vp);
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perTab, kGather_, kGatherWarps * 32, withTab);
                    if (perTab >= per) {
                        gatherTab_ = true;
                        gatherSmem_ = withTab;
                        per = perTab;
                    }
                }
                cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
                gatherBlocks_ = std::max(1, per) * std::max(1, nsm);  // persistent: one wave
                const bool rows32 = (unsigned long long)std::max(a.nA, a.nC) * (a.Vp / npl_) < (1ull << 32);
                std::vector<int> kind(m.nC);
                for (int c = 0; c < m.nC; ++c) {
                    kind[c] = rows32 ? cfOff[c + 1] - cfOff[c] : 0;
                    for (int j = m.cellOff[c]; j < m.cellOff[c + 1]; ++j)
                        if (m.cellFace[j] >= m.nI) kind[c] = 0;
                    if (kind[c] > gatherMF_) kind[c] = 0;
                }
                args_.cfKind = upload(kind);
                // Order of the gather: the cells as numbered, or tile by tile
                // (by number within a tile), whichever separates fewer
                // neighbours by windows of 256 places: cells that run together
                // share face values through L2.  Row-major hexes 48^3: 39 % ->
                // 22 % of the faces, k_cell_gather 6.09 -> 5.72 ms; 128^2
                // quads: 25 % -> 7 %, 173 -> 137 us (as numbered, some warps
                // met nothing but wall cells); triangles along a Morton curve:
                // 9 % as numbered, 11 % by tiles, 547 / 563 us.
                std::vector<int> ord, pos(m.nC);
                for (const TileHdr& h : plan_.hdr) {
                    ord.insert(ord.end(), plan_.cells.begin() + h.cellStart, plan_.cells.begin() + h.cellStart + h.nT);
                    std::sort(ord.end() - h.nT, ord.end());
                }
                for (int i = 0; i < m.nC; ++i) pos[ord[i]] = i;
                long long byTile = 0, asIs = 0;
                for (int f = 0; f < m.nI; ++f) {
                    byTile += pos[m.owner[f]] / 256 != pos[m.neighbour[f]] / 256;
                    asIs += m.owner[f] / 256 != m.neighbour[f] / 256;
                }
                if (asIs <= byTile)
                    for (int i = 0; i < m.nC; ++i) ord[i] = i;
                // Few cells per warp (the last of `rounds` + 1 rounds holds
                // `rem` cells): the cells with boundary faces, which take about
                // 1.5 times as long, go to warps without a cell in the last
                // round, one each.  k_cell_gather: 61^2 quads x 28^2 47.0 ->
                // 39.8 us, 90x45 channel x 24^2 48.6 -> 41.3, 14^3 hexes x 18^3
                // 267 -> 200.
                const int warps = gatherBlocks_ * kGatherWarps, rounds = m.nC / warps, rem = m.nC % warps;
                const long long slow = std::count(kind.begin(), kind.end(), 0);
                if (rounds >= 1 && rounds <= 3 && slow <= warps - rem) {
                    const int at = (rounds - 1) * warps + rem, quick = warps - rem - (int)slow;  // place; other cells there
                    std::vector<int> before, there, after;
                    int n = 0;
                    for (int c : ord) {
                        if (kind[c] == 0) there.push_back(c);
                        else if (n++ < at) before.push_back(c);
                        else (n <= at + quick ? there : after).push_back(c);
                    }
                    ord = before;
                    ord.insert(ord.end(), there.begin(), there.end());
                    ord.insert(ord.end(), after.begin(), after.end());
                }
                args_.cellOrd = upload(ord);
                args_.cfOff = upload(cfOff);
                args_.cfEnt = upload(cfEnt);
                std::vector<float> iv(m.nC);
                for (int c = 0; c < m.nC; ++c) iv[c] = (float)(1.0 / m.V[c]);
                args_.invVf = upload(iv);
                args_.gF = alloc<float>((size_t)a.nA * a.Vp);
                args_.hF = H_ ? alloc<float>((size_t)a.nA * a.Vp) : nullptr;
                args_.feqT = alloc<float4>(3 * (size_t)a.nA);
                args_.faceMom = alloc<double>((size_t)a.nA * 2 * 32);
            }
            std::vector<float4> w4(std::max(a.nW, 1), make_float4(0, 0, 0, 0));
            std::vector<double> Tw(a.nW);
            if (a.nW) cudaMemcpy(Tw.data(), a.Tw, a.nW * 8, cudaMemcpyDeviceToHost);
            for (int w = 0; w < a.nW; ++w) {
                // .y: 1/deltaCoeff of the lagged-gradient boundary value; 0 on
                // symmetryPlane (a constraint patch of gbar+: value = internal value)
                // .z: 0 wall, 1 open boundary, 2 symmetryPlane (relaxed twice outgoing)
                const int kind = m.wallKind[w];
                const bool plane = kind == DUGKS_PATCH_SYMMETRY_PLANE;
                w4[w] = make_float4((float)((a.R * Tw[w]) * (a.K + 3 - a.D)), plane ? 0.f : (float)(1.0 / m.dcW[w]),
                                    kind == DUGKS_PATCH_MAXWELL ? 0.f : (plane ? 2.f : 1.f), 0.f);
            }
            args_.wall4 = upload(w4);
            if (a.bcMask & ((1 << kBcSymmetryMod) | (1 << kBcSymmetryPlane))) {
                args_.symG = alloc<float>((size_t)a.nW * a.Vp);
                args_.symH = H_ ? alloc<float>((size_t)a.nW * a.Vp) : nullptr;
            }
            args_.rhoWs = alloc<float>(std::max(a.nW, 1));
        } else {
            args_.stEnt = upload(plan_.stEnt);
            args_.stL = upload(plan_.stL);
            std::vector<double> fgeo(9 * nRec);
            for (size_t k = 0; k < nRec; ++k) {
                const TileFace& r = plan_.faces[k];
                const int f = r.a < m.nI ? r.a : m.wallFace[r.a - m.nI];
                const int o = m.owner[f];
                for (int q = 0; q < 3; ++q) {
                    fgeo[9 * k + q] = m.Sf[3 * (size_t)f + q];
                    fgeo[9 * k + 3 + q] = m.Cf[3 * (size_t)f + q] - m.C[3 * (size_t)o + q];
                    fgeo[9 * k + 6 + q] =
                        r.a < m.nI ? m.Cf[3 * (size_t)f + q] - m.C[3 * (size_t)m.neighbour[f] + q] : 0.0;
                }
            }
            args_.fgeo = upload(fgeo);
        }
        // ---- DV arrays in storage precision
        std::vector<double> xh(3 * (size_t)a.Vp), wh(a.Vp);
        cudaMemcpy(xh.data(), a.xi, xh.size() * 8, cudaMemcpyDeviceToHost);
        cudaMemcpy(wh.data(), a.w, wh.size() * 8, cudaMemcpyDeviceToHost);
        args_.xi = upload(std::vector<S>(xh.begin(), xh.end()));
        args_.w = upload(std::vector<S>(wh.begin(), wh.end()));
        // ---- state
        const size_t nCV = (size_t)a.nC * a.Vp, nWV = (size_t)std::max(a.nW, 1) * a.Vp;
        for (int i = 0; i < 2; ++i) {
            gT_[i] = alloc<S>(nCV);
            hT_[i] = H_ ? alloc<S>(nCV) : nullptr;
            Gg_[i] = alloc<S>(nWV);
            Gh_[i] = H_ ? alloc<S>(nWV) : nullptr;
            cc_[i] = sizeof(S) == 4 ? alloc<float>((size_t)a.nC * kNCoef) : nullptr;
        }
        args_.Mw = mw_ = alloc<S>(nWV);
        min_ = alloc<double>((size_t)std::max(a.nW, 1) * 32);
        args_.Min = min_;
        args_.fc = sizeof(S) == 4 ? alloc<float>((size_t)a.nA * kNCoef) : nullptr;
        if (sizeof(S) == 4) {
            mref_ = alloc<float>(a.Vp);
            refMom_ = alloc<double>(32);
            wallRefOut_ = alloc<double>((size_t)std::max(a.nW, 1) * 32);
            args_.mref = mref_;
            args_.refMom = refMom_;
            args_.wallRefOut = wallRefOut_;
        }
        rhoN_ = alloc<double>(a.nC); UN_ = alloc<double>(3 * (size_t)a.nC); TN_ = alloc<double>(a.nC);
        qN_ = alloc<double>(3 * (size_t)a.nC); tauN_ = alloc<double>(a.nC);
        if (oom_) { err = "fused pipeline: device allocation failed"; return false; }
        // density scale of the stored distributions: O(1) values in FP32
        if (sizeof(S) == 4) {
            std::vector<double> r0(a.nC), t0(a.nC);
            cudaMemcpy(r0.data(), a.rho, a.nC * 8, cudaMemcpyDeviceToHost);
            cudaMemcpy(t0.data(), a.T, a.nC * 8, cudaMemcpyDeviceToHost);
            double rs = 0, ts = 0;
            for (int c = 0; c < a.nC; ++c) { rs += r0[c]; ts += t0[c]; }
            rs /= a.nC; ts /= a.nC;
            gscale_ = std::pow(2.0 * 3.14159265358979323846 * a.R * ts, 0.5 * D_) / rs;
            T0_ = ts;
            hrefFac_ = a.R * ts * (a.K + 3 - a.D);
            args_.hrefFac = (float)hrefFac_;
        } else {
            gscale_ = 1.0;
        }
        args_.gscale = gscale_;
        args_.invGscale = 1.0 / gscale_;
        return true;
    }

    double gscale() const override { return gscale_; }

    void initState(const StepArgs& a, int sms, cudaStream_t s) override {
        if constexpr (sizeof(S) == 4) {
            kRef_<<<1 + a.nW, 128, 0, s>>>(a, T0_, hrefFac_, mref_, refMom_, wallRefOut_);
            k_init_dev32<<<sms * 8, 256, 0, s>>>(a, mref_, gscale_, hrefFac_, gT_[0], hT_[0]);
        } else {
            launch_init_state<S>(a, gT_[0], hT_[0], gscale_, sms, s);
        }
        if (sizeof(S) == 4) {
            if (D_ == 2) k_cell_coef<2><<<sms * 4, 256, 0, s>>>(a, cc_[0], gscale_);
            else k_cell_coef<3><<<sms * 4, 256, 0, s>>>(a, cc_[0], gscale_);
        }
        if (a.nW > 0) kTables_<<<a.nW, 128, 0, s>>>(a, mw_, min_);
    }

    int nKernels() const override { return fp32_ ? 3 : 2; }
    const char* kernelName(int k) const override {
        if (fp32_) return k == 0 ? "k_face_sides" : (k == 1 ? "k_face_macros" : "k_cell_gather");
        return k == 0 ? "k_sweep_face" : "k_sweep_cell";
    }

    // Arguments of the step `parity` steps ahead (0: this step, 1: the next).
    FusedArgs<S> stepArgs(const StepArgs& a, int parity) const {
        FusedArgs<S> A = args_;
        A.b = a;
        A.dt = (S)a.dt;
        const int c = (cur_ + parity) & 1;
        A.gT = gT_[c]; A.hT = hT_[c];
        A.gTn = gT_[1 - c]; A.hTn = hT_[1 - c];
        A.Gbg = Gg_[c]; A.Gbh = Gh_[c];
        A.Gbgn = Gg_[1 - c]; A.Gbhn = Gh_[1 - c];
        A.cc = cc_[c]; A.ccn = cc_[1 - c];
        A.rhoN = rhoN_; A.UN = UN_; A.TN = TN_; A.qN = qN_; A.tauN = tauN_;
        if (parity & 1) {  // endStep swaps the cell macros into the base arguments
            std::swap(A.b.rho, A.rhoN); std::swap(A.b.U, A.UN); std::swap(A.b.T, A.TN);
            std::swap(A.b.q, A.qN); std::swap(A.b.tau, A.tauN);
        }
        return A;
    }

    bool batchable() const override { return fp32_; }
    bool batchKernels() const override { return fp32_ && (bcMask_ & ~(1 << kBcMaxwell)) == 0; }
    void batchArgs(const StepArgs& a, int parity, void* out) const override {
        const FusedArgs<S> A = stepArgs(a, parity);
        std::memcpy(out, &A, sizeof(A));
    }
    size_t batchArgsBytes() const override { return sizeof(FusedArgs<S>); }
    int batchTiles() const override { return plan_.nTiles; }
    size_t batchSmemFace() const override { return smemA_; }
    int batchGatherMF() const override { return gatherMF_; }
    int batchNpl() const override { return npl_; }

    void launchParity(const StepArgs& a, int parity, int sms, cudaStream_t s) override {
        for (int k = 0; k < nKernels(); ++k) launchArgs(k, stepArgs(a, parity), a, sms, s);
    }

    void launch(int k, const StepArgs& a, int sms, cudaStream_t s) override { launchArgs(k, stepArgs(a, 0), a, sms, s); }

    // Launch that may start while the kernel before it in the stream ends, if
    // that one allows it (early() in fused32.cuh); after any other kernel, copy
    // or event it starts as usual.  For the FP32 face sweep behind the gather
    // only: a step of 24^2 quads x 8^2 31.0 -> 26.9 us, 61^2 quads x 28^2 103 ->
    // 99.4, 18k triangles x 29^2 257 -> 253, 100k triangles and 48^3 hexes
    // unchanged.  Not for the other two: the gather beside the macros finds the
    // SM set up for the face sweep's shared memory and runs with half its L1
    // (48^3 hexes 15.6 -> 17.4 ms), and the macros' blocks, let in while the
    // sweep ends, crowd the SMs that end first (61^2 quads 103 -> 122 us).
    template <class... P, class... Q>
    static void launch_beside(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t s, const Q&... args) {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(grid);
        c.blockDim = dim3(block);
        c.dynamicSmemBytes = smem;
        c.stream = s;
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        c.attrs = &at;
        c.numAttrs = 1;
        cudaLaunchKernelEx(&c, k, P(args)...);
    }

    void launchArgs(int k, const FusedArgs<S>& A, const StepArgs& a, int sms, cudaStream_t s) {
        if (k == 0) {
            if (fp32_) launch_beside(kFace_, plan_.nTiles, kWarps * 32, smemA_, s, A);
            else kFace_<<<plan_.nTiles, kWarps * 32, smemA_, s>>>(A);
            if (kOpen_) kOpen_<<<std::max(1, std::min((a.nW + 3) / 4, sms * 8)), 128, 0, s>>>(A);
        }
        else if (!fp32_) kCell_<<<plan_.nTiles, kWarps * 32, smemB_, s>>>(A);
        else if (k == 1) {  // one face per thread; blocks of one warp while they leave SMs without work
            const int t = a.nA <= 128 * 4 * sms ? 32 : 128;
            kMacros_<<<std::max(1, (a.nA + t - 1) / t), t, 0, s>>>(A);
        }
        else {
            kGather_<<<std::min((a.nC + kGatherWarps - 1) / kGatherWarps, gatherBlocks_), kGatherWarps * 32, gatherSmem_,
                       s>>>(A, gatherMF_, gatherTab_ ? 1 : 0);
            if (a.zgMask || (a.bcMask & ((1 << kBcPressureIn) | (1 << kBcPressureOut)))) {
                StepArgs n = A.b;  // zeroGradient U/T patches, then P10, from the macros this step wrote
                n.rho = A.rhoN; n.U = A.UN; n.T = A.TN;
                launch_zero_gradient_tu(n, s);
                if (a.bcMask & ((1 << kBcPressureIn) | (1 << kBcPressureOut))) launch_pressure_bc(n, s);
            }
        }
    }

    void endStep(StepArgs& base) override {
        cur_ = 1 - cur_;
        std::swap(base.rho, rhoN_);
        std::swap(base.U, UN_);
        std::swap(base.T, TN_);
        std::swap(base.q, qN_);
        std::swap(base.tau, tauN_);
    }

    void refreshDerived(const StepArgs& a, int sms, cudaStream_t s) override {
        if (sizeof(S) == 4) {
            if (D_ == 2) k_cell_coef<2><<<sms * 4, 256, 0, s>>>(a, cc_[cur_], gscale_);
            else k_cell_coef<3><<<sms * 4, 256, 0, s>>>(a, cc_[cur_], gscale_);
        }
    }

    void exportDist(const StepArgs& a, int which, double* dst, int sms, cudaStream_t s) override {
        if constexpr (sizeof(S) == 4)
            k_export_dev32<<<sms * 8, 256, 0, s>>>(a, which ? hT_[cur_] : gT_[cur_], mref_, which ? hrefFac_ : 1.0,
                                                   1.0 / gscale_, dst);
        else
            launch_export_dist<S>(a, which ? hT_[cur_] : gT_[cur_], dst, 1.0 / gscale_, sms, s);
    }
    void importDist(const StepArgs& a, int which, const double* src, int sms, cudaStream_t s) override {
        if constexpr (sizeof(S) == 4)
            k_import_dev32<<<sms * 8, 256, 0, s>>>(a, src, mref_, which ? hrefFac_ : 1.0, gscale_,
                                                   which ? hT_[cur_] : gT_[cur_]);
        else
            launch_import_dist<S>(a, src, which ? hT_[cur_] : gT_[cur_], gscale_, sms, s);
    }
    void* distPtr(int which) override { return which ? (void*)hT_[cur_] : (void*)gT_[cur_]; }
    void* gradBPtr(int which) override { return which ? (void*)Gh_[cur_] : (void*)Gg_[cur_]; }
    size_t bytes() const override { return bytes_; }
    std::string describe() const override {
        char buf[256];
        snprintf(buf, sizeof(buf), "tiles=%d maxT=%d meanT=%.1f halo=%.2f maxT2=%d maxFB=%d npl=%d row=%d smemA=%zu smemB=%zu gatherMF=%d",
                 plan_.nTiles, plan_.maxT, (double)plan_.sumT / std::max(1, plan_.nTiles),
                 (double)plan_.sumT2 / std::max(1LL, plan_.sumT), plan_.maxT2, plan_.maxFB, npl_, (int)row_, smemA_, smemB_, gatherMF_);
        return buf;
    }

private:
    static constexpr int kWarps = sizeof(S) == 4 ? kFaceWarps : 16;  // warps per tile block (one tile per SM)

    template <typename T>
    T* alloc(size_t n) {
        void* p = nullptr;
        const size_t by = std::max<size_t>(n, 1) * sizeof(T);
        if (device_malloc(&p, by) != cudaSuccess) { cudaGetLastError(); oom_ = true; return nullptr; }
        cudaMemset(p, 0, by);
        allocs_.push_back(p);
        bytes_ += by;
        return static_cast<T*>(p);
    }
    template <typename T>
    T* upload(const std::vector<T>& v) {
        T* p = alloc<T>(v.size());
        if (p && !v.empty()) cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
        return p;
    }

    template <int D, bool H>
    void set64() {
        kFace_ = k_sweep_face<S, D, H, 1, kWarps>;
        kCell_ = k_sweep_cell<S, D, H, 1, kWarps>;
        kTables_ = k_wall_tables<S, D, H>;
        smemFaceFn_ = &SmemLayout<S, D, H, 1>::face;
        smemCellFn_ = &SmemLayout<S, D, H, 1>::cell;
    }
    void pick() {
        if constexpr (sizeof(S) == 4) {
            const Kernels32 k = kernels32(D_, H_, npl_, row_, (bcMask_ & ~(1 << kBcMaxwell)) != 0);
            kFace_ = k.face;
            kMacros_ = k.macros;
            kOpen_ = k.open;
            kGather_ = k.gather;
            kTables_ = k.tables;
            kRef_ = k.ref;
            smemFaceFn_ = k.smemFace;
        } else {
            if (D_ == 2) { H_ ? set64<2, true>() : set64<2, false>(); }
            else { H_ ? set64<3, true>() : set64<3, false>(); }
        }
    }
    size_t smemFace(const TileDims& d) const { return smemFaceFn_(d); }
    size_t smemCell(const TileDims& d) const { return smemCellFn_(d); }

    int D_ = 2, npl_ = 1;
    bool fp32_ = false, row_ = false;
    int bcMask_ = 1 << kBcMaxwell;
    KernelFn kMacros_ = nullptr;
    KernelFn kOpen_ = nullptr;  // open boundary faces after sweep A (when the case has any)
    int gatherMF_ = 0, gatherBlocks_ = 1;
    bool gatherTab_ = false;
    size_t gatherSmem_ = 0;
    void (*kGather_)(FusedArgs<S>, int, int) = nullptr;
    bool H_ = true;
    TilePlan plan_;
    FusedArgs<S> args_{};
    KernelFn kFace_ = nullptr, kCell_ = nullptr;
    void (*kTables_)(StepArgs, S*, double*) = nullptr;
    void (*kRef_)(StepArgs, double, double, float*, double*, double*) = nullptr;
    float* mref_ = nullptr;
    double* refMom_ = nullptr;
    double* wallRefOut_ = nullptr;
    double T0_ = 273.0, hrefFac_ = 0.0;
    size_t (*smemFaceFn_)(const TileDims&) = nullptr;
    size_t (*smemCellFn_)(const TileDims&) = nullptr;
    size_t smemA_ = 0, smemB_ = 0;
    S* gT_[2] = {nullptr, nullptr};
    S* hT_[2] = {nullptr, nullptr};
    S* Gg_[2] = {nullptr, nullptr};
    S* Gh_[2] = {nullptr, nullptr};
    float* cc_[2] = {nullptr, nullptr};
    S* mw_ = nullptr;
    double* min_ = nullptr;
    double *rhoN_ = nullptr, *UN_ = nullptr, *TN_ = nullptr, *qN_ = nullptr, *tauN_ = nullptr;
    double gscale_ = 1.0;
    int cur_ = 0;
    std::vector<void*> allocs_;
    size_t bytes_ = 0;
    bool oom_ = false;
};

}  // namespace dugks
