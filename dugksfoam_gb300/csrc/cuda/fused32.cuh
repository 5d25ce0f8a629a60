// FP32 step (fast path): three launches per step.
//
//  k_face_sides32  (tiles of cells T with a one-ring halo H1, DV chunks of
//                   KC = 32*NPL velocities): gbar+ rows of T u H1 (P1), the
//                   least-squares gradient of each T cell (P2) and the upwind
//                   reconstruction of every face side whose cell is in T (P3),
//                   one warp per cell; lagged wall gradients, stored face
//                   values and per-side face moments;
//  k_face_macros32 (one thread per face): Maxwell-wall density (P4), incoming
//                   wall moments (P5), face macros and equilibrium tables (P6);
//  k_cell_gather32 (one warp per cell): face relaxation (P7), flux sum and
//                   g~ update (P8), cell moments and macros (P9).
//
// Layout and arithmetic choices:
//  * each lane owns NPL consecutive discrete velocities held as NPL/2 packed
//    float2 pairs (f32x2 FMA/ADD/MUL), so every per-velocity operation is one
//    packed instruction per pair and the per-face fixed costs (metadata, the
//    warp reduce-scatter of the moments) are paid once per KC velocities;
//  * the distributions are stored as deviations from a fixed rest Maxwellian:
//      G = gscale * g - Mref(xi),   Mref = exp(-|xi|^2 / (2 R T0)),
//    gscale = (2 pi R T0)^(D/2) / rho0 (h likewise with Href = Mref R T0 (K+3-D)).
//    Every pass is linear in g, Mref is uniform in space, so the gradient,
//    reconstruction, flux and update act on G unchanged; the relaxations use
//    g = G + Mref; the moments of Mref about any reference velocity are added
//    back exactly in FP64.  Storing the O(0.01-0.1) deviation instead of the
//    O(1) distribution cuts the FP32 storage rounding by the same factor.
//    (The Mref part of the face flux, Mref xi.sum_f(+-S_f), vanishes for a
//    closed cell and is not formed.)
//  * no FP64 instruction runs inside the DV chunk loops (GB300 issues FP64 at
//    1/64 of the FP32 rate): the face sweep's per-chunk warp totals go into
//    FP32 Kahan pairs per face side; the gather keeps per-lane FP32 partial
//    sums over all chunks of a cell and reduces them across the warp once;
//    both are finished in FP64, batched so that whole warps do the FP64 work.
#pragma once

#include <type_traits>

#include "fused_impl.cuh"

namespace dugks {


// Moment slots of the FP32 step: raw moments (about xi = 0) of the stored
// deviation.  sum w xi_i (|xi|^2 g + h) is one slot per direction: the heat
// flux needs the two terms only together.
template <int D, bool H>
struct Slots32 {
    static constexpr int M1 = 1;
    static constexpr int M2 = 1 + D;                  // xx,xy,(xz),yy,(yz),(zz)
    static constexpr int Q = M2 + D * (D + 1) / 2;
    static constexpr int H0 = Q + D;
    static constexpr int NM = H0 + (H ? 1 : 0);
    static constexpr int FLUX = NM;                   // outgoing wall flux
    static constexpr int NS = 16;
    static constexpr int P = NM + 1;                  // slots of one cell side in the face sweep
    static constexpr int FG = 32 / P;                 // cell sides that share one warp reduction
};

// 2^x by the hardware approximation (ex2.approx.ftz.f32, PTX ISA).  Flushing
// a result below 2^-126 to zero moves an equilibrium value by less than 1e-38
// of its peak (the grids here reach |xi - U|^2 / 2RT = 48 at T = T0).
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Packed FP32 pair arithmetic (sm_100+): each lane's NPL velocities are held
// as NPL/2 float2 pairs and every per-velocity operation is one packed
// instruction per pair.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 sel2(bool x0, bool x1, float2 a, float2 b) {  // per element: x ? a : b
    return make_float2(x0 ? a.x : b.x, x1 ? a.y : b.y);
}

template <int NP>
__device__ __forceinline__ void ldp(float2 (&d)[NP], const float* p) {
    if constexpr (NP == 2) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        d[0] = make_float2(t.x, t.y);
        d[1] = make_float2(t.z, t.w);
    } else {
        d[0] = *reinterpret_cast<const float2*>(p);
    }
}
template <int NP>
__device__ __forceinline__ void stp(float* p, const float2 (&d)[NP]) {
    if constexpr (NP == 2) *reinterpret_cast<float4*>(p) = make_float4(d[0].x, d[0].y, d[1].x, d[1].y);
    else *reinterpret_cast<float2*>(p) = d[0];
}
// Streaming (evict-first) store of the g~new rows: written once, read next step.
template <int NP>
__device__ __forceinline__ void stp_cs(float* p, const float2 (&d)[NP]) {
    if constexpr (NP == 2) __stcs(reinterpret_cast<float4*>(p), make_float4(d[0].x, d[0].y, d[1].x, d[1].y));
    else __stcs(reinterpret_cast<float2*>(p), d[0]);
}

// Per-tile metadata block (int4 units), staged into shared memory once per tile:
//   [nEnt][3] cell-face entries of the cells of T, cell by cell in global face
//             order: {Lx, Ly, Lz, local row of the other cell or -(wall+1)}
//             {S out of the cell, 2 face + side} {Cf - C_cell, 1/|S|}
//   cells (nT2), 2 x first entry of each cell of T (nT + 1), + 1 when none of
//   its faces is a boundary face, as ints padded to whole int4.
__host__ __device__ constexpr int tile_meta32_bound(int nEnt, int nT2) {
    return 3 * nEnt + (nT2 + 3) / 4 + (nT2 + 4) / 4;
}

// Shared memory of the face-sides sweep (all offsets multiples of 16 bytes):
//   2 x rows(T u H1) | moments of the cell sides | metadata | cell equilibria
// (the next DV chunk's raw rows stream into the second row buffer).
template <int D, bool H, int NPL>
struct SmemLayout32 {
    static constexpr int KC = 32 * NPL, P = Slots32<D, H>::P;
    __host__ __device__ static size_t rows(int n) { return (size_t)n * KC * sizeof(float) * (H ? 2 : 1); }
    __host__ __device__ static size_t mom(int nRows) { return 2 * rows(nRows); }
    __host__ __device__ static size_t meta(int nRows, int nEnt) {
        return mom(nRows) + (size_t)((nEnt + 1) & ~1) * P * sizeof(Acc<float>);
    }
    static size_t sides(const TileDims& d) {
        return meta(d.nT2, d.nEnt) + 16 * (size_t)tile_meta32_bound(d.nEnt, d.nT2) + 48 * (size_t)d.nT2;
    }
};

struct TileMeta32 {
    const float4* E;  // cell-face entries [nEnt][3]
    const int* C;     // local -> global cell
    const int* S;     // 2 x first entry of each cell of T (+ 1: no boundary face) [nT+1]
    float4* dyn;      // per-step tables after the block
};

// Copy the tile's block into shared memory (caller synchronises).
template <int NT>
__device__ __forceinline__ TileMeta32 stage_meta(const FusedArgs<float>& A, const TileHdr& hd, int tile,
                                                 unsigned char* at) {
    int4* sm = reinterpret_cast<int4*>(at);
    const int o0 = A.metaOff[tile], n16 = A.metaOff[tile + 1] - o0;
    const int4* gm = A.meta + o0;
    for (int i = threadIdx.x; i < n16; i += NT) sm[i] = __ldg(gm + i);
    TileMeta32 m;
    m.E = reinterpret_cast<const float4*>(sm);
    m.C = reinterpret_cast<const int*>(sm + 3 * hd.nEnt);
    m.S = reinterpret_cast<const int*>(sm + 3 * hd.nEnt + (hd.nT2 + 3) / 4);
    m.dyn = reinterpret_cast<float4*>(sm + tile_meta32_bound(hd.nEnt, hd.nT2));
    return m;
}

#if defined(DUGKS_CHECKED) && DUGKS_CHECKED
// Checked build: every index of a staged tile block within its range (rows
// of T u H1, faces, walls, entries, cells); an index outside is replaced by 0
// in the staged copy and reported (chk).
template <int NT>
__device__ void check_tile_meta32(const FusedArgs<float>& A, const TileHdr& hd, unsigned char* at) {
    int4* sm = reinterpret_cast<int4*>(at);
    int* st = A.b.status;
    float4* E = reinterpret_cast<float4*>(sm);
    for (int k = threadIdx.x; k < hd.nEnt; k += NT) {
        const int o = __float_as_int(E[3 * k].w), f = __float_as_int(E[3 * k + 1].w);
        const int ok = o >= 0 ? chk(o, hd.nT2, st) : -1 - chk(-o - 1, A.b.nW, st);
        E[3 * k].w = __int_as_float(ok);
        E[3 * k + 1].w = __int_as_float(chk(f, 2 * A.b.nA, st));
    }
    int* C = reinterpret_cast<int*>(sm + 3 * hd.nEnt);
    for (int k = threadIdx.x; k < hd.nT2; k += NT) C[k] = chk(C[k], A.b.nC, st);
    int* S = reinterpret_cast<int*>(sm + 3 * hd.nEnt + (hd.nT2 + 3) / 4);
    for (int k = threadIdx.x; k <= hd.nT; k += NT) S[k] = chk(S[k], 2 * hd.nEnt + 2, st);
}
#endif

// Equilibrium table entry {U, kexp} {1/RT, q'} {a, a A, RT, 0} from a
// coefficient block and the relaxation weight a.
__device__ __forceinline__ void eq_table(float4* q, const float* blk, float a) {
    const float4* b = reinterpret_cast<const float4*>(blk);
    const float4 b2 = b[2];
    q[0] = b[0];
    q[1] = b[1];
    q[2] = make_float4(a, a * b2.x, b2.y, 0.0f);
}
// cell weight 1.5dt/(2tau+dt), face weight h/(2tau+h) with h = dt/2
__device__ __forceinline__ float cell_weight(float dt, const float* blk) { return 1.5f * dt / (2.0f * blk[10] + dt); }
__device__ __forceinline__ float face_weight(float dt, const float* blk) {
    const float hh = 0.5f * dt;
    return hh / (2.0f * blk[10] + hh);
}

// DV constants of this lane's NPL consecutive velocities in the current chunk.
// ROW: the velocity count per direction is a multiple of NPL, so that the
// lane's velocities lie in one row of the tensor-product grid and share xi_y
// and xi_z: everything that depends on those is one scalar instruction per
// lane instead of one packed instruction per pair (and no copy of a scalar
// into both halves of a pair).  Other grids (4Z + 1 velocities) hold y and z
// per pair.  Chosen per case by M % NPL.
template <int D, int NPL, bool ROW>
struct Lane32 {
    static constexpr int NP = NPL / 2, NY = ROW ? 1 : NP;
    float2 x[NP], y[NY], z[NY], w[NP], mr[NP];  // ROW: y[0].x, z[0].x
    __device__ __forceinline__ void yz(const float* py, const float* pz) {
        if constexpr (ROW) {
            y[0] = make_float2(*py, 0.f);
            z[0] = make_float2(D == 3 ? *pz : 0.f, 0.f);
        } else {
            ldp<NP>(y, py);
            if (D == 3) ldp<NP>(z, pz);
            else
#pragma unroll
                for (int p = 0; p < NP; ++p) z[p] = f2(0.0f);
        }
    }
    __device__ __forceinline__ void load(const FusedArgs<float>& A, int v0, int lane) {
        const int Vp = A.b.Vp, v = v0 + lane * NPL;
        ldp<NP>(x, A.xi + v);
        yz(A.xi + Vp + v, A.xi + 2 * Vp + v);
        ldp<NP>(w, A.w + v);
        ldp<NP>(mr, A.mref + v);
    }
    // from a shared-memory copy [x | y | (z) | w | mref], Vp each (dv_table32)
    __device__ __forceinline__ void load_tab(const float* tab, int Vp, int v0, int lane) {
        const int v = v0 + lane * NPL;
        ldp<NP>(x, tab + v);
        yz(tab + Vp + v, tab + 2 * Vp + v);
        ldp<NP>(w, tab + D * Vp + v);
        ldp<NP>(mr, tab + (D + 1) * Vp + v);
    }
    // xi.S of pair p, rounded term by term: a velocity lying in the face gives exactly 0
    __device__ __forceinline__ float2 dot(int p, float Sx, float Sy, float Sz) const {
        if constexpr (ROW) {
            float s = __fmul_rn(y[0].x, Sy);
            if (D == 3) s = __fadd_rn(s, __fmul_rn(z[0].x, Sz));
            return add2(mul2(x[p], f2(Sx)), f2(s));
        } else {
            float2 s = add2(mul2(x[p], f2(Sx)), mul2(y[p], f2(Sy)));
            if (D == 3) s = add2(s, mul2(z[p], f2(Sz)));
            return s;
        }
    }
    // dot with the terms added in the order of ROW lanes
    __device__ __forceinline__ float2 dot_row(int p, float Sx, float Sy, float Sz) const {
        static_assert(!ROW, "ROW lanes have one order");
        float2 s = mul2(y[p], f2(Sy));
        if (D == 3) s = add2(s, mul2(z[p], f2(Sz)));
        return add2(mul2(x[p], f2(Sx)), s);
    }
    // xi.S of pair p for use as a factor
    __device__ __forceinline__ float2 lin(int p, float Sx, float Sy, float Sz) const {
        if constexpr (ROW) {
            float s = y[0].x * Sy;
            if (D == 3) s = fmaf(z[0].x, Sz, s);
            return fma2(x[p], f2(Sx), f2(s));
        } else {
            float2 s = fma2(y[p], f2(Sy), mul2(x[p], f2(Sx)));
            if (D == 3) s = fma2(z[p], f2(Sz), s);
            return s;
        }
    }
    // |xi - u|^2 and q.(xi - u) of pair p
    __device__ __forceinline__ void rel(int p, float ux, float uy, float uz, float qx, float qy, float qz, float2& c2,
                                        float2& phi) const {
        const float2 cx = add2(x[p], f2(-ux));
        if constexpr (ROW) {
            const float cy = y[0].x - uy;
            float s2 = cy * cy, sp = cy * qy;
            if (D == 3) {
                const float cz = z[0].x - uz;
                s2 = fmaf(cz, cz, s2);
                sp = fmaf(cz, qz, sp);
            }
            c2 = fma2(cx, cx, f2(s2));
            phi = fma2(cx, f2(qx), f2(sp));
        } else {
            const float2 cy = add2(y[p], f2(-uy));
            c2 = fma2(cy, cy, mul2(cx, cx));
            phi = fma2(cy, f2(qy), mul2(cx, f2(qx)));
            if (D == 3) {
                const float2 cz = add2(z[p], f2(-uz));
                c2 = fma2(cz, cz, c2);
                phi = fma2(cz, f2(qz), phi);
            }
        }
    }
};

// d - xi dt/2 of a lane's velocities (the shift from a cell's centre to the
// foot of the characteristic through a face centre).
template <int D, int NPL, bool ROW>
struct Shift32 {
    static constexpr int NP = NPL / 2, NY = ROW ? 1 : NP;
    float2 x[NP], y[NY], z[NY];
    __device__ __forceinline__ void set(const Lane32<D, NPL, ROW>& L, float dt, float dx, float dy, float dz) {
        const float h = -0.5f * dt;
#pragma unroll
        for (int p = 0; p < NP; ++p) x[p] = fma2(L.x[p], f2(h), f2(dx));
        if constexpr (ROW) {
            y[0].x = fmaf(L.y[0].x, h, dy);
            if (D == 3) z[0].x = fmaf(L.z[0].x, h, dz);
        } else {
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                y[p] = fma2(L.y[p], f2(h), f2(dy));
                if (D == 3) z[p] = fma2(L.z[p], f2(h), f2(dz));
            }
        }
    }
    // L . shift of pair p
    __device__ __forceinline__ float2 dot(int p, float lx, float ly, float lz) const {
        if constexpr (ROW) {
            float t = y[0].x * ly;
            if (D == 3) t = fmaf(z[0].x, lz, t);
            return fma2(x[p], f2(lx), f2(t));
        } else {
            float2 t = fma2(y[p], f2(ly), mul2(x[p], f2(lx)));
            if (D == 3) t = fma2(z[p], f2(lz), t);
            return t;
        }
    }
    // component k of pair p
    __device__ __forceinline__ float2 comp(int k, int p) const {
        if (k == 0) return x[p];
        if constexpr (ROW) return f2(k == 1 ? y[0].x : z[0].x);
        else return k == 1 ? y[p] : z[p];
    }
};

// The velocity constants of Lane32 for all Vp velocities, copied by a block
// into shared memory (caller synchronises); its size in bytes.
__host__ __device__ inline size_t dv_table32_bytes(int D, int Vp) { return (size_t)(D + 2) * Vp * sizeof(float); }
template <int D>
__device__ __forceinline__ void dv_table32(const FusedArgs<float>& A, float* tab) {
    const int Vp = A.b.Vp;
    for (int q = threadIdx.x; q < (D + 2) * Vp; q += blockDim.x) {
        const int k = q / Vp, v = q - k * Vp;
        tab[q] = k < D ? A.xi[k * Vp + v] : (k == D ? A.w[v] : A.mref[v]);
    }
}

// Shakhov relaxation in deviation form: out = G - a (G + Mref) + a g^S, with
//   a g^S = aA e [1 + phi u],   e = exp(-c^2 / 2RT),  u = c^2/RT - (D+2),
//   a h^S = RT (K+3-D) [a g^S + ck aA e phi],   ck = 2 - 2K/(K+3-D)
// (phi = the Shakhov heat-flux term q'.c; the h form is the reference's
// ((c^2/RT - D)(K+3-D) - 2K) regrouped about u, so that g and h share a g^S).
template <int D, bool H>
struct Eq32 {
    float ux, uy, uz, kexp, invRT, qx, qy, qz, a, aA, KDRT, ck, hf;
    __device__ __forceinline__ void load(const float4* q, int K, float hrefFac) {  // an eq_table entry
        const float4 b0 = q[0], b1 = q[1], b2 = q[2];
        ux = b0.x; uy = b0.y; uz = b0.z; kexp = b0.w;
        invRT = b1.x; qx = b1.y; qy = b1.z; qz = b1.w;
        a = b2.x;
        aA = b2.y;
        KDRT = (float)(K + 3 - D) * b2.z;
        ck = D == 2 ? (K == 0 ? 2.0f : 2.0f / (float)(K + 1)) : 0.0f;  // (6 - 2D) / (K + 3 - D)
        hf = hrefFac;
    }
    template <int NPL, bool ROW>
    __device__ __forceinline__ void relax(const Lane32<D, NPL, ROW>& L, int p, float2& g, float2& h) const {
        float2 c2, phi;
        L.rel(p, ux, uy, uz, qx, qy, qz, c2, phi);
        const float2 t = mul2(c2, f2(kexp));
        const float2 e = mul2(make_float2(ex2f(t.x), ex2f(t.y)), f2(aA));
        const float2 u = fma2(c2, f2(invRT), f2(-(float)(D + 2)));
        const float2 ep = mul2(e, phi);
        const float2 ags = fma2(ep, u, e);
        g = fma2(f2(-a), add2(g, L.mr[p]), add2(g, ags));
        if (H) {
            const float2 z = D == 2 ? fma2(ep, f2(ck), ags) : ags;
            h = fma2(f2(-a), fma2(L.mr[p], f2(hf), h), fma2(z, f2(KDRT), h));
        }
    }
};


// The next step's face sweep may start beside the cell gather (programmatic
// stream serialisation, see launch_beside): early() in the gather lets its
// blocks onto SMs as they become free, where they stage their tile data, which
// are constant; after_previous() then waits until the gather has ended and its
// writes are visible.  The gather itself is launched as usual, so that with it
// all kernels before it have ended.
__device__ __forceinline__ void early() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Asynchronous global -> shared copies (each lane copies, and later reads,
// only its own NPL floats of a row, so a lane's wait_group is all the
// ordering it needs).
__device__ __forceinline__ void cp_async_row(float* dst, const float* src, int npl) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    if (npl == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The rows of a tile that a warp copies and relaxes: first, first + step, ...
// below end.  Warp w forms the sides of cells w, w + NW, ...; the warps that
// get one cell less than the others take kCellRows rows more, so that all reach
// the chunk's barrier together (rows dealt out evenly -> so; kCellRows 4 / 8 and
// 10 / 20 are 1 % slower, two rows at a time keep the loop as fast as one with a
// constant step): 48^3 hexes x 20^3 10.30 -> 9.81 ms, 128^2 quads x 32^2
// 172 -> 167 us, 61^2 quads x 28^2 50.8 -> 48.0 us; 100k triangles x 32^2, whose
// tiles of 61 cells leave three warps a cell short, unchanged at 0.71 ms.
struct RowPart {
    int first, step, end;
};
template <int D, int NW>
__device__ __forceinline__ RowPart row_part(const TileHdr& hd, int warp) {
    constexpr int kCellRows = D == 2 ? 7 : 14;
    const int heavy = hd.nT % NW, light = NW - heavy;
    if (heavy == 0) return {warp, NW, hd.nT2};
    const int x = max(0, hd.nT2 - kCellRows * light) / NW;  // rows of a warp with one cell more
    if (warp < heavy) return {warp, heavy, heavy * x};
    return {heavy * x + warp - heavy, light, hd.nT2};
}

// Raw g~ (and h~) rows of T u H1 for the DV chunk at v0 into shared memory,
// 16-byte asynchronous copies (one commit group).  A warp copies the rows it
// relaxes, so that after its own wait_group and a __syncwarp it may relax them
// without a block barrier.
// sg: g rows, sh: h rows of this buffer.
template <int NPL, bool H>
__device__ __forceinline__ void issue_rows32(const FusedArgs<float>& A, const RowPart& rp, const int* C, float* sg,
                                             float* sh, int v0, int lane) {
    constexpr int KC = 32 * NPL, SEG = KC / 4;
#pragma unroll 2
    for (int r = rp.first; r < rp.end; r += rp.step) {
        const size_t gr = (size_t)C[r] * A.b.Vp + v0;
        for (int sgm = lane; sgm < SEG; sgm += 32) {
            cp_async_row(sg + r * KC + sgm * 4, A.gT + gr + sgm * 4, 4);
            if (H) cp_async_row(sh + r * KC + sgm * 4, A.hT + gr + sgm * 4, 4);
        }
    }
    cp_async_commit();
}

// gbar+ = relaxation of the raw rows in place (shared memory only).
template <int D, bool H, int NPL, bool ROW>
__device__ __forceinline__ void relax_rows32(const FusedArgs<float>& A, const RowPart& rp, const float4* ceq,
                                             const Lane32<D, NPL, ROW>& L, int lane, float* rg, float* rh) {
    constexpr int KC = 32 * NPL, NP = NPL / 2;
#pragma unroll 2
    for (int r = rp.first; r < rp.end; r += rp.step) {
        float2 g[NP], h[NP];
        float* sg = rg + r * KC;
        float* sh = rh + r * KC;
        ldp<NP>(g, sg + lane * NPL);
        if (H) ldp<NP>(h, sh + lane * NPL);
        Eq32<D, H> e;
        e.load(ceq + 3 * r, A.b.K, A.hrefFac);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            if (!H) h[p] = f2(0.f);
            e.relax(L, p, g[p], h[p]);
        }
        stp<NP>(sg + lane * NPL, g);
        if (H) stp<NP>(sh + lane * NPL, h);
    }
}

// Upwind weight of a cell's side of a face for one velocity from s = xi.S (S
// out of the cell): 1 for s > 0, 0 for s < 0, 1/2 for s == 0 (one saturating
// FMA; |s| below 2^-101 would count as a partial tie, far below any xi.S of a
// real face).  The other cell's weight, from -s, is exactly the rest.
__device__ __forceinline__ float2 upwind_w2(float2 s) {
    return make_float2(__saturatef(fmaf(s.x, 0x1p100f, 0.5f)), __saturatef(fmaf(s.y, 0x1p100f, 0.5f)));
}

// Raw moments of the lane's velocities into its slots from m[off] (mask:
// per-velocity weight, a cell side's upwind share or a wall's outgoing half);
// ASSIGN: the slots of the moments are set, else added to.
// Moments about xi = 0 need no reference velocity per face or cell, and in
// ROW lanes the powers of xi_x are summed over the lane's velocities before
// the lane's xi_y, xi_z multiply them: 16 packed and ~14 scalar instructions
// per face and lane in 2D (40 packed and 11 scalar about a face velocity).
// The FP64 combination takes T and the heat flux as differences of sums that
// grow with the flow's U^2 and U^3.  L2 errors against FP64 after 6 steps,
// sums about the face's velocity -> about 0 (U in units of sqrt(2RT)):
//   24^2 quads x 28^2  U = 0.2: T 5.1e-9 -> 4.8e-9, q 3.2e-6 -> 3.9e-6
//                      U = 1:   T 3.0e-8 -> 4.6e-8, q 1.4e-6 -> 1.6e-6
//                      U = 2:   T 1.1e-7 -> 1.7e-7, q 1.1e-6 -> 1.9e-6
//   8^3 hexes x 12^3   U = 0.2: T 2.7e-8 -> 2.8e-8, q 3.2e-6 -> 3.5e-6
//                      U = 2:   T 1.3e-7 -> 1.2e-7, q 9.9e-7 -> 1.1e-6
template <int D, bool H, int NPL, bool ROW, int NS, bool ASSIGN = false>
__device__ __forceinline__ void mom32(float (&m)[NS], int off, const Lane32<D, NPL, ROW>& L, const float2 (&g)[NPL / 2],
                                      const float2 (&h)[NPL / 2], const float2* mask) {
    using SL = Slots32<D, H>;
    constexpr int NP = NPL / 2;
    auto put = [&](int slot, float v) {
        if (ASSIGN) m[off + slot] = v;
        else m[off + slot] += v;
    };
    if constexpr (ROW) {
        float2 s[4], t0, t1;  // sum w xi_x^j g, sum w h, sum w xi_x h
#pragma unroll
        for (int p = 0; p < NP; ++p) {  // pair 0 sets the packed sums, the others add
            const bool first = p == 0;
            float2 w = L.w[p];
            if (mask) w = mul2(w, mask[p]);
            float2 t = mul2(w, g[p]);
            s[0] = first ? t : add2(s[0], t);
            t = mul2(t, L.x[p]);
            s[1] = first ? t : add2(s[1], t);
            t = mul2(t, L.x[p]);
            s[2] = first ? t : add2(s[2], t);
            s[3] = first ? mul2(t, L.x[p]) : fma2(t, L.x[p], s[3]);
            if (H) {
                const float2 wh = mul2(w, h[p]);
                t0 = first ? wh : add2(t0, wh);
                t1 = first ? mul2(wh, L.x[p]) : fma2(wh, L.x[p], t1);
            }
        }
        const float y = L.y[0].x, z = L.z[0].x, r2 = D == 3 ? fmaf(z, z, y * y) : y * y;
        const float S0 = s[0].x + s[0].y, S1 = s[1].x + s[1].y, S2 = s[2].x + s[2].y, S3 = s[3].x + s[3].y;
        const float H0 = H ? t0.x + t0.y : 0.f, H1 = H ? t1.x + t1.y : 0.f;
        const float yS0 = y * S0;
        float E = fmaf(r2, S0, S2);  // sum w (|xi|^2 g + h)
        if (H) E += H0;
        put(0, S0);
        put(SL::M1, S1);
        put(SL::M1 + 1, yS0);
        put(SL::M2, S2);
        put(SL::M2 + 1, y * S1);
        put(SL::Q, fmaf(r2, S1, S3) + H1);
        put(SL::Q + 1, y * E);
        if (D == 2) {
            put(SL::M2 + 2, y * yS0);
        } else {
            const float zS0 = z * S0;
            put(SL::M1 + 2, zS0);
            put(SL::M2 + 2, z * S1);
            put(SL::M2 + 3, y * yS0);
            put(SL::M2 + 4, z * yS0);
            put(SL::M2 + 5, z * zS0);
            put(SL::Q + 2, z * E);
        }
        if (H) put(SL::H0, H0);
        return;
    } else {
        float2 m2[SL::NM];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const bool first = p == 0;
            const float2 c[3] = {L.x[p], L.y[p], L.z[p]};
            float2 w = L.w[p];
            if (mask) w = mul2(w, mask[p]);
            const float2 wg = mul2(w, g[p]);
            m2[0] = first ? wg : add2(m2[0], wg);
            float2 E = mul2(c[0], c[0]);
#pragma unroll
            for (int i = 1; i < D; ++i) E = fma2(c[i], c[i], E);
            E = mul2(E, wg);
            if (H) {
                const float2 wh = mul2(w, h[p]);
                m2[SL::H0] = first ? wh : add2(m2[SL::H0], wh);
                E = add2(E, wh);
            }
#pragma unroll
            for (int i = 0; i < D; ++i) {
                const float2 t = mul2(wg, c[i]);
                m2[SL::M1 + i] = first ? t : add2(m2[SL::M1 + i], t);
#pragma unroll
                for (int k = i; k < D; ++k) {
                    const int j = SL::M2 + sym<D>(i, k);
                    m2[j] = first ? mul2(t, c[k]) : fma2(t, c[k], m2[j]);
                }
                m2[SL::Q + i] = first ? mul2(E, c[i]) : fma2(E, c[i], m2[SL::Q + i]);
            }
        }
#pragma unroll
        for (int q = 0; q < SL::NM; ++q) put(q, m2[q].x + m2[q].y);
    }
}

// Macros from raw moment totals (FP64, Slots32 layout): rho, U, T, tau, the
// heat flux
//   q_i = fac/2 [Q_i - 2 M2_ij U_j - U_i (tr M2 + H0) + 2 M0 U_i |U|^2],
// fac = 2 tau / (2 tau + facA), and the FP32 equilibrium block (each entry
// rounded once).  Three FP64 divisions in all (1/rho, 1/RT, fac): a division
// is a chain of some ten FP64 instructions, and on small meshes these chains
// are what the macro steps take.
// FAST_TAU: the viscosity power (T/Tref)^omega by the FP32 hardware log2 /
// exp2 (relative error ~1e-7), for the face macros, whose relaxation weights
// are FP32 (the cell macros keep the FP64 power: the cell values are the
// reported fields).
template <int D, bool H, bool FAST_TAU>
__device__ __forceinline__ void macros32(const double* M, const StepArgs& b, double facA, double gs, double& rho,
                                         double* U, double& T, double& tau, double* q, double& fac, float* blk) {
    using SL = Slots32<D, H>;
    rho = M[0];
    const double irho = 1.0 / rho;
    double uu = 0.0, E = H ? M[SL::H0] : 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) U[i] = i < D ? M[SL::M1 + i] * irho : 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        E += M[SL::M2 + sym<D>(i, i)];
        uu += U[i] * U[i];
    }
    const double RT = (E * irho - uu) * b.iK3, iRT = 1.0 / RT;
    T = RT * b.iR;
    double p;
    if (FAST_TAU) {
        float pf;
        asm("lg2.approx.f32 %0, %1;" : "=f"(pf) : "f"((float)(T * b.iTref)));
        pf *= (float)b.omega;
        asm("ex2.approx.f32 %0, %1;" : "=f"(pf) : "f"(pf));
        p = (double)pf;
    } else {
        p = exp(b.omega * log(T * b.iTref));
    }
    tau = b.muRef * p * irho * iRT;
    fac = 2.0 * tau / (2.0 * tau + facA);
    const double s = 2.0 * rho * uu - E;
    const double qs = (1.0 - b.Pr) * 0.2 * irho * iRT * iRT;
    float qc[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 3; ++i) q[i] = 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        double m2u = 0.0;
#pragma unroll
        for (int j = 0; j < D; ++j) m2u += M[SL::M2 + (i <= j ? sym<D>(i, j) : sym<D>(j, i))] * U[j];
        q[i] = 0.5 * fac * (M[SL::Q + i] - 2.0 * m2u + U[i] * s);
        qc[i] = (float)(q[i] * qs);
    }
    const double t = iRT * (0.5 / kPi);  // 1/(2 pi RT)
    const double ipw = D == 2 ? t : t * sqrt(t);
    float4* o = reinterpret_cast<float4*>(blk);
    o[0] = make_float4((float)U[0], (float)U[1], (float)U[2], (float)(-0.72134752044448170 * iRT));  // -log2(e)/(2RT)
    o[1] = make_float4((float)iRT, qc[0], qc[1], qc[2]);
    o[2] = make_float4((float)(rho * gs * ipw), (float)RT, (float)tau, 0.0f);
}

// Face macros (FP64) from the deviation moment totals M of face a (wall w or
// -1): P4 Maxwell-wall density, P5 incoming wall moments, P6 face macros, wall
// heat flux and stress; then the face equilibrium table.
template <int D, bool H>
__device__ __forceinline__ void finalize_face32(const FusedArgs<float>& A, int a, int w, double* M) {
    using SL = Slots32<D, H>;
    constexpr int NS = SL::NS;
    const StepArgs& b = A.b;
    double rw = 0.0;
    if (w >= 0) {  // outgoing: deviation + reference parts; incoming: rho_w * Mw
        const double* RO = A.wallRefOut + (size_t)w * NS;
        for (int s = 0; s <= SL::FLUX; ++s) M[s] += RO[s];
        rw = M[SL::FLUX] / b.incAbs[w];
        for (int s = 0; s < SL::NM; ++s) M[s] += rw * A.Min[(size_t)w * NS + s];
    } else {
        for (int s = 0; s < SL::NM; ++s) M[s] += A.refMom[s];
    }
    for (int s = 0; s < SL::NM; ++s) M[s] *= A.invGscale;
    double rho, U[3], T, tau, q[3], fac;
    float* blk = A.fc + (size_t)a * kNCoef;
    macros32<D, H, true>(M, b, 0.5 * b.dt * b.Pr, A.gscale, rho, U, T, tau, q, fac, blk);
    b.rhoF[a] = rho;
    b.TF[a] = T;
    b.tauF[a] = tau;
    for (int k = 0; k < 3; ++k) { b.UF[3 * a + k] = U[k]; b.qF[3 * a + k] = q[k]; }
    if (A.feqT) eq_table(A.feqT + 3 * (size_t)a, blk, face_weight(A.dt, blk));
    if (w < 0) return;
    b.rhoW[w] = rw * A.invGscale;
    A.rhoWs[w] = (float)rw;
    const double fs = 2.0 * tau / (2.0 * tau + 0.5 * b.dt);
    // heat flux about the wall velocity u:
    //   1/2 [Q_i - 2 M2_ij u_j - u_i (tr M2 + H0) + M1_i |u|^2 + 2 u_i M1.u - u_i |u|^2 M0]
    const double* u = b.Uw + 3 * w;
    double uu = 0.0, m1u = 0.0, E = H ? M[SL::H0] : 0.0;
    for (int i = 0; i < D; ++i) {
        uu += u[i] * u[i];
        m1u += M[SL::M1 + i] * u[i];
        E += M[SL::M2 + sym<D>(i, i)];
    }
    for (int i = 0; i < 3; ++i) {
        double v = 0.0;
        if (i < D) {
            double m2u = 0.0;
            for (int j = 0; j < D; ++j) m2u += M[SL::M2 + (i <= j ? sym<D>(i, j) : sym<D>(j, i))] * u[j];
            v = 0.5 * (M[SL::Q + i] - 2.0 * m2u - u[i] * E + M[SL::M1 + i] * uu + 2.0 * u[i] * m1u - u[i] * uu * M[0]);
        }
        b.qWall[3 * w + i] = fac * v;
    }
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            b.stressWall[9 * w + 3 * i + j] =
                i < D && j < D ? fs * M[SL::M2 + (i <= j ? sym<D>(i, j) : sym<D>(j, i))] : 0.0;
}

// ---------------------------------------------------------------- sweep A, face sides
// One cell of T for one DV chunk (one warp): the least-squares gradient of
// gbar+ in registers (P2; a wall entry adds L_b G_b / deltaCoeff, the lagged
// boundary gradient), then for each face of the cell the upwind reconstruction
// from this side, gbar+_c + grad_c.(Cf - C_c - xi dt/2) (P3), stored for the
// velocities this side owns (xi.S_out > 0; tie values are never read: their
// flux is zero) and its raw moments with the upwind weights (ties half).  Wall
// faces store every velocity, their moments take the outgoing half, and
// grad.n becomes the next lagged gradient.  FG sides share one 32-slot warp
// reduction (31 shuffles for three triangle sides; 16 each apart), whose
// totals go into FP32 Kahan pairs per side and slot.
//
// A cell's rows are read once per chunk (1 + its neighbours) instead of twice
// per face: with one warp per face, both stencils summed per face, the sweep
// kept the shared-memory pipe busy on 77 % of the cycles (247 wavefronts per
// triangle and chunk; now 188).  Bound by issue and instruction latency at 16
// warps per SM (612 warp instructions per triangle and chunk, 57 % of issue
// slots).  20 or 24 warps per block: 0.83 / 1.05 ms against 0.80 on 100k
// triangles x 32^2.
//
// NF > 0: a cell of NF faces, none of them on the boundary: unrolled, without
// the boundary branches (705 -> 612 instructions per triangle and chunk; 100k
// triangles 0.80 -> 0.71 ms, 48^3 hexes 11.1 -> 10.3); NF = 0 takes every cell.
template <int D, bool H, int NPL, bool ROW, int NF>
__device__ __forceinline__ void cell_sides32(const FusedArgs<float>& A, const TileMeta32& tm, const Lane32<D, NPL, ROW>& L,
                                             const float* sg, const float* sh, int lc, int e0, int nfc, int lane, int v0,
                                             Acc<float>* mom) {
    using SL = Slots32<D, H>;
    constexpr int KC = 32 * NPL, NP = NPL / 2, P = SL::P, FG = SL::FG;
    const int Vp = A.b.Vp, col = lane * NPL;
    const int nf = NF > 0 ? NF : nfc;
    float2 c[NP], hc[NP], gg[D][NP], hg[D][NP];
    ldp<NP>(c, sg + lc * KC + col);
    if (H) ldp<NP>(hc, sh + lc * KC + col);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        if (!H) hc[p] = f2(0.f);
#pragma unroll
        for (int k = 0; k < D; ++k) { gg[k][p] = f2(0.f); hg[k][p] = f2(0.f); }
    }
    auto stencil = [&](int e) {
        const float4 ent = tm.E[3 * e];
        const int o = __float_as_int(ent.w);
        const float Lk[3] = {ent.x, ent.y, ent.z};
        float2 dg[NP], dh[NP];
        if (NF > 0 || o >= 0) {
            ldp<NP>(dg, sg + o * KC + col);
            if (H) ldp<NP>(dh, sh + o * KC + col);
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                dg[p] = sub2(dg[p], c[p]);
                if (H) dh[p] = sub2(dh[p], hc[p]);
            }
        } else {
            const int wf = -o - 1;
            const float idc = A.wall4[wf].y;
            ldp<NP>(dg, A.Gbg + (size_t)wf * Vp + v0 + col);
            if (H) ldp<NP>(dh, A.Gbh + (size_t)wf * Vp + v0 + col);
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                dg[p] = mul2(dg[p], f2(idc));
                if (H) dh[p] = mul2(dh[p], f2(idc));
            }
        }
#pragma unroll
        for (int k = 0; k < D; ++k)
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                gg[k][p] = fma2(f2(Lk[k]), dg[p], gg[k][p]);
                if (H) hg[k][p] = fma2(f2(Lk[k]), dh[p], hg[k][p]);
            }
    };
    if constexpr (NF > 0) {
#pragma unroll
        for (int j = 0; j < NF; ++j) stencil(e0 + j);
    } else {
        for (int j = 0; j < nf; ++j) stencil(e0 + j);
    }
    // one side into the slots m[off ..]
    auto side = [&](int e, auto& m, int off) {
        const float4 s4 = tm.E[3 * e + 1], d4 = tm.E[3 * e + 2];
        const int o = __float_as_int(tm.E[3 * e].w), a = __float_as_int(s4.w) >> 1;
        float2 xs[NP], gf[NP], hf[NP], wt[NP];
        Shift32<D, NPL, ROW> dk;
        dk.set(L, A.dt, d4.x, d4.y, d4.z);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            xs[p] = L.dot(p, s4.x, s4.y, s4.z);
            gf[p] = c[p];
            hf[p] = hc[p];
#pragma unroll
            for (int k = 0; k < D; ++k) {
                gf[p] = fma2(gg[k][p], dk.comp(k, p), gf[p]);
                if (H) hf[p] = fma2(hg[k][p], dk.comp(k, p), hf[p]);
            }
        }
        float* dg = A.gF + (size_t)a * Vp + v0 + col;
        float* dh = H ? A.hF + (size_t)a * Vp + v0 + col : nullptr;
        if (NF > 0 || o >= 0) {
            bool up[NPL], all = true;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                wt[p] = upwind_w2(xs[p]);
                up[2 * p] = xs[p].x > 0.f;
                up[2 * p + 1] = xs[p].y > 0.f;
                all = all && up[2 * p] && up[2 * p + 1];
            }
            if (all) {
                stp<NP>(dg, gf);
                if (H) stp<NP>(dh, hf);
            } else {
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    if (up[2 * p]) {
                        dg[2 * p] = gf[p].x;
                        if (H) dh[2 * p] = hf[p].x;
                    }
                    if (up[2 * p + 1]) {
                        dg[2 * p + 1] = gf[p].y;
                        if (H) dh[2 * p + 1] = hf[p].y;
                    }
                }
            }
            m[off + SL::FLUX] = 0.f;
        } else {  // boundary face
            const int w = -o - 1;
            const float nx = s4.x * d4.w, ny = s4.y * d4.w, nz = s4.z * d4.w;
            float2 gn[NP], hn[NP];
            float fl = 0.0f;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                gn[p] = fma2(gg[1][p], f2(ny), mul2(gg[0][p], f2(nx)));
                if (D == 3) gn[p] = fma2(gg[D - 1][p], f2(nz), gn[p]);
                if (H) {
                    hn[p] = fma2(hg[1][p], f2(ny), mul2(hg[0][p], f2(nx)));
                    if (D == 3) hn[p] = fma2(hg[D - 1][p], f2(nz), hn[p]);
                }
                wt[p] = make_float2(xs[p].x > 0.f ? 1.f : 0.f, xs[p].y > 0.f ? 1.f : 0.f);
                const float2 fx = mul2(mul2(mul2(L.w[p], xs[p]), gf[p]), wt[p]);
                fl += fx.x + fx.y;
            }
            const size_t wi = (size_t)w * Vp + v0 + col;
            stp<NP>(A.Gbgn + wi, gn);
            if (H) stp<NP>(A.Gbhn + wi, hn);
            stp<NP>(dg, gf);
            if (H) stp<NP>(dh, hf);
            m[off + SL::FLUX] = fl;
        }
        mom32<D, H, NPL, ROW, (int)(sizeof(m) / sizeof(float)), true>(m, off, L, gf, hf, wt);
    };
    const int s32 = slot_of<32>(lane), j32 = s32 / P;
    auto group = [&](int j, int n) {  // sides j .. j + n - 1, n <= FG
        float m[32];
#pragma unroll
        for (int s = FG * P; s < 32; ++s) m[s] = 0.f;
#pragma unroll
        for (int q = 0; q < FG; ++q) {
            if (q < n) side(e0 + j + q, m, q * P);
            else
#pragma unroll
                for (int s = 0; s < P; ++s) m[q * P + s] = 0.f;
        }
        const float tot = reduce_scatter<32, float, FG * P>(m, lane);
        if (j32 < n) mom[(size_t)(e0 + j) * P + s32].add(tot);
    };
    auto single = [&](int j) {
        float m[16];
#pragma unroll
        for (int s = P; s < 16; ++s) m[s] = 0.f;
        side(e0 + j, m, 0);
        const float tot = reduce_scatter<16, float, P>(m, lane);
        const int s16 = slot_of<16>(lane);
        if ((lane & 1) == 0 && s16 < P) mom[(size_t)(e0 + j) * P + s16].add(tot);
    };
    if constexpr (NF > 0) {
#pragma unroll
        for (int j = 0; j + 1 < NF; j += FG) group(j, NF - j < FG ? NF - j : FG);
        if constexpr (NF % FG == 1) single(NF - 1);
    } else {
        int j = 0;
        for (; j + 1 < nf; j += FG) group(j, min(FG, nf - j));
        if (j < nf) single(j);
    }
}

// Sweep A on tiles with a one-ring halo (rows of T u H1): every cell of T
// forms its sides of its faces (cell_sides32); the other side of a face is
// formed by the other cell's warp or tile.  Per-side moment totals go to
// faceMom[a][side] (side 0: owner or boundary face) and k_face_macros32 forms
// the face macros.  Raw rows of the next DV chunk stream into the second row
// buffer while this chunk's cells run.
// BESIDE: the kernel was started beside the one before it; tile data are constant.
template <int D, bool H, int NPL, int NW, bool ROW, bool BESIDE = false>
__device__ __forceinline__ void face_sides_body(const FusedArgs<float>& A, int tile, unsigned char* smem) {
    using SL = Slots32<D, H>;
    constexpr int KC = 32 * NPL, P = SL::P;
    const TileHdr hd = A.hdr[tile];
    const StepArgs& b = A.b;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int Vp = b.Vp;
    using LY = SmemLayout32<D, H, NPL>;
    float* const rowBase = reinterpret_cast<float*>(smem);
    const size_t nRK = (size_t)hd.nT2 * KC;
    auto rowsG = [&](int bf) { return rowBase + (size_t)bf * (H ? 2 : 1) * nRK; };  // g rows, then h rows
    Acc<float>* mom = reinterpret_cast<Acc<float>*>(smem + LY::mom(hd.nT2));
    for (int i = threadIdx.x; i < hd.nEnt * P; i += NW * 32) mom[i].zero();
    const TileMeta32 tm = stage_meta<NW * 32>(A, hd, tile, smem + LY::meta(hd.nT2, hd.nEnt));
    float4* ceq = tm.dyn;  // [nT2][3] cell equilibria
    __syncthreads();
    if (BESIDE) after_previous();
#if defined(DUGKS_CHECKED) && DUGKS_CHECKED
    check_tile_meta32<NW * 32>(A, hd, smem + LY::meta(hd.nT2, hd.nEnt));
    __syncthreads();
#endif
    for (int i = threadIdx.x; i < hd.nT2; i += NW * 32) {
        const float* blk = A.cc + (size_t)tm.C[i] * kNCoef;
        eq_table(ceq + 3 * i, blk, cell_weight(A.dt, blk));
    }
    const RowPart rp = row_part<D, NW>(hd, warp);
    issue_rows32<NPL, H>(A, rp, tm.C, rowsG(0), rowsG(0) + nRK, 0, lane);
    const int nChunks = Vp / KC;
    __syncthreads();  // cell equilibria

    // One block barrier per chunk: a warp relaxes the rows it copied itself
    // as soon as its copies have landed (a warp still in the previous
    // chunk's cells reads the other buffer), the barrier after the
    // relaxation releases the cells, and only then are the next chunk's
    // rows copied into the buffer that the previous chunk's cells read.
    for (int ch = 0; ch < nChunks; ++ch) {
        const int v0 = ch * KC;
        Lane32<D, NPL, ROW> L;
        L.load(A, v0, lane);
        cp_async_wait<0>();
        __syncwarp();
        float* cg = rowsG(ch & 1);
        float* chh = cg + nRK;
        relax_rows32<D, H, NPL, ROW>(A, rp, ceq, L, lane, cg, chh);
        __syncthreads();
        if (ch + 1 < nChunks) {
            float* ng = rowsG((ch + 1) & 1);
            issue_rows32<NPL, H>(A, rp, tm.C, ng, ng + nRK, v0 + KC, lane);
        }
        for (int lc = warp; lc < hd.nT; lc += NW) {
            const int s0 = tm.S[lc], e0 = s0 >> 1, nf = (tm.S[lc + 1] >> 1) - e0;
            constexpr int N1 = D == 2 ? 3 : 6;
            if ((s0 & 1) && nf == N1) cell_sides32<D, H, NPL, ROW, N1>(A, tm, L, cg, chh, lc, e0, nf, lane, v0, mom);
            else if ((s0 & 1) && nf == 4) cell_sides32<D, H, NPL, ROW, 4>(A, tm, L, cg, chh, lc, e0, nf, lane, v0, mom);
            else cell_sides32<D, H, NPL, ROW, 0>(A, tm, L, cg, chh, lc, e0, nf, lane, v0, mom);
        }
    }
    __syncthreads();
    // ---- per-side totals (FP64) to faceMom[a][side]
    for (int i = threadIdx.x; i < hd.nEnt * P; i += NW * 32) {
        const int e = i / P, s = i - e * P;
        const int f = __float_as_int(tm.E[3 * e + 1].w);
        double* dst = A.faceMom + ((size_t)(f >> 1) * 2 + (f & 1)) * SL::NS + s;
        *dst = mom[i].value();
        if (__float_as_int(tm.E[3 * e].w) < 0) dst[SL::NS] = 0.0;  // boundary: no other side
    }
}

template <int D, bool H, int NPL, int NW, bool ROW>
__global__ void __launch_bounds__(NW * 32, 1) k_face_sides32(FusedArgs<float> A) {
    extern __shared__ __align__(16) unsigned char smem[];
    face_sides_body<D, H, NPL, NW, ROW, true>(A, blockIdx.x, smem);
}

// Several independent cases in one launch: block b runs tile work[b].y of
// case work[b].x.  The cases' arguments are read through a read-only
// pointer; every case shares D, H and NPL.
template <int D, bool H, int NPL, int NW>
__global__ void __launch_bounds__(NW * 32, 1) k_face_sides32_batch(const FusedArgs<float>* __restrict__ AA,
                                                                   const int2* __restrict__ work) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ FusedArgs<float> sA;
    const int2 w = work[blockIdx.x];
    {
        const long long* src = reinterpret_cast<const long long*>(AA + w.x);
        long long* dst = reinterpret_cast<long long*>(&sA);
        for (int k = threadIdx.x; k < (int)(sizeof(FusedArgs<float>) / 8); k += blockDim.x) dst[k] = src[k];
    }
    __syncthreads();
    if (sA.b.M % NPL == 0) face_sides_body<D, H, NPL, NW, true>(sA, w.y, smem);
    else face_sides_body<D, H, NPL, NW, false>(sA, w.y, smem);
}

// Open boundary faces (zeroGradient, fixedValue -> mixed, farField, pressureIn,
// pressureOut), one warp per face, after sweep A stored their owner-side
// reconstruction for every velocity: the complete face values (deviation
// form) and their moments over all velocities, so that the face macros take
// the internal-face path.  zeroGradient: every velocity takes the owner's
// gbar+ (discreteVelocity.C:551-555); the others keep the outgoing
// reconstruction and set the incoming velocities (xi.S <= 0) to
// rho_b M(U of the owner cell, T_b) (:570-600) -- fixedValue to the
// Maxwellian of its patch rho, U, T, which stays as it was at the start
// (:302-345).  Symmetry faces (symmetryMod, symmetryPlane): the incoming
// velocities (xi.S0 <= 0, S0 the patch's first face) take their mirror
// velocity's value (discreteVelocity.C:733-817), read from a snapshot of the
// face row; symmetryPlane assigns in index order, so a mirror that is itself
// an earlier incoming velocity passes its own mirror's value on (the chain
// ends after one step on grids symmetric about 0).  A separate kernel keeps
// the sweep's code unchanged.
template <int D, bool H, int NPL>
__global__ void k_open_faces32(FusedArgs<float> A) {
    using SL = Slots32<D, H>;
    constexpr int NS = SL::NS, KC = 32 * NPL, NP = NPL / 2;
    const StepArgs& b = A.b;
    const int lane = threadIdx.x & 31, Vp = b.Vp, col = lane * NPL;
    const int myslot = slot_of<NS>(lane);
    const bool writer = NS == 16 ? (lane & 1) == 0 : true;
    for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < b.nW; w += gridDim.x * (blockDim.x >> 5)) {
        const int kind = b.bKind[w];
        if (kind == kBcMaxwell) continue;  // warp-uniform
        const int a = b.nI + w, own = chk(b.own[a], b.nC, b.status);
        const float sx = (float)b.Sf[3 * a], sy = (float)b.Sf[3 * a + 1], sz = (float)b.Sf[3 * a + 2];
        // xi.S rounded as in the sweep and the gather, which take ROW lanes on such grids: a
        // velocity within FP32 rounding of an oblique face (0.1 % of 20^3 velocities on lattice
        // directions) is incoming here and there alike
        const bool row = b.M % NPL == 0;
        Eq32<D, H> ec;
        float ng = 0.f, i2 = 0.f, hw = 0.f, ux = 0.f, uy = 0.f, uz = 0.f;
        const bool sym = kind == kBcSymmetryMod || kind == kBcSymmetryPlane;
        const double* S0 = b.bS0 + 3 * w;
        auto incoming = [&](int u) {
            return b.xi[u] * S0[0] + b.xi[Vp + u] * S0[1] + b.xi[2 * Vp + u] * S0[2] <= 0;
        };
        if (sym) {  // snapshot of the row
            const size_t fb = (size_t)a * Vp, wb = (size_t)w * Vp;
            for (int v = lane; v < Vp; v += 32) {
                A.symG[wb + v] = A.gF[fb + v];
                if (H) A.symH[wb + v] = A.hF[fb + v];
            }
            __syncwarp();
        } else if (kind == kBcZeroGradient) {
            const float* cblk = A.cc + (size_t)own * kNCoef;
            float4 q[3];
            eq_table(q, cblk, cell_weight(A.dt, cblk));
            ec.load(q, b.K, A.hrefFac);
        } else {
            const double Tb = b.TbM[w], RT = b.R * Tb;
            const double* U = kind == kBcFixedValue ? b.Uw + 3 * w : b.U + 3 * own;
            const double sq = sqrt(2.0 * kPi * RT);
            ng = (float)(A.gscale * b.rhoB[w] / (D == 2 ? sq * sq : sq * sq * sq));
            i2 = (float)(-0.5 / RT);
            hw = (float)(RT * (b.K + 3 - D));
            ux = (float)U[0]; uy = (float)U[1]; uz = (float)U[2];
        }
        Acc<float> acc;
        acc.zero();
        for (int v0 = 0; v0 < Vp; v0 += KC) {
            Lane32<D, NPL, false> L;
            L.load(A, v0, lane);
            const size_t fi = (size_t)a * Vp + v0 + col;
            float2 gf[NP], hf[NP];
            if (sym) {
                ldp<NP>(gf, A.gF + fi);
                if (H) ldp<NP>(hf, A.hF + fi);
                float* gs = reinterpret_cast<float*>(gf);
                float* hs = reinterpret_cast<float*>(hf);
                const int* tab = b.symTab + (size_t)b.symOff[w] * b.nV;
                const float* snG = A.symG + (size_t)w * Vp;
                const float* snH = H ? A.symH + (size_t)w * Vp : nullptr;
#pragma unroll
                for (int j = 0; j < NPL; ++j) {
                    const int v = v0 + col + j;
                    if (v >= b.nV || !incoming(v)) continue;
                    int cur = v, u = chk(tab[v], b.nV, b.status);
                    if (kind == kBcSymmetryPlane)
                        for (int guard = 0; guard < b.nV && u < cur && incoming(u); ++guard) {
                            cur = u;
                            u = chk(tab[u], b.nV, b.status);
                        }
                    gs[j] = snG[u];
                    if (H) hs[j] = snH[u];
                }
                if (!H)
#pragma unroll
                    for (int p = 0; p < NP; ++p) hf[p] = f2(0.f);
            } else if (kind == kBcZeroGradient) {
                const size_t ci = (size_t)own * Vp + v0 + col;
                ldp<NP>(gf, A.gT + ci);
                if (H) ldp<NP>(hf, A.hT + ci);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    if (!H) hf[p] = f2(0.f);
                    ec.relax(L, p, gf[p], hf[p]);
                }
            } else {
                ldp<NP>(gf, A.gF + fi);
                if (H) ldp<NP>(hf, A.hF + fi);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const float2 xs = row ? L.dot_row(p, sx, sy, sz) : L.dot(p, sx, sy, sz);
                    const float2 cx = sub2(L.x[p], f2(ux)), cy = sub2(L.y[p], f2(uy));
                    float2 cc = fma2(cy, cy, mul2(cx, cx));
                    if (D == 3) {
                        const float2 cz = sub2(L.z[p], f2(uz));
                        cc = fma2(cz, cz, cc);
                    }
                    const float2 m = make_float2(ng * expf(i2 * cc.x), ng * expf(i2 * cc.y));
                    const bool o0 = xs.x > 0.f, o1 = xs.y > 0.f;
                    gf[p] = sel2(o0, o1, gf[p], sub2(m, L.mr[p]));
                    if (H) hf[p] = sel2(o0, o1, hf[p], sub2(mul2(m, f2(hw)), mul2(L.mr[p], f2(A.hrefFac))));
                }
            }
            stp<NP>(A.gF + fi, gf);
            if (H) stp<NP>(A.hF + fi, hf);
            float m[NS];
#pragma unroll
            for (int s2 = 0; s2 < NS; ++s2) m[s2] = 0.0f;
            mom32<D, H, NPL, false, NS>(m, 0, L, gf, hf, nullptr);
            acc.add(reduce_scatter<NS, float, SL::FLUX + 1>(m, lane));
        }
        double* dst = A.faceMom + (size_t)a * 2 * NS;
        if (writer && myslot < NS) {
            dst[myslot] = myslot < SL::FLUX ? acc.value() : 0.0;
            dst[NS + myslot] = 0.0;
        }
    }
}

// Face macros of every active face from the two per-side moment totals.
template <int D, bool H>
__device__ __forceinline__ void face_macros_one(const FusedArgs<float>& A, int a) {
    using SL = Slots32<D, H>;
    const double* src = A.faceMom + (size_t)a * 2 * SL::NS;
    double M[SL::NS];
#pragma unroll
    for (int s = 0; s <= SL::FLUX; ++s) M[s] = src[s] + src[SL::NS + s];
    const int w = a >= A.b.nI && A.b.bKind[a - A.b.nI] == kBcMaxwell ? a - A.b.nI : -1;
    finalize_face32<D, H>(A, a, w, M);
}

template <int D, bool H>
__global__ void k_face_macros32(FusedArgs<float> A) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < A.b.nA; a += gridDim.x * blockDim.x)
        face_macros_one<D, H>(A, a);
}

// Case of a global item index: off[] holds the first item of each case (n+1 entries).
__device__ __forceinline__ int case_of(const int* __restrict__ off, int n, int g) {
    int lo = 0, hi = n;  // off[lo] <= g < off[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <int D, bool H>
__global__ void k_face_macros32_batch(const FusedArgs<float>* __restrict__ AA, const int* __restrict__ faceOff,
                                      int nCases) {
    const int total = faceOff[nCases];
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const int i = case_of(faceOff, nCases, g);
        face_macros_one<D, H>(AA[i], g - faceOff[i]);
    }
}

// ---------------------------------------------------------------- sweep B, gather form
// Shared memory of the gather sweep: per warp two stages of (1 + MF) rows of
// g (and h): the cell's g~ row and its first MF faces' stored values.
__host__ __device__ inline size_t gather_smem(int nw, int mf, int kc, bool h) {
    return (size_t)nw * 2 * (1 + mf) * (h ? 2 : 1) * kc * sizeof(float);
}

// Cell macros (FP64) from the deviation moment totals (slots as Slots32).
template <int D, bool H, typename TT = double>
__device__ __forceinline__ void finalize_cell32(const FusedArgs<float>& A, int c, const TT* tot) {
    using SL = Slots32<D, H>;
    const StepArgs& b = A.b;
    double M[SL::NM];
#pragma unroll
    for (int s = 0; s < SL::NM; ++s) M[s] = (tot[s] + A.refMom[s]) * A.invGscale;
    double rho, U[3], T, tau, q[3], fac;
    macros32<D, H, false>(M, b, b.dt * b.Pr, A.gscale, rho, U, T, tau, q, fac, A.ccn + (size_t)c * kNCoef);
    A.rhoN[c] = rho;
    A.TN[c] = T;
    A.tauN[c] = tau;
    for (int k = 0; k < 3; ++k) { A.UN[3 * c + k] = U[k]; A.qN[3 * c + k] = q[k]; }
    if (!(rho > 0.0) || !(T > 0.0) || !isfinite(U[0] + U[1] + U[2] + q[0] + q[1] + q[2])) atomicExch(b.status, 5);
}

// Cells per warp batch of the gather sweep's FP64 macro step (one lane per cell).
constexpr int kGatherBatch = 32;

// Cells left in the warps' last, partly filled batches (n < B each) are
// finished by the whole block, one thread per cell: finish(warp, place).  A
// warp that finished its own few cells held the FP64 pipe as long as one with
// 32 (61^2 quads: 1.5 cells per warp, 16 warps per SM: 61 -> 50 us per sweep).
// The counts go into the batches' last places, ids[w * B + B - 1]: 32 bytes
// more of shared memory would cost the two blocks of an SM half of the L1
// (100k triangles: 0.62 -> 0.73 ms).
template <int NW, int B, class F>
__device__ __forceinline__ void finish_rest(int n, int* ids, F&& finish) {
    if ((threadIdx.x & 31) == 0) ids[(threadIdx.x >> 5) * B + B - 1] = n;
    __syncthreads();
    int t = threadIdx.x, w = 0;
    while (w < NW && t >= ids[w * B + B - 1]) t -= ids[w++ * B + B - 1];
    if (w < NW) finish(w, t);
}

// One cell of NF faces, none of them on the boundary: gather_cell with the
// faces unrolled, their indices in registers and rows addressed by 32-bit
// counts of NPL floats (the host marks such cells, A.cfKind, when every row
// fits): 527 -> 344 warp instructions per triangle and chunk, 100k triangles
// x 32^2 0.61 -> 0.55 ms, where DRAM moves 5.1 TB/s; 48^3 hexes x 20^3 6.96 ->
// 6.09 ms.
template <int D, bool H, int NPL, bool ROW, int NF>
__device__ __forceinline__ float gather_inner(const FusedArgs<float>& A, int c, int MF, float* wb, int lane,
                                              const float* tab) {
    using SL = Slots32<D, H>;
    using Row = typename std::conditional<NPL == 4, float4, float2>::type;
    constexpr int NS = SL::NS, KC = 32 * NPL, NP = NPL / 2, NR = H ? 2 : 1;
    const StepArgs& b = A.b;
    const int Vp = b.Vp;
    const unsigned Vq = (unsigned)Vp / NPL, rc = (unsigned)c * Vq + lane;
    const int stageFloats = (1 + MF) * NR * KC;
    const float4* ce = A.cfEnt + A.cfOff[c];
    int a[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) a[f] = chk(__float_as_int(ce[f].w), b.nA, b.status);
    const Row *gT = reinterpret_cast<const Row*>(A.gT), *hT = reinterpret_cast<const Row*>(A.hT),
              *gF = reinterpret_cast<const Row*>(A.gF), *hF = reinterpret_cast<const Row*>(A.hF);
    auto issue = [&](int stage, unsigned q) {
        float* st = wb + stage * stageFloats;
        cp_async_row(st, reinterpret_cast<const float*>(gT + (rc + q)), NPL);
        if (H) cp_async_row(st + KC, reinterpret_cast<const float*>(hT + (rc + q)), NPL);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const unsigned r = (unsigned)a[f] * Vq + (lane + q);
            cp_async_row(st + (1 + f) * NR * KC, reinterpret_cast<const float*>(gF + r), NPL);
            if (H) cp_async_row(st + ((1 + f) * NR + 1) * KC, reinterpret_cast<const float*>(hF + r), NPL);
        }
        cp_async_commit();
    };
    const float* cblk = A.cc + (size_t)c * kNCoef;
    Eq32<D, H> ec;
    {
        float4 q[3];
        eq_table(q, cblk, cell_weight(A.dt, cblk));
        ec.load(q, b.K, A.hrefFac);
    }
    const float kv = -A.dt * A.invVf[c];
    float m[NS];
#pragma unroll
    for (int s2 = 0; s2 < NS; ++s2) m[s2] = 0.0f;
    const int nChunks = Vp / KC;
    issue(0, 0);
    for (int ch = 0; ch < nChunks; ++ch) {
        if (ch + 1 < nChunks) {
            issue((ch + 1) & 1, 32u * (ch + 1));
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        const float* st = wb + (ch & 1) * stageFloats;
        Lane32<D, NPL, ROW> L;
        if (tab) L.load_tab(tab, Vp, ch * KC, lane);
        else L.load(A, ch * KC, lane);
        float2 g0[NP], h0[NP], t[NP], th[NP];
        ldp<NP>(g0, st);
        if (H) ldp<NP>(h0, st + KC);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            float2 g = g0[p], h = H ? h0[p] : f2(0.f);
            ec.relax(L, p, g, h);
            t[p] = fma2(sub2(g, g0[p]), f2(1.0f / 3.0f), g);  // exact when g+ == g~
            th[p] = H ? fma2(sub2(h, h0[p]), f2(1.0f / 3.0f), h) : f2(0.f);
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const float4 ent = ce[f];
            float2 gf[NP], hf[NP];
            ldp<NP>(gf, st + (1 + f) * NR * KC);
            if (H) ldp<NP>(hf, st + ((1 + f) * NR + 1) * KC);
            Eq32<D, H> eq;
            eq.load(A.feqT + 3 * (size_t)a[f], b.K, A.hrefFac);
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                if (!H) hf[p] = f2(0.f);
                eq.relax(L, p, gf[p], hf[p]);
                const float2 kx = L.lin(p, kv * ent.x, kv * ent.y, kv * ent.z);
                t[p] = fma2(kx, gf[p], t[p]);
                if (H) th[p] = fma2(kx, hf[p], th[p]);
            }
        }
        stp_cs<NP>(A.gTn + (size_t)(rc + 32u * ch) * NPL, t);
        if (H) stp_cs<NP>(A.hTn + (size_t)(rc + 32u * ch) * NPL, th);
        mom32<D, H, NPL, ROW, NS>(m, 0, L, t, th, nullptr);
    }
    return reduce_scatter<NS, float, SL::NM>(m, lane);
}

// One cell of the gather sweep, all DV chunks; returns this lane's slot total
// of the new cell moments (slot slot_of(lane)).  wb: the warp's two stages,
// offset by the lane's column.
// OPEN: the case has open boundary faces (instantiated apart so that
// wall-only cases run the same code as before those existed).
// tab: the velocity constants in shared memory (dv_table32), or null.
template <int D, bool H, int NPL, bool ROW, bool OPEN = false>
__device__ __forceinline__ float gather_cell(const FusedArgs<float>& A, int c, int MF, float* wb, int lane,
                                             const float* tab = nullptr) {
    using SL = Slots32<D, H>;
    constexpr int NS = SL::NS, KC = 32 * NPL, NP = NPL / 2, NR = H ? 2 : 1;
    const StepArgs& b = A.b;
    const int Vp = b.Vp, col = lane * NPL;
    constexpr int N1 = D == 2 ? 3 : 6;
    const int kind = A.cfKind[c];
    if (kind == N1) return gather_inner<D, H, NPL, ROW, N1>(A, c, MF, wb, lane, tab);
    if (kind == 4) return gather_inner<D, H, NPL, ROW, 4>(A, c, MF, wb, lane, tab);
    const int stageRows = (1 + MF) * NR;
    const int e0 = A.cfOff[c], e1 = A.cfOff[c + 1];
    const int nfs = min(e1 - e0, MF);  // faces staged through shared memory
    auto issue = [&](int stage, int v0) {
        float* st = wb + (size_t)stage * stageRows * KC;
        const size_t gi = (size_t)c * Vp + v0 + col;
        cp_async_row(st, A.gT + gi, NPL);
        if (H) cp_async_row(st + KC, A.hT + gi, NPL);
        for (int f = 0; f < nfs; ++f) {
            const int a = chk(__float_as_int(A.cfEnt[e0 + f].w), b.nA, b.status);
            const size_t fi = (size_t)a * Vp + v0 + col;
            cp_async_row(st + (1 + f) * NR * KC, A.gF + fi, NPL);
            if (H) cp_async_row(st + ((1 + f) * NR + 1) * KC, A.hF + fi, NPL);
        }
        cp_async_commit();
    };
    const float* cblk = A.cc + (size_t)c * kNCoef;
    Eq32<D, H> ec;
    {
        float4 q[3];
        eq_table(q, cblk, cell_weight(A.dt, cblk));
        ec.load(q, b.K, A.hrefFac);
    }
    const float kv = -A.dt * A.invVf[c];
    // cell moments: per-lane partial sums over all chunks, one warp reduction per cell
    float m[NS];
#pragma unroll
    for (int s2 = 0; s2 < NS; ++s2) m[s2] = 0.0f;
    const int nChunks = Vp / KC;
    issue(0, 0);
    for (int ch = 0; ch < nChunks; ++ch) {
        const int v0 = ch * KC;
        if (ch + 1 < nChunks) {
            issue((ch + 1) & 1, v0 + KC);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        const float* st = wb + (size_t)(ch & 1) * stageRows * KC;
        Lane32<D, NPL, ROW> L;
        if (tab) L.load_tab(tab, Vp, v0, lane);
        else L.load(A, v0, lane);
        float2 g0[NP], h0[NP], t[NP], th[NP];
        ldp<NP>(g0, st);
        if (H) ldp<NP>(h0, st + KC);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            float2 g = g0[p], h = H ? h0[p] : f2(0.f);
            ec.relax(L, p, g, h);
            t[p] = fma2(sub2(g, g0[p]), f2(1.0f / 3.0f), g);  // exact when g+ == g~
            th[p] = H ? fma2(sub2(h, h0[p]), f2(1.0f / 3.0f), h) : f2(0.f);
        }
#pragma unroll 3  // a triangle's three faces: independent relaxations interleave
        for (int e = e0; e < e1; ++e) {
            const int f = e - e0;
            const float4 ent = A.cfEnt[e];
            const int a = chk(__float_as_int(ent.w), b.nA, b.status);
            float2 gf[NP], hf[NP];
            if (f < nfs) {
                ldp<NP>(gf, st + (1 + f) * NR * KC);
                if (H) ldp<NP>(hf, st + ((1 + f) * NR + 1) * KC);
            } else {
                const size_t fi = (size_t)a * Vp + v0 + col;
                ldp<NP>(gf, A.gF + fi);
                if (H) ldp<NP>(hf, A.hF + fi);
            }
            if (!H)
#pragma unroll
                for (int p = 0; p < NP; ++p) hf[p] = f2(0.f);
            Eq32<D, H> eq;
            eq.load(A.feqT + 3 * (size_t)a, b.K, A.hrefFac);
            if (a >= b.nI) {  // boundary: the cell is the owner; outgoing where xi.S > 0
                const int w = a - b.nI;
                const float4 w4 = A.wall4[w];
                if (OPEN && w4.z != 0.f) {  // open boundary: incoming stored, unrelaxed
                    const bool plane = w4.z == 2.f;  // symmetryPlane: every DV once, outgoing twice
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        if (plane) eq.relax(L, p, gf[p], hf[p]);
                        float2 go = gf[p], ho = hf[p];
                        eq.relax(L, p, go, ho);
                        const float2 xs = L.dot(p, ent.x, ent.y, ent.z);
                        const bool o0 = xs.x > 0.f, o1 = xs.y > 0.f;
                        gf[p] = sel2(o0, o1, go, gf[p]);
                        if (H) hf[p] = sel2(o0, o1, ho, hf[p]);
                    }
                } else {  // diffuse wall: incoming rho_w Mw
                    const float rws = A.rhoWs[w], hwf = w4.x;
                    float2 mw[NP];
                    ldp<NP>(mw, A.Mw + (size_t)w * Vp + v0 + col);
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        float2 go = gf[p], ho = hf[p];
                        eq.relax(L, p, go, ho);
                        const float2 gw = mul2(f2(rws), mw[p]);
                        const float2 xs = L.dot(p, ent.x, ent.y, ent.z);
                        const bool o0 = xs.x > 0.f, o1 = xs.y > 0.f;
                        gf[p] = sel2(o0, o1, go, sub2(gw, L.mr[p]));
                        if (H) hf[p] = sel2(o0, o1, ho, sub2(mul2(gw, f2(hwf)), mul2(L.mr[p], f2(A.hrefFac))));
                    }
                }
            } else {
#pragma unroll
                for (int p = 0; p < NP; ++p) eq.relax(L, p, gf[p], hf[p]);
            }
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const float2 kx = L.lin(p, kv * ent.x, kv * ent.y, kv * ent.z);
                t[p] = fma2(kx, gf[p], t[p]);
                if (H) th[p] = fma2(kx, hf[p], th[p]);
            }
        }
        const size_t gi = (size_t)c * Vp + v0 + col;
        stp_cs<NP>(A.gTn + gi, t);
        if (H) stp_cs<NP>(A.hTn + gi, th);
        mom32<D, H, NPL, ROW, NS>(m, 0, L, t, th, nullptr);
    }
    return reduce_scatter<NS, float, SL::NM>(m, lane);
}

// Warps stride over the cells (persistent grid); per cell, all DV chunks:
//   g~new = g+ + (g+ - g~)/3 - dt/V sum_f (xi.S_f) g^f_f,
// with g+ the cell relaxation of g~ (P1), g^f_f the face value stored by
// sweep A relaxed toward the face equilibrium (P7; incoming wall DVs take
// rho_w Mw unrelaxed) and the sum over the cell's faces in face order (P8),
// then the cell moments (P9).  Faces are relaxed once from each side; no
// tiles or block barriers.  The rows of chunk k+1 are copied into the warp's
// other stage while chunk k is computed; the FP64 macros of a batch of cells
// are finished together, one lane per cell.
// dvTab: the launch gave room after the stages for the velocity constants
// (dv_table32), read from there per chunk instead of from global memory.
// The batch of warp totals is kept in FP32: each total is an FP32 warp sum.
template <int D, bool H, int NPL, int NW, bool ROW, bool OPEN = false>
__global__ void __launch_bounds__(NW * 32, 2) k_cell_gather32(FusedArgs<float> A, int MF, int dvTab) {
    constexpr int NS = Slots32<D, H>::NS, KC = 32 * NPL, NR = H ? 2 : 1;
    // 3D: half the batch -- the finalize is a small share of a 63-chunk cell,
    // and the smaller buffer leaves the L1 more room (8.40 -> 8.21 ms, 48^3 hexes)
    constexpr int GB = D == 3 ? kGatherBatch / 2 : kGatherBatch;
    __shared__ float sM[NW][GB][NS];
    __shared__ int sC[NW][GB];
    extern __shared__ __align__(16) float gsm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* wb = gsm + (size_t)warp * 2 * (1 + MF) * NR * KC + lane * NPL;
    early();
    float* tab = nullptr;
    if (dvTab) {
        tab = gsm + gather_smem(NW, MF, KC, H) / sizeof(float);
        dv_table32<D>(A, tab);
        __syncthreads();
    }
    const int myslot = slot_of<NS>(lane);
    const bool writer = NS == 16 ? (lane & 1) == 0 : true;
    const int TW = gridDim.x * NW, nC = A.b.nC;
    int nb = 0;
    for (int i = blockIdx.x * NW + warp; i < nC; i += TW) {
        const int c = A.cellOrd[i];
        const float tot = gather_cell<D, H, NPL, ROW, OPEN>(A, c, MF, wb, lane, tab);
        if (writer) sM[warp][nb][myslot] = tot;
        if (lane == 0) sC[warp][nb] = c;
        if (++nb == GB) {
            __syncwarp();
            if (lane < nb) finalize_cell32<D, H>(A, sC[warp][lane], sM[warp][lane]);
            __syncwarp();
            nb = 0;
        }
    }
    finish_rest<NW, GB>(nb, &sC[0][0], [&](int w, int k) { finalize_cell32<D, H>(A, sC[w][k], sM[w][k]); });
}

// Several independent cases in one launch: warps stride over the cells of
// all cases (cellOff: first global cell of each case, nCases+1 entries).
template <int D, bool H, int NPL, int NW>
__global__ void __launch_bounds__(NW * 32, 2) k_cell_gather32_batch(const FusedArgs<float>* __restrict__ AA,
                                                                    const int* __restrict__ cellOff, int nCases, int MF) {
    constexpr int NS = Slots32<D, H>::NS, KC = 32 * NPL, NR = H ? 2 : 1;
    __shared__ float sM[NW][kGatherBatch][NS];  // FP32 warp totals, exact
    __shared__ int sC[NW][kGatherBatch], sI[NW][kGatherBatch];
    __shared__ FusedArgs<float> sA[NW];  // the warp's current case
    extern __shared__ __align__(16) float gsm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* wb = gsm + (size_t)warp * 2 * (1 + MF) * NR * KC + lane * NPL;
    const int myslot = slot_of<NS>(lane);
    const bool writer = NS == 16 ? (lane & 1) == 0 : true;
    const int TW = gridDim.x * NW, total = cellOff[nCases];
    int nb = 0, cur = -1;
    for (int g = blockIdx.x * NW + warp; g < total; g += TW) {
        const int i = case_of(cellOff, nCases, g), k0 = g - cellOff[i];
        if (i != cur) {  // consecutive cells mostly share a case: copy its arguments once
            static_assert(sizeof(FusedArgs<float>) % 8 == 0, "argument block is copied in 8-byte words");
            const long long* src = reinterpret_cast<const long long*>(AA + i);
            long long* dst = reinterpret_cast<long long*>(&sA[warp]);
            __syncwarp();
            for (int k = lane; k < (int)(sizeof(FusedArgs<float>) / 8); k += 32) dst[k] = src[k];
            __syncwarp();
            cur = i;
        }
        const int c = sA[warp].cellOrd[k0];
        const float tot = sA[warp].b.M % NPL == 0 ? gather_cell<D, H, NPL, true>(sA[warp], c, MF, wb, lane)
                                                   : gather_cell<D, H, NPL, false>(sA[warp], c, MF, wb, lane);
        if (writer) sM[warp][nb][myslot] = tot;
        if (lane == 0) { sC[warp][nb] = c; sI[warp][nb] = i; }
        if (++nb == kGatherBatch) {
            __syncwarp();
            if (lane < nb) finalize_cell32<D, H>(AA[sI[warp][lane]], sC[warp][lane], sM[warp][lane]);
            __syncwarp();
            nb = 0;
        }
    }
    finish_rest<NW, kGatherBatch>(nb, &sC[0][0],
                                  [&](int w, int k) { finalize_cell32<D, H>(AA[sI[w][k]], sC[w][k], sM[w][k]); });
}

// ------------------------------------------------- persistent batched step
// Grid-wide barrier of a cooperative launch (every block resident): an
// arrival counter bar[0] and a generation bar[1] in global memory (zeroed
// before the launch).  Arrival is an acquire-release add, the last arrival
// releases the generation and the waiters acquire it, so that after the
// barrier every block sees what every block wrote before it (the acquire
// also keeps stale L1 lines from being read).  A wait polls at most `cap`
// times; then it sets *status = DUGKS_ERR_TIMEOUT (6) and the barrier returns
// false in every block that reaches it afterwards, so all blocks leave the
// kernel.  Callers reach it only with no asynchronous copy in flight.
constexpr int kStatusTimeout = 6;
__device__ __forceinline__ bool grid_barrier(unsigned* bar, long long cap, int* status) {
    __shared__ int sOk;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned gen = *(volatile unsigned*)(bar + 1);
        unsigned old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(bar) : "memory");
        if (old == gridDim.x - 1) {  // last to arrive: reset, release the others
            atomicExch(bar, 0u);
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar + 1) : "memory");
        } else {
            long long it = 0;
            for (;;) {
                unsigned g;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(g) : "l"(bar + 1) : "memory");
                if (g != gen) break;
                if (++it > cap) {
                    ok = 0;
                    atomicExch(status, kStatusTimeout);
                    break;
                }
                __nanosleep(64);
            }
        }
        if (*(volatile int*)status == kStatusTimeout) ok = 0;
        sOk = ok;
    }
    __syncthreads();
    return sOk != 0;
}

// Cells finished per warp batch in the persistent kernel's gather pass.
constexpr int kPersistBatch = 16;

// Dynamic shared memory of the persistent kernel's gather pass: the warps'
// row stages, their case-argument copies, slot totals and cell / case ids.
template <int D, bool H>
__host__ __device__ inline size_t persist_gather_smem(int nw, int mf, int kc) {
    return gather_smem(nw, mf, kc, H) + (size_t)nw * sizeof(FusedArgs<float>) +
           (size_t)nw * kPersistBatch * Slots32<D, H>::NS * sizeof(double) + 2 * (size_t)nw * kPersistBatch * sizeof(int);
}

// Several independent cases, nSteps whole steps in one cooperative launch:
// per step the face-side tiles of all cases (blocks stride over the work
// list), a grid barrier, the face macros of all cases (threads stride over
// the faces), a barrier, the cell gather of all cases (warps stride over the
// cells), a barrier.  Step s uses the argument arrays of parity
// (parity0 + s) & 1 (double buffers swapped).  The pass bodies are those of
// the single-case kernels.
template <int D, bool H, int NPL, int NW>
__global__ void __launch_bounds__(NW * 32, 1)
    k_batch_persistent32(const FusedArgs<float>* __restrict__ AA0, const FusedArgs<float>* __restrict__ AA1,
                         const int2* __restrict__ work, int nWork, const int* __restrict__ faceOff,
                         const int* __restrict__ cellOff, int nCases, int MF, int nSteps, int parity0, unsigned* bar,
                         long long cap, int* status) {
    using SL = Slots32<D, H>;
    constexpr int NS = SL::NS, KC = 32 * NPL, NR = H ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ FusedArgs<float> sA;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int W8 = (int)(sizeof(FusedArgs<float>) / 8);
    static_assert(sizeof(FusedArgs<float>) % 8 == 0, "argument block is copied in 8-byte words");
    // gather-pass carve-up of the dynamic shared memory
    float* gsm = reinterpret_cast<float*>(smem);
    const size_t stBytes = gather_smem(NW, MF, KC, H);
    FusedArgs<float>* sAw = reinterpret_cast<FusedArgs<float>*>(smem + stBytes);
    double* sM = reinterpret_cast<double*>(smem + stBytes + NW * sizeof(FusedArgs<float>));
    int* sC = reinterpret_cast<int*>(sM + (size_t)NW * kPersistBatch * NS);
    int* sI = sC + NW * kPersistBatch;
    float* wb = gsm + (size_t)warp * 2 * (1 + MF) * NR * KC + lane * NPL;
    const int myslot = slot_of<NS>(lane);
    const bool writer = NS == 16 ? (lane & 1) == 0 : true;
    const int totalFaces = faceOff[nCases], totalCells = cellOff[nCases];
    for (int s = 0; s < nSteps; ++s) {
        const FusedArgs<float>* AA = ((parity0 + s) & 1) ? AA1 : AA0;
        // ---- face sides (P1-P3 and the per-side face moments)
        for (int w = blockIdx.x; w < nWork; w += gridDim.x) {
            const int2 wk = work[w];
            const long long* src = reinterpret_cast<const long long*>(AA + wk.x);
            long long* dst = reinterpret_cast<long long*>(&sA);
            for (int k = threadIdx.x; k < W8; k += blockDim.x) dst[k] = src[k];
            __syncthreads();
            if (sA.b.M % NPL == 0) face_sides_body<D, H, NPL, NW, true>(sA, wk.y, smem);
            else face_sides_body<D, H, NPL, NW, false>(sA, wk.y, smem);
            __syncthreads();
        }
        if (!grid_barrier(bar, cap, status)) return;
        // ---- face macros (P4-P6)
        for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < totalFaces; g += gridDim.x * blockDim.x) {
            const int i = case_of(faceOff, nCases, g);
            face_macros_one<D, H>(AA[i], g - faceOff[i]);
        }
        if (!grid_barrier(bar, cap, status)) return;
        // ---- cell gather (P7-P9)
        int nb = 0, cur = -1;
        const int TW = gridDim.x * NW;
        for (int g = blockIdx.x * NW + warp; g < totalCells; g += TW) {
            const int i = case_of(cellOff, nCases, g), k0 = g - cellOff[i];
            if (i != cur) {
                const long long* src = reinterpret_cast<const long long*>(AA + i);
                long long* dst = reinterpret_cast<long long*>(sAw + warp);
                __syncwarp();
                for (int k = lane; k < W8; k += 32) dst[k] = src[k];
                __syncwarp();
                cur = i;
            }
            const int c = sAw[warp].cellOrd[k0];
            const float tot = sAw[warp].b.M % NPL == 0 ? gather_cell<D, H, NPL, true>(sAw[warp], c, MF, wb, lane)
                                                        : gather_cell<D, H, NPL, false>(sAw[warp], c, MF, wb, lane);
            double* mw = sM + ((size_t)warp * kPersistBatch + nb) * NS;
            if (writer) mw[myslot] = tot;
            if (lane == 0) { sC[warp * kPersistBatch + nb] = c; sI[warp * kPersistBatch + nb] = i; }
            if (++nb == kPersistBatch) {
                __syncwarp();
                if (lane < nb)
                    finalize_cell32<D, H>(AA[sI[warp * kPersistBatch + lane]], sC[warp * kPersistBatch + lane],
                                          sM + ((size_t)warp * kPersistBatch + lane) * NS);
                __syncwarp();
                nb = 0;
            }
        }
        finish_rest<NW, kPersistBatch>(nb, sC, [&](int w, int k) {
            finalize_cell32<D, H>(AA[sI[w * kPersistBatch + k]], sC[w * kPersistBatch + k],
                                  sM + ((size_t)w * kPersistBatch + k) * NS);
        });
        if (!grid_barrier(bar, cap, status)) return;
    }
}

// ------------------------------------------------------------ set-up kernels
// Raw moments of one velocity's (g, h) added into m (FP64, Slots32 layout).
template <int D, bool H>
__device__ __forceinline__ void add_raw32(double* m, double w, double g, double h, const double* x) {
    using SL = Slots32<D, H>;
    const double wg = w * g;
    double x2 = 0.0;
    for (int i = 0; i < D; ++i) x2 += x[i] * x[i];
    const double E = x2 * wg + (H ? w * h : 0.0);
    m[0] += wg;
    for (int i = 0; i < D; ++i) {
        m[SL::M1 + i] += wg * x[i];
        for (int j = i; j < D; ++j) m[SL::M2 + sym<D>(i, j)] += wg * x[i] * x[j];
        m[SL::Q + i] += E * x[i];
    }
    if (H) m[SL::H0] += w * h;
}

// Reference Maxwellian per DV (scaled: exp(-|xi|^2/(2 R T0))), its raw moments
// (scaled) and, per wall face, the reference moments over the outgoing
// velocities plus the reference outgoing flux.
template <int D, bool H>
__global__ void k_ref_tables(StepArgs b, double T0, double hrefFac, float* mref, double* refMom, double* wallRefOut) {
    using SL = Slots32<D, H>;
    constexpr int NS = SL::NS;
    __shared__ double red[32 * NS];
    const int blk = blockIdx.x;  // 0: raw moments; 1 + w: wall face w
    double m[NS];
    for (int s = 0; s < NS; ++s) m[s] = 0.0;
    const double* Sf = blk > 0 ? b.Sf + 3 * (b.nI + blk - 1) : nullptr;
    for (int v = threadIdx.x; v < b.Vp; v += blockDim.x) {
        const double x[3] = {b.xi[v], b.xi[b.Vp + v], b.xi[2 * b.Vp + v]};
        const double M = exp(-(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]) / (2.0 * b.R * T0));
        if (blk == 0) mref[v] = (float)M;
        const double Mf = (double)(float)M;  // moments of the FP32 value actually subtracted
        const double xs = blk == 0 ? 1.0 : x[0] * Sf[0] + x[1] * Sf[1] + x[2] * Sf[2];
        if (xs > 0 && v < b.nV) {
            add_raw32<D, H>(m, b.w[v], Mf, Mf * hrefFac, x);
            if (blk > 0) m[SL::FLUX] += b.w[v] * xs * Mf;
        }
    }
    block_sum<NS>(m, red);
    if (threadIdx.x == 0) {
        double* out = blk == 0 ? refMom : wallRefOut + (size_t)(blk - 1) * NS;
        for (int s = 0; s < NS; ++s) out[s] = m[s];
    }
}

// Wall Maxwellian per unit density of every wall face and its raw moments over
// the incoming velocities.
template <int D, bool H>
__global__ void k_wall_tables32(StepArgs b, float* Mw, double* Min) {
    constexpr int NS = Slots32<D, H>::NS;
    __shared__ double red[32 * NS];
    const int w = blockIdx.x;
    const double* Sf = b.Sf + 3 * (b.nI + w);
    const double Tw = b.Tw[w];
    const double* Uw = b.Uw + 3 * w;
    double m[NS];
    for (int s = 0; s < NS; ++s) m[s] = 0.0;
    for (int v = threadIdx.x; v < b.Vp; v += blockDim.x) {
        const double x[3] = {b.xi[v], b.xi[b.Vp + v], b.xi[2 * b.Vp + v]};
        const double M = maxwell_by_rho_ref(Uw[0], Uw[1], Uw[2], Tw, x[0], x[1], x[2], b.R, b.D);
        Mw[(size_t)w * b.Vp + v] = (float)M;
        if (x[0] * Sf[0] + x[1] * Sf[1] + x[2] * Sf[2] <= 0 && v < b.nV)
            add_raw32<D, H>(m, b.w[v], M, M * (b.R * Tw) * (b.K + 3 - D), x);
    }
    block_sum<NS>(m, red);
    if (threadIdx.x == 0)
        for (int s = 0; s < NS; ++s) Min[(size_t)w * NS + s] = m[s];
}

// Deviation-form state from FP64 values: G = gscale g - Mref, H = gscale h - Href.
__global__ static void k_init_dev32(StepArgs b, const float* mref, double gs, double hrefFac, float* gT, float* hT) {
    const long long n = (long long)b.nC * b.Vp;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i / b.Vp), v = (int)(i - (long long)c * b.Vp);
        double ge, he;
        shakhov_ref(b.rho[c], b.U[3 * c], b.U[3 * c + 1], b.U[3 * c + 2], b.T[c], 0.0, 0.0, 0.0, b.xi[v],
                    b.xi[b.Vp + v], b.xi[2 * b.Vp + v], b.R, b.Pr, b.D, b.K, ge, he);
        const double mr = mref[v];
        gT[i] = (float)(ge * gs - mr);
        if (b.hasH) hT[i] = (float)(he * gs - mr * hrefFac);
        if (v == 0) b.tau[c] = tau_ref(b.T[c], b.rho[c], b.muRef, b.omega, b.Tref, b.R);
    }
}

__global__ static void k_export_dev32(StepArgs b, const float* src, const float* mref, double fac, double inv, double* dst) {
    const long long n = (long long)b.nC * b.nV;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i / b.nV), v = (int)(i - (long long)c * b.nV);
        dst[i] = ((double)src[(long long)c * b.Vp + v] + (double)mref[v] * fac) * inv;
    }
}

__global__ static void k_import_dev32(StepArgs b, const double* src, const float* mref, double fac, double gs, float* dst) {
    const long long n = (long long)b.nC * b.nV;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i / b.nV), v = (int)(i - (long long)c * b.nV);
        dst[(long long)c * b.Vp + v] = (float)(src[i] * gs - (double)mref[v] * fac);
    }
}

}  // namespace dugks
