// Kernels of the FP32 step for one case (fused32.cuh), instantiated in
// fused_fp32_2d.cu and fused_fp32_3d.cu (apart, so that they compile in
// parallel).
#pragma once

#include "fused32.cuh"

namespace dugks {

constexpr int kFaceWarps = 16;   // warps per tile block of the face sweep (one tile per SM)
constexpr int kGatherWarps = 8;  // warps (cells) per block of the gather sweep

struct Kernels32 {
    void (*face)(FusedArgs<float>) = nullptr;
    void (*macros)(FusedArgs<float>) = nullptr;
    void (*open)(FusedArgs<float>) = nullptr;  // only with boundary types other than diffuse walls
    void (*gather)(FusedArgs<float>, int, int) = nullptr;
    void (*tables)(StepArgs, float*, double*) = nullptr;
    void (*ref)(StepArgs, double, double, float*, double*, double*) = nullptr;
    size_t (*smemFace)(const TileDims&) = nullptr;
};
// row: a lane's velocities share xi_y and xi_z; open: some boundary face is no diffuse wall.
Kernels32 kernels32_2d(bool h, int npl, bool row, bool open);
Kernels32 kernels32_3d(bool h, int npl, bool row, bool open);
inline Kernels32 kernels32(int D, bool h, int npl, bool row, bool open) {
    return D == 2 ? kernels32_2d(h, npl, row, open) : kernels32_3d(h, npl, row, open);
}

template <int D, bool H, int NPL, bool ROW>
Kernels32 kernels32_of(bool open) {
    Kernels32 k;
    k.face = k_face_sides32<D, H, NPL, kFaceWarps, ROW>;
    k.macros = k_face_macros32<D, H>;
    if (open) k.open = k_open_faces32<D, H, NPL>;
    k.gather = open ? k_cell_gather32<D, H, NPL, kGatherWarps, ROW, true> : k_cell_gather32<D, H, NPL, kGatherWarps, ROW, false>;
    k.tables = k_wall_tables32<D, H>;
    k.ref = k_ref_tables<D, H>;
    k.smemFace = &SmemLayout32<D, H, NPL>::sides;
    return k;
}
template <int D>
Kernels32 kernels32_d(bool h, int npl, bool row, bool open) {
    if (npl == 4) {
        if (h) return row ? kernels32_of<D, true, 4, true>(open) : kernels32_of<D, true, 4, false>(open);
        return row ? kernels32_of<D, false, 4, true>(open) : kernels32_of<D, false, 4, false>(open);
    }
    if (h) return row ? kernels32_of<D, true, 2, true>(open) : kernels32_of<D, true, 2, false>(open);
    return row ? kernels32_of<D, false, 2, true>(open) : kernels32_of<D, false, 2, false>(open);
}

}  // namespace dugks
