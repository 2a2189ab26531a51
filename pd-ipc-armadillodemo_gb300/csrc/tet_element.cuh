// tet_element.cuh — the strain projection inside the persistent solves (pd_tile.cu,
// pd_persistent.cuh).
#pragma once

#include "svd3.cuh"

namespace pdipc {

namespace {

// One tet's strain projection (solveVolumetricStrainConstraintKernel,
// PdIpcGpuFunc.cu:439-599): Ds from the current positions (the float-float mirror in
// the correction form), w R G of its four vertices (three of a cloth triangle's strain
// element) to Out.  Out of line: once per tet and local-global iteration, its registers
// stay out of the sweeps.  Positions come from L2 (written by other CTAs earlier in the
// launch).
template <typename S, bool kCorr>
__device__ __noinline__ void tet_element(int e, const int4* __restrict__ Tets, const float* __restrict__ Idm,
                                         const float* __restrict__ W, const V4<S>* P, const V4<float>* Ph,
                                         const V4<float>* Pl, V4<float>* Out) {
    const int4 q = Tets[e];
    const bool tri = q.w < 0;
    const int id[4] = {q.x, q.y, q.z, tri ? q.x : q.w};
    float Ds[3][3];
    if constexpr (kCorr) {
        const float4 h0 = __ldcg((const float4*)Ph + id[0]), l0 = __ldcg((const float4*)Pl + id[0]);
        for (int c = 0; c < 3; ++c) {
            const float4 h = __ldcg((const float4*)Ph + id[c + 1]), l = __ldcg((const float4*)Pl + id[c + 1]);
            Ds[0][c] = diff_ff(h.x, l.x, h0.x, l0.x);
            Ds[1][c] = diff_ff(h.y, l.y, h0.y, l0.y);
            Ds[2][c] = diff_ff(h.z, l.z, h0.z, l0.z);
        }
    } else {
        const float4 x0 = __ldcg((const float4*)P + id[0]);
        for (int c = 0; c < 3; ++c) {
            const float4 x = __ldcg((const float4*)P + id[c + 1]);
            Ds[0][c] = x.x - x0.x;
            Ds[1][c] = x.y - x0.y;
            Ds[2][c] = x.z - x0.z;
        }
    }
    float idm[9];
    for (int k = 0; k < 9; ++k) idm[k] = __ldg(Idm + 9 * (size_t)e + k);
    float out[4][3];
    if (tri) {
        const float D2[3][2] = {{Ds[0][0], Ds[0][1]}, {Ds[1][0], Ds[1][1]}, {Ds[2][0], Ds[2][1]}};
        float o3[3][3];
        svd::tri_project<float>(D2, idm, __ldg(W + e), o3);
        for (int c = 0; c < 3; ++c)
            for (int r = 0; r < 3; ++r) out[c][r] = o3[c][r];
        out[3][0] = out[3][1] = out[3][2] = 0.f;
    } else {
        svd::tet_project<float>(Ds, idm, __ldg(W + e), out);
    }
    for (int c = 0; c < 4; ++c)
        __stcg((float4*)Out + 4 * (size_t)e + c, make_float4(out[c][0], out[c][1], out[c][2], 0.f));
}

}  // namespace

}  // namespace pdipc
