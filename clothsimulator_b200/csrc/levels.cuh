// Tile levels of the on-chip solvers' preconditioner (resident.cu, group.cu).  The loader orders a
// tile's rows by recursive bisection, so every eight consecutive rows (an octet of lanes) and every 32
// (a slice, one warp) are a compact patch of the sheet.  With F and G summing a vector over the octets
// and the slices, per component,
//     z = D^-1 r + F^T D_F^-1 F r + G^T D_G^-1 G r (+ R^T A_c^-1 R r),
// D_F and D_G the 3x3 diagonal blocks of F A F^T and G A G^T: additive, SPD, and 15 warp shuffles per
// iteration with no barrier.  It takes the place of a Chebyshev polynomial in the tile's block of A
// together with a larger coarse space: on a 64 x 64 sheet 76 CG iterations of one SpMV each instead of
// 61 of one SpMV and two polynomial steps, and 54 coarse unknowns to invert instead of 162.
#pragma once
#include "cs_internal.h"

namespace {

// The inverse of the symmetrised 3x3 sum `m` as the six entries 00 01 02 11 12 22 (FP64 inside);
// zeros unless it is positive definite.
__device__ __forceinline__ void level_inverse(const float (&m)[9], float* out) {
    const double a00 = m[0], a11 = m[4], a22 = m[8];
    const double a01 = 0.5 * ((double)m[1] + m[3]), a02 = 0.5 * ((double)m[2] + m[6]), a12 = 0.5 * ((double)m[5] + m[7]);
    const double c00 = a11 * a22 - a12 * a12, c01 = a02 * a12 - a01 * a22, c02 = a01 * a12 - a02 * a11;
    const double m2 = a00 * a11 - a01 * a01, det = a00 * c00 + a01 * c01 + a02 * c02, id = 1.0 / det;
    const bool on = a00 > 0.0 && m2 > 0.0 && det > 0.0 && isfinite((float)id);
    out[0] = on ? (float)(c00 * id) : 0.f;
    out[1] = on ? (float)(c01 * id) : 0.f;
    out[2] = on ? (float)(c02 * id) : 0.f;
    out[3] = on ? (float)((a00 * a22 - a02 * a02) * id) : 0.f;
    out[4] = on ? (float)((a01 * a02 - a00 * a12) * id) : 0.f;
    out[5] = on ? (float)(m2 * id) : 0.f;
}
__device__ __forceinline__ void level_apply(const float* inv, const float (&s)[3], float (&u)[3]) {
    const float4 a = reinterpret_cast<const float4*>(inv)[0], b = reinterpret_cast<const float4*>(inv)[1];
    u[0] += a.x * s[0] + a.y * s[1] + a.z * s[2];
    u[1] += a.y * s[0] + a.w * s[1] + b.x * s[2];
    u[2] += a.z * s[0] + b.x * s[1] + b.y * s[2];
}

// The inverse diagonal blocks of one warp's octets (lev[0..3]) and of its slice (lev[4]), from the stored
// blocks of its rows: the first ks slots in shared memory (sp), the others in global memory (gp), `code`
// the slots' columns as row slots of the CTA (others from the halo's first slot on).
__device__ __forceinline__ void level_blocks(const float* sp, const float* gp, int ks, int width, const int* __restrict__ code,
                                             int w, int lane, bool live, float (*lev)[8]) {
    float a8[9], a32[9];
#pragma unroll
    for (int e = 0; e < 9; e++) a8[e] = a32[e] = 0.f;
    for (int k = 0; k < width; k++) {
        const int at = __ldg(code + k * CS_SLICE + lane);
        if (!live || (at >> 5) != w) continue;
        const float* pk = (k < ks ? sp : gp) + (size_t)k * CS_PANEL_FLOATS;
        const float4 b0 = reinterpret_cast<const float4*>(pk)[lane], b1 = reinterpret_cast<const float4*>(pk + 128)[lane];
        const float a[9] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w, pk[256 + lane]};
        const float in8 = ((at ^ lane) & 24) == 0 ? 1.f : 0.f;
#pragma unroll
        for (int e = 0; e < 9; e++) {
            a32[e] += a[e];
            a8[e] = fmaf(in8, a[e], a8[e]);
        }
    }
#pragma unroll
    for (int e = 0; e < 9; e++) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) a8[e] += __shfl_xor_sync(0xffffffffu, a8[e], o);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) a32[e] += __shfl_xor_sync(0xffffffffu, a32[e], o);
    }
    if ((lane & 7) == 0) level_inverse(a8, lev[lane >> 3]);
    if (lane == 0) level_inverse(a32, lev[4]);
    __syncwarp();
}

// u += the octet's and the slice's corrections of r (zero in lanes without a row)
__device__ __forceinline__ void level_correction(const float (*lev)[8], const float (&r)[3], int lane, float (&u)[3]) {
    float t[3] = {r[0], r[1], r[2]};
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int c = 0; c < 3; c++) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
    level_apply(lev[lane >> 3], t, u);
#pragma unroll
    for (int o = 8; o < 32; o <<= 1)
#pragma unroll
        for (int c = 0; c < 3; c++) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
    level_apply(lev[4], t, u);
}

}  // namespace
