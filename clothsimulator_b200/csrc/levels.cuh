// Parts of the on-chip solvers (resident.cu, group.cu) that work on a tile: warp sums, the product of a
// row with the tile's u array, and the preconditioner's levels.  The loader orders a
// tile's rows by recursive bisection into cells: every eight rows in that order (an octet) and every 32
// (a patch) are a compact piece of the sheet.  Lane l of warp w holds place 32 w + l of that order; the rows
// are stored by block count, so a vector's values go to their places and the corrections back through
// shared memory.  With F and G summing a vector over the octets
// and the patches, per component,
//     z = D^-1 r + F^T D_F^-1 F r + G^T D_G^-1 G r (+ R^T A_c^-1 R r),
// D_F and D_G the 3x3 diagonal blocks of F A F^T and G A G^T: additive, SPD, and 15 warp shuffles per
// iteration with two barriers.  It takes the place of a Chebyshev polynomial in the tile's block of A
// together with a larger coarse space: on a 64 x 64 sheet about 75 CG iterations of one SpMV each instead of
// 61 of one SpMV and two polynomial steps, and 54 coarse unknowns to invert instead of 162.
#pragma once
#include "cs_internal.h"

namespace {

// Warp sums of two (lanes 0-15 return the first, 16-31 the second) and of three values (lanes 0-7, 8-15,
// 16-23), by exchanges that halve the values a lane carries: 5 and 8 additions instead of 10 and 15.
template <class T>
__device__ __forceinline__ T tile_sum2(T a, T b) {
    const bool up = threadIdx.x & 16;
    T v = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <class T>
__device__ __forceinline__ T tile_sum3(T a, T b, T c) {
    const bool up = threadIdx.x & 16, odd = threadIdx.x & 8;
    T x = __shfl_xor_sync(0xffffffffu, up ? a : c, 16), y = __shfl_xor_sync(0xffffffffu, up ? b : T(0), 16);
    x += up ? c : a;
    y += up ? T(0) : b;
    T v = (odd ? y : x) + __shfl_xor_sync(0xffffffffu, odd ? x : y, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ void block_times(const float4 a0, const float4 a1, const float a8, const float4 pv, float& q0,
                                            float& q1, float& q2) {
    q0 = fmaf(a0.z, pv.z, fmaf(a0.y, pv.y, fmaf(a0.x, pv.x, q0)));
    q1 = fmaf(a1.y, pv.z, fmaf(a1.x, pv.y, fmaf(a0.w, pv.x, q1)));
    q2 = fmaf(a8, pv.z, fmaf(a1.w, pv.y, fmaf(a1.z, pv.x, q2)));
}

// w += (row of A) u.  The first ks slots of a slice (uniform in the warp) are in shared memory, slots ks ..
// width - 1 (beyond the budget, spread evenly over the slices) in global memory, the first of those
// requested by row_tail_load before the halo wait.  A warp's time is its count of instructions and the
// latencies between them, so the slots go CHUNK at a time without branches, a chunk's loads in flight
// together, over own rows and halo copies alike (a pass over the own rows while the halo values travel
// and a second over the halo's took longer than the wait it hid).  `cw`: the byte offsets of the slots'
// entries in the u array, two 16-bit ones per word (of a zero entry for the slots beyond ks).
struct RowTail {
    float4 a0, a1;
    float a8;
    int idx;
};
__device__ __forceinline__ RowTail row_tail_load(const float* __restrict__ gp, int ks, int width, const int* __restrict__ code,
                                                 int lane) {
    RowTail t;
    t.a0 = t.a1 = make_float4(0.f, 0.f, 0.f, 0.f);
    t.a8 = 0.f;
    t.idx = 0;
    if (ks < width) {
        const float* pk = gp + (size_t)ks * CS_PANEL_FLOATS;
        t.a0 = __ldg(reinterpret_cast<const float4*>(pk) + lane);
        t.a1 = __ldg(reinterpret_cast<const float4*>(pk + 128) + lane);
        t.a8 = __ldg(pk + 256 + lane);
        t.idx = __ldg(code + ks * CS_SLICE + lane);
    }
    return t;
}
// LOCAL: only the columns that are the CTA's own rows (entries below `halo0`; the one before it is zero).
template <int W, int CHUNK, bool LOCAL>
__device__ __forceinline__ void row_times(const float* __restrict__ sp, const float* __restrict__ gp, int ks, int width,
                                          const uint32_t (&cw)[W / 2], const int* __restrict__ code,
                                          const RowTail& t, const float4* su, int halo0, int lane, bool live, float& q0, float& q1,
                                          float& q2) {
    static_assert(W % CHUNK == 0, "whole chunks");
    const unsigned char* const sb = reinterpret_cast<const unsigned char*>(su);
#pragma unroll
    for (int k0 = 0; k0 < W; k0 += CHUNK) {
        if (k0 >= ks) break;
        float4 a0[CHUNK], a1[CHUNK], pv[CHUNK];
        float a8[CHUNK];
#pragma unroll
        for (int j = 0; j < CHUNK; j++) {
            const int k = k0 + j;
            const float* pk = sp + (k < ks ? k : k0) * CS_PANEL_FLOATS;
            const uint32_t at = (k & 1) ? cw[k >> 1] >> 16 : cw[k >> 1] & 0xffffu;
            a0[j] = reinterpret_cast<const float4*>(pk)[lane];
            a1[j] = reinterpret_cast<const float4*>(pk + 128)[lane];
            a8[j] = pk[256 + lane];
            pv[j] = *reinterpret_cast<const float4*>(sb + (LOCAL ? min(at, 16u * (halo0 - 1)) : at));
        }
#pragma unroll
        for (int j = 0; j < CHUNK; j++) block_times(a0[j], a1[j], a8[j], pv[j], q0, q1, q2);
    }
    if (ks < width) {
        if (live && (!LOCAL || t.idx < halo0)) block_times(t.a0, t.a1, t.a8, su[t.idx], q0, q1, q2);
        for (int k = ks + 1; k < width; k++) {
            const int idx = __ldg(code + k * CS_SLICE + lane);
            if (!live || (LOCAL && idx >= halo0)) continue;
            const float* pk = gp + (size_t)k * CS_PANEL_FLOATS;
            block_times(__ldg(reinterpret_cast<const float4*>(pk) + lane), __ldg(reinterpret_cast<const float4*>(pk + 128) + lane),
                        __ldg(pk + 256 + lane), su[idx], q0, q1, q2);
        }
    }
}

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

// A thread's part in the levels: the octet of its row (its place in cell order / 8), and the slot of the row whose
// place is the thread's number.  Threads without a row have their own number for both.
struct LevelPlace {
    uint32_t v;  // slot | place << 16
    __device__ __forceinline__ int slot() const { return (int)(v & 0xffffu); }
    __device__ __forceinline__ int place() const { return (int)(v >> 16); }
    __device__ __forceinline__ int octet() const { return (int)(v >> 19); }
};

// The inverse diagonal blocks of the octets (lev[0..3]) and of the patch (lev[4]) at one warp's places in cell
// order, from the stored blocks of the rows: the first ks slots of a slice in shared memory (sp), the others
// in global memory (gp), `code` the slots' columns as row slots of the CTA (from `own` on: others).  `cells`: the
// {slot, place} of all row slots; `buf`: room for a float4 per row slot.  Every thread of the CTA calls it.
__device__ __forceinline__ void level_blocks(const float* sp, const float* gp, int ks, int width, const int* __restrict__ code,
                                             const uint32_t* __restrict__ cells, int own, LevelPlace at, int lane, bool live,
                                             float4* buf,
                                             float (*lev)[8]) {
    float m[20];  // the row's part of its octet's block, of its patch's
#pragma unroll
    for (int e = 0; e < 20; e++) m[e] = 0.f;
    for (int k = 0; k < width; k++) {
        const int col = __ldg(code + k * CS_SLICE + lane);
        if (!live || col >= own) continue;
        const int other = (int)(__ldg(cells + col) >> 16);
        if ((other >> 5) != (at.place() >> 5)) continue;
        const float* pk = (k < ks ? sp : gp) + (size_t)k * CS_PANEL_FLOATS;
        const float4 b0 = reinterpret_cast<const float4*>(pk)[lane], b1 = reinterpret_cast<const float4*>(pk + 128)[lane];
        const float a[9] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w, pk[256 + lane]};
        const float in8 = (other >> 3) == at.octet() ? 1.f : 0.f;
#pragma unroll
        for (int e = 0; e < 9; e++) {
            m[e] = fmaf(in8, a[e], m[e]);
            m[9 + e] += a[e];
        }
    }
#pragma unroll
    for (int q = 0; q < 20; q += 4) {
        __syncthreads();
        buf[threadIdx.x] = make_float4(m[q], m[q + 1], m[q + 2], m[q + 3]);
        __syncthreads();
        const float4 x = buf[at.slot()];
        m[q] = x.x;
        m[q + 1] = x.y;
        m[q + 2] = x.z;
        m[q + 3] = x.w;
    }
    float a8[9], a32[9];
#pragma unroll
    for (int e = 0; e < 9; e++) {
        a8[e] = m[e];
        a32[e] = m[9 + e];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) a8[e] += __shfl_xor_sync(0xffffffffu, a8[e], o);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) a32[e] += __shfl_xor_sync(0xffffffffu, a32[e], o);
    }
    if ((lane & 7) == 0) level_inverse(a8, lev[lane >> 3]);
    if (lane == 0) level_inverse(a32, lev[4]);
    __syncthreads();  // `buf` is free
}

// The corrections by the octets and the patch at one warp's places of a vector, into `z`, a float4 per octet.  `x`:
// the value of the row whose place is the thread's, which that row's thread stored in shared memory before a
// barrier (zero without a row).  A barrier then lies before level_add; `z` may be overwritten after the next.
__device__ __forceinline__ void level_sums(const float (*lev)[8], const float4 x, float4* z, int w, int lane) {
    float t[3] = {x.x, x.y, x.z}, c[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int k = 0; k < 3; k++) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
    level_apply(lev[lane >> 3], t, c);
#pragma unroll
    for (int o = 8; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < 3; k++) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
    level_apply(lev[4], t, c);
    if ((lane & 7) == 0) z[4 * w + (lane >> 3)] = make_float4(c[0], c[1], c[2], 0.f);
}
__device__ __forceinline__ void level_add(const float4* z, LevelPlace at, float (&u)[3]) {
    const float4 y = z[at.octet()];
    u[0] += y.x;
    u[1] += y.y;
    u[2] += y.z;
}

}  // namespace
