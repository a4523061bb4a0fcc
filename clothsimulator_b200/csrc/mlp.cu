// Learned warm start: a one-ring message-passing MLP that predicts the step's dv, with its
// layers on tcgen05 tensor cores (BF16 operands, FP32 accumulation in tensor memory).
// The reference has no learned component; this is project design (see the header's
// cs_mlp_* functions for the network definition).
#include <cuda_bf16.h>

#include "../../include/clothstep.h"
#include "cs_internal.h"
#include "mlp.h"
#include "tc.cuh"

// ---------------------------------------------------------------------------------------
// Tile GEMM check: D[128 x N] = A[128 x K] B[N x K]^T through the same tcgen05 path the MLP
// layers use.  K in {16, 32, ..., 128}, N in {16, 32, ..., 128}.
__global__ void __launch_bounds__(128) cs_tc_gemm_check_kernel(const __nv_bfloat16* __restrict__ A,
                                                             const __nv_bfloat16* __restrict__ Bm, float* __restrict__ D,
                                                             int K, int N, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;                       // 128 x K bf16
    unsigned char* sB = smem + 128 * 128 * 2;       // N x K bf16
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 2 * 128 * 128 * 2);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
    const int t = threadIdx.x, warp = t >> 5;
    for (int k = 0; k < K; k++) tc::st_bf16(sA, 128, t, k, __bfloat162float(A[t * K + k]));
    for (int r = t; r < N; r += 128)
        for (int k = 0; k < K; k++) tc::st_bf16(sB, N, r, k, __bfloat162float(Bm[r * K + k]));
    if (t == 0) tc::mbar_init(bar, 1);
    if (warp == 0) tc::tmem_alloc(slot, 128);
    tc::fence_async_shared();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;
    if (t == 0) {
        tc::gemm_tile(tmem, tc::smem_u32(sA), tc::smem_u32(sB), K, N, false);
        tc::mma_commit(bar);
    }
    bool ok = tc::mbar_wait(bar, 0);
    tc::fence_after_sync();
    if (ok) {
        for (int c = 0; c < N / 16; c++) {
            float v[16];
            tc::tmem_ld16(tc::tmem_addr(tmem, warp, 16 * c), v);
            for (int i = 0; i < 16; i++) D[t * N + 16 * c + i] = v[i];
        }
    } else if (t == 0) {
        atomicExch(err, 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 128);
}

extern "C" cs_status cs_tc_gemm_check(const uint16_t* A, const uint16_t* B, float* D, int K, int N) {
    if (!A || !B || !D || K < 16 || K > 128 || K % 16 || N < 16 || N > 128 || N % 16) return CS_ERR_INVALID_ARG;
    __nv_bfloat16 *dA = nullptr, *dB = nullptr;
    float* dD = nullptr;
    int* derr = nullptr;
    cudaError_t e = cudaMalloc(&dA, 128 * K * 2);
    if (e == cudaSuccess) e = cudaMalloc(&dB, N * K * 2);
    if (e == cudaSuccess) e = cudaMalloc(&dD, 128 * N * 4);
    if (e == cudaSuccess) e = cudaMalloc(&derr, 4);
    if (e == cudaSuccess) e = cudaMemcpy(dA, A, 128 * K * 2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dB, B, N * K * 2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(derr, 0, 4);
    const int smem = 2 * 128 * 128 * 2 + 64;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(cs_tc_gemm_check_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) {
        cs_tc_gemm_check_kernel<<<1, 128, smem>>>(dA, dB, dD, K, N, derr);
        e = cudaDeviceSynchronize();
    }
    int herr = 0;
    if (e == cudaSuccess) e = cudaMemcpy(D, dD, 128 * N * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&herr, derr, 4, cudaMemcpyDeviceToHost);
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dD);
    cudaFree(derr);
    if (e != cudaSuccess) return CS_ERR_CUDA;
    return herr ? CS_ERR_TIMEOUT : CS_OK;
}

// ---------------------------------------------------------------------------------------
// Network (project design; the reference has no learned component).
//
// Per node i, 16 raw features (scale-free where the physics allows):
//   b_i / d_i (3), upper triangle of the diagonal block A_ii / d_i (6), v_i (3),
//   previous dv_i (3), m_i / d_i (1),   with d_i = trace(A_ii) / 3,
// standardised with the training set's mean and spread.  Two rounds of one-ring mean
// aggregation (agg(h)_i = mean of h_j over mesh neighbours j of i):
//   u1 = [x_i, agg(x)_i]              (32)  -> z1 = W1 u1 + b1 (64),  h1 = SiLU(z1)
//   u2 = [h1_i, agg(h1)_i]            (128) -> z2 = W2 u2 + b2 (64),  h2 = SiLU(z2)
//   z3 = W3 h2 + b3 (64), h3 = SiLU(z3);   y = W4 h3 + b4 (3)
//   prediction dv_i = previous dv_i + sigma_y * y + mu_y.
// MMA operands (u1, u2, h2 and the weights) are BF16; accumulation is FP32 in tensor memory;
// h1 is stored in BF16.  The three 64-wide layers and the backward products dz3 W3, dz2 W2
// run on tcgen05 with 128-node tiles; the 3-wide output layer runs on CUDA cores.
namespace {

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
    float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}
__device__ __forceinline__ float bf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

struct Nbr {
    int beg, end, off;
};
__device__ __forceinline__ Nbr neighbours(const Batch& B, int node) {
    const SheetDesc& sh = B.sheets[B.node_sheet[node]];
    const int local = node - sh.node_off;
    Nbr r;
    r.beg = sh.nbr_off + B.nbr_ptr[sh.nbr_ptr_off + local];
    r.end = sh.nbr_off + B.nbr_ptr[sh.nbr_ptr_off + local + 1];
    r.off = sh.node_off;
    return r;
}

// Loads a row-major [rows x cols] BF16 weight matrix (optionally transposed) into a K-major
// canonical tile with R = rows (or cols if transposed) rows.
__device__ void load_weight_tile(const __nv_bfloat16* __restrict__ W, int rows, int cols, bool transpose,
                                 unsigned char* tile) {
    const int R = transpose ? cols : rows, K = transpose ? rows : cols;
    for (int e = threadIdx.x; e < R * K; e += blockDim.x) {
        const int r = e / K, k = e % K;
        const __nv_bfloat16 w = transpose ? W[k * cols + r] : W[r * cols + k];
        *reinterpret_cast<__nv_bfloat16*>(tile + tc::kmajor_offset(R, r, k)) = w;
    }
}

__device__ __forceinline__ void sync_tmem() {
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
}

}  // namespace

// Raw features of every node from the assembled system (diagonal block from the SELL panel
// of slot 0), the velocities and the previous dv held in B.warm.
__global__ void cs_mlp_features_kernel(Batch B, MlpDev M, float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.N) return;
    const SheetDesc& sh = B.sheets[B.node_sheet[i]];
    const int local = i - sh.node_off;
    const int ts = B.row2slot[sh.row2slot_off + local];
    const SliceDesc& sd = B.slices[sh.slice_off + ts / CS_SLICE];
    const int lane = ts % CS_SLICE;
    const float* panel = B.A + (size_t)sd.panel0 * CS_PANEL_FLOATS;
    const float4 a0 = reinterpret_cast<const float4*>(panel)[lane];
    const float4 a1 = reinterpret_cast<const float4*>(panel + 128)[lane];
    const float a8 = panel[256 + lane];
    const float d = (a0.x + a1.x + a8) / 3.0f;
    const float id = d > 0.f ? 1.0f / d : 0.f;
    float* o = out + 16 * (size_t)i;
    o[0] = B.b[3 * i] * id;
    o[1] = B.b[3 * i + 1] * id;
    o[2] = B.b[3 * i + 2] * id;
    o[3] = a0.x * id;
    o[4] = a0.y * id;
    o[5] = a0.z * id;
    o[6] = a1.x * id;
    o[7] = a1.y * id;
    o[8] = a8 * id;
    o[9] = B.v[3 * i];
    o[10] = B.v[3 * i + 1];
    o[11] = B.v[3 * i + 2];
    o[12] = B.warm[3 * i];
    o[13] = B.warm[3 * i + 1];
    o[14] = B.warm[3 * i + 2];
    o[15] = B.mass[i] * id;
}

// Layer 1 over nodes [n0, n1): u1 = [x, agg(x)] -> h1 (BF16) and, when z1 != nullptr, z1.
__global__ void __launch_bounds__(128) cs_mlp_l1_kernel(Batch B, MlpDev M, const float* __restrict__ fsrc, int n0,
                                                      int n1, float* __restrict__ z1) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;              // 128 x 32 bf16: 8 KB
    unsigned char* sW = smem + 8192;       // 64 x 32 bf16: 4 KB
    float* sb = reinterpret_cast<float*>(smem + 12288);  // b1 (64), mu (16), sigma (16)
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 12288 + 512);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
    const int t = threadIdx.x, warp = t >> 5;
    load_weight_tile(M.wb + MLP_W1, 64, 32, false, sW);
    for (int e = t; e < 64; e += 128) sb[e] = M.w[MLP_B1 + e];
    for (int e = t; e < 32; e += 128) sb[64 + e] = M.stats[e];
    if (t == 0) tc::mbar_init(bar, 1);
    if (warp == 0) tc::tmem_alloc(slot, 64);
    tc::fence_async_shared();
    sync_tmem();
    const uint32_t tmem = *slot;
    uint32_t phase = 0;
    bool ok = true;
    const int ntiles = (n1 - n0 + 127) / 128;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int node = n0 + tile * 128 + t;
        const bool valid = node < n1;
        float u[32];
        if (valid) {
            // feature rows are 16 floats = 4 x 16 bytes
            const float4* x = reinterpret_cast<const float4*>(fsrc + 16 * (size_t)node);
            float acc[16];
#pragma unroll
            for (int g = 0; g < 4; g++) {
                const float4 xv = __ldg(x + g);
                u[4 * g] = (xv.x - sb[64 + 4 * g]) / sb[80 + 4 * g];
                u[4 * g + 1] = (xv.y - sb[65 + 4 * g]) / sb[81 + 4 * g];
                u[4 * g + 2] = (xv.z - sb[66 + 4 * g]) / sb[82 + 4 * g];
                u[4 * g + 3] = (xv.w - sb[67 + 4 * g]) / sb[83 + 4 * g];
            }
#pragma unroll
            for (int c = 0; c < 16; c++) acc[c] = 0.f;
            Nbr nb = neighbours(B, node);
            for (int k = nb.beg; k < nb.end; k++) {
                const float4* xj = reinterpret_cast<const float4*>(fsrc + 16 * (size_t)(B.nbr[k] + nb.off));
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    const float4 xv = __ldg(xj + g);
                    acc[4 * g] += xv.x;
                    acc[4 * g + 1] += xv.y;
                    acc[4 * g + 2] += xv.z;
                    acc[4 * g + 3] += xv.w;
                }
            }
            const float inv = nb.end > nb.beg ? 1.0f / (nb.end - nb.beg) : 0.f;
#pragma unroll
            for (int c = 0; c < 16; c++) u[16 + c] = nb.end > nb.beg ? (acc[c] * inv - sb[64 + c]) / sb[80 + c] : 0.f;
        } else {
#pragma unroll
            for (int c = 0; c < 32; c++) u[c] = 0.f;
        }
#pragma unroll
        for (int g = 0; g < 4; g++) {
            __align__(16) __nv_bfloat16 ub[8];
#pragma unroll
            for (int c = 0; c < 8; c++) ub[c] = __float2bfloat16_rn(u[8 * g + c]);
            *reinterpret_cast<uint4*>(sA + tc::kmajor_offset(128, t, 8 * g)) = *reinterpret_cast<const uint4*>(ub);
        }
        tc::fence_async_shared();
        sync_tmem();
        if (t == 0) {
            tc::gemm_tile(tmem, tc::smem_u32(sA), tc::smem_u32(sW), 32, 64, false);
            tc::mma_commit(bar);
        }
        ok = __syncthreads_and(tc::mbar_wait(bar, phase) ? 1 : 0) != 0;
        phase ^= 1;
        tc::fence_after_sync();
        if (ok) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float zz[16];
                tc::tmem_ld16(tc::tmem_addr(tmem, warp, 16 * q), zz);
                if (valid) {
                    __align__(16) __nv_bfloat16 hb[16];
#pragma unroll
                    for (int c = 0; c < 16; c++) {
                        const float z = zz[c] + sb[16 * q + c];
                        hb[c] = __float2bfloat16_rn(silu(z));
                        if (z1) z1[64 * (size_t)node + 16 * q + c] = z;
                    }
                    uint4* dst = reinterpret_cast<uint4*>(M.h1 + 64 * (size_t)node + 16 * q);
                    dst[0] = reinterpret_cast<uint4*>(hb)[0];
                    dst[1] = reinterpret_cast<uint4*>(hb)[1];
                }
            }
        } else if (t == 0) {
            atomicExch(M.err, 1);
        }
        sync_tmem();
    }
    if (warp == 0) tc::tmem_dealloc(tmem, 64);
}

// Layers 2, 3 and the output over nodes [n0, n1).  Inference (z2 == nullptr): the prediction
// previous dv + sigma_y y + mu_y is written to pred (may alias B.warm).  Training: z2, z3, y.
__global__ void __launch_bounds__(128, 4) cs_mlp_l23_kernel(Batch B, MlpDev M, int n0, int n1, float* __restrict__ z2,
                                                       float* __restrict__ z3, float* __restrict__ yout,
                                                       float* pred) {
    // 51 KB, so that four CTAs (4 x 128 TMEM columns) share an SM: the u2 tile is free once
    // layer 2's MMA is done, and then holds h2 and layer 3's weights
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;                  // 128 x 128 bf16: 32 KB
    unsigned char* sH = smem;                  // after layer 2's MMA: 128 x 64, 16 KB
    unsigned char* sW3 = smem + 16384;         // after layer 2's MMA: 64 x 64, 8 KB
    unsigned char* sW2 = smem + 32768;         // 64 x 128: 16 KB
    float* sf = reinterpret_cast<float*>(smem + 49152);  // W4 (192), b2 (64), b3 (64), b4 (3), mu_y, sigma_y
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 49152 + 2048);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
    const int t = threadIdx.x, warp = t >> 5;
    load_weight_tile(M.wb + MLP_W2, 64, 128, false, sW2);
    for (int e = t; e < 192; e += 128) sf[e] = __bfloat162float(M.wb[MLP_W4 + e]);
    for (int e = t; e < 64; e += 128) {
        sf[192 + e] = M.w[MLP_B2 + e];
        sf[256 + e] = M.w[MLP_B3 + e];
    }
    if (t < 3) {
        sf[320 + t] = M.w[MLP_B4 + t];
        sf[323 + t] = M.stats[32 + t];
        sf[326 + t] = M.stats[35 + t];
    }
    if (t == 0) tc::mbar_init(bar, 1);
    if (warp == 0) tc::tmem_alloc(slot, 128);
    tc::fence_async_shared();
    sync_tmem();
    const uint32_t tmem = *slot;
    uint32_t phase = 0;
    bool ok = true;
    const int ntiles = (n1 - n0 + 127) / 128;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int node = n0 + tile * 128 + t;
        const bool valid = node < n1;
        // u2 = [h1_i, bf16(mean h1_j)]
        if (valid) {
            // rows of h1 are 64 BF16 = 8 x 16 bytes; a K-major tile keeps 8 consecutive k of a
            // row contiguous, so both the gathers and the tile stores move 16 bytes at a time
            const uint4* hi = reinterpret_cast<const uint4*>(M.h1 + 64 * (size_t)node);
            Nbr nb = neighbours(B, node);
            const float inv = nb.end > nb.beg ? 1.0f / (nb.end - nb.beg) : 0.f;
            // the first kNbr neighbours' rows, looked up once for the four quarters of the row;
            // their loads are issued kBatch at a time before the (ordered) additions
            constexpr int kNbr = 8, kBatch = 4;
            const int cnt = nb.end - nb.beg;
            const uint4* nrow[kNbr];
#pragma unroll
            for (int j = 0; j < kNbr; j++)
                nrow[j] = reinterpret_cast<const uint4*>(M.h1 + 64 * (size_t)(j < cnt ? B.nbr[nb.beg + j] + nb.off : node));
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float acc[16];
#pragma unroll
                for (int c = 0; c < 16; c++) acc[c] = 0.f;
                auto add_row = [&](const uint4& v0, const uint4& v1) {
                    const __nv_bfloat16* e0 = reinterpret_cast<const __nv_bfloat16*>(&v0);
                    const __nv_bfloat16* e1 = reinterpret_cast<const __nv_bfloat16*>(&v1);
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        acc[c] += __bfloat162float(e0[c]);
                        acc[8 + c] += __bfloat162float(e1[c]);
                    }
                };
#pragma unroll
                for (int j0 = 0; j0 < kNbr; j0 += kBatch) {
                    uint4 v0[kBatch], v1[kBatch];
#pragma unroll
                    for (int j = 0; j < kBatch; j++)
                        if (j0 + j < cnt) {
                            v0[j] = __ldg(nrow[j0 + j] + 2 * q);
                            v1[j] = __ldg(nrow[j0 + j] + 2 * q + 1);
                        }
#pragma unroll
                    for (int j = 0; j < kBatch; j++)
                        if (j0 + j < cnt) add_row(v0[j], v1[j]);
                }
                for (int k = nb.beg + kNbr; k < nb.end; k++) {
                    const uint4* hj = reinterpret_cast<const uint4*>(M.h1 + 64 * (size_t)(B.nbr[k] + nb.off) + 16 * q);
                    add_row(__ldg(hj), __ldg(hj + 1));
                }
                *reinterpret_cast<uint4*>(sA + tc::kmajor_offset(128, t, 16 * q)) = __ldg(hi + 2 * q);
                *reinterpret_cast<uint4*>(sA + tc::kmajor_offset(128, t, 16 * q + 8)) = __ldg(hi + 2 * q + 1);
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    __align__(16) __nv_bfloat16 ab[8];
#pragma unroll
                    for (int c = 0; c < 8; c++) ab[c] = __float2bfloat16_rn(acc[8 * hh + c] * inv);
                    *reinterpret_cast<uint4*>(sA + tc::kmajor_offset(128, t, 64 + 16 * q + 8 * hh)) =
                        *reinterpret_cast<const uint4*>(ab);
                }
            }
        } else {
            const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
            for (int c = 0; c < 128; c += 8) *reinterpret_cast<uint4*>(sA + tc::kmajor_offset(128, t, c)) = zero;
        }
        tc::fence_async_shared();
        sync_tmem();
        if (t == 0) {
            tc::gemm_tile(tmem, tc::smem_u32(sA), tc::smem_u32(sW2), 128, 64, false);
            tc::mma_commit(bar);
        }
        ok = __syncthreads_and(tc::mbar_wait(bar, phase) ? 1 : 0) != 0;
        phase ^= 1;
        tc::fence_after_sync();
        if (!ok) break;
        // the u2 tile is free: layer 3's weights (row-major 64 x 64, this thread's 16 pairs, all
        // loads issued before the stores) into its second quarter; h2 goes into its first half
        {
            const uint32_t* w3g = reinterpret_cast<const uint32_t*>(M.wb + MLP_W3);
            uint32_t w3r[16];
#pragma unroll
            for (int i = 0; i < 16; i++) w3r[i] = __ldg(w3g + t + 128 * i);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int e = 2 * (t + 128 * i), r = e >> 6, k = e & 63;
                *reinterpret_cast<uint32_t*>(sW3 + tc::kmajor_offset(64, r, k)) = w3r[i];
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float zz[16];
            tc::tmem_ld16(tc::tmem_addr(tmem, warp, 16 * q), zz);
#pragma unroll
            for (int c = 0; c < 16; c++) {
                const float z = zz[c] + sf[192 + 16 * q + c];
                if (z2 && valid) z2[64 * (size_t)node + 16 * q + c] = z;
                tc::st_bf16(sH, 128, t, 16 * q + c, valid ? silu(z) : 0.f);
            }
        }
        tc::fence_async_shared();
        sync_tmem();
        if (t == 0) {
            tc::gemm_tile(tmem + 64, tc::smem_u32(sH), tc::smem_u32(sW3), 64, 64, false);
            tc::mma_commit(bar);
        }
        ok = __syncthreads_and(tc::mbar_wait(bar, phase) ? 1 : 0) != 0;
        phase ^= 1;
        tc::fence_after_sync();
        if (!ok) break;
        float y0 = sf[320], y1 = sf[321], y2 = sf[322];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float zz[16];
            tc::tmem_ld16(tc::tmem_addr(tmem, warp, 64 + 16 * q), zz);
#pragma unroll
            for (int c = 0; c < 16; c++) {
                const int j = 16 * q + c;
                const float z = zz[c] + sf[256 + j];
                if (z3 && valid) z3[64 * (size_t)node + j] = z;
                const float h = silu(z);
                y0 += sf[j] * h;
                y1 += sf[64 + j] * h;
                y2 += sf[128 + j] * h;
            }
        }
        if (valid) {
            if (yout) {
                yout[3 * (size_t)node] = y0;
                yout[3 * (size_t)node + 1] = y1;
                yout[3 * (size_t)node + 2] = y2;
            }
            if (pred) {
                const float p0 = B.warm[3 * node] + sf[326] * y0 + sf[323];
                const float p1 = B.warm[3 * node + 1] + sf[327] * y1 + sf[324];
                const float p2 = B.warm[3 * node + 2] + sf[328] * y2 + sf[325];
                pred[3 * node] = p0;
                pred[3 * node + 1] = p1;
                pred[3 * node + 2] = p2;
            }
        }
        sync_tmem();
    }
    if (!ok && t == 0) atomicExch(M.err, 1);
    sync_tmem();
    if (warp == 0) tc::tmem_dealloc(tmem, 128);
}

// Backward through the output layer, layer 3 and layer 2 over nodes [n0, n1) (one training
// minibatch of whole sheets, ntot nodes).  With a target: loss = sum_i ||y_i - t_i||^2 / ntot
// with t_i = (target_i - mu_y) / sigma_y.  Without (target == nullptr): the energy-norm loss,
// whose gradient with respect to the prediction, ga A p - gb b, the energy kernels left (A p in
// M.dy, ga and gb per sheet in M.sheet_scale; dL/dy = sigma_y dL/dp); its value comes from those
// kernels.  Writes du2 (N x 128) for
// layer 1's backward and this CTA's gradient partials of W2, b2, W3, b3, W4, b4 and of the loss.
//
// 512 threads per CTA (one CTA per SM: the tile's FP32 operands fill its shared memory).  What
// bounds it: the FP32 products of the weight gradients (12,288 multiply-adds a node) and their
// shared-memory reads, so a warp owns four rows of dW2 and dW3 (one broadcast 16-byte read of dz
// per node) and a lane 4 or 2 of their columns; element-wise phases run over contiguous memory, and
// TMEM rows are read by four warps each, a quarter of the columns per warp.  With 128 threads, a
// node per thread in the element-wise phases and a row per thread pair in the products, a minibatch
// of 16 sheets of 64 x 64 took 499 us on a B200.  Every sum runs over the tile's nodes in order.
#define MLP_BWD_LD 68  // floats per node row of the shared operands: 16-byte rows, 4 banks apart
__global__ void __launch_bounds__(MLP_BWD_THREADS, 1) cs_mlp_bwd23_kernel(Batch B, MlpDev M, int n0, int n1,
                                                                        const float* __restrict__ target) {
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int LD = MLP_BWD_LD, TILE = 128 * LD * 4;
    float* sDZ = reinterpret_cast<float*>(smem);                 // 128 x 64 fp32 (dz3, then dz2)
    float* sX = reinterpret_cast<float*>(smem + TILE);           // 128 x 64 fp32 (h3, then h2)
    __nv_bfloat16* sU = reinterpret_cast<__nv_bfloat16*>(smem + 2 * TILE);  // 128 x 128 bf16 (u2), rows of 136
    unsigned char* sA = smem + 3 * TILE;                         // 128 x 64 bf16 MMA operand
    unsigned char* sW3t = sA + 16384;                            // 64 x 64 bf16 (W3^T)
    unsigned char* sW2t = sW3t + 8192;                           // 128 x 64 bf16 (W2^T)
    float* sf = reinterpret_cast<float*>(sW2t + 16384);          // W4 (192), mu_y, sigma_y, dy (128 x 4), loss (128)
    uint64_t* bar = reinterpret_cast<uint64_t*>(sf + 840);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
    float* sDY = sf + 200;
    float* sL = sf + 712;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    load_weight_tile(M.wb + MLP_W3, 64, 64, true, sW3t);
    load_weight_tile(M.wb + MLP_W2, 64, 128, true, sW2t);
    for (int e = t; e < 192; e += MLP_BWD_THREADS) sf[e] = __bfloat162float(M.wb[MLP_W4 + e]);
    if (t < 3) {
        sf[192 + t] = M.stats[32 + t];
        sf[195 + t] = M.stats[35 + t];
    }
    if (t == 0) tc::mbar_init(bar, 1);
    if (warp == 0) tc::tmem_alloc(slot, 256);
    tc::fence_async_shared();
    sync_tmem();
    const uint32_t tmem = *slot;
    uint32_t phase = 0;
    bool ok = true;
    const float scale = 2.0f / (float)max(n1 - n0, 1);
    // rows 4 warp .. 4 warp + 3 of W2 (columns 4 lane ..) and W3 (columns 2 lane ..)
    float acc2[4][4], acc3[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int c = 0; c < 4; c++) acc2[i][c] = 0.f;
        acc3[i][0] = acc3[i][1] = 0.f;
    }
    float acc4 = 0.f, accb2 = 0.f, accb3 = 0.f, accb4 = 0.f, loss = 0.f;
    // this thread's TMEM row (a node of the tile) and quarter of the columns
    const int trow = 32 * (warp & 3) + lane, tq = warp >> 2;
    const int ntiles = (n1 - n0 + 127) / 128;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int base = n0 + tile * 128, rows = min(128, n1 - base);
        // 1. dy, h3, dz3
        if (t < 128) {
            const int node = base + t;
            float dy[3] = {0.f, 0.f, 0.f};
            if (t < rows && target) {
                for (int i = 0; i < 3; i++) {
                    const float tt = (target[3 * (size_t)node + i] - sf[192 + i]) / sf[195 + i];
                    const float d = M.y[3 * (size_t)node + i] - tt;
                    loss += d * d;
                    dy[i] = scale * d;
                }
            } else if (t < rows) {
                const int sh = B.node_sheet[node];
                const float ga = M.sheet_scale[2 * sh], gb = M.sheet_scale[2 * sh + 1];
                for (int i = 0; i < 3; i++)
                    dy[i] = (ga * M.dy[3 * (size_t)node + i] - gb * B.b[3 * (size_t)node + i]) * sf[195 + i];
            }
            for (int i = 0; i < 3; i++) sDY[4 * t + i] = dy[i];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int e = t + MLP_BWD_THREADS * k, n = e >> 4, j = 4 * (e & 15);
            const float4 z = n < rows ? __ldg(reinterpret_cast<const float4*>(M.z3 + 64 * (size_t)(base + n) + j))
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
            const float zz[4] = {z.x, z.y, z.z, z.w};
            float h[4], dz[4];
            __align__(8) __nv_bfloat16 db[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                h[c] = n < rows ? silu(zz[c]) : 0.f;
                const float dh = sDY[4 * n] * sf[j + c] + sDY[4 * n + 1] * sf[64 + j + c] + sDY[4 * n + 2] * sf[128 + j + c];
                dz[c] = n < rows ? dh * silu_grad(zz[c]) : 0.f;
                db[c] = __float2bfloat16_rn(dz[c]);
            }
            *reinterpret_cast<float4*>(sX + LD * n + j) = make_float4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<float4*>(sDZ + LD * n + j) = make_float4(dz[0], dz[1], dz[2], dz[3]);
            *reinterpret_cast<uint2*>(sA + tc::kmajor_offset(128, n, j)) = *reinterpret_cast<const uint2*>(db);
        }
        tc::fence_async_shared();
        sync_tmem();
        // 2. dh2 = bf16(dz3) W3 on the tensor cores, meanwhile dW4, db4, db3
        if (t == 0) {
            tc::gemm_tile(tmem, tc::smem_u32(sA), tc::smem_u32(sW3t), 64, 64, false);
            tc::mma_commit(bar);
        }
        if (t < 192) {
            const int i = t >> 6, j = t & 63;
#pragma unroll 8
            for (int n = 0; n < 128; n++) acc4 += sDY[4 * n + i] * sX[LD * n + j];
        } else if (t < 195) {
            for (int n = 0; n < 128; n++) accb4 += sDY[4 * n + (t - 192)];
        } else if (t >= 256 && t < 320) {
#pragma unroll 8
            for (int n = 0; n < 128; n++) accb3 += sDZ[LD * n + (t - 256)];
        }
        __syncthreads();
        // 3. h2 = bf16(SiLU(z2)) and dW3
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int e = t + MLP_BWD_THREADS * k, n = e >> 4, j = 4 * (e & 15);
            float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            if (n < rows) {
                z = __ldg(reinterpret_cast<const float4*>(M.z2 + 64 * (size_t)(base + n) + j));
                z = make_float4(bf(silu(z.x)), bf(silu(z.y)), bf(silu(z.z)), bf(silu(z.w)));
            }
            *reinterpret_cast<float4*>(sX + LD * n + j) = z;
        }
        __syncthreads();
#pragma unroll 4
        for (int n = 0; n < 128; n++) {
            const float4 d = *reinterpret_cast<const float4*>(sDZ + LD * n + 4 * warp);
            const float2 x = *reinterpret_cast<const float2*>(sX + LD * n + 2 * lane);
            const float dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc3[i][0] += dd[i] * x.x;
                acc3[i][1] += dd[i] * x.y;
            }
        }
        ok = __syncthreads_and(tc::mbar_wait(bar, phase) ? 1 : 0) != 0;
        phase ^= 1;
        tc::fence_after_sync();
        if (!ok) break;
        // 4. dz2 = dh2 * SiLU'(z2); u2 rebuilt, four threads per node
        float dz2[16];
        {
            float dh[16];
            tc::tmem_ld16(tc::tmem_addr(tmem, warp & 3, 16 * tq), dh);
            const float4* z = reinterpret_cast<const float4*>(M.z2 + 64 * (size_t)(base + trow) + 16 * tq);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float4 v = trow < rows ? __ldg(z + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                dz2[4 * c] = trow < rows ? dh[4 * c] * silu_grad(v.x) : 0.f;
                dz2[4 * c + 1] = trow < rows ? dh[4 * c + 1] * silu_grad(v.y) : 0.f;
                dz2[4 * c + 2] = trow < rows ? dh[4 * c + 2] * silu_grad(v.z) : 0.f;
                dz2[4 * c + 3] = trow < rows ? dh[4 * c + 3] * silu_grad(v.w) : 0.f;
            }
        }
        {
            const int n = t >> 2, q = t & 3;
            uint4 own[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
            float acc[16];
#pragma unroll
            for (int c = 0; c < 16; c++) acc[c] = 0.f;
            float inv = 0.f;
            if (n < rows) {
                const uint4* hi = reinterpret_cast<const uint4*>(M.h1 + 64 * (size_t)(base + n) + 16 * q);
                own[0] = __ldg(hi);
                own[1] = __ldg(hi + 1);
                const Nbr nb = neighbours(B, base + n);
                inv = nb.end > nb.beg ? 1.0f / (nb.end - nb.beg) : 0.f;
                for (int k0 = nb.beg; k0 < nb.end; k0 += 4) {
                    uint4 v[4][2];
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (k0 + k < nb.end) {
                            const uint4* hj =
                                reinterpret_cast<const uint4*>(M.h1 + 64 * (size_t)(__ldg(B.nbr + k0 + k) + nb.off) + 16 * q);
                            v[k][0] = __ldg(hj);
                            v[k][1] = __ldg(hj + 1);
                        }
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (k0 + k < nb.end) {
                            const __nv_bfloat16* hv = reinterpret_cast<const __nv_bfloat16*>(v[k]);
#pragma unroll
                            for (int c = 0; c < 16; c++) acc[c] += __bfloat162float(hv[c]);
                        }
                }
            }
            __align__(16) __nv_bfloat16 ab[16];
#pragma unroll
            for (int c = 0; c < 16; c++) ab[c] = __float2bfloat16_rn(acc[c] * inv);
            uint4* u = reinterpret_cast<uint4*>(sU + 136 * n + 16 * q);
            u[0] = own[0];
            u[1] = own[1];
            u[8] = reinterpret_cast<const uint4*>(ab)[0];
            u[9] = reinterpret_cast<const uint4*>(ab)[1];
        }
        sync_tmem();  // every thread is done reading dz3 (sDZ) for dW3
        {
            __align__(16) __nv_bfloat16 db[16];
#pragma unroll
            for (int c = 0; c < 4; c++)
                *reinterpret_cast<float4*>(sDZ + LD * trow + 16 * tq + 4 * c) =
                    make_float4(dz2[4 * c], dz2[4 * c + 1], dz2[4 * c + 2], dz2[4 * c + 3]);
#pragma unroll
            for (int c = 0; c < 16; c++) db[c] = __float2bfloat16_rn(dz2[c]);
            *reinterpret_cast<uint4*>(sA + tc::kmajor_offset(128, trow, 16 * tq)) = reinterpret_cast<const uint4*>(db)[0];
            *reinterpret_cast<uint4*>(sA + tc::kmajor_offset(128, trow, 16 * tq + 8)) = reinterpret_cast<const uint4*>(db)[1];
        }
        tc::fence_async_shared();
        sync_tmem();
        // 5. du2 = bf16(dz2) W2 on the tensor cores, meanwhile dW2 and db2
        if (t == 0) {
            tc::gemm_tile(tmem + 64, tc::smem_u32(sA), tc::smem_u32(sW2t), 64, 128, false);
            tc::mma_commit(bar);
        }
#pragma unroll 4
        for (int n = 0; n < 128; n++) {
            const float4 d = *reinterpret_cast<const float4*>(sDZ + LD * n + 4 * warp);
            const uint2 xb = *reinterpret_cast<const uint2*>(sU + 136 * n + 4 * lane);
            const __nv_bfloat16* xv = reinterpret_cast<const __nv_bfloat16*>(&xb);
            const float dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float x = __bfloat162float(xv[c]);
#pragma unroll
                for (int i = 0; i < 4; i++) acc2[i][c] += dd[i] * x;
            }
        }
        if (t < 64)
#pragma unroll 8
            for (int n = 0; n < 128; n++) accb2 += sDZ[LD * n + t];
        ok = __syncthreads_and(tc::mbar_wait(bar, phase) ? 1 : 0) != 0;
        phase ^= 1;
        tc::fence_after_sync();
        if (!ok) break;
        // 6. du2 out
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float du[16];
            tc::tmem_ld16(tc::tmem_addr(tmem, warp & 3, 64 + 32 * tq + 16 * h), du);
            if (trow < rows) {
                float4* dst = reinterpret_cast<float4*>(M.du2 + 128 * (size_t)(base + trow) + 32 * tq + 16 * h);
#pragma unroll
                for (int c = 0; c < 4; c++) dst[c] = make_float4(du[4 * c], du[4 * c + 1], du[4 * c + 2], du[4 * c + 3]);
            }
        }
        sync_tmem();
    }
    if (!ok && t == 0) atomicExch(M.err, 1);
    sync_tmem();
    if (warp == 0) tc::tmem_dealloc(tmem, 256);
    // this CTA's partials
    float* gp = M.gpart + (size_t)blockIdx.x * MLP_P;
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int c = 0; c < 4; c++) gp[MLP_W2 + 128 * (4 * warp + i) + 4 * lane + c] = acc2[i][c];
#pragma unroll
        for (int c = 0; c < 2; c++) gp[MLP_W3 + 64 * (4 * warp + i) + 2 * lane + c] = acc3[i][c];
    }
    if (t < 64) gp[MLP_B2 + t] = accb2;
    if (t >= 256 && t < 320) gp[MLP_B3 + t - 256] = accb3;
    if (t < 192) gp[MLP_W4 + t] = acc4;
    else if (t < 195) gp[MLP_B4 + t - 192] = accb4;
    // loss partial (fixed-order block sum)
    if (t < 128) sL[t] = loss;
    __syncthreads();
    if (t == 0) {
        float s = 0.f;
        for (int i = 0; i < 128; i++) s += sL[i];
        M.loss_part[blockIdx.x] = s / (float)max(n1 - n0, 1);
    }
}

// Backward into layer 1 over nodes [n0, n1): dh1_i = du2_i[0:64] + sum over neighbours j of
// du2_j[64:128] / deg_j (the transpose of the mean aggregation), dz1 = dh1 * SiLU'(z1),
// and this CTA's partials of W1, b1.  Four threads per node gather 16 of its 64 columns each; a warp
// owns four rows of dW1, a lane one column (as in cs_mlp_bwd23_kernel; 233 us before, with a node
// per thread, for a minibatch of 16 sheets of 64 x 64).
__global__ void __launch_bounds__(MLP_BWD_THREADS) cs_mlp_bwd1_kernel(Batch B, MlpDev M, const float* __restrict__ fsrc,
                                                                    int n0, int n1) {
    extern __shared__ __align__(16) float dyn[];
    constexpr int LD = MLP_BWD_LD, LU = 36;
    float* sDZ = dyn;               // 128 x 64
    float* sU = dyn + 128 * LD;     // 128 x 32
    float* sst = sU + 128 * LU;     // 32
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t < 32) sst[t] = M.stats[t];
    __syncthreads();
    float acc1[4] = {0.f, 0.f, 0.f, 0.f}, accb1 = 0.f;
    const int n = t >> 2, q = t & 3;
    const int ntiles = (n1 - n0 + 127) / 128;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int node = n0 + tile * 128 + n;
        const bool valid = node < n1;
        if (valid) {
            const SheetDesc& sh = B.sheets[B.node_sheet[node]];
            const int* np = B.nbr_ptr + sh.nbr_ptr_off;  // the neighbours are of the same sheet
            const int beg = sh.nbr_off + np[node - sh.node_off], end = sh.nbr_off + np[node - sh.node_off + 1];
            float dh[16];
            {
                const float4* d = reinterpret_cast<const float4*>(M.du2 + 128 * (size_t)node + 16 * q);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float4 v = __ldg(d + c);
                    dh[4 * c] = v.x;
                    dh[4 * c + 1] = v.y;
                    dh[4 * c + 2] = v.z;
                    dh[4 * c + 3] = v.w;
                }
            }
            const float4 x = __ldg(reinterpret_cast<const float4*>(fsrc + 16 * (size_t)node) + q);
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            for (int k0 = beg; k0 < end; k0 += 2) {
                float4 v[2][4], xj[2];
                float w[2];
#pragma unroll
                for (int k = 0; k < 2; k++)
                    if (k0 + k < end) {
                        const int lg = __ldg(B.nbr + k0 + k);
                        w[k] = 1.0f / (float)(__ldg(np + lg + 1) - __ldg(np + lg));
                        const float4* d = reinterpret_cast<const float4*>(M.du2 + 128 * (size_t)(lg + sh.node_off) + 64 + 16 * q);
#pragma unroll
                        for (int c = 0; c < 4; c++) v[k][c] = __ldg(d + c);
                        xj[k] = __ldg(reinterpret_cast<const float4*>(fsrc + 16 * (size_t)(lg + sh.node_off)) + q);
                    }
#pragma unroll
                for (int k = 0; k < 2; k++)
                    if (k0 + k < end) {
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            dh[4 * c] += v[k][c].x * w[k];
                            dh[4 * c + 1] += v[k][c].y * w[k];
                            dh[4 * c + 2] += v[k][c].z * w[k];
                            dh[4 * c + 3] += v[k][c].w * w[k];
                        }
                        acc[0] += xj[k].x;
                        acc[1] += xj[k].y;
                        acc[2] += xj[k].z;
                        acc[3] += xj[k].w;
                    }
            }
            const float4* z = reinterpret_cast<const float4*>(M.z1 + 64 * (size_t)node + 16 * q);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float4 v = __ldg(z + c);
                *reinterpret_cast<float4*>(sDZ + LD * n + 16 * q + 4 * c) =
                    make_float4(dh[4 * c] * silu_grad(v.x), dh[4 * c + 1] * silu_grad(v.y), dh[4 * c + 2] * silu_grad(v.z),
                                dh[4 * c + 3] * silu_grad(v.w));
            }
            // u1 = bf16([x, agg(x)]) as in the forward pass
            const float xs[4] = {x.x, x.y, x.z, x.w};
            const float inv = end > beg ? 1.0f / (end - beg) : 0.f;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float mu = sst[4 * q + c], sg = sst[16 + 4 * q + c];
                sU[LU * n + 4 * q + c] = bf((xs[c] - mu) / sg);
                sU[LU * n + 16 + 4 * q + c] = end > beg ? bf((acc[c] * inv - mu) / sg) : 0.f;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 16; c++) sDZ[LD * n + 16 * q + c] = 0.f;
#pragma unroll
            for (int c = 0; c < 8; c++) sU[LU * n + 8 * q + c] = 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < 128; k++) {
            const float4 d = *reinterpret_cast<const float4*>(sDZ + LD * k + 4 * warp);
            const float u = sU[LU * k + lane];
            acc1[0] += d.x * u;
            acc1[1] += d.y * u;
            acc1[2] += d.z * u;
            acc1[3] += d.w * u;
        }
        if (t < 64)
#pragma unroll 8
            for (int k = 0; k < 128; k++) accb1 += sDZ[LD * k + t];
        __syncthreads();
    }
    float* gp = M.gpart + (size_t)blockIdx.x * MLP_P;
#pragma unroll
    for (int i = 0; i < 4; i++) gp[MLP_W1 + 32 * (4 * warp + i) + lane] = acc1[i];
    if (t < 64) gp[MLP_B1 + t] = accb1;
}

// Sums the per-CTA gradient partials in CTA order (deterministic), then one Adam step
// (Kingma & Ba 2015) on the FP32 master weights and a refresh of their BF16 copies.  With
// lr == 0 only the summed gradient is written to grad_out (gradient checks).
__global__ void cs_mlp_adam_kernel(MlpDev M, int ncta, float lr, float b1, float b2, float eps, int step,
                                   float* grad_out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= MLP_P) return;
    float g = 0.f;
    for (int c = 0; c < ncta; c++) g += M.gpart[(size_t)c * MLP_P + p];
    if (grad_out) grad_out[p] = g;
    if (lr == 0.f) return;
    const float m = b1 * M.m[p] + (1.f - b1) * g;
    const float v = b2 * M.v[p] + (1.f - b2) * g * g;
    M.m[p] = m;
    M.v[p] = v;
    const float mh = m / (1.f - powf(b1, (float)step));
    const float vh = v / (1.f - powf(b2, (float)step));
    const float w = M.w[p] - lr * mh / (sqrtf(vh) + eps);
    M.w[p] = w;
    M.wb[p] = __float2bfloat16_rn(w);
}

// The same Adam update from a gradient held in a device buffer (summed or averaged over
// ranks by the caller).
__global__ void cs_mlp_adam_ext_kernel(MlpDev M, const float* __restrict__ grad, float lr, float b1, float b2,
                                       float eps, int step) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= MLP_P) return;
    const float g = grad[p];
    const float m = b1 * M.m[p] + (1.f - b1) * g;
    const float v = b2 * M.v[p] + (1.f - b2) * g * g;
    M.m[p] = m;
    M.v[p] = v;
    const float mh = m / (1.f - powf(b1, (float)step));
    const float vh = v / (1.f - powf(b2, (float)step));
    const float w = M.w[p] - lr * mh / (sqrtf(vh) + eps);
    M.w[p] = w;
    M.wb[p] = __float2bfloat16_rn(w);
}

// Training pair bookkeeping: the dataset slot receives the raw features of the current
// assembled system (with the previous dv held in B.warm) and, after the solve, the target
// dv - previous dv.
__global__ void cs_mlp_target_kernel(Batch B, const float* __restrict__ feat, float* __restrict__ target) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * B.N) return;
    const int node = i / 3, c = i % 3;
    target[i] = B.dv[i] - feat[16 * (size_t)node + 12 + c];
}

// Sums and sums of squares of the 16 features and 3 targets over nodes (FP64 per block).
__global__ void cs_mlp_moments_kernel(const float* __restrict__ feat, const float* __restrict__ target, long long n,
                                      double* __restrict__ out) {
    __shared__ double sh[38 * 128];
    double acc[38];
    for (int c = 0; c < 38; c++) acc[c] = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        for (int c = 0; c < 16; c++) {
            double x = feat[16 * i + c];
            acc[c] += x;
            acc[19 + c] += x * x;
        }
        for (int c = 0; c < 3; c++) {
            double x = target[3 * i + c];
            acc[16 + c] += x;
            acc[35 + c] += x * x;
        }
    }
    for (int c = 0; c < 38; c++) sh[38 * threadIdx.x + c] = acc[c];
    __syncthreads();
    if (threadIdx.x < 38) {
        double s = 0.0;
        for (int k = 0; k < (int)blockDim.x; k++) s += sh[38 * k + threadIdx.x];
        out[38 * blockIdx.x + threadIdx.x] = s;
    }
}

// Adds this minibatch's loss (sum of the per-CTA partials, in CTA order) to *acc.
__global__ void cs_mlp_loss_acc_kernel(MlpDev M, int ncta, float* acc) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    float s = 0.f;
    for (int c = 0; c < ncta; c++) s += M.loss_part[c];
    *acc += s;
}

// ---------------------------------------------------------------------------------------
// Energy-norm training.  For a sheet with system A dv = b and solution dv*, the warm start the
// solver takes from a prediction p is its Galerkin multiple alpha p, alpha = p^T b / p^T A p
// (warm_scale), whose error in the energy norm is that of the zero guess times sin(theta),
// theta the angle between p and dv* in the A inner product.  The loss is therefore
//     L = sin^2(theta) = 1 - (p^T b)^2 / ((p^T A p)(dv*^T b))      (A dv* = b, in [0, 1]),
// scale-free and bounded; with u = p^T b, w = p^T A p, c = dv*^T b:
//     dL/dp = (2 u / (w c)) (alpha A p - b): one SpMV of the prediction.
// A minibatch's loss is the mean over its sheets.

namespace {
__device__ __forceinline__ double rwsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
}  // namespace

// Per row q = A p into M.dy over slices [sl0, sl1) (a warp per slice, its rows as the SELL
// panels hold them), and per slice the FP64 partials of p.b and p.A p.
__global__ void __launch_bounds__(128) cs_mlp_energy_kernel(Batch B, MlpDev M, int sl0, int sl1) {
    const int slice = sl0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (slice >= sl1) return;
    const SliceDesc sd = B.slices[slice];
    const int node_off = B.sheets[sd.sheet].node_off;
    const float* __restrict__ x = M.pred;
    double pb = 0.0, pq = 0.0;
    if (lane < sd.rows) {
        const int row = sd.row0 + B.rowmap[sd.topo_slice * CS_SLICE + lane];
        float y0 = 0.f, y1 = 0.f, y2 = 0.f;
        for (int k = 0; k < sd.width; k++) {
            const int col = B.tcol[(sd.tpanel0 + k) * CS_SLICE + lane] + node_off;
            const float* panel = B.A + (size_t)(sd.panel0 + k) * CS_PANEL_FLOATS;
            const float4 a0 = reinterpret_cast<const float4*>(panel)[lane];
            const float4 a1 = reinterpret_cast<const float4*>(panel + 128)[lane];
            const float a8 = panel[256 + lane];
            const float p0 = x[3 * col], p1 = x[3 * col + 1], p2 = x[3 * col + 2];
            y0 += a0.x * p0 + a0.y * p1 + a0.z * p2;
            y1 += a0.w * p0 + a1.x * p1 + a1.y * p2;
            y2 += a1.z * p0 + a1.w * p1 + a8 * p2;
        }
        if (B.xptr) {
            for (int m = B.xptr[row]; m < B.xptr[row + 1]; m++) {
                const int col = B.xcol[m];
                const float* a = B.xval + 9 * (size_t)m;
                const float p0 = x[3 * col], p1 = x[3 * col + 1], p2 = x[3 * col + 2];
                y0 += a[0] * p0 + a[1] * p1 + a[2] * p2;
                y1 += a[3] * p0 + a[4] * p1 + a[5] * p2;
                y2 += a[6] * p0 + a[7] * p1 + a[8] * p2;
            }
        }
        const float y[3] = {y0, y1, y2};
#pragma unroll
        for (int c = 0; c < 3; c++) {
            M.dy[3 * row + c] = y[c];
            pb += (double)x[3 * row + c] * (double)B.b[3 * row + c];
            pq += (double)x[3 * row + c] * (double)y[c];
        }
    }
    pb = rwsum(pb);
    pq = rwsum(pq);
    if (lane == 0) {
        M.epart[2 * slice] = pb;
        M.epart[2 * slice + 1] = pq;
    }
}

// Per slice the FP64 partial of dv64 . b (the solution's energy dv*^T A dv* = dv*^T b).
__global__ void __launch_bounds__(128) cs_mlp_energy_norm_kernel(Batch B, MlpDev M, int sl0, int sl1) {
    const int slice = sl0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (slice >= sl1) return;
    const SliceDesc sd = B.slices[slice];
    double e = 0.0;
    if (lane < sd.rows) {
        const int row = sd.row0 + B.rowmap[sd.topo_slice * CS_SLICE + lane];
#pragma unroll
        for (int c = 0; c < 3; c++) e += B.dv64[3 * row + c] * (double)B.b[3 * row + c];
    }
    e = rwsum(e);
    if (lane == 0) {
        M.epart[2 * slice] = e;
        M.epart[2 * slice + 1] = 0.0;
    }
}

// A block per sheet of [s0, s1) sums its slices' partials in a fixed order.  mode 0: the
// solution's energy c into M.sheet_c; mode 1: with u = p.b, w = p.A p, the sheet's loss
// 1 - u^2 / (w c) and the two coefficients of its gradient dL/dp = ga A p - gb b,
// gb = 2 u / (w c (s1 - s0)), ga = gb u / w (a sheet with w <= 0 or c <= 0: loss 1, no gradient).
__global__ void __launch_bounds__(128) cs_mlp_energy_sheet_kernel(Batch B, MlpDev M, int s0, int s1, int mode) {
    __shared__ double sh[8];
    const int s = s0 + blockIdx.x;
    if (s >= s1) return;
    const SheetDesc& d = B.sheets[s];
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < d.n_slices; i += blockDim.x) {
        a += M.epart[2 * (d.slice_off + i)];
        b += M.epart[2 * (d.slice_off + i) + 1];
    }
    a = rwsum(a);
    b = rwsum(b);
    if ((threadIdx.x & 31) == 0) {
        sh[2 * (threadIdx.x >> 5)] = a;
        sh[2 * (threadIdx.x >> 5) + 1] = b;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double u = (sh[0] + sh[2]) + (sh[4] + sh[6]);
    const double w = (sh[1] + sh[3]) + (sh[5] + sh[7]);
    if (mode == 0) {
        M.sheet_c[s] = u;
        return;
    }
    const double c = M.sheet_c[s];
    if (w > 0.0 && c > 0.0) {
        const double gb = 2.0 * u / (w * c * (double)(s1 - s0));
        M.sheet_loss[s] = (float)(1.0 - u * u / (w * c));
        M.sheet_scale[2 * s] = (float)(gb * u / w);
        M.sheet_scale[2 * s + 1] = (float)gb;
    } else {
        M.sheet_loss[s] = 1.f;
        M.sheet_scale[2 * s] = 0.f;
        M.sheet_scale[2 * s + 1] = 0.f;
    }
}

// *acc += the mean of the sheets' losses over [s0, s1), summed in sheet order.
__global__ void cs_mlp_energy_loss_kernel(MlpDev M, int s0, int s1, float* acc) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    float t = 0.f;
    for (int s = s0; s < s1; s++) t += M.sheet_loss[s];
    *acc += t / (float)max(s1 - s0, 1);
}
