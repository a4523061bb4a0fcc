// Allocation-free solve of one block-sparse system, for callers that cannot allocate device
// memory.  It has no counterpart in the reference.
//
// Who needs it: code that runs where cudaMalloc is unavailable or forbidden -- a host that
// owns every byte of device memory through its own allocator (game engines, simulation
// frameworks with fixed arenas), real-time loops that must not allocate for latency
// reasons, or plugins that may not grow the process's device footprint after start-up.
// Such a caller passes its system and output buffers; the solver's scratch vectors live
// in one fixed, file-scope device array instead of memory allocated per call.
//
// Limits and behaviour:
//   * at most CS_NOALLOC_MAX_ROWS (16384) block rows; larger systems are rejected with
//     CS_ERR_INVALID_ARG before anything is launched;
//   * the scratch array (kNoallocBytes, 2 MiB) is a static __device__ variable, so every GPU
//     that loads this library holds it until the process exits;
//   * every call on a device shares that one array and leaves its contents behind; the kernel
//     initialises everything it reads, so nothing has to start at zero between calls, but two
//     calls that overlap on the GPU (different streams, or concurrent host threads) race on
//     it and give wrong results -- serialise them;
//   * the array's device address is looked up with cudaGetSymbolAddress on the first call on
//     each device (with that device current) and cached; make that first call before any
//     stream capture begins;
//   * no cudaMalloc, cudaFree or allocating library routine is called.
//
// Algorithm: the scheme of the cluster-resident solver (resident.cu) for a single system: FP32
// block-Jacobi PCG in Chronopoulos-Gear form (one fused reduction of r.u, w.u, r.r per iteration)
// with FP64 dot products, and FP64 residual replacements that keep the search direction (reliable
// updates), run by one thread-block cluster.
//   * The rows are split evenly over the cluster's CTAs, four lanes per row: lane q of a row
//     takes its blocks q, q + 4, ... and lanes 0-2 then hold the row's three components.
//   * Each CTA keeps its rows' vectors and block-Jacobi inverses in shared memory, and of its
//     blocks as many as fit beside them (read from the caller's arrays once per solve; the rest
//     from L2 every iteration).  u = P^-1 r is exchanged through the scratch array.
//   * Two cluster barriers per iteration (u written; partial sums written to every CTA through
//     distributed shared memory).  Every sum runs in a fixed order: the same bits on every run.
// What bounds it: the two barriers and the latency of the u gather at small sizes, the shared
// memory and L2 reads of the blocks at large ones.  One CTA did all of this before: one SM's
// loads in flight took 31.2 ms for the 4,225 rows of a 64 x 64 sheet at tol 1e-8 on a B200, the
// cluster of 16 takes 2.77 ms (2.48 with a last sweep that ends at the tolerance).
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "../../include/clothstep.h"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32, kRowLanes = 4, kPass = kThreads / kRowLanes;
constexpr int kMaxCtas = 16;
// Scratch: dv64 (3 doubles) and u (4 floats) per block row, then the statistics.
constexpr size_t kRowBytes = 3 * sizeof(double) + 4 * sizeof(float);
constexpr size_t kNoallocBytes = 2u << 20;
static_assert((size_t)CS_NOALLOC_MAX_ROWS * kRowBytes + 256 <= kNoallocBytes, "scratch too small");

// Shared memory of a CTA per own row: the block-Jacobi inverse, r, e, p, s, u, w; and per block
// kept on chip: its nine entries and its column.
constexpr size_t kRowSmem = (9 + 6 * 3) * sizeof(float), kBlockSmem = 9 * sizeof(float) + sizeof(int);
constexpr double kInnerTol = 1e-2;  // residual reduction between FP64 residual replacements
// The last sweep goes below the tolerance: ended at it, x was up to 2.7 times farther from the 64-bit
// solution than that of the solver of one CTA, which overshot it (100 x 100 quads at 1e-8).
constexpr double kLastSweep = 0.2;
constexpr double kDrift = 0.1;      // largest relative drift of r at which the direction is kept
constexpr int kSweeps = 128;

// The fixed scratch array.  Host code must not pass `g_scratch` itself to a kernel: on the host
// that name is only a stand-in, not a device address.  Its address comes from
// cudaGetSymbolAddress (launch_plan below).
static __device__ __align__(256) unsigned char g_scratch[kNoallocBytes];

struct NoallocShared {
    double wsum[kWarps][3];
    double red[2][kMaxCtas][3];  // partial sums by sender, two buffers
    int bad[kMaxCtas];
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Cluster-wide sums of three values: warp butterflies, warp partials in order, CTA partials in
// rank order.  The buffer alternates, and a cluster barrier lies between a buffer's reads and the
// writes of the reduction after next.
__device__ __forceinline__ void cluster_sum3(cg::cluster_group& cl, NoallocShared& S, int& nred, double (&v)[3]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ncta = (int)cl.num_blocks();
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] = warp_sum(v[i]);
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < 3; i++) S.wsum[w][i] = v[i];
    __syncthreads();
    const int b = nred & 1;
    if (w == 0 && lane < ncta) {
        double t[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int j = 0; j < kWarps; j++)
#pragma unroll
            for (int i = 0; i < 3; i++) t[i] += S.wsum[j][i];
        double* dst = cl.map_shared_rank(&S.red[b][cl.block_rank()][0], lane);
#pragma unroll
        for (int i = 0; i < 3; i++) dst[i] = t[i];
    }
    cl.sync();
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] = 0.0;
    for (int c = 0; c < ncta; c++)
#pragma unroll
        for (int i = 0; i < 3; i++) v[i] += S.red[b][c][i];
    nred++;
}

// The three components of a row summed over its four lanes (q = lane of the row); lane q < 3
// returns component q.
template <class T>
__device__ __forceinline__ T row_component(T y0, T y1, T y2, int q) {
#pragma unroll
    for (int o = 1; o < kRowLanes; o <<= 1) {
        y0 += __shfl_xor_sync(0xffffffffu, y0, o);
        y1 += __shfl_xor_sync(0xffffffffu, y1, o);
        y2 += __shfl_xor_sync(0xffffffffu, y2, o);
    }
    return q == 0 ? y0 : (q == 1 ? y1 : y2);
}

__global__ void __launch_bounds__(kThreads, 1) noalloc_pcg_kernel(int n, int nnzb, const int32_t* __restrict__ rp,
                                                             const int32_t* __restrict__ ci,
                                                             const float* __restrict__ val,
                                                             const float* __restrict__ b, float* __restrict__ x,
                                                             double tol, int max_iters, unsigned char* base, int block_cap) {
    extern __shared__ __align__(16) unsigned char noalloc_smem[];
    __shared__ NoallocShared S;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks();
    const int t = threadIdx.x, q = t & (kRowLanes - 1), g0 = t / kRowLanes;
    const int r0 = (int)((long long)n * rank / ncta), r1 = (int)((long long)n * (rank + 1) / ncta);
    const int R = r1 - r0, RM = (n + ncta - 1) / ncta;
    double* const dv64 = reinterpret_cast<double*>(base);
    float4* const U = reinterpret_cast<float4*>(base + (size_t)3 * CS_NOALLOC_MAX_ROWS * sizeof(double));
    double* const stats = reinterpret_cast<double*>(base + kNoallocBytes - 256);
    float* const Pi = reinterpret_cast<float*>(noalloc_smem);
    float* const sr = Pi + 9 * RM;
    float* const se = sr + 3 * RM;
    float* const sp = se + 3 * RM;
    float* const ss = sp + 3 * RM;
    float* const su = ss + 3 * RM;
    float* const sw = su + 3 * RM;
    float* const sval = sw + 3 * RM;
    int* const scol = reinterpret_cast<int*>(sval + 9 * (size_t)block_cap);
    // Row ranges and column indices are checked first; any entry outside [0, nnzb) x [0, n)
    // ends the call with CS_ERR_INVALID_ARG before the matrix or vectors are read.
    bool mine_bad = false;
    for (int i = r0 + t; i < r1; i += kThreads) {
        const int k0 = rp[i], k1 = rp[i + 1];
        if (k0 < 0 || k1 < k0 || k1 > nnzb) mine_bad = true;
        else
            for (int k = k0; k < k1; k++)
                if ((unsigned)ci[k] >= (unsigned)n) mine_bad = true;
    }
    const int cta_bad = __syncthreads_or(mine_bad ? 1 : 0);
    cl.sync();  // every CTA runs before any write to its shared memory
    if (t < ncta) *cl.map_shared_rank(&S.bad[rank], t) = cta_bad;
    cl.sync();
    int bad = 0;
    for (int c = 0; c < ncta; c++) bad |= S.bad[c];
    if (bad) {
        // x becomes NaN, so that a caller of the asynchronous form (which gets no status from
        // the device) cannot take stale contents of x for a solution
        for (int i = 3 * r0 + t; i < 3 * r1; i += kThreads) x[i] = __int_as_float(0x7fc00000);
        if (rank == 0 && t == 0) {
            stats[0] = 0;
            stats[1] = -1.0;
            stats[2] = CS_ERR_INVALID_ARG;
        }
        return;  // uniform over the cluster, after its last remote access
    }
    // the CTA's blocks, up to the budget, into shared memory (its rows' ranges follow one another)
    const int kbase = R > 0 ? rp[r0] : 0, kcap = kbase + min(block_cap, R > 0 ? rp[r1] - kbase : 0);
    for (int k = t; k < 9 * (kcap - kbase); k += kThreads) sval[k] = val[9 * (size_t)kbase + k];
    for (int k = kbase + t; k < kcap; k += kThreads) scol[k - kbase] = ci[k];
    // set-up: block-Jacobi inverses, dv64 = 0, e = 0, r = b, ||b||
    double bb[3] = {0.0, 0.0, 0.0};
    for (int i = t; i < R; i += kThreads) {
        const int row = r0 + i;
        double m[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int k = rp[row]; k < rp[row + 1]; k++)
            if (ci[k] == row)
                for (int c = 0; c < 9; c++) m[c] = val[9 * (size_t)k + c];
        double c00 = m[4] * m[8] - m[5] * m[7], c01 = m[5] * m[6] - m[3] * m[8], c02 = m[3] * m[7] - m[4] * m[6];
        double det = m[0] * c00 + m[1] * c01 + m[2] * c02;
        double id = det != 0.0 ? 1.0 / det : 0.0;
        float* P = Pi + 9 * i;
        P[0] = (float)(c00 * id);
        P[1] = (float)((m[2] * m[7] - m[1] * m[8]) * id);
        P[2] = (float)((m[1] * m[5] - m[2] * m[4]) * id);
        P[3] = (float)(c01 * id);
        P[4] = (float)((m[0] * m[8] - m[2] * m[6]) * id);
        P[5] = (float)((m[2] * m[3] - m[0] * m[5]) * id);
        P[6] = (float)(c02 * id);
        P[7] = (float)((m[1] * m[6] - m[0] * m[7]) * id);
        P[8] = (float)((m[0] * m[4] - m[1] * m[3]) * id);
        for (int c = 0; c < 3; c++) {
            const float bi = b[3 * row + c];
            dv64[3 * row + c] = 0.0;
            se[3 * i + c] = 0.f;
            sr[3 * i + c] = bi;
            bb[0] += (double)bi * bi;
        }
    }
    int nred = 0;
    cluster_sum3(cl, S, nred, bb);
    const double bn = sqrt(bb[0]);
    int iters = 0, sweep_iters = 0;
    double rel = 0.0, gam = 0.0, gam_prev = 0.0;
    int status = CS_ERR_NOT_CONVERGED;

    // u = P^-1 r for every own row, into shared memory and the exchange array; `step`: first
    // e += alpha p, r -= alpha s
    auto precondition = [&](bool step, float alpha) {
        for (int i0 = 0; i0 < R; i0 += kPass) {
            const int i = i0 + g0;
            const bool on = i < R && q < 3;
            float rc = 0.f;
            if (on) {
                rc = sr[3 * i + q];
                if (step) {
                    se[3 * i + q] = __fmaf_rn(alpha, sp[3 * i + q], se[3 * i + q]);
                    rc = __fmaf_rn(-alpha, ss[3 * i + q], rc);
                    sr[3 * i + q] = rc;
                }
            }
            const int l0 = (t & 31) & ~(kRowLanes - 1);
            const float a0 = __shfl_sync(0xffffffffu, rc, l0), a1 = __shfl_sync(0xffffffffu, rc, l0 + 1),
                        a2 = __shfl_sync(0xffffffffu, rc, l0 + 2);
            float uc = 0.f;
            if (on) {
                const float* P = Pi + 9 * i + 3 * q;
                uc = P[0] * a0 + P[1] * a1 + P[2] * a2;
                su[3 * i + q] = uc;
            }
            const float u0 = __shfl_sync(0xffffffffu, uc, l0), u1 = __shfl_sync(0xffffffffu, uc, l0 + 1),
                        u2 = __shfl_sync(0xffffffffu, uc, l0 + 2);
            if (on && q == 0) U[r0 + i] = make_float4(u0, u1, u2, 0.f);
        }
    };
    // w = A u over the own rows and the sums (r.u, w.u, r.r)
    auto product = [&](double (&v)[3]) {
        v[0] = v[1] = v[2] = 0.0;
        for (int i0 = 0; i0 < R; i0 += kPass) {
            const int i = i0 + g0;
            float y0 = 0.f, y1 = 0.f, y2 = 0.f;
            if (i < R) {
                const int k1 = rp[r0 + i + 1];
#pragma unroll 4
                for (int k = rp[r0 + i] + q; k < k1; k += kRowLanes) {
                    const bool on_chip = k < kcap;
                    const float4 p = __ldcg(&U[on_chip ? scol[k - kbase] : __ldg(&ci[k])]);
                    const float* A = on_chip ? sval + 9 * (k - kbase) : val + 9 * (size_t)k;
                    y0 += A[0] * p.x + A[1] * p.y + A[2] * p.z;
                    y1 += A[3] * p.x + A[4] * p.y + A[5] * p.z;
                    y2 += A[6] * p.x + A[7] * p.y + A[8] * p.z;
                }
            }
            const float wc = row_component(y0, y1, y2, q);
            if (i < R && q < 3) {
                const float rc = sr[3 * i + q], uc = su[3 * i + q];
                sw[3 * i + q] = wc;
                v[0] += (double)rc * uc;
                v[1] += (double)wc * uc;
                v[2] += (double)rc * rc;
            }
        }
    };
    // p = u + beta p, s = w + beta s; returns this thread's part of p.s
    auto directions = [&](float beta) {
        double ps = 0.0;
        for (int i = t; i < 3 * R; i += kThreads) {
            const float p = beta != 0.f ? __fmaf_rn(beta, sp[i], su[i]) : su[i];
            const float s = beta != 0.f ? __fmaf_rn(beta, ss[i], sw[i]) : sw[i];
            sp[i] = p;
            ss[i] = s;
            ps += (double)p * s;
        }
        return ps;
    };

    bool breakdown = false;
    for (int sweep = 0; sweep < kSweeps; sweep++) {
        // dv64 += e; the FP64 residual of dv64 replaces r (the first one is b itself)
        double v[3] = {0.0, 0.0, 0.0};
        if (sweep > 0) {
            __syncthreads();
            for (int i = t; i < 3 * R; i += kThreads) {
                dv64[3 * r0 + i] += (double)se[i];
                se[i] = 0.f;
            }
            cl.sync();
        } else {
            __syncthreads();
        }
        for (int i0 = 0; i0 < R; i0 += kPass) {
            const int i = i0 + g0;
            double y0 = 0.0, y1 = 0.0, y2 = 0.0;
            if (i < R && sweep > 0) {
                const int k1 = rp[r0 + i + 1];
#pragma unroll 2
                for (int k = rp[r0 + i] + q; k < k1; k += kRowLanes) {
                    const bool on_chip = k < kcap;
                    const double* d = dv64 + 3 * (size_t)(on_chip ? scol[k - kbase] : __ldg(&ci[k]));
                    const float* A = on_chip ? sval + 9 * (k - kbase) : val + 9 * (size_t)k;
                    const double d0 = __ldcg(d), d1 = __ldcg(d + 1), d2 = __ldcg(d + 2);
                    y0 += (double)A[0] * d0 + (double)A[1] * d1 + (double)A[2] * d2;
                    y1 += (double)A[3] * d0 + (double)A[4] * d1 + (double)A[5] * d2;
                    y2 += (double)A[6] * d0 + (double)A[7] * d1 + (double)A[8] * d2;
                }
            }
            const double yc = row_component(y0, y1, y2, q);
            if (i < R && q < 3) {
                const double res = (double)b[3 * (r0 + i) + q] - yc, dr = res - (double)sr[3 * i + q];
                sr[3 * i + q] = (float)res;
                v[0] += res * res;
                v[1] += dr * dr;
            }
        }
        cluster_sum3(cl, S, nred, v);
        const double res = sqrt(v[0]);
        rel = bn > 0.0 ? res / bn : 0.0;
        if (res <= tol * bn || bn == 0.0) {
            status = CS_OK;
            break;
        }
        if (iters >= max_iters) break;
        // a reliable update keeps the direction of the last sweep if r had drifted little
        const bool cont = sweep > 0 && sweep_iters > 0 && !breakdown && sqrt(v[1]) <= kDrift * res;
        __syncthreads();
        precondition(false, 0.f);
        cl.sync();
        product(v);
        cluster_sum3(cl, S, nred, v);
        double alpha = 0.0;
        bool kept = false;
        if (cont && v[0] > 0.0 && gam_prev > 0.0 && isfinite(v[0] / gam_prev)) {
            // r left the recursion the step length assumes: alpha = r.u / p.s
            double ps[3] = {directions((float)(v[0] / gam_prev)), 0.0, 0.0};
            cluster_sum3(cl, S, nred, ps);
            alpha = v[0] / ps[0];
            kept = ps[0] > 0.0 && isfinite(alpha);
        }
        gam = v[0];
        sweep_iters = 0;
        breakdown = false;
        if (!kept) {
            alpha = gam / v[1];
            if (!(gam > 0.0) || !(v[1] > 0.0) || !isfinite(alpha)) {
                breakdown = true;
                continue;
            }
            directions(0.f);
        }
        const double stop1 = kInnerTol * res > tol * bn ? kInnerTol * res : kLastSweep * tol * bn, stop2 = stop1 * stop1;
        for (;;) {
            __syncthreads();
            precondition(true, (float)alpha);
            cl.sync();
            product(v);
            cluster_sum3(cl, S, nred, v);
            iters++;
            sweep_iters++;
            const double beta = v[0] / gam, next = v[0] / (v[1] - beta * v[0] / alpha);
            gam_prev = gam;
            gam = v[0];
            if (!(v[0] > 0.0) || !(next > 0.0) || !isfinite(next) || !isfinite(beta)) {
                breakdown = true;
                break;
            }
            if (v[2] <= stop2 || iters >= max_iters) break;
            alpha = next;
            directions((float)beta);
        }
    }
    __syncthreads();
    for (int i = t; i < 3 * R; i += kThreads) x[3 * r0 + i] = (float)dv64[3 * r0 + i];
    if (rank == 0 && t == 0) {
        stats[0] = iters;
        stats[1] = rel;
        stats[2] = status;
    }
    cl.sync();  // no CTA leaves while another may still write its partial sums here
}

// What a launch on one device needs, looked up on the first call there with it current.
struct LaunchPlan {
    unsigned char* scratch = nullptr;
    int ctas = 0;        // per cluster: 16, or 8 where a cluster of 16 cannot run
    size_t smem = 0;     // dynamic shared memory per CTA
};
std::mutex g_mutex;
LaunchPlan g_plan[64];

cudaError_t launch(const LaunchPlan& P, cudaStream_t s, int n, int nnzb, const int32_t* rp, const int32_t* ci, const float* val,
                   const float* b, float* x, double tol, int max_iters) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = P.ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(P.ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const size_t rows = kRowSmem * ((n + P.ctas - 1) / P.ctas);
    // an even share of the blocks and a margin for rows of more than the mean, what fits of it
    const size_t want = (size_t)(nnzb / P.ctas + nnzb / (4 * P.ctas) + 64);
    const int cap = (int)std::min(want, rows < P.smem ? (P.smem - rows) / kBlockSmem : 0);
    cfg.dynamicSmemBytes = rows + kBlockSmem * cap;
    return cudaLaunchKernelEx(&cfg, noalloc_pcg_kernel, n, nnzb, rp, ci, val, b, x, tol, max_iters, P.scratch, cap);
}

cs_status launch_plan(int device, LaunchPlan* out) {
    if (device < 0 || device >= 64) return CS_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lock(g_mutex);
    LaunchPlan& P = g_plan[device];
    if (!P.scratch) {
        void* ptr = nullptr;
        int optin = 0;
        cudaFuncAttributes fa;
        if (cudaGetSymbolAddress(&ptr, g_scratch) != cudaSuccess || !ptr ||
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess ||
            cudaFuncGetAttributes(&fa, noalloc_pcg_kernel) != cudaSuccess)
            return CS_ERR_CUDA;
        P.smem = (size_t)optin - fa.sharedSizeBytes;
        if (cudaFuncSetAttribute(noalloc_pcg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem) != cudaSuccess)
            return CS_ERR_CUDA;
        P.ctas = 8;
        if (cudaFuncSetAttribute(noalloc_pcg_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = kMaxCtas;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(kMaxCtas);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = P.smem;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, noalloc_pcg_kernel, &cfg) == cudaSuccess && clusters > 0)
                P.ctas = kMaxCtas;
        }
        cudaGetLastError();
        P.scratch = static_cast<unsigned char*>(ptr);
    }
    *out = P;
    return CS_OK;
}

}  // namespace

extern "C" cs_status cs_solve_block_csr_noalloc(int n_rows, int nnzb, const int32_t* row_ptr, const int32_t* col,
                                               const float* val, const float* b, float* x, double tol,
                                               int max_iters, void* stream, int* iters, double* rel_residual) {
    if (n_rows <= 0 || n_rows > CS_NOALLOC_MAX_ROWS || nnzb <= 0) return CS_ERR_INVALID_ARG;
    if (!row_ptr || !col || !val || !b || !x || !(tol > 0.0) || max_iters < 0) return CS_ERR_INVALID_ARG;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return CS_ERR_NO_DEVICE;
    LaunchPlan plan;
    cs_status st = launch_plan(device, &plan);
    if (st != CS_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (launch(plan, s, n_rows, nnzb, row_ptr, col, val, b, x, tol, max_iters) != cudaSuccess) {
        cudaGetLastError();
        return CS_ERR_CUDA;
    }
    if (!iters && !rel_residual) return CS_OK;
    double stats[3];
    if (cudaMemcpyAsync(stats, plan.scratch + kNoallocBytes - 256, sizeof(stats), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return CS_ERR_CUDA;
    if (iters) *iters = (int)stats[0];
    if (rel_residual) *rel_residual = stats[1];
    return (cs_status)(int)stats[2];
}
