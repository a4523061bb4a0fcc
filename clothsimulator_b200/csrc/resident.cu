// Cluster-resident PCG: one thread-block cluster solves one sheet with the sheet's system
// held in the cluster's distributed shared memory for the whole solve.
//
// The batched loop of pcg.cu streams every sheet's matrix from HBM once per CG iteration
// (about 1.7 MB per 64x64 sheet, ~300 iterations per step).  A sheet of that size fits in
// the shared memory of a cluster of 8 to 10 CTAs (227 KB each), so here each cluster
//   * takes the next sheet from a device work counter (persistent clusters; a sheet that
//     converges early frees its cluster at once, there is no batch-wide tail),
//   * copies its tile of the sheet's SELL-32 panels (a contiguous range of slices; the loader orders
//     the rows by tiles) into shared memory once per solve (what exceeds the budget, spread evenly
//     over the slices, is read from L2),
//   * runs the per-instance state machine of the batched loop (FP32 CG on the correction
//     system, FP64 dot products and norms, FP64 residual replacements with the search
//     direction kept (reliable updates), warm-start guard, inner and outer stopping tests)
//     with the FP32 vectors in registers, one thread per row.  The CG recurrence is the
//     Chronopoulos-Gear form: per iteration one SpMV w = A u and ONE fused reduction of
//     (r.u, w.u, r.r), instead of two reductions;
//   * preconditions with the 3x3 block-Jacobi inverse; when asked, for a sheet whose rows are ordered
//     by tiles, together with the levels of levels.cuh and, on larger sheets, a coarse-space
//     correction (one constant per component on CS_COARSE_SEGS segments of every tile), or, without
//     that correction, with a Chebyshev polynomial in the block-Jacobi-scaled tile each CTA holds (its
//     SpMVs read only the CTA's own shared memory) if the tiles keep enough of the couplings;
//   * exchanges data without cluster barriers: after u = P^-1 r each CTA pushes the values
//     of its tile's boundary rows into the halo slots of the CTAs that read them with
//     st.async remote stores, which complete bytes on the receiver's mbarrier; reduction
//     partials travel the same way.  A CTA waits only on its own mbarriers.  Sends for step
//     k+1 depend on every CTA's step-k partial, so one halo buffer and two reduction buffers
//     suffice (a sender is never two steps ahead of a receiver);
//   * sums deterministically: lanes, warps and CTAs in fixed orders, every CTA summing the same
//     partials: all CTAs take identical decisions;
//   * forms the sums r.u and r.r while the halo values travel.
// Every wait is bounded.  A CTA whose wait runs out raises an abort flag in all CTAs and an
// error word for the host, and all CTAs leave through the kernel's final cluster barrier (the
// only one after start-up), so no CTA exits while another may still address its memory.
//
// What bounds it: the chain of latencies of one iteration -- its instructions in the slowest warp, two
// exchanges through the cluster (halo, reduction), FP64 sums -- about 8 us for a 64 x 64 sheet on 9 CTAs
// of 15 warps with the levels and the coarse space, 6 us without them, 4 us for a 16 x 16 one.  Measured on the B200 (tol 1e-6, whole steps) against strips of
// rows with a strip-local Chebyshev-3, 162 coarse unknowns and sums by every thread: a lone sheet of 64 x
// 64 quads 1.14 -> 0.82 ms, 48 x 48 0.92 -> 0.52, 32 x 32 0.85 -> 0.34, 16 x 16 0.38 -> 0.30; 96 sheets of
// 45 x 45 4.3 -> 2.9 ms, 700 of 64 x 64 46.0 -> 39.9 ms.
//
// Replaces the reference's per-cloth GPU solve (Cloth.cu:766-809) like pcg.cu does; the
// block-Jacobi preconditioner is the 3x3 block inverse from the gather kernel (the reference
// builds the scalar Jacobi one, PhysicsHelper.cu:479-485).
#include <cooperative_groups.h>

#include "cs_internal.h"
#include "levels.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr uint32_t RES_WAIT_TRIES = 1u << 22;  // polls of a phase before a CTA gives up (about 0.1 s)
#ifndef RES_POLL_NS
#define RES_POLL_NS 32
#endif

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t mapa(uint32_t a, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ void rbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void rbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Non-blocking test of a phase (test_wait, not try_wait: try_wait may suspend the thread for
// a system-defined time).  CLUSTER = false: acquire at CTA scope, enough for data that
// st.async wrote into this CTA's shared memory with completion on this mbarrier; true:
// cluster scope, for the residual signal that orders other CTAs' global-memory writes.
template <bool CLUSTER>
__device__ __forceinline__ bool rbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    if (CLUSTER)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    return ok != 0;
}

// Remote arrive on another CTA's mbarrier, releasing this thread's prior writes cluster-wide.
__device__ __forceinline__ void rbar_arrive_remote(uint32_t cbar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cbar) : "memory");
}

__device__ __forceinline__ void st_async_f4(uint32_t caddr, float4 v, uint32_t cbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(caddr),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(cbar)
                 : "memory");
}

__device__ __forceinline__ void st_async_d2(uint32_t caddr, double a, double b, uint32_t cbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(caddr), "d"(a),
                 "d"(b), "r"(cbar)
                 : "memory");
}

__device__ __forceinline__ void st_async_u32(uint32_t caddr, uint32_t v, uint32_t cbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(caddr), "r"(v), "r"(cbar)
                 : "memory");
}

__device__ __forceinline__ double rwarp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float rwarp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ bool rfinite(double x) { return x == x && x < 1e300 && x > -1e300; }

// Shared control block of one CTA.
struct __align__(16) ResShared {
    double red[2][CS_RES_MAX_CL][4];   // reduction partials by sender rank, two buffers
    double wsum[CS_RES_MAX_WARPS][4];  // warp partials
    float wy[CS_RES_MAX_WARPS][4];     // warp sums of the coarse restriction
    double tot[6];                     // a reduction's sums and the scalars derived from them
    uint64_t bar[5];                   // 0 halo, 1-2 reduction buffers, 3 residual signal, 4 work item
    int next;                          // work item sent by rank 0
    int abort_flag;                    // raised by any CTA whose wait ran out
    // tile-local Chebyshev preconditioner of the current sheet: degree (1: block-Jacobi),
    // 1/theta, and per step k the coefficients of d_k = a_k d_{k-1} + b_k P^-1 (r - A_loc x)
    int cheb_deg;
    float cheb_inv_th;
    float cheb_a[CS_PRECOND_MAX_DEGREE], cheb_b[CS_PRECOND_MAX_DEGREE];
    // inverse diagonal blocks of the levels: per warp its four octets, then its patch (six entries)
    alignas(16) float lev[CS_RES_MAX_WARPS][5][8];
    double sc[CS_RES_MAX_WARPS][7];    // scalars of the solve, per warp
};

constexpr float CHEB_LMAX_MARGIN = 1.1f; // the estimate approaches lambda_max from below
constexpr float CHEB_LMIN_RATIO = 1.0f / 30.0f;

// Waits for `parity` of `bar`, at most RES_WAIT_TRIES polls, giving up early once another CTA raised
// the abort flag (res_poll); on every thread, returning true only if the whole CTA saw the phase
// complete (res_wait).
template <bool CLUSTER = false>
__device__ __forceinline__ bool res_poll(ResShared& S, uint32_t bar, uint32_t parity) {
    bool ok = false;
    for (uint32_t t = 0; t < RES_WAIT_TRIES; t++) {
        if (rbar_test<CLUSTER>(bar, parity)) {
            ok = true;
            break;
        }
        if (*(volatile int*)&S.abort_flag) break;
        // back off: polls share the shared-memory pipe with the remote stores being awaited
        __nanosleep(RES_POLL_NS);
    }
    __syncwarp();
    return ok;
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool res_wait(ResShared& S, uint32_t bar, uint32_t parity) {
    return __syncthreads_and(res_poll<CLUSTER>(S, bar, parity) ? 1 : 0) != 0;
}

// Barrier of the first n warps of the CTA.
__device__ __forceinline__ void warps_sync(int n) { asm volatile("bar.sync 1, %0;" ::"r"(32 * n) : "memory"); }

// Raises the abort flag in every CTA of the cluster and the error word for the host.
__device__ __forceinline__ void res_abort(const cg::cluster_group& cl, ResShared& S, int ncta, int* err) {
    if (threadIdx.x == 0) {
        for (int c = 0; c < ncta; c++) *(volatile int*)cl.map_shared_rank(&S.abort_flag, c) = 1;
        atomicExch(err, 1);
    }
}

// The coarse vectors in one CTA's shared memory, sized by the loader with coarseSmemBytes (CP = 3K
// rounded up to 4 floats):
//   part  this CTA's segment sums before they are sent, CP
//   red   every CTA's segment sums: [buffer][rank][CP]
//   ai    the rows of A_c^-1 of this CTA's segments, 3K x 64 (nc <= 64)
struct CoarseSm {
    unsigned char* base;
    int nc, k3, cp;
    __device__ __forceinline__ CoarseSm(unsigned char* b, int nc_, int k) : base(b), nc(nc_), k3(3 * k), cp((3 * k + 3) / 4 * 4) {}
    __device__ __forceinline__ float* part() const { return reinterpret_cast<float*>(base); }
    __device__ __forceinline__ float* red() const { return part() + cp; }
    __device__ __forceinline__ float* ai(int ncta) const { return red() + 2 * ncta * cp; }
    // entry q of the coarse vector in one buffer of `red` (rank q / 3K, segment and component
    // q % 3K)
    __device__ __forceinline__ int off(int q) const { return (q / k3) * cp + q % k3; }
};

// The warp's part of a reduction: sums 0 and 2, sum 1, or the coarse restriction of y, in shared memory.
__device__ __forceinline__ void put_sum02(ResShared& S, double a, double c, bool fp32) {
    const int lane = threadIdx.x & 31;
    const double t = fp32 ? (double)tile_sum2((float)a, (float)c) : tile_sum2(a, c);
    if ((lane & 15) == 0) S.wsum[threadIdx.x >> 5][lane >> 3] = t;  // lane 0: sum 0, lane 16: sum 2
}
__device__ __forceinline__ void put_sum1(ResShared& S, double a, bool fp32) {
    const double t = fp32 ? (double)rwarp_sum((float)a) : rwarp_sum(a);
    if ((threadIdx.x & 31) == 0) S.wsum[threadIdx.x >> 5][1] = t;
}
__device__ __forceinline__ void put_coarse(ResShared& S, const float (&y)[3]) {
    const int lane = threadIdx.x & 31;
    const float t = tile_sum3(y[0], y[1], y[2]);
    if ((lane & 7) == 0 && lane < 24) S.wy[threadIdx.x >> 5][lane >> 3] = t;
}
// The sums over 16 lanes (each half of the warp) of three values, in FP64 or (fp32) in float.
__device__ __forceinline__ void half_sum3(double (&t)[3], bool fp32) {
    if (fp32) {
        float f[3] = {(float)t[0], (float)t[1], (float)t[2]};
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 3; i++) f[i] += __shfl_xor_sync(0xffffffffu, f[i], o);
#pragma unroll
        for (int i = 0; i < 3; i++) t[i] = (double)f[i];
        return;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 3; i++) t[i] += __shfl_xor_sync(0xffffffffu, t[i], o);
}

// Cluster-wide sum of three values (fp32: in float, the plain FP32 solver; else double) and, with
// COARSE, the coarse vector R y of a per-row vector y, of the warps' sums that put_* stored.  Its time is a chain of latencies, so the stages
// are short and only warp 0 works on the cluster's: a barrier; warp 0 adds the warps' sums
//  (a lane per warp) and sends the CTA's partials by st.async to buffer `nred & 1` of every CTA,
// waits for everyone's, adds them (a lane per CTA), calls `post` on the sums for the scalars that
// depend on them, and publishes both; a barrier.  Fixed orders, the same in every CTA: all threads of
// the cluster return identical sums.  (Sums added serially by every thread and divisions done by every
// thread took 5,900 of the 12,500 cycles of an iteration on a 64 x 64 sheet.)
// R y: every warp's rows are of one segment (the loader cuts a tile's slices into K ranges); after the
// first barrier lane 3k + c of warp 1 adds component c over segment k's warps, in warp order, and sends
// the sums.  On return buffer (nred - 1) & 1 of C.red holds R y, entry q at C.off(q) (q = 3 (rank K + k)
// + c); it may be overwritten by the reduction after next.
// Returns false if the wait gave up (the caller aborts).
template <bool COARSE, class Post>
__device__ __forceinline__ bool cluster_reduce(ResShared& S, int rank, int ncta, uint32_t& nred, double (&v)[3], bool fp32,
                                               int nsl, const CoarseSm& C, Post post) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int b = (int)(nred & 1u);
    __syncthreads();
    bool ok = true;
    if (w == 0) {
        const uint32_t bar = saddr(&S.bar[1 + b]);
        if (lane == 0) rbar_expect(bar, (uint32_t)ncta * (32u + (COARSE ? 4u * (uint32_t)C.cp : 0u)));
        const int h = lane & 15;
        double t[3] = {0.0, 0.0, 0.0};
        if (h < nw)
#pragma unroll
            for (int i = 0; i < 3; i++) t[i] = S.wsum[h][i];
        half_sum3(t, fp32);
        if (lane < ncta) {
            const uint32_t dst = mapa(saddr(&S.red[b][rank][0]), lane);
            const uint32_t dbar = mapa(bar, lane);
            st_async_d2(dst, t[0], t[1], dbar);
            st_async_d2(dst + 16, t[2], 0.0, dbar);
        }
        ok = res_poll(S, bar, (nred >> 1) & 1u);
        t[0] = t[1] = t[2] = 0.0;
        if (h < ncta)
#pragma unroll
            for (int i = 0; i < 3; i++) t[i] = S.red[b][h][i];
        half_sum3(t, fp32);
        double x[3] = {0.0, 0.0, 0.0};
        post(t, x);
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                S.tot[i] = t[i];
                S.tot[3 + i] = x[i];
            }
        }
    } else if (COARSE && w == 1) {
        const uint32_t bar = saddr(&S.bar[1 + b]);
        if (lane < C.cp) {
            float a = 0.f;
            const int K = C.k3 / 3, k = lane / 3, c = lane - 3 * k, q0 = (nsl * k) / K, q1 = k < K ? (nsl * (k + 1)) / K : q0;
#pragma unroll 8
            for (int q = q0; q < q1; q++) a += S.wy[q][c];
            C.part()[lane] = a;
        }
        __syncwarp();
        if (lane < ncta) {
            const uint32_t cdst = mapa(saddr(C.red() + ((size_t)b * ncta + rank) * C.cp), lane);
            const uint32_t dbar = mapa(bar, lane);
            for (int q = 0; q < C.cp / 4; q++)
                st_async_f4(cdst + 16u * q, reinterpret_cast<const float4*>(C.part())[q], dbar);
        }
    }
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    nred++;
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] = S.tot[i];
    return ok;
}

// CTA-wide sums of two values in FP64, in a fixed order (warp butterfly, then warp partials in
// warp order); every thread returns the same sums.  Ends with a barrier, so S.wsum is free again.
__device__ __forceinline__ void cta_sum2(ResShared& S, double& a, double& b) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    a = rwarp_sum(a);
    b = rwarp_sum(b);
    if (lane == 0) {
        S.wsum[w][0] = a;
        S.wsum[w][1] = b;
    }
    __syncthreads();
    double sa = 0.0, sb = 0.0;
    for (int j = 0; j < nw; j++) {
        sa += S.wsum[j][0];
        sb += S.wsum[j][1];
    }
    a = sa;
    b = sb;
    __syncthreads();
}

__device__ __forceinline__ void mat3_vec(const float (&M)[9], const float (&x)[3], float (&y)[3]) {
    y[0] = M[0] * x[0] + M[1] * x[1] + M[2] * x[2];
    y[1] = M[3] * x[0] + M[4] * x[1] + M[5] * x[2];
    y[2] = M[6] * x[0] + M[7] * x[1] + M[8] * x[2];
}

}  // namespace

extern __shared__ __align__(16) unsigned char cs_res_smem[];

// Launch: cluster dimension (CL, 1, 1), blockDim = 32 x (slices per CTA, at most
// CS_RES_MAX_WARPS), dynamic shared memory = res_cap panels + the u array (res_halo0 own row
// slots, then the halo slots).  Grid: whole clusters, persistent (each takes sheets until
// none is left).  B.loop[5] is the work counter (zeroed by the solve setup), B.loop[6] the
// error word (set when a wait ran out).
__global__ void __launch_bounds__(CS_RES_MAX_WARPS * 32, 1) cs_resident_pcg_kernel(Batch B) {
    const DevParams& P = *B.params;
    if (P.solver != CS_SOLVER_AUTO_DEV || B.n_resident == 0) return;  // uniform over the grid
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int ncta = (int)cl.num_blocks();
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    const int cap = B.res_cap, halo0 = B.res_halo0;
    const float* sm_panels = reinterpret_cast<const float*>(cs_res_smem);
    float4* su = reinterpret_cast<float4*>(cs_res_smem + (size_t)cap * CS_PANEL_FLOATS * sizeof(float));
    __shared__ ResShared S;
    if (tid == 0) {
        rbar_init(saddr(&S.bar[0]), 1);
        rbar_init(saddr(&S.bar[1]), 1);
        rbar_init(saddr(&S.bar[2]), 1);
        rbar_init(saddr(&S.bar[3]), (uint32_t)ncta);
        rbar_init(saddr(&S.bar[4]), 1);
        S.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cl.sync();  // every CTA's barriers exist before any remote arrive or st.async
    const uint32_t hbar = saddr(&S.bar[0]), sbar = saddr(&S.bar[3]), ibar = saddr(&S.bar[4]);
    uint32_t nhalo = 0, nred = 0, nres = 0, nitem = 0;
    const bool mixed = P.mixed != 0, fp32 = !mixed;
    const int myslot = w * CS_SLICE + lane;
    int* err = B.loop + 6;

    for (;;) {
        // work item: rank 0 takes the next sheet and sends its index to every CTA
        if (tid == 0) rbar_expect(ibar, 4u);
        if (rank == 0 && tid == 0) {
            const int nx = atomicAdd(&B.loop[5], 1);
            for (int c = 0; c < ncta; c++) st_async_u32(mapa(saddr(&S.next), c), (uint32_t)nx, mapa(ibar, c));
        }
        if (!res_wait(S, ibar, nitem & 1u)) {
            res_abort(cl, S, ncta, err);
            break;
        }
        nitem++;
        const int idx = S.next;
        if (idx >= B.n_resident) break;

        const int s = B.rlist[idx];
        const SheetDesc sh = B.sheets[s];
        const int tb = sh.topo * (CS_RES_MAX_CL + 1);
        const int lo = B.rsplit[tb + rank], hi = B.rsplit[tb + rank + 1];
        const int nsl = hi - lo;
        // this CTA's panels into shared memory, up to the budget: what exceeds it are
        // the last slots of the slices (the loader chose how many of each, panels.h)
        bool live = false;
        int width = 0, ks = 0, lp = 0, gp = 0, tp = 0, row = 0;
        {
            const SliceDesc* sl = B.slices + sh.slice_off + lo;
            int at = 0;
            for (int j = 0; j < nsl; j++) {
                const int wd = sl[j].width, p0 = sl[j].panel0, keep = sl[j].keep;
                const float4* src = reinterpret_cast<const float4*>(B.A + (size_t)p0 * CS_PANEL_FLOATS);
                float4* dst = reinterpret_cast<float4*>(cs_res_smem) + (size_t)at * (CS_PANEL_FLOATS / 4);
                for (int i = tid; i < keep * (CS_PANEL_FLOATS / 4); i += blockDim.x) dst[i] = __ldg(src + i);
                if (j == w) {
                    lp = at;
                    ks = keep;
                    width = wd;
                }
                at += keep;
            }
        }
        // this thread's row: slice lo + w, lane
        if (w < nsl) {
            const SliceDesc d = B.slices[sh.slice_off + lo + w];
            live = lane < d.rows;
            gp = d.panel0;
            tp = d.tpanel0;
            if (live) row = B.rowmap[d.topo_slice * CS_SLICE + lane];
        }
        const float* const spn = sm_panels + (size_t)lp * CS_PANEL_FLOATS;
        const float* const gpn = B.A + (size_t)gp * CS_PANEL_FLOATS;
        const int* const code = B.rcode + (size_t)tp * CS_SLICE;
        const int g = sh.node_off + row;
        // byte offsets of the u entries of the slots in shared memory (fewer than 4,096 entries), for the
        // whole solve; others point at the zero entry between the own rows and the halo
        if (tid == 0) su[halo0 - 1] = su[B.res_alt + halo0 - 1] = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t cw[CS_RES_MAX_WIDTH / 2];
#pragma unroll
        for (int j = 0; j < CS_RES_MAX_WIDTH; j++) {
            const uint32_t at = 16u * (live && j < ks ? __ldg(code + j * CS_SLICE + lane) & 0xfff : halo0 - 1);
            cw[j >> 1] = (j & 1) ? cw[j >> 1] | at << 16 : at;
        }
        // halo sends of this CTA (the first one per thread in a register) and bytes it receives
        const int snd0 = B.rsendptr[tb + rank], snd1 = B.rsendptr[tb + rank + 1];
        const uint32_t my_send = snd0 + tid < snd1 ? __ldg(&B.rsend[snd0 + tid]) : 0u;
        const uint32_t halo_bytes = (uint32_t)B.rhalo[tb + rank] * 16u;

        // the multilevel preconditioner, and its coarse-space correction (both uniform over the cluster)
        const bool levels = P.coarse && P.cheb_degree >= 3 && (B.rcheb[tb + rank] & 2);
        const int4 cinfo = B.rcoarse[sh.topo];
        const bool coarse = levels && cinfo.x == B.res_cnc && cinfo.x > 0 && B.cvalid[idx] && nw >= 2;
#define C CoarseSm(cs_res_smem + B.res_coff, B.res_cnc, B.res_ck)
        // Every warp keeps the whole coarse residual R r and direction R s (FP64), entries `lane` and
        // `lane + 32` per lane (nc <= 64): applying and updating the correction takes no barrier.  `coff`:
        // those entries' places in a buffer of C.red (16 bits each), `rw` R w of the last CG reduction
        // there (read at once: a reduction later, the buffer may be overwritten).
        int coff = 0;
        float rw[2] = {0.f, 0.f};
        const float* cai = C.ai(ncta) + lane;  // this warp's segment's rows of A_c^-1
        double cr[2] = {0.0, 0.0}, cs[2] = {0.0, 0.0};
        if (coarse) {
            int seg = 0;
            while (seg + 1 < B.res_ck && w >= (nsl * (seg + 1)) / B.res_ck) seg++;
            cai += 3 * 64 * seg;
            const float* src = B.cinv + (size_t)idx * B.res_cnc * B.res_cnc + (size_t)rank * C.k3 * C.nc;
            for (int i = tid; i < C.k3 * 64; i += blockDim.x) C.ai(ncta)[i] = (i & 63) < C.nc ? __ldcg(src + (i >> 6) * C.nc + (i & 63)) : 0.f;
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (lane + 32 * h < C.nc) coff |= C.off(lane + 32 * h) << (16 * h);
        }

        float Pi[9];
        float e[3] = {0.f, 0.f, 0.f}, r[3] = {0.f, 0.f, 0.f}, u[3], wv[3], p[3] = {0.f, 0.f, 0.f},
              sv3[3] = {0.f, 0.f, 0.f};
        if (live) {
#pragma unroll
            for (int k = 0; k < 9; k++) Pi[k] = B.Pinv[9 * (size_t)g + k];
#pragma unroll
            for (int c = 0; c < 3; c++) r[c] = B.b[3 * g + c];
        } else {
#pragma unroll
            for (int k = 0; k < 9; k++) Pi[k] = 0.f;
        }
        // a node without a face has an empty row, which no correction may move
        bool moves = false;
#pragma unroll
        for (int k = 0; k < 9; k++) moves |= Pi[k] != 0.f;
        moves |= r[0] != 0.f || r[1] != 0.f || r[2] != 0.f;
        // scalars used once per iteration or less live in shared memory, a copy per warp (every lane
        // writes the same value and reads its own write)
        double &bn = S.sc[w][0], &res0 = S.sc[w][1], &resnorm = S.sc[w][2], &first_res = S.sc[w][3], &rr = S.sc[w][4],
               &delta = S.sc[w][5], &thr = S.sc[w][6];
        bn = res0 = sqrt(B.inst[s].bnorm2);
        rr = delta = thr = 0.0;
        resnorm = first_res = -1.0;
        double gam = 0.0, gam_prev = 0.0, alpha_d = 0.0;
        bool cont = false;  // the next PH_INIT keeps the search direction (reliable update)
        // dv64 and e are known to be zero (zero guess before its first CG step, or a rejected
        // warm start just cleared): the next FP64 residual is b itself and needs no SpMV
        bool dv_zero = !P.warm;
        // the warm start was just scaled by affine_a: the next residual is the affine combination
        // (1 - a) b + a r of b and the residual r of the unscaled start, no SpMV either
        bool affine = false;
        double affine_a = 0.0;
        // the warm start's scaling pass (warm_scale): its first residual gives d.b and d.r
        bool scale_pass = P.warm && P.warm_scale;
        // 1 / gam and 1 / (gam alpha), computed when gam and alpha are set, so that the next
        // iteration's step length costs one division after the reduction instead of three
        double inv_gam = 0.0, inv_ga = 0.0;
        float alpha = 0.f, beta = 0.f;
        int iters = 0, sweeps = 0, sweep_iters = 0, flags = 0, trips = 0;
        // with the coarse correction every solve starts with an FP64 residual: its reduction
        // carries the coarse residual R r that the first preconditioner application needs
        int phase = (P.warm || coarse) ? PH_RES : PH_INIT;
        bool ok = true;

        // The next iteration's scalars from the reduction's sums (r.u, w.u, r.r), by warp 0: the step
        // length alpha = gnew / (dnew - beta gnew / alpha_prev), 1 / gnew and 1 / (gnew alpha)
        auto no_post = [](const double (&)[3], double (&)[3]) {};
        auto next_step = [&](const double (&t)[3], double (&x)[3]) {
            if (!mixed || phase != PH_CG) return;
            x[0] = t[0] / (t[1] - t[0] * t[0] * inv_ga);
            x[1] = 1.0 / t[0];
            x[2] = 1.0 / (t[0] * x[0]);
        };
        // q = A_loc x over this CTA's own rows and columns (the tile's diagonal block of A), x in `buf`
        float4* const su_alt = su + B.res_alt;
        auto local_spmv = [&](const float4* buf, float (&q)[3]) {
            q[0] = q[1] = q[2] = 0.f;
            row_times<CS_RES_MAX_WIDTH, 4, true>(spn, gpn, ks, width, cw, code, row_tail_load(gpn, ks, width, code, lane), buf, halo0, lane, live,
                            q[0], q[1], q[2]);
        };
        // The coarse images of the CG recurrences: with s = w + beta s and the next iteration's
        // r -= alpha s, R s = R w + beta R s and R r -= alpha R s (R w from the reduction just done); R r
        // is what the next preconditioner application reads.  An FP64 residual replaces R r exactly
        // (PH_RES).
        auto coarse_step = [&](double beta_c, double alpha_c) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                cs[h] = (double)rw[h] + beta_c * cs[h];
                cr[h] -= alpha_c * cs[h];
            }
        };
        // The levels' diagonal blocks (levels.cuh); its first barrier also covers the panel copy
        LevelPlace at{(uint32_t)myslot * 0x10001u};
        if (levels) {
            __syncthreads();
            const uint32_t* cells = B.rcell + (size_t)B.slices[sh.slice_off + lo].topo_slice * CS_SLICE;
            if (live) at.v = __ldg(cells + myslot);
            level_blocks(spn, gpn, ks, width, code, cells, halo0 - 1, at, lane, live, su_alt, S.lev[w]);
        }
        // Tile-local Chebyshev preconditioner: the largest eigenvalue of P^-1 A_loc by power
        // iteration from a hashed +-1 vector (the first barrier also covers the panel copy),
        // then the coefficients of the Chebyshev iteration on [lmax / 30, lmax].  An odd
        // degree keeps the polynomial positive on all of (0, inf), so the preconditioner is
        // SPD whatever the estimate.
        const bool poly = !levels && P.cheb_degree >= 3 && (B.rcheb[tb + rank] & 1);  // uniform over the cluster
        if (poly) {
            float v[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const uint32_t h = (uint32_t)(3 * row + c) * 0x9E3779B1u;
                v[c] = live ? (((h >> 16) & 1u) ? 1.f : -1.f) : 0.f;
            }
            double lam = 0.0;
            for (int it = 0; it < CS_CHEB_POWER_ITERS; it++) {
                su_alt[myslot] = make_float4(v[0], v[1], v[2], 0.f);
                __syncthreads();
                float q[3], z[3];
                local_spmv(su_alt, q);
                mat3_vec(Pi, q, z);
                double zz = (double)z[0] * z[0] + (double)z[1] * z[1] + (double)z[2] * z[2];
                double vv = (double)v[0] * v[0] + (double)v[1] * v[1] + (double)v[2] * v[2];
                cta_sum2(S, zz, vv);
                lam = vv > 0.0 ? sqrt(zz / vv) : 0.0;
                const float sc = zz > 0.0 ? (float)(1.0 / sqrt(zz)) : 0.f;
#pragma unroll
                for (int c = 0; c < 3; c++) v[c] = z[c] * sc;
            }
            if (tid == 0) {
                int deg = P.cheb_degree;
                if (!(lam > 0.0) || !rfinite(lam)) deg = 1;
                const float lmax = CHEB_LMAX_MARGIN * (float)lam, lmin = lmax * CHEB_LMIN_RATIO;
                const float th = 0.5f * (lmax + lmin), de = 0.5f * (lmax - lmin), sig = th / de;
                float rho = 1.f / sig;
                S.cheb_inv_th = 1.f / th;
                for (int k = 1; k < deg; k++) {
                    const float rn = 1.f / (2.f * sig - rho);
                    S.cheb_a[k] = rn * rho;
                    S.cheb_b[k] = 2.f * rn / de;
                    rho = rn;
                }
                S.cheb_deg = deg;
            }
        } else if (tid == 0) {
            S.cheb_deg = 1;
        }
        __syncthreads();
        const int cdeg = S.cheb_deg;

        while (phase != PH_FINISH) {
            if (++trips > P.loop_cap) {
                flags |= CS_IF_CAPPED;
                break;
            }
            if (phase == PH_RES) {
                // fold the FP32 correction into the FP64 solution; every CTA signals that its
                // rows are written; then r = b - A dv64 in FP64 over global dv64 (r = b when
                // dv64 is known to be zero: no signal, no SpMV; the decision is uniform)
                const bool zero = dv_zero, aff = affine;
                dv_zero = false;
                affine = false;
                if (live) {
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        B.dv64[3 * g + c] += (double)e[c];
                        e[c] = 0.f;
                    }
                }
                if (!zero && !aff) {
                    __syncthreads();
                    if (tid == 0) {
                        asm volatile("fence.acq_rel.cluster;" ::: "memory");
                        for (int c = 0; c < ncta; c++) rbar_arrive_remote(mapa(sbar, c));
                    }
                    ok = res_wait<true>(S, sbar, nres & 1u);
                    nres++;
                    if (!ok) break;
                }
                double v[3] = {0.0, 0.0, 0.0};
                if (live) {
                    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
                    // four slots' column and dv64 loads in flight at a time; sums in slot order
#pragma unroll
                    for (int k0 = 0; k0 < CS_RES_MAX_WIDTH; k0 += 4) {
                        if (zero || aff || k0 >= width) break;
                        int col[4];
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            col[j] = k0 + j < width ? __ldg(&B.tcol[(tp + k0 + j) * CS_SLICE + lane]) + sh.node_off : g;
                        double d[4][3];
#pragma unroll
                        for (int j = 0; j < 4; j++)
#pragma unroll
                            for (int c = 0; c < 3; c++) d[j][c] = __ldcg(&B.dv64[3 * col[j] + c]);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            if (k0 + j >= width) break;
                            const int k = k0 + j;
                            const float* pk = k < ks ? spn + k * CS_PANEL_FLOATS : gpn + (size_t)k * CS_PANEL_FLOATS;
                            const float4 a0 = reinterpret_cast<const float4*>(pk)[lane];
                            const float4 a1 = reinterpret_cast<const float4*>(pk + 128)[lane];
                            const float a8 = pk[256 + lane];
                            y0 += (double)a0.x * d[j][0] + (double)a0.y * d[j][1] + (double)a0.z * d[j][2];
                            y1 += (double)a0.w * d[j][0] + (double)a1.x * d[j][1] + (double)a1.y * d[j][2];
                            y2 += (double)a1.z * d[j][0] + (double)a1.w * d[j][1] + (double)a8 * d[j][2];
                        }
                    }
                    double r0 = (double)B.b[3 * g] - y0, r1 = (double)B.b[3 * g + 1] - y1, r2 = (double)B.b[3 * g + 2] - y2;
                    if (aff) {
                        r0 = (1.0 - affine_a) * (double)B.b[3 * g] + affine_a * (double)r[0];
                        r1 = (1.0 - affine_a) * (double)B.b[3 * g + 1] + affine_a * (double)r[1];
                        r2 = (1.0 - affine_a) * (double)B.b[3 * g + 2] + affine_a * (double)r[2];
                    }
                    // drift of the recursive residual it replaces
                    const double q0 = r0 - (double)r[0], q1 = r1 - (double)r[1], q2 = r2 - (double)r[2];
                    r[0] = (float)r0;
                    r[1] = (float)r1;
                    r[2] = (float)r2;
                    if (scale_pass) {
                        const double d0 = B.dv64[3 * g], d1 = B.dv64[3 * g + 1], d2 = B.dv64[3 * g + 2];
                        v[0] = d0 * (double)B.b[3 * g] + d1 * (double)B.b[3 * g + 1] + d2 * (double)B.b[3 * g + 2];
                        v[1] = d0 * r0 + d1 * r1 + d2 * r2;
                    } else {
                        v[0] = r0 * r0 + r1 * r1 + r2 * r2;
                        v[1] = q0 * q0 + q1 * q1 + q2 * q2;
                    }
                }
                put_sum02(S, v[0], v[2], false);
                put_sum1(S, v[1], false);
                if (coarse) {
                    // the coarse residual R r of the replaced r travels with the norms
                    put_coarse(S, r);
                    ok = cluster_reduce<true>(S, rank, ncta, nred, v, false, nsl, C, no_post);
                    const float* red = C.red() + (size_t)((nred - 1) & 1u) * ncta * C.cp;
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        if (lane + 32 * h < C.nc) cr[h] = (double)red[(coff >> (16 * h)) & 0xffff];
                } else {
                    ok = cluster_reduce<false>(S, rank, ncta, nred, v, false, nsl, C, no_post);
                }
                if (!ok) break;
                if (scale_pass) {
                    // d becomes alpha d, alpha = d.b / d.A d (d.A d = d.b - d.r): the multiple of d
                    // nearest to the solution in the energy norm; the next residual is its guard's.
                    // Every CTA holds the same sums, so all take the same branch; each scales its
                    // own rows once every CTA's reads of them are done (they precede the sums).
                    scale_pass = false;
                    const double dad = v[0] - v[1], a = v[0] / dad;
                    if (dad > 0.0 && rfinite(a)) {
                        if (live) {
#pragma unroll
                            for (int c = 0; c < 3; c++) B.dv64[3 * g + c] *= a;
                        }
                        affine = true;  // b - A (a d) = (1 - a) b + a (b - A d)
                        affine_a = a;
                        continue;       // phase stays PH_RES
                    }
                    flags |= CS_IF_WARM_REJECTED;
                    sweeps = 1;
                    res0 = bn;
                    phase = PH_INIT;
                    if (coarse) {
                        if (live) {
#pragma unroll
                            for (int c = 0; c < 3; c++) B.dv64[3 * g + c] = 0.0;
                        }
                        dv_zero = true;
                        phase = PH_RES;
                    }
                    continue;
                }
                const double res = sqrt(v[0]);
                resnorm = res;
                sweeps += 1;
                if (sweeps == 1) {
                    first_res = res;
                    if (P.warm && !(res <= bn)) {
                        // the warm start is worse than the zero guess: discard it
                        flags |= CS_IF_WARM_REJECTED;
                        res0 = bn;
                        phase = PH_INIT;
                        if (coarse) {
                            // r = b and its coarse residual come from one more residual of dv = 0
                            if (live) {
#pragma unroll
                                for (int c = 0; c < 3; c++) B.dv64[3 * g + c] = 0.0;
                            }
                            dv_zero = true;
                            phase = PH_RES;
                        }
                        continue;
                    }
                }
                if (aff && (res <= P.tol * bn || bn == 0.0 || iters >= P.max_iters)) {
                    // the solve would end on the affine residual (built from an FP32 copy of r):
                    // an FP64 residual of the scaled start decides instead, so the residual a
                    // finished sheet reports is always an FP64 one
                    phase = PH_RES;
                } else if (res <= P.tol * bn || bn == 0.0) {
                    flags |= CS_IF_CONVERGED;
                    phase = PH_FINISH;
                } else if (iters >= P.max_iters) {
                    flags |= CS_IF_CAPPED;
                    phase = PH_FINISH;
                } else if (mixed || gam == 0.0) {
                    // mixed: a reliable update (the FP64 residual replaced r; the direction
                    // of the last sweep is kept if it ran and r had drifted little); plain:
                    // the first sweep after a warm start
                    res0 = res;
                    cont = mixed && sweep_iters > 0 && !(flags & CS_IF_BREAKDOWN) && sqrt(v[1]) <= CS_RELIABLE_DRIFT * res;
                    phase = PH_INIT;
                } else {
                    // plain FP32 CG stopped on its recursive residual and the FP64 check failed
                    flags |= CS_IF_CAPPED;
                    phase = PH_FINISH;
                }
                continue;
            }
            // PH_INIT (start of a sweep) or PH_CG: u = P^-1 r, halo exchange, w = A u, and
            // one reduction of (r.u, w.u, r.r)
            if (phase == PH_INIT && (flags & CS_IF_WARM_REJECTED) && sweeps == 1 && live) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    B.dv64[3 * g + c] = 0.0;
                    r[c] = B.b[3 * g + c];
                }
            }
            if (phase == PH_CG) {
                dv_zero = false;  // e (folded into dv64 by the next residual) leaves zero here
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    e[c] = __fmaf_rn(alpha, p[c], e[c]);
                    r[c] = __fmaf_rn(-alpha, sv3[c], r[c]);
                }
            }
            mat3_vec(Pi, r, u);
            if (cdeg >= 3) {
                // u = x after cdeg steps of the Chebyshev iteration for A_loc x = r from x = 0.
                // Steps alternate between the two own-row buffers, ending on su_alt (cdeg - 1
                // is even), so one barrier per step orders every write after the reads of the
                // buffer's previous contents, the final su write included.
                float d[3];
                const float ith = S.cheb_inv_th;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    d[c] = u[c] * ith;
                    u[c] = d[c];
                }
                for (int k = 1; k < cdeg; k++) {
                    float4* const buf = (k & 1) ? su : su_alt;
                    buf[myslot] = make_float4(u[0], u[1], u[2], 0.f);
                    __syncthreads();
                    float q[3], t[3];
                    local_spmv(buf, q);
#pragma unroll
                    for (int c = 0; c < 3; c++) q[c] = r[c] - q[c];
                    mat3_vec(Pi, q, t);
                    const float ca = S.cheb_a[k], cb = S.cheb_b[k];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        d[c] = ca * d[c] + cb * t[c];
                        u[c] += d[c];
                    }
                }
            }
            if (levels && w < nsl) {
                // + the segment's, the octet's and the patch's corrections (additive); the barriers are of the
                // warps with a slice alone, few of a small sheet's in a batch with large ones
                su[myslot] = make_float4(r[0], r[1], r[2], 0.f);
                if (coarse) {
                    const float r0 = (float)cr[0], r1 = (float)cr[1];
#pragma unroll
                    for (int c = 0; c < 3; c++) u[c] += rwarp_sum(fmaf(cai[64 * c + 32], r1, cai[64 * c] * r0));
                }
                warps_sync(nsl);
                level_sums(S.lev[w], su[at.slot()], su_alt, w, lane);
                warps_sync(nsl);
                level_add(su_alt, at, u);
            }
            if (!moves) u[0] = u[1] = u[2] = 0.f;  // the corrections reach lanes without a row and empty rows
            su[myslot] = make_float4(u[0], u[1], u[2], 0.f);
            __syncthreads();
            if (tid == 0) rbar_expect(hbar, halo_bytes);
            for (int i = snd0 + tid; i < snd1; i += blockDim.x) {
                const uint32_t m = i == snd0 + tid ? my_send : __ldg(&B.rsend[i]);
                const int d = (int)((m >> 12) & 0xfu);
                st_async_f4(mapa(saddr(&su[halo0 + (int)(m >> 16)]), d), su[m & 0xfffu], mapa(hbar, d));
            }
            // while the halo values travel: the sums r.u and r.r, the first slot in global memory
            const RowTail tail = row_tail_load(gpn, ks, width, code, lane);
            if (mixed)
                put_sum02(S, (double)r[0] * u[0] + (double)r[1] * u[1] + (double)r[2] * u[2],
                          (double)r[0] * r[0] + (double)r[1] * r[1] + (double)r[2] * r[2], false);
            else
                put_sum02(S, (double)(r[0] * u[0] + r[1] * u[1] + r[2] * u[2]), (double)(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]), true);
            ok = res_wait(S, hbar, nhalo & 1u);
            nhalo++;
            if (!ok) break;
            wv[0] = wv[1] = wv[2] = 0.f;
            row_times<CS_RES_MAX_WIDTH, 4, false>(spn, gpn, ks, width, cw, code, tail, su, halo0, lane, live, wv[0], wv[1], wv[2]);
            double v[3] = {0.0, 0.0, 0.0};
            if (mixed)
                put_sum1(S, (double)wv[0] * u[0] + (double)wv[1] * u[1] + (double)wv[2] * u[2], false);
            else
                put_sum1(S, (double)(wv[0] * u[0] + wv[1] * u[1] + wv[2] * u[2]), true);
            if (coarse) {
                // R w travels with the dot products (the coarse recurrences below)
                put_coarse(S, wv);
                ok = cluster_reduce<true>(S, rank, ncta, nred, v, fp32, nsl, C, next_step);
                const float* red = C.red() + (size_t)((nred - 1) & 1u) * ncta * C.cp;
#pragma unroll
                for (int h = 0; h < 2; h++) rw[h] = lane + 32 * h < C.nc ? red[(coff >> (16 * h)) & 0xffff] : 0.f;
            } else {
                ok = cluster_reduce<false>(S, rank, ncta, nred, v, fp32, nsl, C, next_step);
            }
            if (!ok) break;
            const double gnew = v[0], dnew = v[1];
            rr = v[2];
            if (phase == PH_INIT) {
                // a sweep ends when r fell by inner_tol, the last one at half the tolerance at the latest; with the
                // levels or the polynomial it goes to CS_LAST_SWEEP of it: at equal residuals the levels
                // leave up to 1.6 times the error in dv that a larger coarse space did (32 x 32 quads)
                const double ti = mixed ? P.inner_tol * res0 : 0.0, tt = P.tol * bn;
                const double t = !mixed ? tt : levels || poly ? (ti > tt ? ti : CS_LAST_SWEEP * tt) : fmax(ti, 0.5 * tt);
                thr = t * t;
            }
            if (phase == PH_INIT && cont) {
                // p = u + beta p and s = w + beta s with beta = (r.u) / (the last iteration's
                // r.u); r no longer follows the recursion that the Chronopoulos-Gear step
                // length assumes, so alpha = r.u / p.s is computed with one more reduction
                cont = false;
                const double bd = gnew / gam_prev;
                if (gnew > 0.0 && rfinite(gnew) && rfinite(bd)) {
                    const float bc = (float)bd;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        p[c] = __fmaf_rn(bc, p[c], u[c]);
                        sv3[c] = __fmaf_rn(bc, sv3[c], wv[c]);
                    }
                    double v2[3] = {0.0, 0.0, 0.0};
                    if (live) v2[0] = (double)p[0] * sv3[0] + (double)p[1] * sv3[1] + (double)p[2] * sv3[2];
                    put_sum02(S, v2[0], 0.0, false);
                    put_sum1(S, 0.0, false);
                    ok = cluster_reduce<false>(S, rank, ncta, nred, v2, false, nsl, C, no_post);
                    if (!ok) break;
                    if (v2[0] > 0.0 && rfinite(v2[0]) && rfinite(gnew / v2[0])) {
                        gam = gnew;
                        delta = dnew;
                        sweep_iters = 0;
                        beta = bc;
                        alpha_d = gnew / v2[0];
                        alpha = (float)alpha_d;
                        inv_gam = 1.0 / gam;
                        inv_ga = 1.0 / (gam * alpha_d);
                        if (coarse) coarse_step((double)bc, alpha_d);
                        phase = PH_CG;
                        continue;
                    }
                }
                // otherwise: restart from p = u below
            }
            if (phase == PH_INIT) {
                gam = gnew;
                delta = dnew;
                sweep_iters = 0;
                beta = 0.f;
                if (!(gam > 0.0 && rfinite(gam))) {
                    phase = PH_RES;
                    continue;
                }
                if (mixed) {
                    alpha_d = gam / delta;
                    alpha = (float)alpha_d;
                    inv_gam = 1.0 / gam;
                    inv_ga = 1.0 / (gam * alpha_d);
                } else {
                    alpha = (float)gam / (float)delta;
                    alpha_d = (double)alpha;
                }
                if (!(delta > 0.0) || !rfinite((double)alpha)) {
                    flags |= CS_IF_BREAKDOWN;
                    phase = PH_RES;
                    continue;
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    p[c] = u[c];
                    sv3[c] = wv[c];
                }
                if (coarse) coarse_step(0.0, alpha_d);
                phase = PH_CG;
                continue;
            }
            // PH_CG: the iteration's x and r updates are done; stopping test on ||r||
            iters += 1;
            sweep_iters += 1;
            // ||r|| against the sweep's threshold, squared (no square root on the critical path)
            bool stop = v[2] <= thr || (mixed && sweep_iters >= P.sweep_cap);
            float nb, na;
            double na_d;
            if (mixed) {
                // beta = gnew / gam; alpha = gnew / (dnew - beta gnew / alpha_prev)
                const double bd = gnew * inv_gam;
                na_d = S.tot[3];
                nb = (float)bd;
                na = (float)na_d;
            } else {
                nb = (float)gnew / (float)gam;
                na = (float)gnew / ((float)dnew - nb * (float)gnew / alpha);
                na_d = (double)na;
            }
            if (!isfinite(nb) || !isfinite(na) || !(gnew > 0.0) || !(na > 0.f)) {
                flags |= CS_IF_BREAKDOWN;
                stop = true;
            }
            gam_prev = gam;
            gam = gnew;
            delta = dnew;
            if (stop || iters >= P.max_iters) {
                phase = PH_RES;
                continue;
            }
            beta = nb;
            alpha = na;
            alpha_d = na_d;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                p[c] = __fmaf_rn(beta, p[c], u[c]);
                sv3[c] = __fmaf_rn(beta, sv3[c], wv[c]);
            }
            if (coarse) coarse_step((double)beta, alpha_d);
            if (mixed) {
                inv_gam = S.tot[4];
                inv_ga = S.tot[5];
            }
        }
        if (!ok) {
            res_abort(cl, S, ncta, err);
            flags |= CS_IF_BREAKDOWN;
        }
        if (live && (!ok || trips > P.loop_cap)) {
#pragma unroll
            for (int c = 0; c < 3; c++) B.dv64[3 * g + c] += (double)e[c];
        }
        if (rank == 0 && tid == 0) {
            InstState& I = B.inst[s];
            I.rz = gam;
            I.rr = rr;
            I.pq = delta;
            I.res0 = res0;
            I.resnorm = resnorm;
            I.first_res = first_res;
            I.alpha = alpha;
            I.beta = beta;
            I.iters = iters;
            I.sweeps = sweeps;
            I.sweep_iters = sweep_iters;
            I.flags = flags;
            I.phase = PH_DONE;
        }
        if (!ok) break;
    }
#undef C
    cl.sync();  // no CTA leaves while another may still address its shared memory
}
