// Group-resident PCG: a sheet too large for a thread-block cluster (resident.cu) is solved by a
// group of CTAs spread over the whole chip, one per SM, with its system held in their shared
// memory for the whole solve.
//
// The batched loop of pcg.cu streams such a sheet's matrix from L2 or HBM and launches seven
// kernels per CG iteration: 45 us per iteration for a sheet of 66,049 nodes, whose 31 MB fit the
// 33 MB of shared memory the chip has.  Here one cooperative launch solves all such sheets:
//   * The loader orders the sheet's rows by tiles (recursive bisection of the rest (u, v)
//     coordinates), one tile of at most CS_GROUP_MAX_WARPS slices per CTA, and assigns every sheet a
//     range of CTAs and a place in the order each CTA works through (several sheets at a time
//     where they fit side by side).
//   * A CTA holds its tile's SELL-32 panels in shared memory (what exceeds it, spread evenly over
//     the slices, is read from L2), one row per thread with the CG vectors in registers, as
//     resident.cu does, and runs the same iteration: Chronopoulos-Gear CG with one fused
//     reduction, the levels of levels.cuh (without the coarse correction the tile-local
//     Chebyshev preconditioner), the additive coarse-space correction (one constant per segment of a
//     tile and component, its residual carried by recurrence within the reduction), FP64 residual
//     replacements with the search direction kept.
//   * CTAs exchange values through global memory (L2) in 16-byte packets {three words, epoch},
//     each written and read by one 128-bit access: a reader polls the packet itself, so a value's
//     arrival needs no flag, fence or barrier.
//     After u = P^-1 r every CTA publishes its boundary rows and gathers its halo; reduction
//     partials go to a slot per CTA that every CTA of the group polls.  A CTA publishes u for
//     step k + 1 only after the reduction of step k, to which every reader contributes after it
//     read u of step k: one halo buffer suffices; the partials alternate between two.  The
//     packets are zeroed before the launch and epochs start at 1.
//   * Sums are deterministic: warp butterflies, warp partials in order, CTA partials in a fixed
//     order that is the same in every CTA, so all take identical decisions.
// Every wait is bounded by a number of polls (Batch::g_polls: about 0.3 s; for a sheet's first exchange, whose
// CTAs may still solve others, g_polls_first: more than a minute); a CTA whose wait runs out sets the error word,
// which ends the others' waits, and the host reports CS_ERR_TIMEOUT.
//
// What bounds it: per iteration two trips through L2 (halo, reduction) of about 1 us each, the chain of
// instructions between them and the shared-memory reads of the tile.  Measured against the batched
// loop (whole steps, B200): a sheet of 66,049 nodes at 1e-10 15.4 -> 3.6 ms (4.2 with Chebyshev-3), 10,201
// nodes 9.1 -> 1.33 ms, a lone sheet of 72 x 72 quads 8.1 -> 0.92 ms, an irregular sheet of 261 x 261
// nodes (Chebyshev-3) 13.0 -> 3.4 ms, 64 sheets of 4 to 128 quads a side 15.5 -> 8.1 ms.
#include "cs_internal.h"
#include "levels.cuh"

namespace {

constexpr float G_LMAX_MARGIN = 1.1f;            // as in resident.cu
constexpr float G_LMIN_RATIO = 1.0f / 30.0f;

__device__ __forceinline__ void put_packet(uint4* p, uint32_t a, uint32_t b, uint32_t c, uint32_t epoch) {
    const unsigned long long lo = ((unsigned long long)b << 32) | a, hi = ((unsigned long long)epoch << 32) | c;
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p), "l"(lo),
                 "l"(hi)
                 : "memory");
}
__device__ __forceinline__ uint4 get_packet(const uint4* p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}

template <class T>
__device__ __forceinline__ T gwarp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ bool gfinite(double x) { return x == x && x < 1e300 && x > -1e300; }

__device__ __forceinline__ void gmat3_vec(const float (&M)[9], const float (&x)[3], float (&y)[3]) {
    y[0] = M[0] * x[0] + M[1] * x[1] + M[2] * x[2];
    y[1] = M[3] * x[0] + M[4] * x[1] + M[5] * x[2];
    y[2] = M[6] * x[0] + M[7] * x[1] + M[8] * x[2];
}

struct __align__(16) GroupShared {
    double wsum[CS_GROUP_MAX_WARPS][3];  // warp partials
    float wseg[CS_GROUP_MAX_WARPS][4];   // the warps' sums of a vector (coarse restriction)
    double tot[4];
    // scalars of the solve that are used once per iteration or less (kept out of the registers)
    double bn, res0, rr, delta, resnorm, first_res;
    int cheb_deg;
    float cheb_inv_th;
    float cheb_a[CS_PRECOND_MAX_DEGREE], cheb_b[CS_PRECOND_MAX_DEGREE];
    alignas(16) float lev[CS_GROUP_MAX_WARPS][5][8];
};

// The dynamic shared memory after the panels and the three parts of the u array, each part
// rounded up to 16 bytes; sizes for the batch's largest group (B.g_max, B.g_cnc, B.g_ck3).
struct GroupSm {
    double *red, *r64, *s64;  // 3 per CTA; coarse residual R r and direction R s, nc each
    float *rw, *r32, *ai, *ce;  // R w of the last reduction; R r in FP32; rows of A_c^-1; correction, in parts
    __device__ __forceinline__ GroupSm(unsigned char* base, const Batch& B) {
        red = reinterpret_cast<double*>(base);
        r64 = red + ((3 * B.g_max + 1) & ~1);
        s64 = r64 + ((B.g_cnc + 1) & ~1);
        rw = reinterpret_cast<float*>(s64 + ((B.g_cnc + 1) & ~1));
        r32 = rw + ((B.g_cnc + 3) & ~3);
        ce = r32 + ((B.g_cnc + 3) & ~3);
        ai = ce + ((CS_GROUP_CE_PARTS * B.g_ck3 + 3) & ~3);
    }
};

}  // namespace

extern __shared__ __align__(16) unsigned char cs_group_smem[];

// Cooperative launch, one CTA per SM (the CTAs wait on one another).  CTA c works through items
// B.gcta_item[B.gcta_ptr[c] .. B.gcta_ptr[c + 1]), each a sheet of which it holds one tile.
__global__ void __launch_bounds__(CS_GROUP_MAX_WARPS * 32, 1) cs_group_pcg_kernel(Batch B) {
    const DevParams& P = *B.params;
    if (P.solver != CS_SOLVER_AUTO_DEV || !P.mixed) return;  // uniform over the grid
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int halo0 = B.g_own;
    const float* sm_panels = reinterpret_cast<const float*>(cs_group_smem);
    float4* const su = reinterpret_cast<float4*>(cs_group_smem + (size_t)B.g_cap * CS_PANEL_FLOATS * sizeof(float));
    float4* const su_alt = su + B.g_own + B.g_halo;
    __shared__ GroupShared S;
    const GroupSm C(cs_group_smem + B.g_coff, B);
    const int myslot = w * CS_SLICE + lane;
    int* const err = B.loop + 6;

    for (int it = B.gcta_ptr[blockIdx.x]; it < B.gcta_ptr[blockIdx.x + 1]; it++) {
        const GroupItem gi = B.gitem[B.gcta_item[it]];
        const int s = gi.sheet;
        // sheets with proximity blocks outside the pattern are the batched loop's
        if (B.sheet_prox && (B.sheet_prox[s] & 2)) continue;
        const SheetDesc& sh = B.sheets[s];
        const int G = gi.ctas, rank = (int)blockIdx.x - gi.cta0, K = gi.segs, ns = sh.n_slices;
        const int lo = (int)((long long)ns * rank / G), hi = (int)((long long)ns * (rank + 1) / G), nsl = hi - lo;
        uint4* const upk = B.gupk + gi.slot0;  // one per row slot of the sheet
        uint4* const rpk = B.grpk + gi.red0;   // 2 x G x (K + 2)
        const int rstride = K + 2;
        __syncthreads();  // the previous item's shared memory is free
        // this thread's row: slice lo + w, lane.  The panels beyond the shared-memory budget are
        // the last slots of the slices (the loader chose how many of each, panels.h).
        bool live = false;
        int width = 0, ks = 0, lp = 0, gp = 0, tp = 0, row = 0, slot = 0, pub = 0;
        {
            const SliceDesc* sl = B.slices + sh.slice_off + lo;
            int at = 0;
            for (int j = 0; j < nsl; j++) {
                const int wd = sl[j].width, keep = sl[j].keep;
                // cooperative copy of the slice's kept panels
                const float4* src = reinterpret_cast<const float4*>(B.A + (size_t)sl[j].panel0 * CS_PANEL_FLOATS);
                float4* dst = reinterpret_cast<float4*>(cs_group_smem) + (size_t)at * (CS_PANEL_FLOATS / 4);
                for (int i = tid; i < keep * (CS_PANEL_FLOATS / 4); i += blockDim.x) dst[i] = __ldg(src + i);
                if (j == w) {
                    lp = at;
                    ks = keep;
                    width = wd;
                }
                at += keep;
            }
        }
        if (w < nsl) {
            const SliceDesc d = B.slices[sh.slice_off + lo + w];
            live = lane < d.rows;
            gp = d.panel0;
            tp = d.tpanel0;
            slot = (lo + w) * CS_SLICE + lane;
            if (live) {
                row = B.rowmap[d.topo_slice * CS_SLICE + lane];
                pub = B.gpub[gi.pub0 + slot];
            }
        }
        const int g = sh.node_off + row;
        const float* const spn = sm_panels + (size_t)lp * CS_PANEL_FLOATS;
        const float* const gpn = B.A + (size_t)gp * CS_PANEL_FLOATS;
        const int* const code = B.rcode + (size_t)tp * CS_SLICE;
        // byte offsets of the u entries of the slots in shared memory (the zero entry before the halo's for
        // others)
        uint32_t cw[CS_GROUP_MAX_WIDTH / 2];
        if (tid == 0) su[halo0 - 1] = su_alt[halo0 - 1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < CS_GROUP_MAX_WIDTH; j++) {
            const uint32_t at = 16u * (uint32_t)(live && j < ks ? __ldg(code + j * CS_SLICE + lane) : halo0 - 1);
            cw[j >> 1] = (j & 1) ? cw[j >> 1] | at << 16 : at;
        }
        const int h0 = B.ghalo_ptr[gi.halo0 + rank], nh = B.ghalo_ptr[gi.halo0 + rank + 1] - h0;
        const int my_halo = tid < nh ? __ldg(&B.ghalo[h0 + tid]) : 0;
        // the segment of this warp's rows: the tile's slices cut into K ranges
        int seg = 0;
        while (seg + 1 < K && w >= (nsl * (seg + 1)) / K) seg++;
        const int nc = 3 * G * K, k3 = 3 * K;
        const bool coarse = P.coarse && nc <= B.g_cnc && gi.mat >= 0 && B.gc_ok[s];
        if (coarse) {
            const float* src = B.gc_inv + gi.mat + (size_t)rank * k3 * nc;
            for (int i = tid; i < k3 * nc; i += blockDim.x) C.ai[i] = __ldcg(src + i);
            for (int i = tid; i < nc; i += blockDim.x) C.s64[i] = 0.0;
        }
        float Pi[9];
        float e[3] = {0.f, 0.f, 0.f}, r[3] = {0.f, 0.f, 0.f}, u[3], wv[3], p[3] = {0.f, 0.f, 0.f}, sv[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 9; k++) Pi[k] = live ? B.Pinv[9 * (size_t)g + k] : 0.f;
        if (live)
#pragma unroll
            for (int c = 0; c < 3; c++) r[c] = B.b[3 * g + c];
        // a node without a face has an empty row, which no correction may move
        bool moves = false;
#pragma unroll
        for (int k = 0; k < 9; k++) moves |= Pi[k] != 0.f;
        moves |= r[0] != 0.f || r[1] != 0.f || r[2] != 0.f;
        if (tid == 0) {
            S.bn = S.res0 = sqrt(B.inst[s].bnorm2);
            S.rr = S.delta = 0.0;
            S.resnorm = S.first_res = -1.0;
        }
        uint32_t nred = 0, nhalo = 0, tries = B.g_polls_first;

        // Waits for the packet at `q` to carry `epoch`; zeros with ok = false where that runs out.
        auto wait_packet = [&](const uint4* q, uint32_t epoch, bool& ok) -> uint4 {
            uint4 v = get_packet(q);
            for (uint32_t t = 0; v.w != epoch; t++) {
                if (t >= tries || ((t & 255u) == 255u && *(volatile int*)err)) {
                    ok = false;
                    return make_uint4(0u, 0u, 0u, 0u);
                }
                if (t > 64) __nanosleep(t > 4096 ? 256 : 32);
                v = get_packet(q);
            }
            return v;
        };
        // The warp's part of a reduction: sums 0 and 2, sum 1, the restriction of y
        auto put_sum02 = [&](double a, double c) {
            const double t = tile_sum2(a, c);
            if ((lane & 15) == 0) S.wsum[w][lane >> 3] = t;  // lane 0: sum 0, lane 16: sum 2
        };
        auto put_sum1 = [&](double a) {
            a = gwarp_sum(a);
            if (lane == 0) S.wsum[w][1] = a;
        };
        auto put_coarse = [&](const float (&y)[3]) {
            const float t = tile_sum3(y[0], y[1], y[2]);
            if ((lane & 7) == 0 && lane < 24) S.wseg[w][lane >> 3] = t;
        };
        // Group-wide sums v of the warps' (identical in every CTA) and, with `y`, R y into C.rw.  Packet i < 3 of
        // a CTA carries its part of sum i and component i of its first segment's sum of y, packet
        // 2 + k the three components of segment k > 0.
        auto group_sum = [&](double (&v)[3], bool y) -> bool {
            const uint32_t epoch = nred + 1, buf = nred & 1u;
            nred++;
            const int np = y ? rstride : 3;
            __syncthreads();
            uint4* const mine = rpk + ((size_t)buf * G + rank) * rstride;
            if (tid < 3) {
                double a = 0.0;
                float f = 0.f;
#pragma unroll
                for (int j = 0; j < CS_GROUP_MAX_WARPS; j++) {
                    if (j < nsl) a += S.wsum[j][tid];
                    if (j < nsl / K) f += S.wseg[j][tid];
                }
                put_packet(mine + tid, (uint32_t)__double2loint(a), (uint32_t)__double2hiint(a), __float_as_uint(f), epoch);
            } else if (y && tid > 32 && tid < 32 + K) {
                const int k = tid - 32;
                float f[3] = {0.f, 0.f, 0.f};
                for (int j = (nsl * k) / K; j < (nsl * (k + 1)) / K; j++)
#pragma unroll
                    for (int c = 0; c < 3; c++) f[c] += S.wseg[j][c];
                put_packet(mine + 2 + k, __float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), epoch);
            }
            bool ok = true;
            for (int q = tid; q < G * np; q += blockDim.x) {
                const int c = q / np, k = q - c * np;
                const uint4 x = wait_packet(rpk + ((size_t)buf * G + c) * rstride + k, epoch, ok);
                if (k < 3) {
                    C.red[3 * c + k] = __hiloint2double((int)x.y, (int)x.x);
                    if (y) C.rw[c * k3 + k] = __uint_as_float(x.z);
                } else {
                    float* o = C.rw + c * k3 + 3 * (k - 2);
                    o[0] = __uint_as_float(x.x);
                    o[1] = __uint_as_float(x.y);
                    o[2] = __uint_as_float(x.z);
                }
            }
            tries = B.g_polls;
            if (!ok) atomicExch(err, 1);
            if (!__syncthreads_and(ok ? 1 : 0)) return false;
            // with fewer than three warps, a warp takes more than one sum
            for (int i = w; i < 3; i += (int)(blockDim.x >> 5)) {
                double a = 0.0;
                for (int c = lane; c < G; c += 32) a += C.red[3 * c + i];
                a = gwarp_sum(a);
                if (lane == 0) S.tot[i] = a;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 3; i++) v[i] = S.tot[i];
            return true;
        };
        auto local_spmv = [&](const float4* buf, float (&q)[3]) {
            q[0] = q[1] = q[2] = 0.f;
            row_times<CS_GROUP_MAX_WIDTH, 3, true>(spn, gpn, ks, width, cw, code, row_tail_load(gpn, ks, width, code, lane), buf,
                                                   halo0, lane, live, q[0], q[1], q[2]);
        };
        auto cta_sum2 = [&](double& a, double& b) {
            a = gwarp_sum(a);
            b = gwarp_sum(b);
            if (lane == 0) {
                S.wsum[w][0] = a;
                S.wsum[w][1] = b;
            }
            __syncthreads();
            a = b = 0.0;
            for (int j = 0; j < nsl; j++) {
                a += S.wsum[j][0];
                b += S.wsum[j][1];
            }
            __syncthreads();
        };
        // ce = this CTA's rows of A_c^-1 R r, a row's columns shared out over `parts` warps whose sums
        // are added where the correction is used
        const int parts = max(1, min(CS_GROUP_CE_PARTS, (int)(blockDim.x >> 5) / k3));
        auto coarse_matvec = [&]() {
            for (int j = w; j < k3 * parts; j += (int)(blockDim.x >> 5)) {
                const float* ai = C.ai + (j / parts) * nc;
                float a = 0.f, b = 0.f;
                int t = (j % parts) * 32 + lane;
                for (; t + 32 * parts < nc; t += 64 * parts) {
                    a = fmaf(ai[t], C.r32[t], a);
                    b = fmaf(ai[t + 32 * parts], C.r32[t + 32 * parts], b);
                }
                if (t < nc) a = fmaf(ai[t], C.r32[t], a);
                a = gwarp_sum(a + b);
                if (lane == 0) C.ce[j] = a;
            }
        };
        auto coarse_step = [&](double beta_c, double alpha_c) {
            for (int q = tid; q < nc; q += blockDim.x) {
                const double sq = (double)C.rw[q] + beta_c * C.s64[q];
                C.s64[q] = sq;
                const double rq = C.r64[q] - alpha_c * sq;
                C.r64[q] = rq;
                C.r32[q] = (float)rq;
            }
        };
        // The tile-local Chebyshev polynomial's interval: power iteration for P^-1 A_loc, as in
        // resident.cu (an odd degree keeps the preconditioner SPD whatever the estimate).
        const bool levels = P.coarse && P.cheb_degree >= 3;
        __syncthreads();
        LevelPlace at{(uint32_t)myslot * 0x10001u};
        if (levels) {
            const uint32_t* cells = B.rcell + (size_t)B.slices[sh.slice_off + lo].topo_slice * CS_SLICE;
            if (live) at.v = __ldg(cells + myslot);
            level_blocks(spn, gpn, ks, width, code, cells, halo0 - 1, at, lane, live, su_alt, S.lev[w]);
        }
        if (!levels && P.cheb_degree >= 3) {
            float v[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const uint32_t h = (uint32_t)(3 * row + c) * 0x9E3779B1u;
                v[c] = live ? (((h >> 16) & 1u) ? 1.f : -1.f) : 0.f;
            }
            double lam = 0.0;
            for (int k = 0; k < CS_CHEB_POWER_ITERS; k++) {
                su_alt[myslot] = make_float4(v[0], v[1], v[2], 0.f);
                __syncthreads();
                float q[3], z[3];
                local_spmv(su_alt, q);
                gmat3_vec(Pi, q, z);
                double zz = (double)z[0] * z[0] + (double)z[1] * z[1] + (double)z[2] * z[2];
                double vv = (double)v[0] * v[0] + (double)v[1] * v[1] + (double)v[2] * v[2];
                cta_sum2(zz, vv);
                lam = vv > 0.0 ? sqrt(zz / vv) : 0.0;
                const float sc = zz > 0.0 ? (float)(1.0 / sqrt(zz)) : 0.f;
#pragma unroll
                for (int c = 0; c < 3; c++) v[c] = z[c] * sc;
            }
            if (tid == 0) {
                int deg = P.cheb_degree;
                if (!(lam > 0.0) || !gfinite(lam)) deg = 1;
                const float lmax = G_LMAX_MARGIN * (float)lam, lmin = lmax * G_LMIN_RATIO;
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

        double gam = 0.0, gam_prev = 0.0, alpha_d = 0.0;
        double inv_gam = 0.0, inv_ga = 0.0;
        bool cont = false;         // the next PH_INIT keeps the search direction (reliable update)
        bool dv_zero = !P.warm;    // dv64 and e are zero: the next FP64 residual is b
        bool scale_pass = P.warm && P.warm_scale;
        float alpha = 0.f, beta = 0.f;
        int iters = 0, sweeps = 0, sweep_iters = 0, flags = 0, trips = 0;
        int phase = PH_RES;
        bool ok = true;
        while (phase != PH_FINISH) {
            if (++trips > P.loop_cap) {
                flags |= CS_IF_CAPPED;
                break;
            }
            if (phase == PH_RES) {
                const bool zero = dv_zero;
                dv_zero = false;
                if (live) {
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        B.dv64[3 * g + c] += (double)e[c];
                        e[c] = 0.f;
                    }
                }
                double v[3] = {0.0, 0.0, 0.0};
                if (!zero) {
                    // every CTA's rows of dv64 are written before any is read
                    __threadfence();
                    put_sum02(0.0, 0.0);
                    put_sum1(0.0);
                    ok = group_sum(v, false);
                    if (!ok) break;
                    __threadfence();
                }
                v[0] = v[1] = v[2] = 0.0;
                float rn[3] = {0.f, 0.f, 0.f};
                if (live) {
                    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
                    for (int k0 = 0; k0 < width && !zero; k0 += 4) {
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
                            const float* pk = (k0 + j < ks ? spn : gpn) + (size_t)(k0 + j) * CS_PANEL_FLOATS;
                            const float4 a0 = reinterpret_cast<const float4*>(pk)[lane];
                            const float4 a1 = reinterpret_cast<const float4*>(pk + 128)[lane];
                            const float a8 = pk[256 + lane];
                            y0 += (double)a0.x * d[j][0] + (double)a0.y * d[j][1] + (double)a0.z * d[j][2];
                            y1 += (double)a0.w * d[j][0] + (double)a1.x * d[j][1] + (double)a1.y * d[j][2];
                            y2 += (double)a1.z * d[j][0] + (double)a1.w * d[j][1] + (double)a8 * d[j][2];
                        }
                    }
                    const double b0 = B.b[3 * g], b1 = B.b[3 * g + 1], b2 = B.b[3 * g + 2];
                    const double r0 = b0 - y0, r1 = b1 - y1, r2 = b2 - y2;
                    const double q0 = r0 - (double)r[0], q1 = r1 - (double)r[1], q2 = r2 - (double)r[2];
                    rn[0] = (float)r0;
                    rn[1] = (float)r1;
                    rn[2] = (float)r2;
                    if (scale_pass) {
                        const double d0 = B.dv64[3 * g], d1 = B.dv64[3 * g + 1], d2 = B.dv64[3 * g + 2];
                        v[0] = d0 * b0 + d1 * b1 + d2 * b2;
                        v[1] = d0 * r0 + d1 * r1 + d2 * r2;
                    } else {
                        v[0] = r0 * r0 + r1 * r1 + r2 * r2;
                        v[1] = q0 * q0 + q1 * q1 + q2 * q2;
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; c++) r[c] = rn[c];
                // the coarse residual R r of the replaced r travels with the norms
                put_sum02(v[0], v[2]);
                put_sum1(v[1]);
                if (coarse) put_coarse(r);
                ok = group_sum(v, coarse);
                if (!ok) break;
                if (coarse)
                    for (int q = tid; q < nc; q += blockDim.x) {
                        C.r64[q] = (double)C.rw[q];
                        C.r32[q] = C.rw[q];
                    }
                if (scale_pass) {
                    // d becomes a d, a = d.b / d.A d (d.A d = d.b - d.r), the multiple of d nearest to
                    // the solution in the energy norm; the next residual judges it
                    scale_pass = false;
                    const double dad = v[0] - v[1], a = v[0] / dad;
                    const bool good = dad > 0.0 && gfinite(a);
                    if (live) {
#pragma unroll
                        for (int c = 0; c < 3; c++) B.dv64[3 * g + c] = good ? B.dv64[3 * g + c] * a : 0.0;
                    }
                    if (!good) {
                        flags |= CS_IF_WARM_REJECTED;
                        dv_zero = true;
                        sweeps = 1;
                    }
                    continue;  // phase stays PH_RES
                }
                const double res = sqrt(v[0]), bn = S.bn;
                sweeps += 1;
                if (tid == 0) {
                    S.resnorm = res;
                    if (sweeps == 1) S.first_res = res;
                }
                if (sweeps == 1) {
                    if (P.warm && !(res <= bn)) {
                        // the warm start is worse than the zero guess: discard it
                        flags |= CS_IF_WARM_REJECTED;
                        if (live) {
#pragma unroll
                            for (int c = 0; c < 3; c++) B.dv64[3 * g + c] = 0.0;
                        }
                        dv_zero = true;
                        continue;  // the residual of dv = 0
                    }
                }
                if (res <= P.tol * bn || bn == 0.0) {
                    flags |= CS_IF_CONVERGED;
                    phase = PH_FINISH;
                } else if (iters >= P.max_iters) {
                    flags |= CS_IF_CAPPED;
                    phase = PH_FINISH;
                } else {
                    // a reliable update keeps the direction of the last sweep if r drifted little
                    if (tid == 0) S.res0 = res;  // read after the next barriers
                    cont = sweep_iters > 0 && !(flags & CS_IF_BREAKDOWN) && sqrt(v[1]) <= CS_RELIABLE_DRIFT * res;
                    phase = PH_INIT;
                }
                continue;
            }
            // PH_INIT (start of a sweep) or PH_CG: u = P^-1 r, halo exchange, w = A u, and one
            // reduction of (r.u, w.u, r.r)
            if (phase == PH_CG) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    e[c] = __fmaf_rn(alpha, p[c], e[c]);
                    r[c] = __fmaf_rn(-alpha, sv[c], r[c]);
                }
            }
            gmat3_vec(Pi, r, u);
            if (cdeg >= 3) {
                float d[3];
                const float ith = S.cheb_inv_th;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    d[c] = u[c] * ith;
                    u[c] = d[c];
                }
                // alternating own-row buffers, ending on su_alt: one barrier per step orders every
                // write after the reads of the buffer's previous contents
                for (int k = 1; k < cdeg; k++) {
                    float4* const buf = (k & 1) ? su : su_alt;
                    buf[myslot] = make_float4(u[0], u[1], u[2], 0.f);
                    __syncthreads();
                    if (coarse && k == 1) coarse_matvec();
                    float q[3], t[3];
                    local_spmv(buf, q);
#pragma unroll
                    for (int c = 0; c < 3; c++) q[c] = r[c] - q[c];
                    gmat3_vec(Pi, q, t);
                    const float ca = S.cheb_a[k], cb = S.cheb_b[k];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        d[c] = ca * d[c] + cb * t[c];
                        u[c] += d[c];
                    }
                }
            } else if (levels || coarse) {
                if (levels) su[myslot] = make_float4(r[0], r[1], r[2], 0.f);
                __syncthreads();
                if (levels) level_sums(S.lev[w], su[at.slot()], su_alt, w, lane);
                if (coarse) coarse_matvec();
                __syncthreads();
                if (levels) level_add(su_alt, at, u);
            }
            if (coarse && live) {
                // u = C r + R^T A_c^-1 R r: the additive coarse-space correction
#pragma unroll
                for (int c = 0; c < 3; c++)
                    for (int q = 0; q < parts; q++) u[c] += C.ce[(3 * seg + c) * parts + q];
            }
            nhalo++;
            if (!moves) u[0] = u[1] = u[2] = 0.f;  // the corrections reach lanes without a row and empty rows
            su[myslot] = make_float4(u[0], u[1], u[2], 0.f);
            if (live && pub)
                put_packet(upk + slot, __float_as_uint(u[0]), __float_as_uint(u[1]), __float_as_uint(u[2]), nhalo);
            // while the halo values travel: the sums r.u and r.r, the first slot in global memory
            const RowTail tail = row_tail_load(gpn, ks, width, code, lane);
            put_sum02((double)r[0] * u[0] + (double)r[1] * u[1] + (double)r[2] * u[2],
                      (double)r[0] * r[0] + (double)r[1] * r[1] + (double)r[2] * r[2]);
            for (int i = tid; i < nh; i += blockDim.x) {
                const uint4 x = wait_packet(upk + (i == tid ? my_halo : __ldg(&B.ghalo[h0 + i])), nhalo, ok);
                su[halo0 + i] = make_float4(__uint_as_float(x.x), __uint_as_float(x.y), __uint_as_float(x.z), 0.f);
            }
            if (!ok) atomicExch(err, 1);
            ok = __syncthreads_and(ok ? 1 : 0) != 0;
            if (!ok) break;
            wv[0] = wv[1] = wv[2] = 0.f;
            row_times<CS_GROUP_MAX_WIDTH, 3, false>(spn, gpn, ks, width, cw, code, tail, su, halo0, lane, live, wv[0], wv[1], wv[2]);
            put_sum1((double)wv[0] * u[0] + (double)wv[1] * u[1] + (double)wv[2] * u[2]);
            if (coarse) put_coarse(wv);
            double v[3];
            ok = group_sum(v, coarse);
            if (!ok) break;
            const double gnew = v[0], dnew = v[1], rr = v[2];
            if (tid == 0) {
                S.rr = rr;
                S.delta = dnew;
            }
            if (phase == PH_INIT && cont) {
                // p = u + beta p, s = w + beta s with beta = (r.u) / (the last iteration's r.u); r
                // left the recursion that the Chronopoulos-Gear step length assumes, so alpha =
                // r.u / p.s takes one more reduction
                cont = false;
                const double bd = gnew / gam_prev;
                if (gnew > 0.0 && gfinite(gnew) && gfinite(bd)) {
                    const float bc = (float)bd;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        p[c] = __fmaf_rn(bc, p[c], u[c]);
                        sv[c] = __fmaf_rn(bc, sv[c], wv[c]);
                    }
                    double v2[3] = {0.0, 0.0, 0.0};
                    if (live) v2[0] = (double)p[0] * sv[0] + (double)p[1] * sv[1] + (double)p[2] * sv[2];
                    put_sum02(v2[0], 0.0);
                    put_sum1(0.0);
                    ok = group_sum(v2, false);
                    if (!ok) break;
                    if (v2[0] > 0.0 && gfinite(v2[0]) && gfinite(gnew / v2[0])) {
                        gam = gnew;
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
                sweep_iters = 0;
                beta = 0.f;
                if (!(gam > 0.0 && gfinite(gam))) {
                    phase = PH_RES;
                    continue;
                }
                alpha_d = gam / dnew;
                alpha = (float)alpha_d;
                inv_gam = 1.0 / gam;
                inv_ga = 1.0 / (gam * alpha_d);
                if (!(dnew > 0.0) || !gfinite((double)alpha)) {
                    flags |= CS_IF_BREAKDOWN;
                    phase = PH_RES;
                    continue;
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    p[c] = u[c];
                    sv[c] = wv[c];
                }
                if (coarse) coarse_step(0.0, alpha_d);
                phase = PH_CG;
                continue;
            }
            // PH_CG: the iteration's x and r updates are done; stopping test on ||r||
            iters += 1;
            sweep_iters += 1;
            // the sweep's end, as in resident.cu
            const double ti = P.inner_tol * S.res0, tt = P.tol * S.bn;
            const double t = P.cheb_degree >= 3 ? (ti > tt ? ti : CS_LAST_SWEEP * tt) : fmax(ti, 0.5 * tt);
            bool stop = rr <= t * t || sweep_iters >= P.sweep_cap;
            const double bd = gnew * inv_gam, na = gnew / (dnew - gnew * gnew * inv_ga);
            if (!gfinite((double)(float)bd) || !gfinite((double)(float)na) || !(gnew > 0.0) || !((float)na > 0.f)) {
                flags |= CS_IF_BREAKDOWN;
                stop = true;
            }
            gam_prev = gam;
            gam = gnew;
            if (stop || iters >= P.max_iters) {
                phase = PH_RES;
                continue;
            }
            beta = (float)bd;
            alpha = (float)na;
            alpha_d = na;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                p[c] = __fmaf_rn(beta, p[c], u[c]);
                sv[c] = __fmaf_rn(beta, sv[c], wv[c]);
            }
            if (coarse) coarse_step((double)beta, alpha_d);
            inv_gam = 1.0 / gam;
            inv_ga = 1.0 / (gam * alpha_d);
        }
        if (!ok) flags |= CS_IF_BREAKDOWN;
        if (live && (!ok || trips > P.loop_cap)) {
#pragma unroll
            for (int c = 0; c < 3; c++) B.dv64[3 * g + c] += (double)e[c];
        }
        if (rank == 0 && tid == 0) {
            InstState& I = B.inst[s];
            I.rz = gam;
            I.rr = S.rr;
            I.pq = S.delta;
            I.res0 = S.res0;
            I.resnorm = S.resnorm;
            I.first_res = S.first_res;
            I.alpha = alpha;
            I.beta = beta;
            I.iters = iters;
            I.sweeps = sweeps;
            I.sweep_iters = sweep_iters;
            I.flags = flags;
            I.phase = PH_DONE;
        }
        if (!ok) return;
    }
}
