// The collision step on the device (cs_collision_step): Simulator::collisionStep as the
// reference's GPU path runs it after the implicit step (Simulator.cu:602-684).
//
// Each round: candidate face pairs from the contact grid over the start-of-step and current
// positions (contact.cu with ccd bounds, dilated by the collision thickness), then
//   cs_impact_kernel         per (pair, test) the shared-node and swept-box filters, the
//                            survivors compacted per block, then the continuous impact test
//                            of checkVertexFaceImpact / checkEdgeEdgeImpact
//                            (CollisionHelper.cu:61-136: the cubic for coplanarity along the
//                            linear trajectories, solveCubic / solveQuadratic /
//                            newtonsMethod :3-59, the distance and side at the root);
//   cs_impact_keys/gather_kernel  keys of the stable radix sorts by impact time (ties by node
//                            ids, type, index; the sorts are CUB's, in ctx.cu), then the gather;
//   cs_select_*_kernel       the independent impacts, earliest first, one per node
//                            (Simulator.cu:394-420), by rounds of per-node minima;
//   cs_opt_*_kernel          the impact zone's nodes (ascending), each impact's node slots,
//                            each node's constraint list in constraint order;
//   cs_opt_kernel            one cluster: CollisionOptimization (CollisionOptimization.cu) solved
//                            by Optimization::solve's augmented Lagrangian gradient descent
//                            (Optimization.cu:94-137).  Element terms are computed in
//                            parallel; every sum has the CPU loop's order and rounding,
//                            so the iterates are the FP32 CPU path's bit for bit.
// After the rounds, cs_collide_velocity_kernel sets v = (x - x0) / dt (Mesh.cu:238-247).
// Built without FMA contraction.
#include <cooperative_groups.h>

#include "cs_internal.h"

namespace cg = cooperative_groups;

namespace {

struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 ld(const float* p, int i) { return mk(p[3 * i], p[3 * i + 1], p[3 * i + 2]); }
__device__ __forceinline__ void st(float* p, int i, f3 a) {
    p[3 * i] = a.x;
    p[3 * i + 1] = a.y;
    p[3 * i + 2] = a.z;
}
__device__ __forceinline__ f3 sub(f3 a, f3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ f3 add(f3 a, f3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ f3 scl(float s, f3 a) { return mk(s * a.x, s * a.y, s * a.z); }
// Vector.cuh:126-176 (dot and norm2 from zero, division by the reciprocal)
__device__ __forceinline__ float dot0(f3 a, f3 b) {
    float s = 0.0f;
    s += a.x * b.x;
    s += a.y * b.y;
    s += a.z * b.z;
    return s;
}
__device__ __forceinline__ f3 dvd(f3 a, float s) {
    const float inv = 1.0f / s;
    return mk(a.x * inv, a.y * inv, a.z * inv);
}
__device__ __forceinline__ f3 normalized(f3 a) { return dvd(a, sqrtf(dot0(a, a))); }
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
    return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float mixed(f3 a, f3 b, f3 c) { return dot0(a, cross(b, c)); }  // MathHelper.cuh:43-45
__device__ __forceinline__ float mn(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float mx(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float ab(float x) { return x < 0.0f ? -x : x; }

// signedVertexFaceDistance / signedEdgeEdgeDistance (MathHelper.cu:38-69); false for INFINITY
__device__ bool signed_vf(f3 x, f3 y0, f3 y1, f3 y2, f3& n, float w[4], float& h) {
    n = cross(normalized(sub(y1, y0)), normalized(sub(y2, y0)));
    if (dot0(n, n) < 1e-6f) return false;
    n = normalized(n);
    h = dot0(sub(x, y0), n);
    const float b0 = mixed(sub(y1, x), sub(y2, x), n);
    const float b1 = mixed(sub(y2, x), sub(y0, x), n);
    const float b2 = mixed(sub(y0, x), sub(y1, x), n);
    w[0] = 1.0f;
    w[1] = -b0 / (b0 + b1 + b2);
    w[2] = -b1 / (b0 + b1 + b2);
    w[3] = -b2 / (b0 + b1 + b2);
    return true;
}
__device__ bool signed_ee(f3 x0, f3 x1, f3 y0, f3 y1, f3& n, float w[4], float& h) {
    n = cross(normalized(sub(x1, x0)), normalized(sub(y1, y0)));
    if (dot0(n, n) < 1e-6f) return false;
    n = normalized(n);
    h = dot0(sub(x0, y0), n);
    const float a0 = mixed(sub(y1, x1), sub(y0, x1), n);
    const float a1 = mixed(sub(y0, x0), sub(y1, x0), n);
    const float b0 = mixed(sub(x0, y1), sub(x1, y1), n);
    const float b1 = mixed(sub(x1, y0), sub(x0, y0), n);
    w[0] = a0 / (a0 + a1);
    w[1] = a1 / (a0 + a1);
    w[2] = -b0 / (b0 + b1);
    w[3] = -b1 / (b0 + b1);
    return true;
}

// CollisionHelper.cu:3-20
__device__ float newtons_method(float a, float b, float c, float d, float x0, int dir) {
    if (dir != 0) {
        const float y0 = d + x0 * (c + x0 * (b + x0 * a));
        const float ddy0 = 2.0f * b + x0 * (6.0f * a);
        x0 += (float)dir * sqrtf(ab(2.0f * y0 / ddy0));
    }
    for (int iter = 0; iter < 100; iter++) {
        const float y = d + x0 * (c + x0 * (b + x0 * a));
        const float dy = c + x0 * (2.0f * b + 3.0f * x0 * a);
        if (dy == 0) return x0;
        const float x1 = x0 - y / dy;
        if (ab(x0 - x1) < 1e-6f) return x0;
        x0 = x1;
    }
    return x0;
}

// CollisionHelper.cu:22-37
__device__ int solve_quadratic(float a, float b, float c, float x[2]) {
    const float d = b * b - 4.0f * a * c;
    if (d < 0.0f) {
        x[0] = -b / (2.0f * a);
        return 0;
    }
    const float q = -(b + (float)(b < 0.0f ? -1 : 1) * sqrtf(d)) * 0.5f;
    int i = 0;
    if (ab(a) > 1e-12f * ab(q)) x[i++] = q / a;
    if (ab(q) > 1e-12f * ab(c)) x[i++] = c / q;
    if (i == 2 && x[0] > x[1]) {
        const float t = x[0];
        x[0] = x[1];
        x[1] = t;
    }
    return i;
}

// CollisionHelper.cu:39-59.  Where solve_quadratic finds no root without writing one (both of
// its guards fail: a degenerate derivative), Newton's method starts from 0, as the oracle does
// (the reference reads an uninitialised value there).
__device__ int solve_cubic(float a, float b, float c, float d, float x[3]) {
    float xc[2] = {0.0f, 0.0f};
    const int n = solve_quadratic(3.0f * a, 2.0f * b, c, xc);
    if (n == 0) {
        x[0] = newtons_method(a, b, c, d, xc[0], 0);
        return 1;
    }
    if (n == 1) return solve_quadratic(b, c, d, x);
    const float yc[2] = {d + xc[0] * (c + xc[0] * (b + xc[0] * a)), d + xc[1] * (c + xc[1] * (b + xc[1] * a))};
    int i = 0;
    if (yc[0] * a >= 0.0f) x[i++] = newtons_method(a, b, c, d, xc[0], -1);
    if (yc[0] * yc[1] <= 0.0f) {
        const int closer = ab(yc[0]) < ab(yc[1]) ? 0 : 1;
        x[i++] = newtons_method(a, b, c, d, xc[closer], closer == 0 ? 1 : -1);
    }
    if (yc[1] * a <= 0.0f) x[i++] = newtons_method(a, b, c, d, xc[1], 1);
    return i;
}

// checkImpact (CollisionHelper.cu:61-110)
__device__ bool check_impact(int type, const f3 p[4], const f3 q[4], ImpactRec& r) {
    const f3 x0 = p[0];
    const f3 v0 = sub(q[0], x0);
    const f3 x1 = sub(p[1], x0), x2 = sub(p[2], x0), x3 = sub(p[3], x0);
    const f3 v1 = sub(sub(q[1], p[1]), v0), v2 = sub(sub(q[2], p[2]), v0), v3 = sub(sub(q[3], p[3]), v0);
    const float a0 = mixed(x1, x2, x3);
    const float a1 = mixed(v1, x2, x3) + mixed(x1, v2, x3) + mixed(x1, x2, v3);
    const float a2 = mixed(x1, v2, v3) + mixed(v1, x2, v3) + mixed(v1, v2, x3);
    const float a3 = mixed(v1, v2, v3);
    float t[3] = {0.0f, 0.0f, 0.0f};
    const int ns = solve_cubic(a3, a2, a1, a0, t);
    for (int i = 0; i < ns; i++) {
        if (t[i] < 0.0f || t[i] > 1.0f) continue;
        f3 y[4];
        for (int k = 0; k < 4; k++) y[k] = add(p[k], scl(t[i], sub(q[k], p[k])));  // Node::position
        f3 n;
        float w[4], h;
        bool inside;
        if (type == 0) {
            if (!signed_vf(y[0], y[1], y[2], y[3], n, w, h)) continue;
            inside = mn(-w[1], mn(-w[2], -w[3])) >= -1e-6f;
        } else {
            if (!signed_ee(y[0], y[1], y[2], y[3], n, w, h)) continue;
            inside = mn(mn(w[0], w[1]), mn(-w[2], -w[3])) >= -1e-6f;
        }
        if (dot0(n, add(add(scl(w[1], v1), scl(w[2], v2)), scl(w[3], v3))) > 0.0f) n = mk(-n.x, -n.y, -n.z);
        if (ab(h) < 1e-6f && inside) {
            r.type = type;
            r.t = t[i];
            for (int k = 0; k < 4; k++) r.w[k] = w[k];
            r.n[0] = n.x;
            r.n[1] = n.y;
            r.n[2] = n.z;
            return true;
        }
    }
    return false;
}

// Bounds of a node set over its start and current positions (Node/Face/Edge::bounds(ccd)).
__device__ void ccd_box(const Batch& B, const int* nodes, int k, float lo[3], float hi[3]) {
    for (int c = 0; c < 3; c++) {
        lo[c] = 3.0e38f;
        hi[c] = -3.0e38f;
    }
    for (int i = 0; i < k; i++) {
        const float* a = B.x + 3 * (size_t)nodes[i];
        const float* b = B.x0 + 3 * (size_t)nodes[i];
        for (int c = 0; c < 3; c++) {
            lo[c] = mn(mn(lo[c], a[c]), b[c]);
            hi[c] = mx(mx(hi[c], a[c]), b[c]);
        }
    }
}
// Bounds::overlap(b, thickness) (Bounds.cu:85-101): a against b dilated
__device__ bool overlap(const float alo[3], const float ahi[3], const float blo[3], const float bhi[3], float t) {
    for (int c = 0; c < 3; c++) {
        if (alo[c] > bhi[c] + t) return false;
        if (ahi[c] < blo[c] - t) return false;
    }
    return true;
}

// The swept-box filter of checkVertexFaceImpact / checkEdgeEdgeImpact (type 0: vertex-face,
// 1: edge-edge): false where the bounds of the two elements over the step stay apart.
__device__ bool impact_boxes_meet(const Batch& B, const Collide& K, int type, const int nodes[4]) {
    float alo[3], ahi[3], blo[3], bhi[3];
    if (type == 0) {
        ccd_box(B, nodes, 1, alo, ahi);
        ccd_box(B, nodes + 1, 3, blo, bhi);
    } else {
        ccd_box(B, nodes, 2, alo, ahi);
        ccd_box(B, nodes + 2, 2, blo, bhi);
    }
    return overlap(alo, ahi, blo, bhi, K.thickness);
}

// The continuous test of one element pair that passed the filters; an impact is appended.
__device__ void impact_test(const Batch& B, const Collide& K, int type, const int nodes[4]) {
    f3 p[4], q[4];
    for (int k = 0; k < 4; k++) {
        p[k] = ld(B.x0, nodes[k]);
        q[k] = ld(B.x, nodes[k]);
    }
    ImpactRec r;
    if (!check_impact(type, p, q, r)) return;
    for (int k = 0; k < 4; k++) r.nodes[k] = nodes[k];
    const int slot = atomicAdd(&K.counters[0], 1);
    if (slot < K.found_cap) K.found[slot] = r;
}

// The nodes of test k (0-5 vertex-face, 6-14 edge-edge) of candidate pair pr, or false where
// the two elements share a node (checkImpacts skips those, Simulator.cu:369-381).
__device__ bool impact_nodes(const Batch& B, const Contact& C, int2 pr, int k, int& type, int nodes[4]) {
    if (k < 6) {
        // vertex-face: corner k % 3 of one face against the other face
        const int f = k < 3 ? pr.x : pr.y, g = k < 3 ? pr.y : pr.x;
        const int4 y = B.face_nodes[f], z = B.face_nodes[g];
        const int i = k % 3;
        const int node = i == 0 ? y.x : i == 1 ? y.y : y.z;
        if (node == z.x || node == z.y || node == z.z) return false;
        type = 0;
        nodes[0] = node;
        nodes[1] = z.x;
        nodes[2] = z.y;
        nodes[3] = z.z;
        return true;
    }
    // edge-edge: edge i of the first face against edge j of the second
    const int4 fe = C.face_edges[pr.x], ge = C.face_edges[pr.y];
    const int i = (k - 6) / 3, j = (k - 6) % 3;
    const int4 a = C.edges[i == 0 ? fe.x : i == 1 ? fe.y : fe.z], b = C.edges[j == 0 ? ge.x : j == 1 ? ge.y : ge.z];
    if (a.x == b.x || a.x == b.y || a.y == b.x || a.y == b.y) return false;
    type = 1;
    nodes[0] = a.x;
    nodes[1] = a.y;
    nodes[2] = b.x;
    nodes[3] = b.y;
    return true;
}

}  // namespace

// checkImpacts (Simulator.cu:369-381): per candidate pair its 6 vertex-face and 9 edge-edge
// tests.  Each block takes kImpactItems consecutive (pair, test) items: first every thread
// applies the cheap filters (shared nodes, swept boxes) to its items and queues the survivors
// in shared memory, then the block's threads share out the queued continuous tests, so the
// cubic solves run with full warps instead of beside threads that have nothing to do.  The
// impacts' order in `found` does not matter: the round sorts them by a total order.
constexpr int kImpactThreads = 256, kImpactPerThread = 8, kImpactItems = kImpactThreads * kImpactPerThread;
__global__ void __launch_bounds__(kImpactThreads) cs_impact_kernel(Batch B, Contact C, Collide K, int npairs) {
    __shared__ int4 qnodes[kImpactItems];
    __shared__ unsigned char qtype[kImpactItems];
    __shared__ int qcount;
    if (threadIdx.x == 0) qcount = 0;
    __syncthreads();
    const long long total = 15LL * npairs, base = (long long)blockIdx.x * kImpactItems;
    for (int j = 0; j < kImpactPerThread; j++) {
        const long long item = base + j * kImpactThreads + threadIdx.x;
        if (item >= total) break;
        const int2 pr = C.pairs[(int)(item / 15)];
        int type, nodes[4];
        if (!impact_nodes(B, C, pr, (int)(item % 15), type, nodes)) continue;
        if (!impact_boxes_meet(B, K, type, nodes)) continue;
        const int slot = atomicAdd(&qcount, 1);
        qnodes[slot] = make_int4(nodes[0], nodes[1], nodes[2], nodes[3]);
        qtype[slot] = (unsigned char)type;
    }
    __syncthreads();
    const int n = qcount;
    for (int q = threadIdx.x; q < n; q += kImpactThreads) {
        const int4 v = qnodes[q];
        const int nodes[4] = {v.x, v.y, v.z, v.w};
        impact_test(B, K, qtype[q], nodes);
    }
}

// Order of the found impacts: by time, then node ids, then type, then index (std::sort in
// Simulator::independentImpacts orders by time; the rest makes the order total).  A least-
// significant-first sequence of stable radix sorts (CUB, in ctx.cu) over the key parts: type,
// (n2, n3), n1, (t, n0).  t >= 0, so its IEEE bits order like its values once -0.0 (which the
// impact tests accept: it is not below 0, and the quadratic's c / q yields it for a start that
// is exactly coplanar) is taken as +0.0, as the oracle's comparison of times does; node ids
// are >= 0.  pass 0 also starts the permutation at the identity.
__global__ void cs_impact_keys_kernel(Collide K, int n, int pass, const int* __restrict__ perm,
                                      unsigned long long* __restrict__ key, int* __restrict__ perm_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int src = pass == 0 ? i : perm[i];
    if (pass == 0) perm_out[i] = i;
    const ImpactRec& r = K.found[src];
    unsigned long long k;
    if (pass == 0) k = (unsigned long long)(unsigned)r.type;
    else if (pass == 1) k = ((unsigned long long)(unsigned)r.nodes[2] << 32) | (unsigned)r.nodes[3];
    else if (pass == 2) k = (unsigned long long)(unsigned)r.nodes[1];
    else k = ((unsigned long long)(r.t == 0.0f ? 0u : __float_as_uint(r.t)) << 32) | (unsigned)r.nodes[0];
    key[i] = k;
}

__global__ void cs_impact_gather_kernel(Collide K, int n, const int* __restrict__ perm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) K.sorted[i] = K.found[perm[i]];
}

// independentImpacts (Simulator.cu:394-420) in parallel: the earliest-first greedy choice of
// impacts with disjoint nodes equals, round by round, the impacts that are the earliest live
// impact at each of their nodes; those are chosen, and the live impacts sharing a node with
// them drop out (the reference's GPU branch uses the same scheme, Simulator.cu:422-468).
__global__ void cs_select_init_kernel(Collide K, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    if (i < n) K.alive[i] = 1;
    K.chosen[i] = 0;
}
__global__ void cs_select_reset_kernel(Collide K, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !K.alive[i]) return;
    for (int k = 0; k < 4; k++) K.nodemin[K.sorted[i].nodes[k]] = 0x7fffffff;
}
__global__ void cs_select_min_kernel(Collide K, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !K.alive[i]) return;
    for (int k = 0; k < 4; k++) atomicMin(&K.nodemin[K.sorted[i].nodes[k]], i);
}
__global__ void cs_select_choose_kernel(Collide K, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !K.alive[i]) return;
    const ImpactRec& r = K.sorted[i];
    bool first = true;
    for (int k = 0; k < 4; k++) first &= K.nodemin[r.nodes[k]] == i;
    if (!first) return;
    K.chosen[i] = 1;
    K.alive[i] = 0;
    for (int k = 0; k < 4; k++) K.used[r.nodes[k]] = 1;
}
__global__ void cs_select_drop_kernel(Collide K, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !K.alive[i]) return;
    const ImpactRec& r = K.sorted[i];
    bool hit = false;
    for (int k = 0; k < 4; k++) hit |= K.used[r.nodes[k]] != 0;
    if (hit) K.alive[i] = 0;
    else atomicAdd(&K.counters[1], 1);  // still live: another round
}
// The chosen impacts (exclusive offsets in chosen) appended in order; the node flags cleared.
__global__ void cs_select_write_kernel(Collide K, int n, int base, int cap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ImpactRec& r = K.sorted[i];
    if (K.chosen[i + 1] > K.chosen[i] && base + K.chosen[i] < cap) K.all[base + K.chosen[i]] = r;
    for (int k = 0; k < 4; k++) K.used[r.nodes[k]] = 0;
}

// The projection's nodes: marked, then (after an exclusive scan of mark) listed ascending.
__global__ void cs_opt_mark_kernel(Collide K, int nc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * nc) return;
    K.mark[K.all[t >> 2].nodes[t & 3]] = 1;
}
__global__ void cs_opt_nodes_kernel(Collide K, int N) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    if (K.mark[i + 1] > K.mark[i]) K.nodes[K.mark[i]] = i;
}
__global__ void cs_opt_idx_kernel(Collide K, int nc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * nc) return;
    const int slot = K.mark[K.all[t >> 2].nodes[t & 3]];
    K.idx[t] = slot;
    atomicAdd(&K.nptr[slot], 1);
}
__global__ void cs_opt_fill_kernel(Collide K, int nc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * nc) return;
    const int slot = K.idx[t];
    K.nlist[K.nptr[slot] + atomicAdd(&K.nfill[slot], 1)] = t;
}
__global__ void cs_opt_sort_kernel(Collide K, int nn) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nn) return;
    const int q0 = K.nptr[s], q1 = K.nptr[s + 1];
    for (int q = q0 + 1; q < q1; q++) {
        const int v = K.nlist[q];
        int r = q - 1;
        while (r >= q0 && K.nlist[r] > v) {
            K.nlist[r + 1] = K.nlist[r];
            r--;
        }
        K.nlist[r + 1] = v;
    }
}

namespace {
constexpr float kMu = 1e3f;          // Optimization::solve (Optimization.cu:96)
constexpr float kEpsS = 1e-12f;      // Optimization.cuh:16
constexpr float kEpsF = 1e-10f;      // Optimization.cuh:17
constexpr int kMaxOptIterations = 100;

constexpr int kOptThreads = CS_OPT_THREADS, kOptMaxCtas = 16;
constexpr int kPer = CS_OPT_STAGE / kOptThreads;  // consecutive terms of an ordered sum per thread at most
constexpr int kSat = 1 << 26;                     // increments saturate above any crossing (2^24)

// Float sums acc + t0 + t1 + ... in that order, as one thread would add them, computed by a block.
// While acc stays in one binade (ulp U, acc = A U with 2^23 <= A < 2^24), adding t >= 0 rounds to
// A + q + r with t = (q + f) U: r = 1 for f > 1/2, 0 for f < 1/2, and for a tie (f = 1/2) whatever
// makes the result even.  So a run of terms acts on A as an integer increment that depends on A's
// parity alone, a pair of integers, and such pairs compose associatively.
struct SumFn {
    int c0, c1;  // increment for even and for odd A
};
struct SumEntry {
    int kind, thread;  // kind < 0: the thread's terms one by one; else a run in binade `kind`
    SumFn f;
};
struct OptShared {
    SumEntry list[kOptThreads];
    float wsum[kOptThreads / 32];
    int wcount[kOptThreads / 32];
    float2 result;
    float2 xch[2][kOptMaxCtas];  // per sending CTA: a sum and its node part, two buffers
};
__device__ __forceinline__ int float_binade(float x) { return max((int)(__float_as_uint(x) >> 23), 1); }
__device__ __forceinline__ SumFn sum_compose(SumFn a, SumFn b) {  // a, then b
    SumFn r;
    r.c0 = min(a.c0 + ((a.c0 & 1) ? b.c1 : b.c0), kSat);
    r.c1 = min(a.c1 + (((a.c1 + 1) & 1) ? b.c1 : b.c0), kSat);
    return r;
}
__device__ __forceinline__ SumFn sum_term(float t, int E) {
    const unsigned u = __float_as_uint(t);
    const int M = (u >> 23) ? (int)((u & 0x7fffffu) | 0x800000u) : (int)u;
    const int sh = float_binade(t) - E;
    if (M == 0 || sh < -24) return {0, 0};
    if (sh >= 0) {
        const int q = sh > 3 ? kSat : min(M << sh, kSat);
        return {q, q};
    }
    const int q = M >> -sh, rem = M & ((1 << -sh) - 1), half = 1 << (-sh - 1);
    const int up = q + (rem > half ? 1 : 0), tie = rem == half ? 1 : 0;
    return {up + (tie & (q & 1)), up + (tie & ((q + 1) & 1))};
}

// a1 = acc + stage[0] + ... + stage[m1 - 1] in order, then a2 = scale(a1) + stage[m1] + ... +
// stage[m1 + m2 - 1], scale(a) = 0.5 a invMass (all terms >= 0); every thread calls it and returns
// (a1, a2).  Thread t owns up to kPer consecutive terms of one of the two parts.  A plain parallel
// prefix sum tells which binade acc is in there; the terms of threads whose prefix stays clear of
// a binade's edge form runs (merged within the warp), the others (some 30 threads: acc crosses some
// ten edges) are added one by one.  Thread 0 walks the runs and the single terms in order.  A run
// that does not start and end in the binade it was computed for sends everything through plain
// addition.  A chain of dependent additions took 17 us for 8,000 terms on a B200.
__device__ float2 ordered_sums(OptShared& S, const float* stage, int m1, int m2, float acc, float invMass) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    int per = (m1 + m2 + kOptThreads - 1) / kOptThreads, T1 = per ? (m1 + per - 1) / per : 0;
    if (per && T1 + (m2 + per - 1) / per > kOptThreads) {
        per++;
        T1 = (m1 + per - 1) / per;
    }
    const bool second = t >= T1;
    auto range = [&](int th, int& i0, int& i1) {
        i0 = th < T1 ? th * per : m1 + (th - T1) * per;
        i1 = min(i0 + per, th < T1 ? m1 : m1 + m2);
    };
    int i0, i1;
    range(t, i0, i1);
    float v[kPer], ls = 0.0f;
#pragma unroll
    for (int k = 0; k < kPer; k++) v[k] = i0 + k < i1 ? stage[i0 + k] : 0.0f;
#pragma unroll
    for (int k = 0; k < kPer; k++) ls += v[k];
    // prefix sums within the part: the second part's start from the scaled first
    float incl = ls, head = second ? 0.0f : ls;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
        head += __shfl_xor_sync(0xffffffffu, head, o);
    }
    if (lane == 31) S.list[w] = {0, 0, {__float_as_int(incl), __float_as_int(head)}};
    __syncthreads();
    if (w == 0) {
        float a = __int_as_float(S.list[lane].f.c0), h = __int_as_float(S.list[lane].f.c1);
        const float self = a;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, a, o);
            if (lane >= o) a += u;
            h += __shfl_xor_sync(0xffffffffu, h, o);
        }
        S.wsum[lane] = a - self;
        if (lane == 0) S.result.x = h;
    }
    __syncthreads();
    const float first = acc + S.result.x;  // a1, about
    const float before = S.wsum[w] + (incl - ls);
    const float start = second ? 0.5f * first * invMass + fmaxf(before - S.result.x, 0.0f) : acc + before;
    const float lo = start * (1.0f - 1.0f / 4096), hi = (start + ls) * (1.0f + 1.0f / 4096);
    const int E = float_binade(lo);
    const bool none = ls == 0.0f;
    const bool single = !none && !(lo > 1e-30f && hi < 1e37f && E == float_binade(hi));
    SumFn f = {0, 0};
    if (!none && !single)
#pragma unroll
        for (int k = 0; k < kPer; k++)
            if (k < per) f = sum_compose(f, sum_term(v[k], E));
    // the warp's runs, composed onto a run's last lane; a run ends at a single thread and at the
    // first part's end
    const unsigned ms = __ballot_sync(0xffffffffu, single), m2nd = __ballot_sync(0xffffffffu, second);
    const unsigned heads = (ms << 1) | (m2nd & ~(m2nd << 1)) | 1u;  // lanes that start a run
    const int begin = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    int Er = none || single ? -1 : E;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        SumFn p;
        p.c0 = __shfl_up_sync(0xffffffffu, f.c0, o);
        p.c1 = __shfl_up_sync(0xffffffffu, f.c1, o);
        const int Ep = __shfl_up_sync(0xffffffffu, Er, o);
        if (lane - o >= begin && !single) {
            f = sum_compose(p, f);
            // one binade per run (-1: nothing yet; 0: two different ones, refused by the walk)
            Er = Er == -1 ? Ep : (Ep == -1 || Ep == Er ? Er : 0);
        }
    }
    const bool ends = lane == 31 || ((ms | heads) >> (lane + 1) & 1u);
    const bool emit = single || (Er != -1 && ends);
    const unsigned me = __ballot_sync(0xffffffffu, emit);
    if (lane == 0) S.wcount[w] = __popc(me);
    __syncthreads();
    const int mine = S.wcount[lane];
    int cum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, cum, o);
        if (lane >= o) cum += u;
    }
    const int total = __shfl_sync(0xffffffffu, cum, 31), pos = __shfl_sync(0xffffffffu, cum - mine, w);
    if (emit) S.list[pos + __popc(me & ((1u << lane) - 1u))] = {single ? -1 : Er, t, f};
    __syncthreads();
    if (t == 0) {
        float a = acc, a1 = acc;
        bool ok = true, scaled = m2 == 0;
        SumEntry e = total > 0 ? S.list[0] : SumEntry{};
        for (int k = 0; k < total; k++) {
            const SumEntry nx = S.list[min(k + 1, total - 1)];
            if (!scaled && e.thread >= T1) {
                a1 = a;
                a = 0.5f * a * invMass;
                scaled = true;
            }
            if (e.kind < 0) {
                int j0, j1;
                range(e.thread, j0, j1);
                float u[kPer];
#pragma unroll
                for (int j = 0; j < kPer; j++) u[j] = j0 + j < j1 ? stage[j0 + j] : 0.0f;
#pragma unroll
                for (int j = 0; j < kPer; j++) a += u[j];  // + 0 leaves a (>= +0) as it is
            } else {
                const unsigned b = __float_as_uint(a);
                int A = (int)((b & 0x7fffffu) | 0x800000u);
                A += (A & 1) ? e.f.c1 : e.f.c0;
                ok &= (int)(b >> 23) == e.kind && A < (1 << 24);
                a = __uint_as_float(((unsigned)e.kind << 23) + (unsigned)(A - (1 << 23)));
            }
            e = nx;
        }
        if (!scaled || m2 == 0) a1 = a;
        if (!scaled) a = 0.5f * a * invMass;  // the second part holds zeros only
        if (!ok) {
            a = acc;
            for (int j = 0; j < m1; j++) a += stage[j];
            a1 = a;
            if (m2 > 0) {
                a = 0.5f * a * invMass;
                for (int j = m1; j < m1 + m2; j++) a += stage[j];
            }
        }
        S.result = make_float2(a1, a);
    }
    __syncthreads();
    const float2 r = S.result;
    __syncthreads();
    return r;
}

// acc + term(0) + ... + term(n - 1) in that order (the CPU loop's).
template <class Term>
__device__ float ordered_sum(OptShared& S, float* stage, int n, float acc, Term term) {
    for (int base = 0; base < n; base += CS_OPT_STAGE) {
        const int m = min(CS_OPT_STAGE, n - base);
#pragma unroll 4
        for (int i = threadIdx.x; i < m; i += kOptThreads) stage[i] = term(base + i);
        __syncthreads();
        acc = ordered_sums(S, stage, m, 0, acc, 0.0f).x;
    }
    return acc;
}
// (a, b): a = 0.5 invMass (first(0) + ... + first(n1 - 1)), b = a + second(0) + ... + second(n2 - 1)
template <class First, class Second>
__device__ float2 ordered_value(OptShared& S, float* stage, int n1, int n2, float invMass, First first, Second second) {
    if (n1 + n2 > CS_OPT_STAGE - kOptThreads) {
        const float a = 0.5f * ordered_sum(S, stage, n1, 0.0f, first) * invMass;
        return make_float2(a, ordered_sum(S, stage, n2, a, second));
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < n1; i += kOptThreads) stage[i] = first(i);
#pragma unroll 2
    for (int i = threadIdx.x; i < n2; i += kOptThreads) stage[n1 + i] = second(i);
    __syncthreads();
    const float2 r = ordered_sums(S, stage, n1, n2, 0.0f, invMass);
    return make_float2(0.5f * r.x * invMass, n2 > 0 ? r.y : 0.5f * r.x * invMass);
}

__device__ __forceinline__ f3 xyz(float4 v) { return mk(v.x, v.y, v.z); }

// CollisionOptimization::constraint (CollisionOptimization.cu:91-103) at the positions x(slot);
// con[3 c ..]: the four slots, the four weights, the normal
template <class X>
__device__ __forceinline__ float constraint(const float4* con, int c, float thickness, X x) {
    const float4 id = con[3 * (size_t)c], wt = con[3 * (size_t)c + 1];
    const f3 n = xyz(con[3 * (size_t)c + 2]);
    const int i[4] = {__float_as_int(id.x), __float_as_int(id.y), __float_as_int(id.z), __float_as_int(id.w)};
    const float wk[4] = {wt.x, wt.y, wt.z, wt.w};
    f3 p[4];
#pragma unroll
    for (int k = 0; k < 4; k++) p[k] = x(i[k]);
    float a = -thickness;
#pragma unroll
    for (int k = 0; k < 4; k++) a += wk[k] * dot0(n, p[k]);
    return a;
}
}  // namespace

// One cluster: Optimization::solve (Optimization.cu:94-137) of CollisionOptimization over the
// accumulated impacts; the result is written back into B.x.  Element terms are spread over the
// cluster, every sum has the CPU loop's order and rounding.  An iteration has two phases with a
// cluster barrier after each:
//   1  per node: the iteration's position (the last one moved by the accepted step) and the gradient
//      (valueAndGradient, Optimization.cu:51-63), each of its constraints evaluated in place; per
//      constraint: the multiplier's update (updateMultiplier, Optimization.cu:85-92) and its term
//      of the value;
//   2  the sums, each by one CTA: rank 0 the value, rank 1 the gradient's square, and each further
//      rank the value at one step length of the backtracking line search, which tries s, 0.7 s,
//      0.49 s, ... until one passes: the first that does is the one the CPU loop takes.
// What bounds it: the latency of the two phases' loads (L2) and of the ordered sums.  By one CTA,
// one trial and one chain of additions at a time, it took 12.2 ms for 4,774 nodes and 3,300
// constraints on a B200 (100 iterations, the first with 26 trials); now 3.9 ms.
__global__ void __launch_bounds__(kOptThreads, 1) cs_opt_kernel(Batch B, Collide K, int nn, int nc) {
    __shared__ OptShared S;
    extern __shared__ float cs_opt_stage[];
    float* const stage = cs_opt_stage;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks(), trials = ncta - 2;
    const int gid = rank * kOptThreads + threadIdx.x, G = ncta * kOptThreads;
    float4 *cur = K.cur, *next = K.next, *grad = K.grad, *gnext = K.grad2;
    float *lam = K.lambda, *lnext = K.lambda2;
    // per slot the position when the collision step began and the mass; per constraint its slots,
    // weights and normal, contiguous
    for (int i = gid; i < nn; i += G) {
        const int node = K.nodes[i];
        const f3 x = ld(B.x, node), x1 = ld(K.x1, node);
        cur[i] = make_float4(x.x, x.y, x.z, 0.0f);
        K.home[i] = make_float4(x1.x, x1.y, x1.z, B.mass[node]);
    }
    for (int c = gid; c < nc; c += G) {
        const ImpactRec& r = K.all[c];
        K.con[3 * (size_t)c] = make_float4(__int_as_float(K.idx[4 * c]), __int_as_float(K.idx[4 * c + 1]),
                                           __int_as_float(K.idx[4 * c + 2]), __int_as_float(K.idx[4 * c + 3]));
        K.con[3 * (size_t)c + 1] = make_float4(r.w[0], r.w[1], r.w[2], r.w[3]);
        K.con[3 * (size_t)c + 2] = make_float4(r.n[0], r.n[1], r.n[2], 0.0f);
        lam[c] = 0.0f;
    }
    // CollisionOptimization.cu:22-35: the mean inverse mass
    const float invMass = ordered_sum(S, stage, nn, 0.0f, [&](int i) { return 1.0f / B.mass[K.nodes[i]]; }) / (float)nn;
    float ss = 1e-3f * (float)nn;
    float sacc = 0.0f;     // the accepted step from cur along grad that gives the iteration's positions
    float nodeSum = 0.0f;  // the value's node part there, already summed by the accepted trial
    bool moved = false;    // the result is one accepted step beyond cur
    int nx = 0;
    // every CTA's (value, node part) to every CTA; returns after a cluster barrier
    auto exchange = [&](float a, float b) {
        if (threadIdx.x < ncta) *cl.map_shared_rank(&S.xch[nx & 1][rank], threadIdx.x) = make_float2(a, b);
        cl.sync();
        return S.xch[nx++ & 1];
    };
    cl.sync();
    for (int iter = 0; iter < kMaxOptIterations; iter++) {
        const bool first = iter == 0;
        auto here = [&](int i) {
            const f3 x = xyz(__ldcg(cur + i));
            return first ? x : sub(x, scl(sacc, xyz(__ldcg(grad + i))));
        };
        // the clamped violation (clampViolation(x, +1)) and the updated multiplier
        auto violation = [&](int c, float& l) {
            const float a = constraint(K.con, c, K.thickness, here);
            l = __ldcg(lam + c);
            if (!first) l = mn(l + kMu * a, 0.0f);
            return mn(a + l / kMu, 0.0f);
        };
        for (int t = gid; t < nn + nc; t += G) {
            if (t >= nn) {
                const int c = t - nn;
                float l;
                const float co = violation(c, l);
                lnext[c] = l;
                // skipped terms (coefficient 0) enter the value as +0: the running sum is >= +0, so
                // adding +0 leaves it unchanged, bit for bit
                K.cterm[c] = co != 0.0f ? 0.5f * kMu * (co * co) : 0.0f;
                continue;
            }
            const float4 hm = K.home[t];
            const f3 x = here(t);
            f3 g = scl(invMass * hm.w, sub(x, xyz(hm)));
            const int q1 = K.nptr[t + 1];
#pragma unroll 2
            for (int q = K.nptr[t]; q < q1; q++) {
                const int c = K.nlist[q] >> 2, k = K.nlist[q] & 3;
                float l;
                const float co = violation(c, l);
                const float4 wt = K.con[3 * (size_t)c + 1];
                const float wk = k == 0 ? wt.x : k == 1 ? wt.y : k == 2 ? wt.z : wt.w;
                if (co != 0.0f) g = add(g, scl((kMu * co) * wk, xyz(K.con[3 * (size_t)c + 2])));
            }
            next[t] = make_float4(x.x, x.y, x.z, 0.0f);
            gnext[t] = make_float4(g.x, g.y, g.z, dot0(g, g));
        }
        cl.sync();
        {
            float4* a = cur;
            cur = next;
            next = a;
            a = grad;
            grad = gnext;
            gnext = a;
            float* l = lam;
            lam = lnext;
            lnext = l;
        }
        // Optimization::value (Optimization.cu:24-35) at cur, or a step s along the gradient from it:
        // (the objective's scaled sum, with the constraints' terms)
        auto node_term = [&](int i, float s, bool step) {
            const f3 x = xyz(__ldcg(cur + i));
            const float4 hm = K.home[i];
            const f3 d = sub(step ? sub(x, scl(s, xyz(__ldcg(grad + i)))) : x, xyz(hm));
            return hm.w * dot0(d, d);
        };
        float f = 0.0f, g2 = 0.0f, ft = 0.0f, ftNode = 0.0f;
        ss /= 0.7f;
        ss *= 0.7f;
        bool stop = false;
        for (int batch = 0; !stop; batch++) {
            if (batch > 0) ss *= 0.7f;
            float2 mine = make_float2(0.0f, 0.0f);
            if (rank == 0) {
                auto cterm = [&](int c) { return __ldcg(K.cterm + c); };
                if (batch == 0 && first)
                    mine = ordered_value(S, stage, nn, nc, invMass, [&](int i) { return node_term(i, 0.0f, false); }, cterm);
                else if (batch == 0) mine = make_float2(nodeSum, ordered_sum(S, stage, nc, nodeSum, cterm));
            } else if (rank == 1) {
                if (batch == 0) mine.y = ordered_sum(S, stage, nn, 0.0f, [&](int i) { return __ldcg(grad + i).w; });
            } else {
                float s = ss;
                for (int k = 2; k < rank; k++) s *= 0.7f;
                mine = ordered_value(S, stage, nn, nc, invMass, [&](int i) { return node_term(i, s, true); }, [&](int c) {
                    const float a = constraint(K.con, c, K.thickness, [&](int i) {
                        return sub(xyz(__ldcg(cur + i)), scl(s, xyz(__ldcg(grad + i))));
                    });
                    const float co = mn(a + __ldcg(lam + c) / kMu, 0.0f);
                    return co != 0.0f ? 0.5f * kMu * (co * co) : 0.0f;
                });
            }
            const float2* x = exchange(mine.x, mine.y);
            if (batch == 0) {
                f = x[0].y;
                g2 = x[1].y;
            }
            for (int k = 0; k < trials && !stop; k++) {
                if (k > 0) ss *= 0.7f;
                ft = x[2 + k].y;
                ftNode = x[2 + k].x;
                stop = !(ft >= f - 0.5f * ss * g2 && ss >= kEpsS && ab(f - ft) >= kEpsF);
            }
        }
        moved = !(ss < kEpsS || ab(f - ft) < kEpsF);
        if (!moved) break;
        sacc = ss;
        nodeSum = ftNode;
    }
    for (int i = gid; i < nn; i += G) {
        const f3 x = xyz(__ldcg(cur + i));
        st(B.x, K.nodes[i], moved ? sub(x, scl(sacc, xyz(__ldcg(grad + i)))) : x);
    }
    cl.sync();  // no CTA leaves while another may still write into its shared memory
}

// Mesh::updateVelocities (Mesh.cu:238-247): v = (x - x0) * (1 / dt)
__global__ void cs_collide_velocity_kernel(Batch B, float invDt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * B.N) return;
    B.v[i] = (B.x[i] - B.x0[i]) * invDt;
}
