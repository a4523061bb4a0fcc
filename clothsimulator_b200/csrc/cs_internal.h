// Internal data layout of the B200 implicit cloth step.  Not part of the C ABI.
//
// HBM layout (one batch of independent sheets = "instances"):
//   nodes   : x, v, dv as 3N floats (xyz interleaved), mass N, handle float4 N (xyz target,
//             w = handle count), FP64 solution accumulator dv64 3N.
//   faces   : int4 {n0, n1, n2, sheet} (global node ids), float4 inverse rest matrix
//             (Face::inverse, Face.cu:16), rest area.
//   edges   : interior edges only (the reference skips boundary edges, Cloth.cu:142):
//             int4 {n0, n1, opposite0, opposite1}, int meta (face-vertex rotations), sheet,
//             float4 {area0 + area1, bias weight side 0, side 1, 0}; per step a 64-byte
//             record of its bending geometry (dtheta, coefficient, theta).
//   system  : SELL-32 block layout.  A sheet's rows (nodes), sorted by block count within
//             windows of sigma rows (sigma chosen per topology to minimise padding), are cut
//             into slices of 32; slice s has `width` block slots per row (padded with zero
//             blocks).  Slot (slice, k, lane) stores its 3x3 block in a "panel" of 32 lanes:
//             entries 0-3 as float4[32], entries 4-7 as float4[32], entry 8 as float[32]
//             (1152 bytes per panel, 128-bit coalesced loads).  Slot k = 0 is the diagonal.
//             Column indices and the assembly's row lists are per *topology* (shared by all
//             sheets with identical connectivity) and hold sheet-local ids.
#ifndef CLOTHSTEP_CS_INTERNAL_H
#define CLOTHSTEP_CS_INTERNAL_H

#include <cuda_runtime.h>
#include <stdint.h>

#include "clothstep.h"

#define CS_SLICE 32
#define CS_PANEL_FLOATS 288  // 32 lanes x 9 entries
#define CS_TABLE_N 30
#define CS_TABLE_ENTRIES (CS_TABLE_N * CS_TABLE_N * CS_TABLE_N)
// Contributor code: bit 31 = edge (1) / face (0); bits 4..30 = sheet-local element id;
// bits 2..3 = local row corner a; bits 0..1 = local column corner b.
#define CS_CODE_EDGE 0x80000000u
__host__ __device__ inline uint32_t cs_code(int is_edge, int elem, int a, int b) {
    return (is_edge ? CS_CODE_EDGE : 0u) | ((uint32_t)elem << 4) | ((uint32_t)a << 2) | (uint32_t)b;
}
// Threads per CTA of the assembly gather (forces.cu) at most; its slot accumulators take
// gather_width x 1152 bytes of shared memory per warp, and a batch whose widest slice would not
// fit four warps in a CTA's shared memory gets fewer.  (One-warp CTAs, 15 warps per SM instead
// of 12, measured slower on the windy batch: 3.82 against 3.35 ms.)
#define CS_GATHER_THREADS 128
// Rows (threads) per block of the proximity row kernel: a warp's, fewer where the blocks and columns of that
// many rows of `width` blocks exceed the shared memory of a block (from 182 blocks a row; the gather
// takes up to 201); and that shared memory.
#define CS_PROX_ROW_THREADS 32
inline size_t cs_prox_row_smem(int width, int rows) { return (size_t)width * 10 * rows * sizeof(float); }
inline int cs_prox_rows(int width, size_t smem) {
    const size_t rows = smem / cs_prox_row_smem(width > 0 ? width : 1, 1);
    return rows < CS_PROX_ROW_THREADS ? (int)rows : CS_PROX_ROW_THREADS;
}

struct SheetDesc {
    int node_off, n_nodes;
    int face_off, n_faces;
    int edge_off, n_edges;      // interior edges
    int slice_off, n_slices;    // global slices
    int topo;                   // shared topology id
    int table;                  // stretching table id
    float bending[15];          // scaled bending samples, 3x5 (Material.cu:38-40)
    float wind_density, wind_drag, wind_v[3];
    int nbr_ptr_off, nbr_off;   // this sheet's topology in the one-ring neighbour arrays
    int row2slot_off;           // this sheet's topology in the row -> slot map
    int resident;               // 1: solved by the cluster-resident kernel (resident.cu), 2: by a
                                // group of CTAs (group.cu)
    int csr_ptr_off;            // this sheet's topology in tcsr_ptr (block CSR for slot lookups)
    int panel_off;              // first value panel: global slot = panel_off * 32 + topology slot
    // coarse space of the batched loop: this sheet's topology in the aggregate arrays, its
    // aggregates, its coarse unknowns' offset in the per-sheet vectors and its matrices' offset
    int bc_node_off, bc_agg_off, bc_pair_off, bc_npair, bc_na, bc_vec_off;
    // the finer cells: the topology's middle and fine cells in their pointer arrays, the middle cells'
    // number, this sheet's offset among the middle and the fine cells of all sheets; levels in use
    // (bit 0: fine, bit 1: middle)
    int bc_mid_off, bc_fine_off, bc_nmid, bc_mvec_off, bc_fvec_off, bc_levels;
    long long bc_mat_off;
};

struct SliceDesc {
    int sheet;
    int topo_slice;  // index into the per-topology slice arrays
    int row0;        // the sheet's first node; lane l holds row row0 + rowmap[topo_slice * 32 + l]
    int rows;        // rows in this slice (<= 32)
    int width;       // block slots per row
    int panel0;      // first global value panel
    int tpanel0;     // first per-topology panel (columns, contributor lists)
    int keep;        // block slots that the on-chip solvers hold in shared memory (panels.h)
};

// Solver phases of one instance (one sheet's system) inside the batched loop.
enum InstPhase : int {
    PH_CG = 0,        // one preconditioned CG iteration on the FP32 correction system
    PH_RES = 1,       // FP64 residual b - A (dv64 + e) and its norm
    PH_INIT = 2,      // start a CG sweep: dv64 += e, e = 0, z = P r, p = z (or, continuing after a
                      // reliable update, p = z + beta p with the FP64 residual in r)
    PH_FINISH = 3,    // dv64 += e, then done
    PH_DONE = 4,
    PH_RESIDENT = 5,  // owned by the cluster-resident kernel this step (skipped by the loop)
    PH_SCALE = 6,     // dv64 *= wscale (the warm start's Galerkin multiple), then PH_RES
};

// Cluster-resident solver limits: CTAs per cluster, warps (slices) per CTA, block slots per
// row (the SpMV over a row is fully unrolled to this width; column codes live in registers).
#define CS_RES_MAX_CL 16
#define CS_RES_MAX_WARPS 16
#define CS_RES_MAX_WIDTH 16
// Reliable updates keep the search direction only while the recursive residual has drifted
// from the FP64 one by at most this fraction of the latter (larger drift: restart).
#define CS_RELIABLE_DRIFT 0.1
#define CS_LAST_SWEEP 0.3  // on-chip solvers beyond block-Jacobi: recursive residual that ends the last sweep, of the tolerance
// power iterations per sheet solve for the tile-local Chebyshev bound
#define CS_CHEB_POWER_ITERS 10
// A sheet uses the tile-local Chebyshev preconditioner only if at least this share of its
// blocks couple rows of one CTA.  Small sheets split into thin strips do better with
// block-Jacobi; measured on the B200 (hanging and windy sheets in strips, tol 1e-6): 24x24 (0.54 of the
// blocks strip-local) and 28x28 (0.59) need fewer or as many iterations with block-Jacobi, 32x32
// (0.71), 40x40 (0.65), 48x48 (0.84) and 64x64 (0.89) fewer with the Chebyshev polynomial.
#define CS_CHEB_MIN_LOCAL 0.62
// Coarse-space correction of the cluster-resident solver: each CTA's tile of rows is cut into K
// segments of whole slices, K = min(CS_COARSE_SEGS, CS_COARSE_AGGS / CTAs per cluster), and the coarse
// space holds one constant per (segment, component): at most 64 unknowns, two per lane of a warp.  With
// the levels below it (levels.cuh) more segments save little: 1, 2, 3 or 6 take 82, 76, 77 or 76
// iterations on a 64 x 64 sheet.
// threads of the per-instance reduction kernels of the batched loop
#define CS_REDUCE_THREADS 256
// coarse-space correction of the batched loop (coarse.cu): a sheet's nodes binned by their rest
// (u, v) into g x g cells (g = round(sqrt(nodes / CS_BC_NODES_PER_AGG)), 1..CS_BC_MAX_G), the
// non-empty cells its aggregates; coarse systems up to CS_BC_SMALL_NC unknowns are inverted by
// one CTA in shared memory, larger ones by a cluster of CS_BC_CLUSTER CTAs
#define CS_BC_NODES_PER_AGG 256
#define CS_BC_MAX_G 16
// Sheets up to this size take at most 8 x 8 cells.  Steps with at most 8 x 8 / 16 x 16 (B200, tol 1e-6): an
// irregular sheet of 301 x 301 nodes 5.9 / 7.1 ms, 401 x 401 9.5 / 13.7, 501 x 501 13.8 / 13.8, 601 x 601
// 19.8 / 19.9, 801 x 801 39.3 / 32.3, 1,001 x 1,001 62 / 51; at tol 1e-8, where the iterations are many,
// a sheet of 301 x 301 18.6 / 19.8 and of 451 x 451 52 / 41.
#define CS_BC_BIG_NODES (1 << 18)
// the finer grids' cells (coarse.cu): nodes of a fine cell, fine cells along the side of a middle one.  Steps
// with 15, 30, 60 nodes (B200, tol 1e-6): irregular 301 x 301 nodes 5.3, 5.9, 8.5 ms, 401 x 401 10.2, 9.5, 11.7,
// 501 x 501 14.4, 13.8, 16.1, 1,001 x 1,001 50.3, 50.7, 65.9, 60 sheets of 64 x 64 in the loop 11.3, 10.8,
// 12.0 (a precision sheet of 601 x 601 at 1e-8 77, 96, 128); with a split of 2, 4, 6: 301 x 301 5.1, 5.9, 9.3,
// 401 x 401 10.5, 9.5, 11.4, 501 x 501 14.8, 13.8, 16.9, 1,001 x 1,001 54, 51, 55 (601 x 601 73, 96, 108).
#define CS_BC_NODES_PER_FINE 30
#define CS_BC_FINE_SPLIT 4
#define CS_BC_RESTRICT_THREADS 512
#define CS_BC_APPLY_THREADS 128
#define CS_BC_UNROLL 4
#define CS_BC_MAX_NC (3 * CS_BC_MAX_G * CS_BC_MAX_G)
#define CS_BC_SMALL_NC 192
#define CS_BC_CLUSTER 16
#define CS_BC_THREADS 512
// Gauss-Jordan pivot blocks of the coarse inversion: CS_BC_PB aggregates, CS_BC_KB rows
#define CS_BC_PB 4
#define CS_BC_KB (3 * CS_BC_PB)
#define CS_COARSE_MAX_K 8
#define CS_COARSE_SEGS 2
#define CS_COARSE_AGGS 21
// Slices per CTA from which the cluster solver takes the coarse correction.  A step without / with it (B200, tol
// 1e-6): one sheet of 32 x 32 quads (3.5 slices) 0.36 / 0.47 ms, of 40 x 40 (5.3) 0.42 / 0.50, of 48 x 48 (7.6)
// 0.50 / 0.57, where a lone sheet waits for the set-up; 90 sheets of 32 x 32 1.27 / 1.45, of 40 x 40
// 2.02 / 1.99, of 48 x 48 3.15 / 3.05, where it runs beside others.
#define CS_COARSE_MIN_SLICES 5
// Threads of the per-sheet set-up kernel that forms and inverts the coarse matrix, and its
// dynamic shared memory: the nc x nc matrix with rows padded to 16 bytes, then one pivot block.
#define CS_COARSE_THREADS 512
__host__ __device__ inline int cs_coarse_ld(int nc) { return (nc + 3) & ~3; }
__host__ __device__ inline size_t cs_coarse_setup_smem(int nc) {
    return ((size_t)nc * cs_coarse_ld(nc) + CS_BC_KB * CS_BC_KB) * sizeof(float);
}
// Launch shapes of the batched SpMV that cs_tune times (pcg.cu, kSpmvShapes): threads per block,
// slices per warp, block slots whose loads are issued together.
struct SpmvShape {
    int threads, spw, unroll;
};
#define CS_SPMV_CANDIDATES 24
// 64 threads, one slice per warp, four slots' loads issued together: at the sizes where the loop is
// bound by the latency of a row's loads one slot at a time costs most (128 threads, no unrolling: 26 us
// for a sheet of 66,049 nodes in L2), and the large ones stream as fast
#define CS_SPMV_DEFAULT 12
struct Batch;
extern const SpmvShape kSpmvShapes[CS_SPMV_CANDIDATES];
void launchSpmvShape(const Batch& B, int shape, cudaStream_t st);
// Group-resident solver (group.cu): block slots per row (column codes live in registers), slices
// per CTA that a sheet's tiles are planned for, its fewest when a batch would leave the chip idle.
#define CS_GROUP_MAX_WIDTH 18
#define CS_GROUP_SLICES 14
#define CS_GROUP_MAX_WARPS CS_RES_MAX_WARPS
#define CS_GROUP_CE_PARTS 4    // warps that share a row of the coarse matrix-vector product, at most
#define CS_GROUP_MIN_SLICES 8
// coarse unknowns up to which a group's segments are cut finer than one per CTA
#define CS_GROUP_NC 192
#define CS_SOLVER_AUTO_DEV 0
#define CS_SOLVER_BATCHED_DEV 1

// Instance flags
#define CS_IF_CONVERGED 1
#define CS_IF_WARM_REJECTED 2
#define CS_IF_BREAKDOWN 4
#define CS_IF_CAPPED 8

struct InstState {
    double bnorm2;      // ||b||^2 (FP64)
    double rz;          // r.z of the current iteration
    double rz_prev;     // r.z of the iteration before (a reliable update's beta)
    double pq;
    double rr;          // ||r||^2 of the recursive residual
    double res0;        // FP64 true residual norm at the start of the current sweep
    double resnorm;     // last FP64 true residual norm
    double first_res;   // FP64 residual of the initial guess
    float alpha, beta;
    int phase;
    int sweep_iters;
    int iters;          // total CG iterations this step
    int sweeps;         // FP64 residual evaluations this step
    int flags;
    int cont;           // the next PH_INIT keeps the search direction (reliable update)
    double wscale;      // Galerkin multiple of the warm start (warm_scale)
    int scaled;         // the warm start's scaling pass is done
    int pad;
};

// Step parameters in device memory (read by every kernel of the captured step graph).
struct DevParams {
    float dt;
    float gravity[3];
    float handle_stiffness;
    double tol;            // FP64-checked relative residual target
    double inner_tol;      // mixed precision: residual reduction between FP64 residual replacements
    int max_iters;         // CG iterations per instance per step
    int sweep_cap;         // CG iterations per sweep
    int mixed;             // 1: FP32 CG + FP64 refinement; 0: plain FP32 CG (FP32 dots)
    int warm;              // 0 zero guess, 1 warm start from dv64 as preloaded
    int loop_cap;          // hard bound on loop trips per step
    int advance;           // 1: v += dv, x += dt v at the end of the step
    int warm_scale;        // 1: the warm start replaced by its Galerkin multiple before the guard
    int solver;            // CS_SOLVER_AUTO_DEV: resident sheets on the cluster kernel; BATCHED: loop only
    int cheb_degree;       // resident solver: 1 block-Jacobi; odd >= 3 levels, or tile-local Chebyshev of that degree without `coarse`
    int coarse;            // resident solver with the Chebyshev preconditioner: 1 adds the coarse-space correction
    int n_motions;         // transformations of this step (cs_step_params.transformations)
    float motion[CS_MAX_MOTIONS][CS_TRANSFORM_FLOATS];
};

// One proximity as seen by one sheet it touches (cs_set_proximities): node[i] is a batch
// node or -1; bit i of `local` marks the nodes of this sheet (their rows and columns get
// blocks); other points enter through their state only.
struct ProxInst {
    int node[4];
    int local, free_mask, sheet;
    float thickness;
    float n[3], w[4], mu, stiffness;
    float xe[4][3], ve[4][3], me[4];  // points outside the batch (node -1)
};

// Per-instance record written by cs_prox_kernel: -dt^2 J of the impulse (12x12), -dt J of
// the friction (12x12), the impulse right-hand side dt (f + dt J v) (12), the friction one dt f.
#define CS_PROX_REC 312

// One sheet of the group-resident solver: its CTAs cta0 .. cta0 + ctas - 1, segments per CTA of its
// coarse space, and where its packets, reduction packets, published-row marks, halo lists and
// inverse coarse matrix (-1: none) start.
struct GroupItem {
    int sheet, cta0, ctas, segs;
    int slot0, red0, pub0, halo0;
    long long mat;
};

struct Batch {
    int N = 0, F = 0, E = 0, S = 0;
    // coarse-space correction of the batched loop (coarse.cu)
    int bc_total_agg = 0;        // aggregates of all sheets (the per-aggregate kernels' work list)
    int bc_max_npair = 0;        // largest coarse pair count of a sheet
    int bc_n_big = 0;            // sheets whose coarse system exceeds CS_BC_SMALL_NC
    int2* bc_agg = nullptr;      // per global aggregate: (sheet, local aggregate)
    int* bc_big = nullptr;       // the sheets inverted by a cluster
    int* bc_node_fine = nullptr; // per topology node: its fine cell
    int* bc_aptr = nullptr;      // per topology aggregate: its middle cells (na + 1 per topology)
    int* bc_fptr = nullptr;      // per topology middle cell: its fine cells (one more per topology)
    int* bc_mptr = nullptr;      // per topology fine cell: its nodes in bc_mem (one more per topology)
    int* bc_mem = nullptr;       // per topology: the nodes by fine cell, ascending
    float* bc_finv = nullptr;    // per sheet fine cell: its diagonal block's inverse (9)
    float* bc_minv = nullptr;    // the same of the middle cells
    float* bc_ef = nullptr;      // per sheet fine cell: its correction, then the sum of all levels' (3)
    float* bc_em = nullptr;      // per sheet middle cell: its correction (3)
    int bc_max_nmid = 0;         // largest number of middle cells of a sheet
    int bc_warps = 1;            // warps per block of the restriction: middle cells of an aggregate, at most 16
    int4* bc_pair = nullptr;     // per topology coarse pair: (a, b, contributor begin, end)
    int* bc_contrib = nullptr;   // topology slots (panel * 32 + lane) of the stored blocks of each pair
    float* bc_mat = nullptr;     // per sheet nc x nc: the coarse matrix R A R^T (then GJ's work)
    float* bc_inv = nullptr;     // per sheet nc x nc: its inverse, symmetrised
    float* bc_rc = nullptr;      // per sheet nc: R r
    int* bc_ok = nullptr;        // per sheet: the coarse inverse of this step is valid
    int n_slices = 0, n_panels = 0, n_tpanels = 0, n_tables = 0;
    // nodes
    float *x = nullptr, *v = nullptr, *dv = nullptr, *mass = nullptr;
    float* x0 = nullptr;     // positions at the start of the last step (Node::x0, Mesh.cu:226-231)
    float4* handle = nullptr;
    int* handle_motion = nullptr;  // per node: the motion of its handle (-1: fixed)
    double* dv64 = nullptr;
    float* warm = nullptr;   // warm-start vector (previous dv or learned prediction)
    // faces
    int4* face_nodes = nullptr;
    float4* face_inv = nullptr;
    float* face_area = nullptr;
    // edges
    int4* edge_nodes = nullptr;
    int* edge_meta = nullptr;
    int* edge_sheet = nullptr;
    float4* edge_par = nullptr;
    float4* edge_geo = nullptr;  // per step: 4 per edge, dtheta (12), coefficient, theta (cs_edge_kernel)
    // sheets, materials, topology
    SheetDesc* sheets = nullptr;
    float4* tables = nullptr;
    SliceDesc* slices = nullptr;
    int* tcol = nullptr;         // per topology panel: 32 local column ids
    // assembly row lists (forces.cu, cs_gather_kernel): per topology node (at row2slot_off),
    // its (face << 2 | corner, slots of the face's corners) in face order and its (interior
    // edge << 2 | corner, slots of the edge's four nodes) in edge order; slots 8 bits each
    int* rface_ptr = nullptr;    // topology nodes of all topologies + 1
    int2* rface = nullptr;
    int* redge_ptr = nullptr;
    int2* redge = nullptr;
    int gather_width = 0;        // widest slice of the batch (the gather's accumulators per lane)
    int* nbr_ptr = nullptr;      // per topology: one-ring neighbour CSR (sheet-local ids)
    int* nbr = nullptr;
    int* node_sheet = nullptr;   // sheet of every node
    int* rowmap = nullptr;       // per topology slice lane: sheet-local row
    uint32_t* rcell = nullptr;   // per topology slice lane of a tiled sheet: LevelPlace (levels.cuh)
    int* row2slot = nullptr;     // per topology row: slice * 32 + lane
    // system
    float* A = nullptr;          // n_panels * 288
    float* b = nullptr;          // 3N
    float* Pinv = nullptr;       // 9N
    // PCG
    float *e = nullptr, *r = nullptr, *z = nullptr, *pA = nullptr, *pB = nullptr, *q = nullptr;
    double* part = nullptr;      // 2 per slice
    InstState* inst = nullptr;
    DevParams* params = nullptr;
    // [0] loop trip counter, [1] instances not done, [2] a trip's finished blocks, [3] go on, [4] trips
    // since load, [5] resident work counter, [6] error word, [7] checksum (cs_tune), [8], [9] the solve
    // set-up's finished blocks and instances that the loop solves
    int* loop = nullptr;
    // cluster-resident solver (resident.cu)
    int n_resident = 0;          // sheets listed in rlist
    int res_cap = 0;             // panels per CTA held in shared memory
    int* rlist = nullptr;        // resident sheets, largest first
    int* rsplit = nullptr;       // per topology: CS_RES_MAX_CL + 1 sheet-relative slice bounds per CTA rank
    int* rcode = nullptr;        // per topology panel slot: index of its column in the reading CTA's p array
    int* rsendptr = nullptr;     // per topology: CS_RES_MAX_CL + 1 offsets into rsend per owner rank
    uint32_t* rsend = nullptr;   // halo sends: src slot | dst rank << 12 | dst halo index << 16
    int* rhalo = nullptr;        // per topology: CS_RES_MAX_CL + 1 halo slot counts per rank
    int* rcheb = nullptr;        // per topology and rank: bit 0, the Chebyshev preconditioner when asked; bit 1, rows tiled (levels)
    int res_halo0 = 0;           // first halo slot of every CTA's u array (after the own slots and a zero entry)
    int res_alt = 0;             // first slot of the second own-row buffer (tile-local Chebyshev)
    // coarse-space correction (resident.cu): per topology {coarse unknowns nc (0: none), segments
    // per tile K, first and last entry of the coarse pattern in cpair}; the coarse pattern's block
    // pairs {aggregate a, aggregate b, first, last contributor in ccontrib} with their stored
    // blocks as topology slots; per resident work item the inverse coarse matrix (nc x nc) and
    // whether it was formed.
    int4* rcoarse = nullptr;
    int4* cpair = nullptr;
    int* ccontrib = nullptr;
    float* cinv = nullptr;
    int* cvalid = nullptr;
    int res_cnc = 0;             // largest nc over the resident topologies (0: no coarse correction)
    int res_ck = 0;              // largest K
    int res_coff = 0;            // byte offset of the coarse region in the resident kernel's shared memory
    // group-resident solver (group.cu): work items, per CTA the items it takes part in (in order);
    // per topology slot (pub0) whether another CTA reads the row, per CTA (halo0) the slots it reads
    // from others; exchange packets; the groups' inverse coarse matrices and per sheet their validity;
    // sizes for the largest group (CTAs, own slots, halo slots, coarse unknowns, 3 segments per CTA,
    // entries of a CTA's rows of the inverse coarse matrix),
    // panels per CTA in shared memory and the byte offset of what follows the u array there
    int n_group = 0, g_max = 0, g_own = 0, g_halo = 0, g_cap = 0, g_coff = 0, g_cnc = 0, g_ck3 = 0, g_cai = 0;
    // polls of an exchange packet before a CTA gives up: within a solve, and for a sheet's first exchange
    uint32_t g_polls = 1u << 19, g_polls_first = 1u << 27;
    GroupItem* gitem = nullptr;
    int *gcta_ptr = nullptr, *gcta_item = nullptr;
    unsigned char* gpub = nullptr;
    int *ghalo_ptr = nullptr, *ghalo = nullptr;
    uint4 *gupk = nullptr, *grpk = nullptr;
    float* gc_inv = nullptr;
    int* gc_ok = nullptr;
    // the batched coarse set-up kernels (coarse.cu) run on the sheets that the loop solves (0), or,
    // on a copy of this struct holding the groups' coarse spaces, on those of the groups (1)
    int bc_resident = 0;
    // per-topology block CSR (local ids, columns ascending) with the SELL slot of each block
    int* tcsr_ptr = nullptr;
    int* tcsr_col = nullptr;
    int* tcsr_slot = nullptr;
    // proximities (cs_set_proximities, cs_detect_proximities)
    int n_pinst = 0, n_px = 0;
    const ProxInst* pinst = nullptr;
    float* prec = nullptr;        // CS_PROX_REC per instance
    const int* prow_ptr = nullptr;   // N + 1: the instances holding each row's node
    const int* prow_inst = nullptr;  // ascending per row
    int* xptr = nullptr;          // N + 1: blocks outside the pattern, per row (null: none)
    int* xcol = nullptr;          // their columns (batch nodes), ascending per row
    float* xval = nullptr;        // 9 per block, summed each step
    int* sheet_prox = nullptr;    // per sheet: bit 0 a proximity touches it, bit 1 it has blocks outside the pattern
};

// Proximity detection (contact.cu, cs_detect_proximities).  Scene-wide ids: nodes and faces as
// in Batch, edges (every edge, not only interior ones) of all sheets concatenated in sheet order.
struct Contact {
    int E = 0;               // edges
    int n_keys = 0;          // 2 N + 2 E + 2 F
    int hash_bits = 0;       // grid buckets = 1 << hash_bits
    float repulsion = 0.f, stiffness = 0.f, friction = 0.f;
    float dilate = 0.f;      // bounds dilation of the candidate pairs (2 x repulsion; collision thickness)
    int ccd = 0;             // 1: face bounds over x0 and x (continuous impacts)
    const int4* face_edges = nullptr;  // 3 edges + collision group per face
    const int4* edges = nullptr;       // node 0, node 1, face side 0, face side 1
    const int* nf_ptr = nullptr;       // N + 1
    const int* nf_code = nullptr;      // face << 2 | corner, faces in index order
    const float* node_area = nullptr;  // Mesh::updateNodeGeometries (Mesh.cu:190-198)
    const float* edge_area = nullptr;  // Edge::area (Edge.cu:89-95)
    float* fn = nullptr;               // face normals (3 per face)
    float* nn = nullptr;               // node normals (3 per node)
    float* box = nullptr;              // face bounds: lo xyz, hi xyz
    unsigned* ext = nullptr;           // [0] largest face extent (float bits), [1] error flags
    int* head = nullptr;               // grid bucket heads (-1: empty)
    int* next = nullptr;               // 8 entries per face: next entry in the bucket
    unsigned long long* keys = nullptr;  // per (node|edge|face, side): distance bits << 32 | other id
    int2* pairs = nullptr;             // candidate face pairs (f, g > f)
    int pair_cap = 0;
    int* pair_count = nullptr;
    int* block_count = nullptr;        // compaction: valid keys per block, then exclusive offsets
    int* total = nullptr;
    cs_proximity_desc* out = nullptr;  // detected proximities
    int out_cap = 0;
};

// Collision step (collide.cu, cs_collision_step): continuous impacts and their projection.
struct ImpactRec {
    int nodes[4];
    float t, w[4], n[3];
    int type;  // 0 vertex-face, 1 edge-edge
    int pad[3];
};

struct Collide {
    float thickness = 0.f;
    ImpactRec* found = nullptr;   // impacts of this round
    int found_cap = 0;
    int* counters = nullptr;      // [0] impacts found, [1] impacts selected
    ImpactRec* sorted = nullptr;  // by time (then node ids)
    // radix sort of the found impacts: key and permutation double buffers, CUB temp storage
    unsigned long long *skey[2] = {nullptr, nullptr};
    int* sperm[2] = {nullptr, nullptr};
    void* stmp = nullptr;
    size_t stmp_bytes = 0;
    ImpactRec* all = nullptr;     // independent impacts accumulated this deformation level
    int* used = nullptr;          // per node: taken by a selected impact of this round
    int* nodemin = nullptr;       // per node: lowest live impact index touching it (selection)
    int* alive = nullptr;         // per found impact: still a candidate of the selection
    int* chosen = nullptr;        // per found impact (+1): selected, then its output offset
    // the projection's nodes and constraints
    int* mark = nullptr;          // N + 1: node in an impact, then its slot (exclusive scan)
    int* nodes = nullptr;         // slot -> node, ascending
    int* idx = nullptr;           // 4 per impact: slots of its nodes
    int* nptr = nullptr;          // slots + 1: each slot's constraint corners
    int* nfill = nullptr;
    int* nlist = nullptr;         // 4 impact + corner, ascending per slot
    float* x1 = nullptr;          // 3N: positions when the collision step began
    float4 *cur = nullptr, *next = nullptr;    // per slot: positions, two buffers
    float4 *grad = nullptr, *grad2 = nullptr;  // per slot: gradient and its square, two buffers
    float4* home = nullptr;                    // per slot: position when the step began, mass
    float4* con = nullptr;                     // 3 per constraint: slots, weights, normal
    float *lambda = nullptr, *lambda2 = nullptr, *cterm = nullptr;  // per constraint
};

// threads per CTA of the impact projection and the terms of an ordered sum staged in its shared memory
#define CS_OPT_THREADS 1024
#define CS_OPT_STAGE 12288
#define CS_CONTACT_ITEMS 4096  // keys per compaction block (256 threads x 16)
#define CS_PAIR_LANES 8        // lanes that share out the cells of a face
#define CS_PAIR_STAGE 16       // candidate pairs staged per thread before appending
#define CS_SCAN_ITEMS 4096     // ints per block of the exclusive scan (1024 threads x 4)

#endif
