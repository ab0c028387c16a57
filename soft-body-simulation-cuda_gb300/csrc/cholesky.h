// Sparse Cholesky of the scalar PD system K: ordering, symbolic analysis and the
// host's numeric factorisation.
//
// The reference assembles A = K (x) I_3 (3n x 3n) from per-tet triplets
// (pdUtil.cu:9-54), orders it with cuSOLVER's host AMD and factors it in
// FP32 with cuSOLVER's low-level sparse Cholesky (cholesky.cu:72-158).  The
// engine orders the n x n scalar K on the host (approximate minimum degree),
// factors it once in FP64, on the GPU (factor.cu) or on the host (supernodal
// multifrontal LL^T both), and solves the three coordinates together on the GPU.
//
// Solve representation.  For every supernode s with pivot columns C_s
// (k_s of them) and off-diagonal rows O_s (m_s - k_s), the GPU stores the
// m_s x k_s matrix
//     M_s = [ L_ss^-1 ; L_os L_ss^-1 ]       (column major, FP32, columns
//                                              m_stride floats apart)
// so that the forward step of s is y_s = L_ss^-1 r_s plus the update
// r_O -= (L_os L_ss^-1) r_s, and the backward step is
// x_s = (L_ss^-1)^T y_s - (L_os L_ss^-1)^T x_O: both are dense
// matrix-vector products with M_s.  Supernodes on the same level of the
// supernodal elimination tree are independent.
#pragma once

#include <cstdint>
#include <vector>

namespace pdgb {

struct SparseSym {
    int n = 0;
    std::vector<int64_t> p;  // CSR row pointers (full symmetric pattern, diagonal included)
    std::vector<int> i;
    std::vector<double> x;
};

// Approximate minimum degree ordering (Amestoy, Davis & Duff, SIAM J. Matrix
// Anal. Appl. 17(4), 1996): quotient graph with element absorption,
// approximate external degrees, mass elimination and supervariable
// detection.  Returns perm (perm[k] = row eliminated k-th).
std::vector<int> amd_order(const SparseSym& A);

// Geometric nested dissection (recursive coordinate bisection), an
// alternative ordering for meshes.  xyz: 3 floats per row.
std::vector<int> nd_order(const SparseSym& A, const float* xyz);

struct SolveLevel {
    int fwd_begin, fwd_end;  // warp work items of the forward pass for this level
    int bwd_begin, bwd_end;  // warp work items of the backward pass
    int blk_begin, blk_end;    // per-level launches: block items (both directions)
    int sml_begin, sml_end;    // per-level launches: small supernodes, one warp each
    int tiny_begin, tiny_end;  // per-level launches: tiny supernodes, a few lanes each
};

// Warp work items, 8 ints each (two int4 loads, no dependent metadata loads):
//   forward : {moff_lo, moff_hi, roff, m, k, r0, c0, c1}: rows r0 .. min(r0+32, m)
//             of M_s (column major) times the right-hand side of pivot
//             columns c0 .. c1
//   backward: {moff_lo, moff_hi, roff, m, k, c, 0, 0}: pivot column c
constexpr int kItemInts = 8;
constexpr int kFwdItemRows = 32;
constexpr int kFwdItemCols = 64;
// Items of the per-level launches (same 8-int layout):
//   block: {moff_lo, moff_hi, roff, m, k, r0, c0, c1}: the tile of M_s with
//          rows r0 .. r0 + kTileRows and pivot columns c0 .. c1 (at most
//          kTileCols), for one CTA and both directions
//   small: {moff_lo, moff_hi, roff, m, k, 0, 0, 0}: a whole supernode of fewer
//          than kSmallRows rows and at most kSmallCols pivots, for a warp
//   tiny : the same for a supernode of one pivot and at most kTinyRows rows
constexpr int kTileRows = 128;
constexpr int kTileCols = 32;
constexpr int kSmallRows = 64;
constexpr int kSmallCols = 32;
constexpr int kTinyRows = 32;
// Shared memory of a warp that takes a small supernode: its block, then z of
// its rows, in floats.
constexpr int kSmallFloats = 896;
constexpr int kWarpFloats = kSmallFloats + 4 * kSmallRows;
static_assert(4 * kWarpFloats >= kTileRows * kTileCols, "a tile fits the same shared memory");

#ifdef __CUDACC__
#define PDGB_HD __host__ __device__
#else
#define PDGB_HD
#endif
// Floats between the columns of M_s: a multiple of 4, so that its rows can be
// loaded 16 bytes at a time; of a supernode that a warp copies whole, an odd
// multiple, so that the 8 lanes of a quarter-warp that read 4 rows of 8
// neighbouring columns in shared memory hit 8 groups of banks.
PDGB_HD inline int m_stride(int m, int k) {
    const int q = (m + 3) / 4;
    return 4 * (k > 1 && k <= kSmallCols && m < kSmallRows ? (q | 1) : q);
}
PDGB_HD inline bool is_small(int m, int k) {
    return m < kSmallRows && k <= kSmallCols && k * m_stride(m, k) <= kSmallFloats;
}

// Numeric factorisation on the GPU (factor.cu): everything the device needs
// beyond the symbolic structure of CholFactor.  Each supernode s has a dense
// front F_s (m_s x m_s, column major, FP64) in one pool, followed by an
// m_s x k_s FP64 block for M_s; F_s receives the entries of K in its pivot
// columns and the Schur complements of its children (extend-add), is
// factored over its first k_s columns, and its own Schur complement
// F_s[k_s:, k_s:] is then added into its parent's front.  Fronts live from
// their level until their parent's level is assembled, and the pool reuses
// the memory of the fronts that are done.
struct FrontPlan {
    bool on = false;                   // mval is left to the GPU
    int64_t pool = 0;                  // doubles in the front pool
    int max_m = 0;                     // largest front
    std::vector<int64_t> foff;         // [nsuper] front offset in the pool
    std::vector<int> parent;           // [nsuper] parent supernode, -1 for a root
    std::vector<int> child_ptr, child; // children of each supernode ([nsuper + 1] / [nsuper])
    std::vector<int> rel_ptr, rel;     // rows of s past its pivots, as positions in its parent's row list
    std::vector<int> kptr;             // [nsuper + 1] entries of K in the pivot columns of s
    std::vector<int> kpos;             // position of the entry in F_s (column * m_s + row)
    std::vector<double> kval;
    std::vector<int> lvl_ptr, lvl_sn;  // supernodes by level (from the leaves, all bodies together)
};

struct CholFactor {
    int n = 0;
    long long nnz_L = 0;             // nnz of the scalar factor (incl. diagonal)
    int nsuper = 0;
    double flops = 0.0;
    // per supernode
    std::vector<int> sk, sm;         // pivot count k_s, row count m_s
    std::vector<int64_t> moff;       // offset of M_s in mval (column major m x k, columns m_stride apart)
    std::vector<int> roff;           // offset of the row list in rows
    std::vector<int> rows;           // row lists (vertex ids; first k = pivots)
    std::vector<float> mval;         // FP32 M_s blocks, column major
    std::vector<int> level;          // level of each supernode (leaves = 0)
    int nlevels = 0;
    // GPU warp work items grouped by level (see kItemInts).
    std::vector<int> fwd_items;
    std::vector<int> bwd_items;
    std::vector<int> blocks;         // items of the per-level launches (see kTileRows)
    std::vector<int> small;
    std::vector<int> tiny;
    std::vector<SolveLevel> levels;  // body-major: body b owns levels[body_level[b] .. body_level[b+1])
    // Per-level launches (block and small items): level L of every body in
    // one launch, levels counted from the leaves.  Equal to `levels` for a
    // single body.
    std::vector<SolveLevel> step_levels;
    std::vector<int> body_level;     // [nbodies + 1]
    std::vector<int> body_order;     // bodies by decreasing stored factor size (batch solve order)
    long long zeros = 0;             // explicit zeros stored by amalgamated supernodes
    // FP64 copy of K for refinement residuals (CSR over vertex ids)
    SparseSym K;
    int64_t mval_size = 0;           // FP32 entries of the M_s blocks (= mval.size() when factored on the host)
    FrontPlan fp;                    // numeric factorisation left to the GPU (fp.on)
    // The inverse of the root's block of the factored system, L^-T L^-1 over its
    // k pivots, stored past the M_s blocks (symmetric, columns
    // m_stride(k, k) floats apart): -1 where there is none (plan_root_inverse).
    int root = -1;                   // the root supernode
    int64_t root_off = 0;            // its inverse's offset in mval
    int64_t mval_total = 0;          // floats of the M_s blocks and the root's inverse
};

// Lets the factorisation on the GPU add the root's inverse to a single body's
// factor (before gpu_factor).  At the root nothing is left between the forward
// and the backward pass, so one product with the inverse takes the place of
// two dependent launches, for the same bytes: a square matrix once instead of
// a triangle twice.  Worth it where a solve is few launches, up to kRootLevels
// levels, and up to kRootCols pivots: an iteration of the 6^3 grid 9.1 -> 7.7 us,
// 12^3 10.1 -> 9.4 us, 14^3 (861 pivots) even, and of 19 x 11 x 23 (1,523) 13.2 ->
// 15.1 us, where every CTA's gather of all right-hand sides costs more than the
// launch.
constexpr int kRootLevels = 3;
constexpr int kRootCols = 1024;
void plan_root_inverse(CholFactor& f);

// Plan of the distributed-shared-memory solve of a single body: an 8-CTA
// cluster, each CTA owning a set of supernodes whose M_s blocks and row
// lists it stages into its shared memory once per solve; the right-hand
// side, y and x live in the cluster's shared memory, vertex v in CTA v % 8
// at slot v / 8.  Items use the warp-item layout with shared-memory offsets:
//   forward : {m_off, r_off, m, k, r0, c0, c1, 0}; backward: {m_off, r_off, m, k, c, 0, 0, 0}.
struct DsmPlan {
    bool ok = false;
    int ctas = 0;                 // cluster size
    int n = 0;                    // vertices
    int slots = 0;                // vector slots per CTA (ceil(n / ctas))
    int nlevels = 0;
    int m_area = 0;               // float index of the staged M area in shared memory
    int r_area = 0;               // int index of the staged row area
    size_t smem_bytes = 0;        // dynamic shared memory per CTA
    // Each CTA's staged areas, laid out as in its shared memory and stored
    // contiguously per CTA, so that staging is one wide copy per CTA.
    std::vector<float> mcopy;     // M_s blocks of CTA c at [mcopy_ptr[c], mcopy_ptr[c+1])
    std::vector<int> mcopy_ptr;   // [ctas + 1], multiples of 4
    std::vector<int> rcopy;       // row lists of CTA c at [rcopy_ptr[c], rcopy_ptr[c+1])
    std::vector<int> rcopy_ptr;   // [ctas + 1], multiples of 4
    std::vector<int> items;       // kItemInts per item, each CTA's items grouped by level
    std::vector<int> lvl;         // [ctas][nlevels] x {fwd_begin, fwd_end, bwd_begin, bwd_end}
};
// Fills the plan for a single-body factor when the busiest CTA's share fits
// max_smem bytes of shared memory; plan.ok tells whether it does.
void build_dsm_plan(const CholFactor& f, int ctas, int warps_per_cta, size_t max_smem, DsmPlan& plan);

// Factors K (vertex-indexed, n x n SPD).  ordering: 0 = AMD, 1 = nested
// dissection (xyz required), 2 = AMD order stored as one dense supernode.  Throws Error(PDGB_ERR_NOT_SPD) if a pivot is
// not positive.
// gpu_numeric: stop after the symbolic analysis and fill out.fp for the
// GPU factorisation (factor.cu) instead of computing mval on the host;
// finish_plan: complete it (finish_front_plan) -- a batch completes the
// combined plan of its bodies instead.
// price: how supernodes are amalgamated for a schedule, a level of the solve
// against stored entries (SolveCost).
enum class SolveKind {
    kSingle,  // one body: a launch, a grid's or a cluster's barrier a level
    kShared,  // bodies that share their launches: they count items instead of
              // entries, however small their share of a level
    kCta,     // one CTA a body: a level is a CTA's barrier
    kDsm,     // one cluster, and every stored entry takes its shared memory
    kLeast,   // as few stored entries as there are
};
// Entries that a level costs.  Launches: about 6 us of dependent ones, forward and
// backward, against 8 bytes an entry at some 5 TB/s.  Batches pay it by size,
// requests of a server 1 / kServerBodies (40 uneven requests of 4 to 19 cells take
// 151, 126 and 112 ms at 4, 16 and 64, 8 of 28^3 323, 307 and 305, one of 28^3 128,
// 134 and 133, one of 10^3 64, 64 and 73, twelve of 1 k to 100 k tets 72, 70 and 71).
// For one CTA a barrier is less and an
// entry more: ten iterations of a 13^3 body, of a 60 x 6 x 3 one and of 16 of 2^3
// beside 32 of 10^3 take 1,715, 1,044 and 1,096 us at 1e4 and 2,297, 1,179 and
// 1,202 with the tree for launches.
constexpr double kLevelEntries = 3.75e6;
constexpr double kServerBodies = 16.0;
constexpr double kCtaLevelEntries = 1e4;
constexpr double kDsmLevelEntries = 1e3;
struct SolveCost {
    SolveKind kind = SolveKind::kSingle;
    double level_entries = kLevelEntries;
};
void cholesky_factor(const SparseSym& K, int ordering, const float* xyz, CholFactor& out,
                     bool gpu_numeric = false, bool finish_plan = true, const SolveCost& price = SolveCost{});

// Factors the block-diagonal system of independent bodies, one block per
// body (vertex range vstart[b]..vstart[b+1], tets tstart[b]..tstart[b+1] in
// the engine's order), in parallel over bodies, and concatenates the
// factors: rows keep engine vertex ids, work items and levels are grouped
// per body.  price: a body's, or with kShared what the level costs all of them.
void cholesky_factor_bodies(int nbodies, const std::vector<int>& vstart, const std::vector<int>& tstart,
                            const uint32_t* tets4, const double* dminv, const double* coef,
                            const std::vector<double>& mdt2, int ordering, const float* xyz, CholFactor& out,
                            bool gpu_numeric, const SolveCost& price);

// Doubles of the pool that supernode s takes: its front and its M_s block.
int64_t front_doubles(const CholFactor& f, int s);

// Numeric factorisation of the plan f.fp on the GPU (factor.cu): writes the
// FP32 M_s blocks and the root's inverse if planned (f.mval_total floats,
// device memory) and returns the device
// time in ms.  Waits for the stream.  Throws Error(PDGB_ERR_NOT_SPD) when a
// pivot is not positive.
double gpu_factor(const CholFactor& f, float* mval, void* stream);

// Completes out.fp once the supernodes of all bodies are in place: children
// lists, supernodes by level, and the front pool (best-fit reuse of the
// fronts whose parents are assembled).
void finish_front_plan(CholFactor& out);

// Applies the factor on the host exactly as the GPU work items do
// (forward by levels with M_s, backward by levels), in double: x = K^-1 b
// for 3 interleaved right-hand sides indexed by vertex id.
void cholesky_solve_host(const CholFactor& f, const double* b3, double* x3);

// Assembles K = diag(mdt2) + sum_t c_t B_t^T B_t for tets given by internal
// vertex ids (tets4), DmInv (9 doubles per tet, row major) and c_t.
SparseSym assemble_system(int nv, int nt, const uint32_t* tets4, const double* dminv, const double* coef,
                          const std::vector<double>& mdt2);

// The scalar system K of a single body's layout, in its internal vertex
// order: M/h^2 from the float coefficients the kernels use (pin weight
// included) and the double geometry.
struct HostLayout;
SparseSym layout_system(const HostLayout& L);

// Rest positions of a layout as 3 floats per vertex (the nested-dissection
// ordering's coordinates).
std::vector<float> layout_xyz(const HostLayout& L);

}  // namespace pdgb
