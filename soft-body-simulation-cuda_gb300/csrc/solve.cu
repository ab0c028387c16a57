// Level-scheduled supernodal triangular solves (sm_103a) and the Cholesky
// path's per-iteration vertex kernel.
//
// Replaces the reference's global step CholeskySpLinearSolver::Solve
// (cholesky.cu:184-192: permute, cusolverSpScsrcholSolve, unpermute) and the
// error check computeError (pdSolver.cu:186-191, 243-253).  The factor is
// stored per supernode as M_s = [L_ss^-1 ; L_os L_ss^-1] (see cholesky.h);
// three right-hand sides (x, y, z) travel together as float4.  Row lists
// hold engine vertex ids, so no permutation pass is needed.
#include "engine.h"
#include "solve.h"
#include "pdl.cuh"
#include "scene.cuh"

#include <cooperative_groups.h>

#include <cstdlib>

namespace pdgb {

// The per-level kernels are launched with programmatic dependent launch
// (pdl.cuh): each triggers its dependents at entry and, before its wait,
// reads only its item descriptors, factor blocks and row ids -- never r, y,
// x, z or the early-exit flag, which earlier kernels write.

// Forward warp item {moff, roff, m, k, r0, c0, c1}: lane = row r0 + lane of
// M_s; sum over pivot columns c0..c1 of M_s[row, c] r[pivot c]; pivot rows
// add the sum to y, off-diagonal rows subtract it from r (ancestor columns,
// solved at a later level).  The chunk's pivot right-hand sides are staged
// in warp-private shared memory 32 at a time; the column loop issues 8
// independent loads of M before using them (memory-level parallelism for
// the few, large supernodes at the top of the tree).
__device__ __forceinline__ void fwd_warp_item(const CholArgs& a, const int* w, float4* stage, int lane) {
    const int4 h0 = __ldg(reinterpret_cast<const int4*>(w));
    const int4 h1 = __ldg(reinterpret_cast<const int4*>(w) + 1);
    const int64_t moff = (int64_t)(uint32_t)h0.x | ((int64_t)h0.y << 32);
    const int roff = h0.z, m = h0.w, k = h1.x, r0 = h1.y, c0 = h1.z, c1 = h1.w;
    const int* rows = a.rows + roff;
    const int row = r0 + lane;
    const bool valid = row < m;
    const int cend = !valid ? c0 : (row < k ? min(c1, row + 1) : c1);
    const float* Mr = a.mval + moff + row;
    const int vid = valid ? __ldg(&rows[row]) : 0;
    float ax = 0.f, ay = 0.f, az = 0.f;
    for (int cb = c0; cb < c1; cb += 32) {
        const int nc = min(32, c1 - cb);
        __syncwarp();
        if (lane < nc) stage[lane] = a.r[__ldg(&rows[cb + lane])];
        __syncwarp();
        for (int c = cb; c < cb + nc; c += 8) {
            float mv[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) mv[q] = (c + q < cend) ? __ldg(Mr + (size_t)(c + q) * m) : 0.f;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (c + q < cb + nc) {
                    const float4 v = stage[c + q - cb];
                    ax = fmaf(mv[q], v.x, ax);
                    ay = fmaf(mv[q], v.y, ay);
                    az = fmaf(mv[q], v.z, az);
                }
            }
        }
    }
    if (!valid) return;
    if (row < k) atomicAdd(&a.y[vid], make_float4(ax, ay, az, 0.f));
    else atomicAdd(&a.r[vid], make_float4(-ax, -ay, -az, 0.f));
}

// Backward warp item {moff, roff, m, k, c}: x[pivot c] = sum_{i >= c}
// M_s[i, c] z_i with z = [y_pivots ; -x_offdiag]; lanes stride over rows
// (a coalesced column of M_s, 4 independent loads in flight per lane),
// then a warp reduction.  One column per warp keeps the large supernodes at
// the top of the tree spread over many warps.  No atomics.
__device__ __forceinline__ void bwd_warp_item(const CholArgs& a, const int* w, float4* stage, int lane) {
    (void)stage;
    const int4 h0 = __ldg(reinterpret_cast<const int4*>(w));
    const int4 h1 = __ldg(reinterpret_cast<const int4*>(w) + 1);
    const int64_t moff = (int64_t)(uint32_t)h0.x | ((int64_t)h0.y << 32);
    const int roff = h0.z, m = h0.w, k = h1.x, c = h1.y;
    const int* rows = a.rows + roff;
    const float* Mc = a.mval + moff + (size_t)c * m;
    float ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll 4
    for (int i = c + lane; i < m; i += 32) {
        const int vid = __ldg(&rows[i]);
        const float mv = __ldg(Mc + i);
        float4 z;
        if (i < k) z = a.y[vid];
        else {
            const float4 xv = a.x[vid];
            z = make_float4(-xv.x, -xv.y, -xv.z, 0.f);
        }
        ax = fmaf(mv, z.x, ax);
        ay = fmaf(mv, z.y, ay);
        az = fmaf(mv, z.z, az);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, off);
        ay += __shfl_xor_sync(0xffffffffu, ay, off);
        az += __shfl_xor_sync(0xffffffffu, az, off);
    }
    if (lane == 0) a.x[__ldg(&rows[c])] = make_float4(ax, ay, az, 0.f);
}

// ---- per-level launches: one per level and direction.  A launch's CTAs
// (kLevelThreads threads) take, by index, first the level's block items, then
// its small supernodes (one warp each), then its tiny ones (kTinyLanes lanes
// each), then -- in the solve's first backward launch, when asked -- the
// resets of the next iteration's vectors.  Each CTA reads its descriptors,
// row ids and factor entries into registers before the grid dependency wait,
// so that a level's factor bytes are under way while the level before drains;
// after the wait come one gather from L2, the products, one reduction and the
// stores.  What bounds a narrow level is that chain of latencies, about 3 us
// with the launch, so a level is one launch and nothing is staged by another.

// Block item {moff, roff, m, k, r0, c0, c1}: the tile rows r0 .. r0 + 128,
// pivot columns c0 .. c1 (at most 32) of M_s; both directions use the same
// items.
struct BlockItem {
    const float* M;   // M_s, column major
    const int* rows;
    int m, k, r0, c0, c1;
};

__device__ __forceinline__ BlockItem block_item(const CholArgs& a, const int* list, int item) {
    const int4* w = reinterpret_cast<const int4*>(list + (size_t)kItemInts * item);
    const int4 h0 = __ldg(w), h1 = __ldg(w + 1);
    const int64_t moff = (int64_t)(uint32_t)h0.x | ((int64_t)h0.y << 32);
    return BlockItem{a.mval + moff, a.rows + h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
}

// Forward block, static part: thread t owns row r0 + t, its (at most 32)
// entries of the tile in registers.  A warp's loads of one column are
// contiguous.
struct FwdBlockPre {
    float mv[kTileCols];
    int vid, sv, ncols, row, k, m;
    bool first;   // the tile holds the first pivot columns
};

__device__ __forceinline__ void fwd_block_load(const CholArgs& a, int item, FwdBlockPre& p) {
    const BlockItem b = block_item(a, a.blocks, item);
    const int row = b.r0 + threadIdx.x;
    const bool active = row < b.m && row >= b.c0;  // rows above the tile's columns have nothing in it
    const int cend = !active ? b.c0 : (row < b.k ? min(b.c1, row + 1) : b.c1);
    const float* Mr = b.M + row;
#pragma unroll
    for (int q = 0; q < kTileCols; ++q) p.mv[q] = (b.c0 + q < cend) ? __ldg(Mr + (size_t)(b.c0 + q) * b.m) : 0.f;
    p.vid = active ? __ldg(&b.rows[row]) : -1;
    p.ncols = b.c1 - b.c0;
    p.sv = (int)threadIdx.x < p.ncols ? __ldg(&b.rows[b.c0 + threadIdx.x]) : 0;
    p.row = row;
    p.k = b.k;
    p.m = b.m;
    p.first = b.c0 == 0;
}

// Vector part: the pivot right-hand sides staged in shared memory, then the
// row's sum into y (pivot rows; stored where no other tile adds to it) or out
// of r (ancestor rows, pivots of later levels).  The backward pass adds the
// partial sums of a supernode with more rows than a tile into x, which is
// cleared here.
__device__ __forceinline__ void fwd_block_run(const CholArgs& a, const FwdBlockPre& p, float4* rs) {
    if (threadIdx.x < kTileCols)
        rs[threadIdx.x] = (int)threadIdx.x < p.ncols ? __ldcg(&a.r[p.sv]) : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    if (p.vid < 0) return;
    float ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll
    for (int q = 0; q < kTileCols; ++q) {
        const float4 v = rs[q];
        ax = fmaf(p.mv[q], v.x, ax);
        ay = fmaf(p.mv[q], v.y, ay);
        az = fmaf(p.mv[q], v.z, az);
    }
    if (p.row >= p.k) {
        atomicAdd(&a.r[p.vid], make_float4(-ax, -ay, -az, 0.f));
        return;
    }
    if (p.row < kTileCols) a.y[p.vid] = make_float4(ax, ay, az, 0.f);
    else atomicAdd(&a.y[p.vid], make_float4(ax, ay, az, 0.f));
    if (p.first && p.m > kTileRows) a.x[p.vid] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// z of a row: y at a pivot, -x at an ancestor.
__device__ __forceinline__ float4 z_of(const CholArgs& a, bool pivot, int vid) {
    if (pivot) return __ldcg(&a.y[vid]);
    const float4 v = __ldcg(&a.x[vid]);
    return make_float4(-v.x, -v.y, -v.z, 0.f);
}

// Sums of 8 columns x 3 coordinates over the 32 lanes of a warp: three
// exchanges that halve the columns a lane holds, then two plain ones.  Lane l
// ends with the sums of column (l >> 2).
__device__ __forceinline__ float3 reduce_cols8(float (&v)[8][3], int lane) {
    float w[4][3], u[2][3], t[3];
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float keep = b4 ? v[j + 4][d] : v[j][d], give = b4 ? v[j][d] : v[j + 4][d];
            w[j][d] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
        }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float keep = b3 ? w[j + 2][d] : w[j][d], give = b3 ? w[j][d] : w[j + 2][d];
            u[j][d] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
        }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float keep = b2 ? u[1][d] : u[0][d], give = b2 ? u[0][d] : u[1][d];
        t[d] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
        t[d] += __shfl_xor_sync(0xffffffffu, t[d], 2);
        t[d] += __shfl_xor_sync(0xffffffffu, t[d], 1);
    }
    return make_float3(t[0], t[1], t[2]);
}

// Backward block, static part: warp w owns the tile's columns c0 + 8 w ..,
// lane l its rows r0 + l, + 32, ..: 4 x 8 entries in registers.
constexpr int kBwdWarpCols = kTileCols / (kLevelThreads / 32);
constexpr int kBwdRows = kTileRows / 32;
static_assert(kBwdWarpCols == 8, "reduce_cols8");
struct BwdBlockPre {
    float mv[kBwdRows][kBwdWarpCols];
    int vid;      // of row r0 + thread, -1 past the last
    int cv;       // vertex of this lane's result column, -1: none
    bool pivot, split;
};

__device__ __forceinline__ void bwd_block_load(const CholArgs& a, int item, BwdBlockPre& p) {
    const BlockItem b = block_item(a, a.blocks, item);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cw = b.c0 + kBwdWarpCols * warp;
    const float* Mc = b.M + (size_t)cw * b.m;
#pragma unroll
    for (int t = 0; t < kBwdRows; ++t) {
        const int i = b.r0 + lane + 32 * t;
#pragma unroll
        for (int j = 0; j < kBwdWarpCols; ++j)
            p.mv[t][j] = (i < b.m && cw + j < b.c1 && i >= cw + j) ? __ldg(Mc + (size_t)j * b.m + i) : 0.f;
    }
    const int row = b.r0 + threadIdx.x;
    p.vid = row < b.m ? __ldg(&b.rows[row]) : -1;
    p.pivot = row < b.k;
    const int c = cw + (lane >> 2);
    p.cv = ((lane & 3) == 0 && c < b.c1) ? __ldg(&b.rows[c]) : -1;
    p.split = b.m > kTileRows;
}

// Vector part: z of the tile's rows staged in shared memory, the products,
// the warp's reduction; sums stored, or added where the supernode's rows take
// several tiles.
__device__ __forceinline__ void bwd_block_run(const CholArgs& a, const BwdBlockPre& p, float4* zs) {
    zs[threadIdx.x] = p.vid >= 0 ? z_of(a, p.pivot, p.vid) : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    float acc[kBwdWarpCols][3];
#pragma unroll
    for (int j = 0; j < kBwdWarpCols; ++j) acc[j][0] = acc[j][1] = acc[j][2] = 0.f;
#pragma unroll
    for (int t = 0; t < kBwdRows; ++t) {
        const float4 z = zs[lane + 32 * t];
#pragma unroll
        for (int j = 0; j < kBwdWarpCols; ++j) {
            acc[j][0] = fmaf(p.mv[t][j], z.x, acc[j][0]);
            acc[j][1] = fmaf(p.mv[t][j], z.y, acc[j][1]);
            acc[j][2] = fmaf(p.mv[t][j], z.z, acc[j][2]);
        }
    }
    const float3 s = reduce_cols8(acc, lane);
    if (p.cv < 0) return;
    if (p.split) atomicAdd(&a.x[p.cv], make_float4(s.x, s.y, s.z, 0.f));
    else a.x[p.cv] = make_float4(s.x, s.y, s.z, 0.f);
}

// Small supernodes {moff, roff, m, k} (m < kBlockMinRows = 64 rows, at most
// kSmallCols pivots): one warp, lane l owns rows l and l + 32.  Forward: the
// first kSmallPre columns before the wait, the rest after it.
constexpr int kSmallPre = 16;
struct SmallPre {
    float mv[2][kSmallPre];
    const float* M;
    int m, k, vid[2];
};

__device__ __forceinline__ void small_load(const CholArgs& a, int item, bool live, int lane, SmallPre& p) {
    p.m = p.k = 0;
    p.M = a.mval;
    p.vid[0] = p.vid[1] = -1;
    if (live) {
        const BlockItem b = block_item(a, a.small, item);
        p.M = b.M;
        p.m = b.m;
        p.k = b.k;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (lane + 32 * h < p.m) p.vid[h] = __ldg(&b.rows[lane + 32 * h]);
    }
#pragma unroll
    for (int c = 0; c < kSmallPre; ++c)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = lane + 32 * h;
            p.mv[h][c] = (c < p.k && row < p.m && row >= c) ? __ldg(p.M + (size_t)c * p.m + row) : 0.f;
        }
}

__device__ __forceinline__ void fwd_small_run(const CholArgs& a, const SmallPre& p, int lane, float4* stage) {
    stage[lane] = lane < p.k ? __ldcg(&a.r[p.vid[0]]) : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    float s[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll
    for (int c = 0; c < kSmallPre; ++c) {
        const float4 v = stage[c];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            s[h][0] = fmaf(p.mv[h][c], v.x, s[h][0]);
            s[h][1] = fmaf(p.mv[h][c], v.y, s[h][1]);
            s[h][2] = fmaf(p.mv[h][c], v.z, s[h][2]);
        }
    }
#pragma unroll 4
    for (int c = kSmallPre; c < p.k; ++c) {
        const float4 v = stage[c];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = lane + 32 * h;
            const float mv = (row < p.m && row >= c) ? __ldg(p.M + (size_t)c * p.m + row) : 0.f;
            s[h][0] = fmaf(mv, v.x, s[h][0]);
            s[h][1] = fmaf(mv, v.y, s[h][1]);
            s[h][2] = fmaf(mv, v.z, s[h][2]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (p.vid[h] < 0) continue;
        if (lane + 32 * h < p.k) a.y[p.vid[h]] = make_float4(s[h][0], s[h][1], s[h][2], 0.f);
        else atomicAdd(&a.r[p.vid[h]], make_float4(-s[h][0], -s[h][1], -s[h][2], 0.f));
    }
}

// Backward: z of the warp's rows in registers, 8 columns at a time.
__device__ __forceinline__ void bwd_small_run(const CholArgs& a, const SmallPre& p, int lane) {
    float4 z[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        z[h] = p.vid[h] >= 0 ? z_of(a, lane + 32 * h < p.k, p.vid[h]) : make_float4(0.f, 0.f, 0.f, 0.f);
    auto columns = [&](int c0, const float (&mv)[2][8]) {
        float acc[8][3];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[j][0] = fmaf(mv[0][j], z[0].x, mv[1][j] * z[1].x);
            acc[j][1] = fmaf(mv[0][j], z[0].y, mv[1][j] * z[1].y);
            acc[j][2] = fmaf(mv[0][j], z[0].z, mv[1][j] * z[1].z);
        }
        const float3 s = reduce_cols8(acc, lane);
        const int c = c0 + (lane >> 2);  // pivots are the first rows: vertex in lane c
        const int vid = __shfl_sync(0xffffffffu, p.vid[0], c & 31);
        if ((lane & 3) == 0 && c < p.k) a.x[vid] = make_float4(s.x, s.y, s.z, 0.f);
    };
    static_assert(kSmallPre % 8 == 0 && kSmallCols <= 32, "column groups");
#pragma unroll
    for (int g = 0; g < kSmallPre / 8; ++g) {
        if (8 * g >= p.k) break;
        float mv[2][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            mv[0][j] = p.mv[0][8 * g + j];
            mv[1][j] = p.mv[1][8 * g + j];
        }
        columns(8 * g, mv);
    }
    for (int c0 = kSmallPre; c0 < p.k; c0 += 8) {
        float mv[2][8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = lane + 32 * h, c = c0 + j;
                mv[h][j] = (c < p.k && row < p.m && row >= c) ? __ldg(p.M + (size_t)c * p.m + row) : 0.f;
            }
        columns(c0, mv);
    }
}

// Tiny supernodes {moff, roff, m, 1} (one pivot, at most kTinyRows rows --
// half the vertices of a grid are eliminated that way): kTinyLanes lanes,
// lane j its rows j, j + kTinyLanes, ..; the first one before the wait.
struct TinyPre {
    const float* M;
    const int* rows;
    int m, vid;
    float mv;
};

__device__ __forceinline__ void tiny_load(const CholArgs& a, int item, bool live, int j, TinyPre& p) {
    p.m = 0;
    p.vid = 0;
    p.mv = 0.f;
    p.M = a.mval;
    p.rows = a.rows;
    if (!live) return;
    const int4 h0 = __ldg(reinterpret_cast<const int4*>(a.tiny + (size_t)kItemInts * item));
    p.M = a.mval + ((int64_t)(uint32_t)h0.x | ((int64_t)h0.y << 32));
    p.rows = a.rows + h0.z;
    p.m = h0.w;
    if (j < p.m) {
        p.vid = __ldg(p.rows + j);
        p.mv = __ldg(p.M + j);
    }
}

__device__ __forceinline__ void fwd_tiny_run(const CholArgs& a, const TinyPre& p, int j) {
    const int piv = __shfl_sync(0xffffffffu, p.vid, 0, kTinyLanes);
    if (p.m == 0) return;
    const float4 r = __ldcg(&a.r[piv]);
    if (j == 0) a.y[piv] = make_float4(p.mv * r.x, p.mv * r.y, p.mv * r.z, 0.f);
    else if (j < p.m) atomicAdd(&a.r[p.vid], make_float4(-p.mv * r.x, -p.mv * r.y, -p.mv * r.z, 0.f));
    for (int i = j + kTinyLanes; i < p.m; i += kTinyLanes) {
        const float mv = __ldg(p.M + i);
        atomicAdd(&a.r[__ldg(p.rows + i)], make_float4(-mv * r.x, -mv * r.y, -mv * r.z, 0.f));
    }
}

__device__ __forceinline__ void bwd_tiny_run(const CholArgs& a, const TinyPre& p, int j) {
    float sx = 0.f, sy = 0.f, sz = 0.f;
    if (j < p.m) {
        const float4 z = z_of(a, j == 0, p.vid);
        sx = p.mv * z.x;
        sy = p.mv * z.y;
        sz = p.mv * z.z;
    }
    for (int i = j + kTinyLanes; i < p.m; i += kTinyLanes) {
        const float4 z = z_of(a, false, __ldg(p.rows + i));
        const float mv = __ldg(p.M + i);
        sx = fmaf(mv, z.x, sx);
        sy = fmaf(mv, z.y, sy);
        sz = fmaf(mv, z.z, sz);
    }
#pragma unroll
    for (int off = kTinyLanes / 2; off > 0; off >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, off);
        sy += __shfl_xor_sync(0xffffffffu, sy, off);
        sz += __shfl_xor_sync(0xffffffffu, sz, off);
    }
    if (j == 0 && p.m > 0) a.x[p.vid] = make_float4(sx, sy, sz, 0.f);
}

// Item ranges of one launch: first item and count of each kind; CTAs past
// them reset vertices (ResetArgs).
struct LevelRange {
    int b0, nb, s0, ns, t0, nt;
};
constexpr int kLevelWarps = kLevelThreads / 32;
constexpr int kTinyPerCta = kLevelThreads / kTinyLanes;
__host__ __device__ inline int small_ctas(int n) { return (n + kLevelWarps - 1) / kLevelWarps; }
__host__ __device__ inline int tiny_ctas(int n) { return (n + kTinyPerCta - 1) / kTinyPerCta; }

__global__ void __launch_bounds__(kLevelThreads, kLevelMinBlocks) k_chol_fwd_level(CholArgs a, LevelRange v) {
    __shared__ float4 rs[kLevelThreads];
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int u = blockIdx.x;
    if (u < v.nb) {
        FwdBlockPre p;
        fwd_block_load(a, v.b0 + u, p);
        pdl_wait();
        if (a.done && *a.done) return;
        fwd_block_run(a, p, rs);
        return;
    }
    u -= v.nb;
    if (u < small_ctas(v.ns)) {
        const int it = u * kLevelWarps + warp;
        SmallPre p;
        small_load(a, v.s0 + it, it < v.ns, lane, p);
        pdl_wait();
        if (a.done && *a.done) return;
        if (it < v.ns) fwd_small_run(a, p, lane, rs + 32 * warp);
        return;
    }
    u -= small_ctas(v.ns);
    const int it = u * kTinyPerCta + (int)threadIdx.x / kTinyLanes, j = threadIdx.x % kTinyLanes;
    TinyPre p;
    tiny_load(a, v.t0 + it, it < v.nt, j, p);
    pdl_wait();
    if (a.done && *a.done) return;
    fwd_tiny_run(a, p, j);
}

__global__ void __launch_bounds__(kLevelThreads, kLevelMinBlocks) k_chol_bwd_level(CholArgs a, LevelRange v, ResetArgs q) {
    __shared__ float4 zs[kLevelThreads];
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int u = blockIdx.x;
    if (u < v.nb) {
        BwdBlockPre p;
        bwd_block_load(a, v.b0 + u, p);
        pdl_wait();
        if (a.done && *a.done) return;
        bwd_block_run(a, p, zs);
        return;
    }
    u -= v.nb;
    if (u < small_ctas(v.ns)) {
        const int it = u * kLevelWarps + warp;
        SmallPre p;
        small_load(a, v.s0 + it, it < v.ns, lane, p);
        pdl_wait();
        if (a.done && *a.done) return;
        if (it < v.ns) bwd_small_run(a, p, lane);
        return;
    }
    u -= small_ctas(v.ns);
    if (u < tiny_ctas(v.nt)) {
        const int it = u * kTinyPerCta + (int)threadIdx.x / kTinyLanes, j = threadIdx.x % kTinyLanes;
        TinyPre p;
        tiny_load(a, v.t0 + it, it < v.nt, j, p);
        pdl_wait();
        if (a.done && *a.done) return;
        bwd_tiny_run(a, p, j);
        return;
    }
    // resets for the next solve: the right-hand side is dead once the forward
    // pass is done, and y_next is the buffer this solve does not use
    u -= tiny_ctas(v.nt);
    const int i = u * kLevelThreads + threadIdx.x;
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < q.nv && q.b) b = __ldg(&q.coef[i]).z != 0.f ? __ldg(&q.pin_rhs[i]) : __ldg(&q.base[i]);
    pdl_wait();
    if ((a.done && *a.done) || i >= q.nv) return;
    q.y_next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q.b) q.b[i] = b;
}

void launch_chol_solve_levels(const CholArgs& a, const std::vector<SolveLevel>& levels, cudaStream_t s,
                              const ResetArgs& reset) {
    const int nl = (int)levels.size();
    auto range = [&](int L) {
        const SolveLevel& v = levels[L];
        return LevelRange{v.blk_begin, v.blk_end - v.blk_begin, v.sml_begin, v.sml_end - v.sml_begin, v.tiny_begin,
                          v.tiny_end - v.tiny_begin};
    };
    for (int L = 0; L < nl; ++L) {
        const LevelRange r = range(L);
        const int grid = r.nb + small_ctas(r.ns) + tiny_ctas(r.nt);
        if (grid > 0) launch_pdl(k_chol_fwd_level, grid, kLevelThreads, 0, s, a, r);
    }
    bool first = reset.y_next != nullptr;
    for (int L = nl - 1; L >= 0; --L) {
        const LevelRange r = range(L);
        int grid = r.nb + small_ctas(r.ns) + tiny_ctas(r.nt);
        if (first) grid += (reset.nv + kLevelThreads - 1) / kLevelThreads;
        if (grid > 0) launch_pdl(k_chol_bwd_level, grid, kLevelThreads, 0, s, a, r, first ? reset : ResetArgs{});
        first = false;
    }
}

// ---- the whole solve in one persistent launch over the GPU.
// All CTAs are resident (cooperative launch), 128 threads each.  Per level
// and direction the CTAs stride over the level's units -- one block item,
// four small supernodes or sixteen tiny ones -- and meet at a grid-wide
// barrier.
// The barrier spins for a bounded time: past the limit it sets a sticky
// timeout word and every CTA returns at its next barrier (the step's result
// is then invalid and the engine reports PDGB_ERR_TIMEOUT).
__device__ __forceinline__ bool grid_sync(GridSync* g, unsigned& gen, unsigned expect, long long spin_limit) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = gen + 1;
        bool good = true;
        __threadfence();  // this CTA's writes before the arrival (cumulative over the CTA barrier)
        const unsigned prev = atomicAdd(&g->arrive, 1u);
        if (prev == expect - 1) {
            atomicExch(&g->arrive, 0u);
            __threadfence();
            atomicExch(&g->gen, target);
        } else {
            long long n = 0;
            for (;;) {
                if (*reinterpret_cast<volatile unsigned*>(&g->gen) == target) break;
                if (*reinterpret_cast<volatile int*>(&g->timeout)) {
                    good = false;
                    break;
                }
                if (++n > spin_limit) {
                    atomicExch(&g->timeout, 1);
                    good = false;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();  // the other CTAs' writes before any read after the barrier
        gen = target;
        ok = good && !*reinterpret_cast<volatile int*>(&g->timeout);
    }
    __syncthreads();
    return ok;
}

__global__ void __launch_bounds__(kLevelThreads) k_chol_solve_persistent(CholArgs a, const SolveLevel* __restrict__ lv,
                                                                         int nl, GridSync* bar, long long spin) {
    __shared__ float4 rs[kLevelThreads];
    if (a.done && *a.done) return;  // set before this launch: the same for every CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned expect = gridDim.x;
    unsigned gen = 0;
    for (int pass = 0; pass < 2 * nl; ++pass) {
        const bool fwd = pass < nl;
        const SolveLevel v = lv[fwd ? pass : 2 * nl - 1 - pass];
        const int nb = v.blk_end - v.blk_begin, ns = v.sml_end - v.sml_begin, nt = v.tiny_end - v.tiny_begin;
        const int nsu = small_ctas(ns), ntu = tiny_ctas(nt);
        for (int u = blockIdx.x; u < nb + nsu + ntu; u += gridDim.x) {
            __syncthreads();  // rs of the previous unit is read
            if (u < nb) {
                if (fwd) {
                    FwdBlockPre p;
                    fwd_block_load(a, v.blk_begin + u, p);
                    fwd_block_run(a, p, rs);
                } else {
                    BwdBlockPre p;
                    bwd_block_load(a, v.blk_begin + u, p);
                    bwd_block_run(a, p, rs);
                }
            } else if (u < nb + nsu) {
                const int it = (u - nb) * kLevelWarps + warp;
                SmallPre p;
                small_load(a, v.sml_begin + it, it < ns, lane, p);
                if (it < ns) {
                    if (fwd) fwd_small_run(a, p, lane, rs + 32 * warp);
                    else bwd_small_run(a, p, lane);
                }
            } else {
                const int it = (u - nb - nsu) * kTinyPerCta + (int)threadIdx.x / kTinyLanes,
                          j = threadIdx.x % kTinyLanes;
                TinyPre p;
                tiny_load(a, v.tiny_begin + it, it < nt, j, p);
                if (fwd) fwd_tiny_run(a, p, j);
                else bwd_tiny_run(a, p, j);
            }
        }
        if (pass + 1 < 2 * nl && !grid_sync(bar, gen, expect, spin)) return;
    }
}

// CTAs of the persistent solve: the resident CTAs per SM (at most
// PDGB_PERSIST_CTAS_PER_SM, default 8) times the SMs.
int persistent_grid() {
    static int grid[64] = {0};
    int dev = 0;
    PDGB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw Error{PDGB_ERR_CUDA, "device index out of range"};
    if (!grid[dev]) {
        int sms = 0, per = 0;
        PDGB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        PDGB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_chol_solve_persistent, kLevelThreads, 0));
        int cap = 8;
        if (const char* e = std::getenv("PDGB_PERSIST_CTAS_PER_SM")) cap = std::max(1, std::atoi(e));
        grid[dev] = sms * std::max(1, std::min(per, cap));
    }
    return grid[dev];
}

void launch_chol_solve_persistent(const CholArgs& a, const SolveLevel* levels, int nl, GridSync* bar,
                                  long long spin_limit, cudaStream_t s) {
    if (nl <= 0) return;
    PDGB_CUDA_TRY(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), s));  // arrival count and generation
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(persistent_grid());
    cfg.blockDim = dim3(kLevelThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PDGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_chol_solve_persistent, a, levels, nl, bar, spin_limit));
}

// Check of the grid barrier on its own: `rounds` barriers of a cooperative
// launch of `ctas` CTAs that wait for `missing` more arrivals than there are
// CTAs (0: the barrier completes; > 0: it can only time out).
__global__ void k_grid_sync_check(GridSync* bar, int rounds, int missing, long long spin) {
    unsigned gen = 0;
    for (int r = 0; r < rounds; ++r)
        if (!grid_sync(bar, gen, gridDim.x + (unsigned)missing, spin)) return;
}

void launch_grid_sync_check(GridSync* bar, int ctas, int rounds, int missing, long long spin_limit, cudaStream_t s) {
    PDGB_CUDA_TRY(cudaMemsetAsync(bar, 0, sizeof(GridSync), s));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kLevelThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PDGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_grid_sync_check, bar, rounds, missing, spin_limit));
}

// ---- one body per CTA: warps stride over the items of a level,
// __syncthreads between levels (global writes of the block become visible
// to the whole block at the barrier).  Bodies are independent, so CTAs
// never wait on each other.
__global__ void __launch_bounds__(kCtaSolveThreads) k_chol_solve_cta(CholArgs a) {
    __shared__ float4 stage[kCtaSolveThreads / 32][32];
    if (a.done && *a.done) return;
    constexpr int kWarps = kCtaSolveThreads / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int body = __ldg(&a.body_order[blockIdx.x]);
    const int L0 = __ldg(&a.body_level[body]), L1 = __ldg(&a.body_level[body + 1]);
    for (int L = L0; L < L1; ++L) {
        const int4 lv = __ldg(&a.levels[L]);
        for (int it = lv.x + warp; it < lv.y; it += kWarps)
            fwd_warp_item(a, a.fwd_items + (size_t)kItemInts * it, stage[warp], lane);
        __syncthreads();
    }
    for (int L = L1 - 1; L >= L0; --L) {
        const int4 lv = __ldg(&a.levels[L]);
        for (int it = lv.z + warp; it < lv.w; it += kWarps)
            bwd_warp_item(a, a.bwd_items + (size_t)kItemInts * it, stage[warp], lane);
        __syncthreads();
    }
}

void launch_chol_solve_cta(const CholArgs& a, int nbodies, cudaStream_t s) {
    if (nbodies > 0) k_chol_solve_cta<<<nbodies, kCtaSolveThreads, 0, s>>>(a);
}

// ---- one body per thread-block cluster: the cluster's warps stride over
// the items of a level, with a cluster barrier between levels.  The barrier
// (arrive with release, wait with acquire semantics at cluster scope) makes
// the level's global writes and atomics of every CTA of the cluster visible
// to all of them.  All CTAs of a cluster run the same level loops, so every
// thread arrives at every barrier; the hardware co-schedules the cluster.
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterSolveThreads)
    k_chol_solve_cluster(CholArgs a) {
    __shared__ float4 stage[kClusterSolveThreads / 32][32];
    if (a.done && *a.done) return;  // the flag is fixed for the kernel: uniform over the cluster
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int kWarps = kClusterSolveThreads / 32;
    constexpr int kStride = kWarps * kClusterCtas;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gw = (int)cl.block_rank() * kWarps + warp;
    const int body = __ldg(&a.body_order[blockIdx.x / kClusterCtas]);
    const int L0 = __ldg(&a.body_level[body]), L1 = __ldg(&a.body_level[body + 1]);
    for (int L = L0; L < L1; ++L) {
        const int4 lv = __ldg(&a.levels[L]);
        for (int it = lv.x + gw; it < lv.y; it += kStride)
            fwd_warp_item(a, a.fwd_items + (size_t)kItemInts * it, stage[warp], lane);
        cl.sync();
    }
    for (int L = L1 - 1; L >= L0; --L) {
        const int4 lv = __ldg(&a.levels[L]);
        for (int it = lv.z + gw; it < lv.w; it += kStride)
            bwd_warp_item(a, a.bwd_items + (size_t)kItemInts * it, stage[warp], lane);
        cl.sync();
    }
}

void launch_chol_solve_cluster(const CholArgs& a, int nbodies, cudaStream_t s) {
    if (nbodies > 0) k_chol_solve_cluster<<<nbodies * kClusterCtas, kClusterSolveThreads, 0, s>>>(a);
}

// ---- one body per cluster, everything in the cluster's shared memory.
// Each CTA stages the M_s blocks and row lists of its supernodes (stored
// back to back per CTA by the plan: one float4-wide copy each), and
// holds the vector slots of vertices v with v % 8 == its rank.  The level
// loops run the warp items of the CTA's supernodes; right-hand side, y and x
// are read and updated in whichever CTA holds the vertex (distributed shared
// memory, float atomics for the forward updates); a cluster barrier
// separates levels.  Nothing but the staging and the final x touches global
// memory.
namespace {
namespace cg = cooperative_groups;

__device__ __forceinline__ float4* dsm_slot(cg::cluster_group& cl, float4* local, int v) {
    return cl.map_shared_rank(local + (v >> 3), (unsigned)(v & (kClusterCtas - 1)));
}

__device__ __forceinline__ void dsm_add(float4* p, float x, float y, float z) {
    atomicAdd(&p->x, x);
    atomicAdd(&p->y, y);
    atomicAdd(&p->z, z);
}

// cnt4 16-byte words from global to shared memory, the whole CTA at once
__device__ __forceinline__ void dsm_copy16(void* dst, const void* src, int cnt4) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
    float4* d4 = reinterpret_cast<float4*>(dst);
    for (int t = threadIdx.x; t < cnt4; t += blockDim.x) d4[t] = __ldg(s4 + t);
}
}  // namespace

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterSolveThreads)
    k_chol_solve_dsm(CholArgs a, DsmArgs d) {
    extern __shared__ float4 dsm_base[];
    if (a.done && *a.done) return;  // the flag is fixed for the kernel: uniform over the cluster
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = kClusterSolveThreads / 32;
    const int S = d.slots;
    float4* vr = dsm_base;
    float4* vy = vr + S;
    float4* vx = vy + S;
    float4* stage = vx + S + warp * 32;
    float* Ms = reinterpret_cast<float*>(dsm_base) + d.m_area;
    int* Rs = reinterpret_cast<int*>(dsm_base) + d.r_area;
    const int m0 = d.mcopy_ptr[rank], r0c = d.rcopy_ptr[rank];
    dsm_copy16(Ms, d.mcopy + m0, (d.mcopy_ptr[rank + 1] - m0) >> 2);
    dsm_copy16(Rs, d.rcopy + r0c, (d.rcopy_ptr[rank + 1] - r0c) >> 2);
    for (int j = threadIdx.x; j < S; j += blockDim.x) {
        const int v = j * kClusterCtas + rank;
        vr[j] = v < d.n ? a.r[v] : make_float4(0.f, 0.f, 0.f, 0.f);
        vy[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        vx[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    cl.sync();
    // forward: y_s = L_ss^-1 r_s (pivot rows), r_O -= L_os L_ss^-1 r_s
    for (int L = 0; L < d.nlevels; ++L) {
        const int4 lv = d.lvl[rank * d.nlevels + L];
        for (int it = lv.x + warp; it < lv.y; it += kWarps) {
            const int* w = d.items + (size_t)kItemInts * it;
            const int moff = w[0], m = w[2], k = w[3], r0 = w[4], c0 = w[5], c1 = w[6];
            const int* rows = Rs + w[1];
            const int row = r0 + lane;
            const bool valid = row < m;
            const int cend = !valid ? c0 : (row < k ? min(c1, row + 1) : c1);
            const float* Mr = Ms + moff + row;
            float ax = 0.f, ay = 0.f, az = 0.f;
            for (int cb = c0; cb < c1; cb += 32) {
                const int nc = min(32, c1 - cb);
                __syncwarp();
                if (lane < nc) stage[lane] = *dsm_slot(cl, vr, rows[cb + lane]);
                __syncwarp();
                for (int c = cb; c < cb + nc; ++c) {
                    const float mv = c < cend ? Mr[(size_t)c * m] : 0.f;
                    const float4 v = stage[c - cb];
                    ax = fmaf(mv, v.x, ax);
                    ay = fmaf(mv, v.y, ay);
                    az = fmaf(mv, v.z, az);
                }
            }
            if (valid) {
                const int vid = rows[row];
                if (row < k) dsm_add(dsm_slot(cl, vy, vid), ax, ay, az);
                else dsm_add(dsm_slot(cl, vr, vid), -ax, -ay, -az);
            }
        }
        cl.sync();
    }
    // backward: x_s = sum_{i >= c} M_s[i, c] z_i, z = [y_pivots ; -x_offdiag]
    for (int L = d.nlevels - 1; L >= 0; --L) {
        const int4 lv = d.lvl[rank * d.nlevels + L];
        for (int it = lv.z + warp; it < lv.w; it += kWarps) {
            const int* w = d.items + (size_t)kItemInts * it;
            const int moff = w[0], m = w[2], k = w[3], c = w[4];
            const int* rows = Rs + w[1];
            const float* Mc = Ms + moff + (size_t)c * m;
            float ax = 0.f, ay = 0.f, az = 0.f;
            for (int i = c + lane; i < m; i += 32) {
                const int vid = rows[i];
                const float mv = Mc[i];
                float4 z;
                if (i < k) {
                    z = *dsm_slot(cl, vy, vid);
                } else {
                    const float4 xv = *dsm_slot(cl, vx, vid);
                    z = make_float4(-xv.x, -xv.y, -xv.z, 0.f);
                }
                ax = fmaf(mv, z.x, ax);
                ay = fmaf(mv, z.y, ay);
                az = fmaf(mv, z.z, az);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                ax += __shfl_xor_sync(0xffffffffu, ax, off);
                ay += __shfl_xor_sync(0xffffffffu, ay, off);
                az += __shfl_xor_sync(0xffffffffu, az, off);
            }
            if (lane == 0) *dsm_slot(cl, vx, rows[c]) = make_float4(ax, ay, az, 0.f);
        }
        cl.sync();
    }
    for (int j = threadIdx.x; j < S; j += blockDim.x) {
        const int v = j * kClusterCtas + rank;
        if (v < d.n) a.x[v] = vx[j];
    }
}

void launch_chol_solve_dsm(const CholArgs& a, const DsmArgs& d, size_t smem_bytes, cudaStream_t s) {
    static size_t allowed = 0;
    if (smem_bytes > allowed) {
        PDGB_CUDA_TRY(cudaFuncSetAttribute(k_chol_solve_dsm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem_bytes));
        allowed = smem_bytes;
    }
    k_chol_solve_dsm<<<kClusterCtas, kClusterSolveThreads, smem_bytes, s>>>(a, d);
}

// Cholesky-path vertex kernel after each solve (new positions in sn, written
// by the backward pass): resets b for the next local step (pinned vertices
// get the pin RHS: computeDBCLocal overwrites b, pdUtil.cu:153-158), clears
// y, and with tol > 0 runs the reference's convergence test
// (computeError, pdSolver.cu:186-191, 243-253): err = mean over the 3n
// coordinates of (sn - prev)^2, prev = sn, stop when sqrt(err) < tol.  The
// last block to finish evaluates the test and sets st->done, which makes
// every later kernel of the step return at entry.
__global__ void __launch_bounds__(256) k_chol_vertex(CholVertexArgs a) {
    __shared__ float red[8];
    __shared__ bool last;
    if (a.st->done) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float e = 0.f;
    if (i < a.nv) {
        const float4 s = a.sn[i];
        a.y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 cf = __ldg(&a.coef[i]);
        a.b[i] = cf.z != 0.f ? __ldg(&a.pin_rhs[i]) : __ldg(&a.base[i]);
        if (a.tol > 0.f) {
            const float4 p = a.prev[i];
            const float dx = p.x - s.x, dy = p.y - s.y, dz = p.z - s.z;
            e = dx * dx + dy * dy + dz * dz;
            a.prev[i] = s;
        }
    }
    if (a.tol <= 0.f) return;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) e += __shfl_xor_sync(0xffffffffu, e, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        float blk = 0.f;
        for (int w = 0; w < 8; ++w) blk += red[w];
        atomicAdd(&a.st->err_acc, blk);
        __threadfence();
        last = atomicAdd(&a.st->count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        const float total = atomicAdd(&a.st->err_acc, 0.0f);
        const float err = (float)((double)total / (3.0 * (double)a.nv));
        if (!(sqrtf(err) >= a.tol)) {
            a.st->done = 1;
            a.st->iterations = a.iteration + 1;
        }
        a.st->err_acc = 0.f;
        a.st->count = 0u;
    }
}

// Multi-request forms (serving, fixed iteration count): CTA i takes 256
// vertices of request list[i].x from list[i].y.
__global__ void __launch_bounds__(256) k_chol_vertex_multi(const CholVertexArgs* __restrict__ req,
                                                           const int2* __restrict__ list,
                                                           const int* __restrict__ count) {
    if ((int)blockIdx.x >= *count) return;
    const int2 w = list[blockIdx.x];
    const CholVertexArgs& a = req[w.x];
    const int i = w.y + threadIdx.x;
    if (i >= a.nv) return;
    a.y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 cf = __ldg(&a.coef[i]);
    a.b[i] = cf.z != 0.f ? __ldg(&a.pin_rhs[i]) : __ldg(&a.base[i]);
}

__global__ void __launch_bounds__(256) k_chol_finish_multi(const CholVertexArgs* __restrict__ req,
                                                           const int2* __restrict__ list,
                                                           const int* __restrict__ count) {
    if ((int)blockIdx.x >= *count) return;
    const int2 w = list[blockIdx.x];
    const CholVertexArgs& a = req[w.x];
    const int i = w.y + threadIdx.x;
    if (i >= a.nv) return;
    finish_vertex(a.sc, i, a.sn[i], a.dt_inv, a.x, a.v);
    a.y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

void launch_chol_vertex_multi(const CholVertexArgs* req, const int2* list, const int* count, int grid,
                              cudaStream_t s) {
    if (grid > 0) k_chol_vertex_multi<<<grid, 256, 0, s>>>(req, list, count);
}

void launch_chol_finish_multi(const CholVertexArgs* req, const int2* list, const int* count, int grid,
                              cudaStream_t s) {
    if (grid > 0) k_chol_finish_multi<<<grid, 256, 0, s>>>(req, list, count);
}

// After the iterations: velocity / position update (updateVelPos,
// pdUtil.cu:180-193), X <- XTilde (pdSolver.cu:227) and the fixed-body
// correction of XTilde and V (pdSolver.cu:228-231).
__global__ void __launch_bounds__(256) k_chol_finish(CholVertexArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nv) return;
    finish_vertex(a.sc, i, a.sn[i], a.dt_inv, a.x, a.v);
    a.y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// ---- iterative refinement
__global__ void __launch_bounds__(256) k_copy_rhs(int nv, const float4* __restrict__ b, float4* bsave,
                                                  const int* done) {
    if (done && *done) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nv) bsave[i] = b[i];
}

// One warp per row: r = bsave - K x0 accumulated in double over the row's
// nonzeros (lanes stride the row, then a warp reduction).
__global__ void __launch_bounds__(256) k_refine_residual(RefineArgs a) {
    if (a.done && *a.done) return;
    const int row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= a.nv) return;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int e = __ldg(&a.rowptr[row]) + lane; e < __ldg(&a.rowptr[row + 1]); e += 32) {
        const double kv = __ldg(&a.val[e]);
        const float4 xv = a.x0[__ldg(&a.colind[e])];
        sx = fma(kv, (double)xv.x, sx);
        sy = fma(kv, (double)xv.y, sy);
        sz = fma(kv, (double)xv.z, sz);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, off);
        sy += __shfl_xor_sync(0xffffffffu, sy, off);
        sz += __shfl_xor_sync(0xffffffffu, sz, off);
    }
    if (lane == 0) {
        const float4 b = a.bsave[row];
        a.b[row] = make_float4((float)((double)b.x - sx), (float)((double)b.y - sy), (float)((double)b.z - sz), 0.f);
        a.y[row] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__global__ void __launch_bounds__(256) k_refine_update(RefineArgs a) {
    if (a.done && *a.done) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nv) return;
    const float4 x = a.x[i], d = a.dx[i];
    a.x[i] = make_float4(x.x + d.x, x.y + d.y, x.z + d.z, 0.f);
}

void launch_copy_rhs(int nv, const float4* b, float4* bsave, const int* done, cudaStream_t s) {
    if (nv > 0) k_copy_rhs<<<(nv + 255) / 256, 256, 0, s>>>(nv, b, bsave, done);
}
void launch_refine_residual(const RefineArgs& a, cudaStream_t s) {
    if (a.nv > 0) k_refine_residual<<<(a.nv + 7) / 8, 256, 0, s>>>(a);
}
void launch_refine_update(const RefineArgs& a, cudaStream_t s) {
    if (a.nv > 0) k_refine_update<<<(a.nv + 255) / 256, 256, 0, s>>>(a);
}

void launch_chol_vertex(const CholVertexArgs& a, cudaStream_t s) {
    const int blocks = (a.nv + 255) / 256;
    if (blocks) k_chol_vertex<<<blocks, 256, 0, s>>>(a);
}

void launch_chol_finish(const CholVertexArgs& a, cudaStream_t s) {
    const int blocks = (a.nv + 255) / 256;
    if (blocks) k_chol_finish<<<blocks, 256, 0, s>>>(a);
}

}  // namespace pdgb
