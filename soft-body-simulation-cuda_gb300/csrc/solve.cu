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
// (pdl.cuh): each, before its wait,
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
    const int ld = m_stride(m, k);
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
            for (int q = 0; q < 8; ++q) mv[q] = (c + q < cend) ? __ldg(Mr + (size_t)(c + q) * ld) : 0.f;
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
    const float* Mc = a.mval + moff + (size_t)c * m_stride(m, k);
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
// (kLevelThreads threads) take, by index, first the level's block items (a
// 128 x 32 tile of M_s, 32 rows a warp), then its small supernodes (one warp
// each), then its tiny ones (kTinyLanes lanes each), then -- in the solve's
// first backward launch, when asked -- the resets of the next iteration's
// vectors.
//
// What bounds a narrow level is the chain launch -> descriptor -> factor
// entries -> gather -> products -> scatter, each a trip to L2 or HBM; what
// bounds a wide one is how many bytes its resident CTAs have on the way and
// how many shared-memory accesses they queue.  So a tile's entries are copied
// 16 bytes a lane, asynchronously, before the grid dependency wait: 16 KB a
// CTA that hold no registers, 11 CTAs on an SM.  A lane copies and uses 4 rows
// of 8 columns: forward it needs one staged right-hand side for 12 products,
// backward its 4 rows' z once for all 96.  After the wait come one gather, the
// products, a few exchanges and the scatter.  A warp uses only its own part of
// the shared memory until the backward tile's last sum.
// Holding the tile in registers instead (8 and 7 CTAs) is 4 to 8 % slower on
// the 40^3 cube and on a batch of 128 bodies; one row or column a lane takes
// twice the shared-memory accesses and sums chains of 32.
__device__ __forceinline__ void cp_async16(void* dst, const float* src, bool live) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct Supernode {
    const float* M;   // M_s, column major, columns ld apart
    const int* rows;
    int m, k, ld;
};

__device__ __forceinline__ Supernode supernode(const CholArgs& a, const int4 h0, int k) {
    const int64_t moff = (int64_t)(uint32_t)h0.x | ((int64_t)h0.y << 32);
    return Supernode{a.mval + moff, a.rows + h0.z, h0.w, k, m_stride(h0.w, k)};
}

// Block item {moff, roff, m, k, r0, c0, c1}: warp w takes the rows
// r0 + 32 w .. + 32 of the tile; lane l holds the rows rw + 4 (l & 7) .. + 4
// of the columns c0 + 4 q + (l >> 3), q < 8 (zero past the last row or
// column), the vertex of row rw + l and that of pivot column c0 + l.
constexpr int kLaneCols = kTileCols / 4;
struct TilePre {
    int vid, cvid;    // -1: none
    int row, k, m;
    bool first;       // the tile holds the first pivot columns
};

__device__ __forceinline__ void tile_load(const CholArgs& a, int item, float4* tile, TilePre& p) {
    const int4* w = reinterpret_cast<const int4*>(a.blocks + (size_t)kItemInts * item);
    const int4 h0 = __ldg(w), h1 = __ldg(w + 1);
    const Supernode s = supernode(a, h0, h1.x);
    const int r0 = h1.y, c0 = h1.z, c1 = h1.w;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rw = r0 + 32 * warp, i = rw + 4 * (lane & 7), cl = c0 + (lane >> 3);
    // rows above the first column hold zeros, and so does the padding of a column
    const int cend = i < s.m && i + 3 >= c0 ? c1 : c0;
    const float* col = s.M + (size_t)cl * s.ld + i;
    float4* t = tile + 32 * kLaneCols * warp + lane;
#pragma unroll
    for (int q = 0; q < kLaneCols; ++q) {
        const bool live = cl + 4 * q < cend;
        cp_async16(t + 32 * q, live ? col + (size_t)(4 * q) * s.ld : a.mval, live);
    }
    p.row = rw + lane;
    p.k = s.k;
    p.m = s.m;
    p.first = c0 == 0;
    p.vid = p.row < s.m && p.row >= c0 ? __ldg(&s.rows[p.row]) : -1;
    p.cvid = c0 + lane < c1 ? __ldg(&s.rows[c0 + lane]) : -1;
}

// Halving exchange between the lanes that differ in bit `off`: each keeps
// half of its 2 n values (the upper half where the bit is set) and adds the
// partner's.
template <int n>
__device__ __forceinline__ void halve(float3 (&v)[2 * n], int lane, int off) {
    const bool up = lane & off;
#pragma unroll
    for (int j = 0; j < n; ++j) {
        const float3 give = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
        v[j] = make_float3(keep.x + __shfl_xor_sync(0xffffffffu, give.x, off),
                           keep.y + __shfl_xor_sync(0xffffffffu, give.y, off),
                           keep.z + __shfl_xor_sync(0xffffffffu, give.z, off));
    }
}

__device__ __forceinline__ void fma3(float3& s, float m, const float4& v) {
    s.x = fmaf(m, v.x, s.x);
    s.y = fmaf(m, v.y, s.y);
    s.z = fmaf(m, v.z, s.z);
}

// Forward: each lane's four row sums over its eight columns, exchanged so
// that lane l ends with the row 4 (l & 7) + 2 (l >> 3 & 1) + (l >> 4); the sum
// goes into y (pivot rows; stored where no other tile adds to it) or out of r
// (ancestor rows, pivots of later levels).  The backward pass adds the partial
// sums of a supernode with more rows than a tile into x, which is cleared
// here.
__device__ __forceinline__ void fwd_tile_run(const CholArgs& a, const TilePre& p, const float4* tile, float4* vec) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4* rs = vec + 32 * warp;
    rs[lane] = p.cvid >= 0 ? __ldcg(&a.r[p.cvid]) : make_float4(0.f, 0.f, 0.f, 0.f);
    const int mine = 4 * (lane & 7) + 2 * (lane >> 3 & 1) + (lane >> 4);
    const int vid = __shfl_sync(0xffffffffu, p.vid, mine), row = p.row - lane + mine;
    cp_async_wait();
    __syncwarp();
    const float4* t4 = tile + 32 * kLaneCols * warp + lane;
    float3 s[4] = {};
#pragma unroll
    for (int q = 0; q < kLaneCols; ++q) {
        const float4 v = rs[4 * q + (lane >> 3)], m = t4[32 * q];
        fma3(s[0], m.x, v);
        fma3(s[1], m.y, v);
        fma3(s[2], m.z, v);
        fma3(s[3], m.w, v);
    }
    halve<2>(s, lane, 8);
    float3 t[2] = {s[0], s[1]};
    halve<1>(t, lane, 16);
    if (vid < 0) return;
    if (row >= p.k) {
        atomicAdd(&a.r[vid], make_float4(-t[0].x, -t[0].y, -t[0].z, 0.f));
        return;
    }
    const float4 sum = make_float4(t[0].x, t[0].y, t[0].z, 0.f);
    if (row < kTileCols) a.y[vid] = sum;
    else atomicAdd(&a.y[vid], sum);
    if (p.first && p.m > kTileRows) a.x[vid] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// z of a row: y at a pivot, -x at an ancestor.
__device__ __forceinline__ float4 z_of(const CholArgs& a, bool pivot, int vid) {
    if (pivot) return __ldcg(&a.y[vid]);
    const float4 v = __ldcg(&a.x[vid]);
    return make_float4(-v.x, -v.y, -v.z, 0.f);
}

// Backward: each lane's eight column sums over its four rows, exchanged so
// that one lane holds the warp's sum of a column, then one warp adds the four
// warps' sums, which are stored, or added where the supernode's rows take
// several tiles.
__device__ __forceinline__ void bwd_tile_run(const CholArgs& a, const TilePre& p, const float4* tile, float4* vec) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4* zs = vec + 32 * warp;
    zs[lane] = p.vid >= 0 ? z_of(a, p.row < p.k, p.vid) : make_float4(0.f, 0.f, 0.f, 0.f);
    cp_async_wait();
    __syncwarp();
    const int r = 4 * (lane & 7);
    const float4 z0 = zs[r], z1 = zs[r + 1], z2 = zs[r + 2], z3 = zs[r + 3];
    const float4* t4 = tile + 32 * kLaneCols * warp + lane;
    float3 s[8];
#pragma unroll
    for (int q = 0; q < kLaneCols; ++q) {
        const float4 m = t4[32 * q];
        s[q] = make_float3(m.x * z0.x, m.x * z0.y, m.x * z0.z);
        fma3(s[q], m.y, z1);
        fma3(s[q], m.z, z2);
        fma3(s[q], m.w, z3);
    }
    halve<4>(s, lane, 4);
    float3 u[4] = {s[0], s[1], s[2], s[3]};
    halve<2>(u, lane, 2);
    float3 t[2] = {u[0], u[1]};
    halve<1>(t, lane, 1);
    __syncwarp();  // every lane has read its z
    // the lane kept q = l & 7 of its columns 4 q + (l >> 3)
    zs[4 * (lane & 7) + (lane >> 3)] = make_float4(t[0].x, t[0].y, t[0].z, 0.f);
    __syncthreads();
    if (warp != 0 || p.cvid < 0) return;
    static_assert(kLevelThreads == 128, "four partial sums");
    const float4 q0 = vec[lane], q1 = vec[32 + lane], q2 = vec[64 + lane], q3 = vec[96 + lane];
    const float4 sum = make_float4((q0.x + q1.x) + (q2.x + q3.x), (q0.y + q1.y) + (q2.y + q3.y),
                                   (q0.z + q1.z) + (q2.z + q3.z), 0.f);
    if (p.m > kTileRows) atomicAdd(&a.x[p.cvid], sum);
    else a.x[p.cvid] = sum;
}

// One column's sum over its first 4 n rows in shared memory (16-byte aligned)
// against z, four rows a load, each row of the four in a chain of its own.
__device__ __forceinline__ float3 column_sum(const float* col, const float4* z, int n) {
    float3 s[4] = {};
#pragma unroll 4
    for (int q = 0; q < n; ++q) {
        const float4 mq = *reinterpret_cast<const float4*>(col + 4 * q);
        fma3(s[0], mq.x, z[4 * q]);
        fma3(s[1], mq.y, z[4 * q + 1]);
        fma3(s[2], mq.z, z[4 * q + 2]);
        fma3(s[3], mq.w, z[4 * q + 3]);
    }
    return make_float3((s[0].x + s[1].x) + (s[2].x + s[3].x), (s[0].y + s[1].y) + (s[2].y + s[3].y),
                       (s[0].z + s[1].z) + (s[2].z + s[3].z));
}

// Small supernodes {moff, roff, m, k} (is_small): one warp copies the whole
// block; forward lane = rows l and l + 32, backward lane = column.
struct SmallPre {
    int m, k, ld, vid[2];
};

__device__ __forceinline__ void small_load(const CholArgs& a, int item, float* blk, int lane, SmallPre& p) {
    const int4* w = reinterpret_cast<const int4*>(a.small + (size_t)kItemInts * item);
    const int4 h0 = __ldg(w);
    const Supernode s = supernode(a, h0, __ldg(a.small + (size_t)kItemInts * item + 4));
    for (int e = 4 * lane; e < s.k * s.ld; e += 128) cp_async16(blk + e, s.M + e, true);
    p.m = s.m;
    p.k = s.k;
    p.ld = s.ld;
#pragma unroll
    for (int h = 0; h < 2; ++h) p.vid[h] = lane + 32 * h < s.m ? __ldg(&s.rows[lane + 32 * h]) : -1;
}

__device__ __forceinline__ void fwd_small_run(const CholArgs& a, const SmallPre& p, const float* blk, float4* rs,
                                              int lane) {
    rs[lane] = lane < p.k ? __ldcg(&a.r[p.vid[0]]) : make_float4(0.f, 0.f, 0.f, 0.f);
    cp_async_wait();
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (p.vid[h] < 0) continue;
        const int row = lane + 32 * h;
        float sx = 0.f, sy = 0.f, sz = 0.f;
        const float* t = blk + row;
#pragma unroll 4
        for (int c = 0; c < p.k; ++c) {
            const float mv = t[c * p.ld];
            const float4 v = rs[c];
            sx = fmaf(mv, v.x, sx);
            sy = fmaf(mv, v.y, sy);
            sz = fmaf(mv, v.z, sz);
        }
        if (row < p.k) a.y[p.vid[h]] = make_float4(sx, sy, sz, 0.f);
        else atomicAdd(&a.r[p.vid[h]], make_float4(-sx, -sy, -sz, 0.f));
    }
}

__device__ __forceinline__ void bwd_small_run(const CholArgs& a, const SmallPre& p, float* blk, int lane) {
    float4* zs = reinterpret_cast<float4*>(blk + kSmallFloats);
#pragma unroll
    for (int h = 0; h < 2; ++h)
        zs[lane + 32 * h] =
            p.vid[h] >= 0 ? z_of(a, lane + 32 * h < p.k, p.vid[h]) : make_float4(0.f, 0.f, 0.f, 0.f);
    cp_async_wait();
    __syncwarp();
    if (lane >= p.k) return;
    const float3 s = column_sum(blk + lane * p.ld, zs, (p.m + 3) / 4);
    a.x[p.vid[0]] = make_float4(s.x, s.y, s.z, 0.f);
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

// Resets of vertex i for the next solve (ResetArgs).  The right-hand side it
// clears is dead: the forward pass is done, or it is another buffer.
__device__ __forceinline__ void reset_vertex(const CholArgs& a, const ResetArgs& q, int i) {
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < q.nv && q.b) b = __ldg(&q.coef[i]).z != 0.f ? __ldg(&q.pin_rhs[i]) : __ldg(&q.base[i]);
    pdl_wait();
    pdl_trigger();
    if ((a.done && *a.done) || i >= q.nv) return;
    if (q.y_next) q.y_next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q.b) q.b[i] = b;
}

__global__ void __launch_bounds__(kLevelThreads, kFwdBlocks) k_chol_fwd_level(CholArgs a, LevelRange v) {
    extern __shared__ float4 tile[];  // a tile, or kWarpFloats a warp
    float* blocks = reinterpret_cast<float*>(tile);
    __shared__ float4 vec[kLevelWarps * 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int u = blockIdx.x;
    if (u < v.nb) {
        TilePre p;
        tile_load(a, v.b0 + u, tile, p);
        pdl_wait();
        pdl_trigger();
        if (a.done && *a.done) {
            cp_async_wait();
            return;
        }
        fwd_tile_run(a, p, tile, vec);
        return;
    }
    u -= v.nb;
    if (u < small_ctas(v.ns)) {
        const int it = u * kLevelWarps + warp;
        SmallPre p{};
        if (it < v.ns) small_load(a, v.s0 + it, blocks + kWarpFloats * warp, lane, p);
        pdl_wait();
        pdl_trigger();
        if (a.done && *a.done) {
            cp_async_wait();
            return;
        }
        if (it < v.ns) fwd_small_run(a, p, blocks + kWarpFloats * warp, vec + 32 * warp, lane);
        return;
    }
    u -= small_ctas(v.ns);
    const int it = u * kTinyPerCta + (int)threadIdx.x / kTinyLanes, j = threadIdx.x % kTinyLanes;
    TinyPre p;
    tiny_load(a, v.t0 + it, it < v.nt, j, p);
    pdl_wait();
    pdl_trigger();
    if (a.done && *a.done) return;
    fwd_tiny_run(a, p, j);
}

__global__ void __launch_bounds__(kLevelThreads, kBwdBlocks) k_chol_bwd_level(CholArgs a, LevelRange v, ResetArgs q) {
    extern __shared__ float4 tile[];  // a tile, or kWarpFloats a warp
    float* blocks = reinterpret_cast<float*>(tile);
    __shared__ float4 vec[kLevelWarps * 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int u = blockIdx.x;
    if (u < v.nb) {
        TilePre p;
        tile_load(a, v.b0 + u, tile, p);
        pdl_wait();
        pdl_trigger();
        if (a.done && *a.done) {
            cp_async_wait();
            return;
        }
        bwd_tile_run(a, p, tile, vec);
        return;
    }
    u -= v.nb;
    if (u < small_ctas(v.ns)) {
        const int it = u * kLevelWarps + warp;
        SmallPre p{};
        if (it < v.ns) small_load(a, v.s0 + it, blocks + kWarpFloats * warp, lane, p);
        pdl_wait();
        pdl_trigger();
        if (a.done && *a.done) {
            cp_async_wait();
            return;
        }
        if (it < v.ns) bwd_small_run(a, p, blocks + kWarpFloats * warp, lane);
        return;
    }
    u -= small_ctas(v.ns);
    if (u < tiny_ctas(v.nt)) {
        const int it = u * kTinyPerCta + (int)threadIdx.x / kTinyLanes, j = threadIdx.x % kTinyLanes;
        TinyPre p;
        tiny_load(a, v.t0 + it, it < v.nt, j, p);
        pdl_wait();
        pdl_trigger();
        if (a.done && *a.done) return;
        bwd_tiny_run(a, p, j);
        return;
    }
    reset_vertex(a, q, (u - tiny_ctas(v.nt)) * kLevelThreads + threadIdx.x);
}

// x = S r over the root's pivots, S its inverse: a CTA takes 8 rows (which are
// 8 rows of every column, 32 bytes of each) and copies them, 32 k bytes, to
// shared memory before the grid dependency wait: the whole inverse is on the
// SMs while the kernel before it still runs.  After the wait come the k
// right-hand sides, 12 products a column and half, and a tree over the CTA.
// What bounds it is the gather (k / 256 float4 a thread from L2) and the
// launch: an iteration of a dense 343-vertex body 6.3 -> 5.1 us against the two
// passes over the triangle.
constexpr int kRootThreads = 256;
constexpr int kRootRows = 8;
constexpr int kRootWarps = kRootThreads / 32;
constexpr int kRootGather = (kRootCols + kRootThreads - 1) / kRootThreads;
size_t root_smem(int k) { return (size_t)k * 3 * sizeof(float4) + kRootWarps * kRootRows * sizeof(float4); }

__global__ void __launch_bounds__(kRootThreads, 2) k_chol_root(CholArgs a, RootArgs q, int tiles, ResetArgs z) {
    extern __shared__ float4 tile[];  // [k][2], then r [k], then the warps' sums
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if ((int)blockIdx.x >= tiles) {
        reset_vertex(a, z, ((int)blockIdx.x - tiles) * kRootThreads + t);
        return;
    }
    float4* rs = tile + 2 * q.k;
    float4* part = rs + q.k;
    const int row0 = kRootRows * blockIdx.x, half = t & 1;
    const bool live = row0 + 4 * half < q.k;
    for (int c = t >> 1; c < q.k; c += kRootThreads / 2)
        cp_async16(tile + 2 * c + half, live ? q.inv + (size_t)c * q.ld + row0 + 4 * half : q.inv, live);
    int vid[kRootGather];
#pragma unroll
    for (int g = 0; g < kRootGather; ++g) vid[g] = t + kRootThreads * g < q.k ? __ldg(&q.rows[t + kRootThreads * g]) : -1;
    const int xv = t < kRootRows && row0 + t < q.k ? __ldg(&q.rows[row0 + t]) : -1;
    pdl_wait();
    pdl_trigger();
    const bool skip = a.done && *a.done;  // the same for every thread
    if (!skip) {
        float4 v[kRootGather];
#pragma unroll
        for (int g = 0; g < kRootGather; ++g) v[g] = vid[g] >= 0 ? __ldcg(&a.r[vid[g]]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int g = 0; g < kRootGather; ++g)
            if (vid[g] >= 0) rs[t + kRootThreads * g] = v[g];
    }
    cp_async_wait();
    if (skip) return;
    __syncthreads();
    float3 s[4] = {};
    for (int c = t >> 1; c < q.k; c += kRootThreads / 2) {
        const float4 m = tile[2 * c + half], v = rs[c];
        fma3(s[0], m.x, v);
        fma3(s[1], m.y, v);
        fma3(s[2], m.z, v);
        fma3(s[3], m.w, v);
    }
    // lanes of one parity hold the same four rows
    halve<2>(s, lane, 16);
    float3 u[2] = {s[0], s[1]};
    halve<1>(u, lane, 8);
    float3 w = u[0];
#pragma unroll
    for (int off = 4; off > 1; off >>= 1) {
        w.x += __shfl_xor_sync(0xffffffffu, w.x, off);
        w.y += __shfl_xor_sync(0xffffffffu, w.y, off);
        w.z += __shfl_xor_sync(0xffffffffu, w.z, off);
    }
    if ((lane & 6) == 0)
        part[kRootRows * warp + 4 * half + 2 * (lane >> 4) + (lane >> 3 & 1)] = make_float4(w.x, w.y, w.z, 0.f);
    __syncthreads();
    if (xv < 0) return;
    float3 x = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int g = 0; g < kRootWarps; ++g) {
        const float4 e = part[kRootRows * g + t];
        x = make_float3(x.x + e.x, x.y + e.y, x.z + e.z);
    }
    a.x[xv] = make_float4(x.x, x.y, x.z, 0.f);
}

void launch_chol_solve_levels(const CholArgs& a, const std::vector<SolveLevel>& levels, cudaStream_t s,
                              const ResetArgs& reset, const RootArgs& root) {
    const int nl = (int)levels.size();
    auto smem = [](const LevelRange& r) {
        return sizeof(float) * (r.ns > 0 ? kLevelWarps * kWarpFloats : r.nb > 0 ? kTileRows * kTileCols : 0);
    };
    auto range = [&](int L) {
        const SolveLevel& v = levels[L];
        return LevelRange{v.blk_begin, v.blk_end - v.blk_begin, v.sml_begin, v.sml_end - v.sml_begin, v.tiny_begin,
                          v.tiny_end - v.tiny_begin};
    };
    const int top = root.k > 0 ? nl - 1 : nl;  // levels of the two passes: the root, alone on its own, has the product
    for (int L = 0; L < top; ++L) {
        const LevelRange r = range(L);
        const int grid = r.nb + small_ctas(r.ns) + tiny_ctas(r.nt);
        if (grid > 0) launch_pdl(k_chol_fwd_level, grid, kLevelThreads, smem(r), s, a, r);
    }
    bool first = reset.nv > 0;
    if (root.k > 0) {
        // with no level below the root the product does the resets
        const int tiles = (root.k + kRootRows - 1) / kRootRows;
        const bool here = first && top == 0;
        const int grid = tiles + (here ? (reset.nv + kRootThreads - 1) / kRootThreads : 0);
        launch_pdl(k_chol_root, grid, kRootThreads, root_smem(root.k), s, a, root, tiles, here ? reset : ResetArgs{});
    }
    for (int L = top - 1; L >= 0; --L) {
        const LevelRange r = range(L);
        int grid = r.nb + small_ctas(r.ns) + tiny_ctas(r.nt);
        if (first) grid += (reset.nv + kLevelThreads - 1) / kLevelThreads;
        if (grid > 0)
            launch_pdl(k_chol_bwd_level, grid, kLevelThreads, smem(r), s, a, r, first ? reset : ResetArgs{});
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
    __shared__ float4 tile[kLevelWarps * kWarpFloats / 4];
    float* blocks = reinterpret_cast<float*>(tile);
    __shared__ float4 vec[kLevelWarps * 32];
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
            __syncthreads();  // the previous unit's shared memory is read
            if (u < nb) {
                TilePre p;
                tile_load(a, v.blk_begin + u, tile, p);
                if (fwd) fwd_tile_run(a, p, tile, vec);
                else bwd_tile_run(a, p, tile, vec);
            } else if (u < nb + nsu) {
                const int it = (u - nb) * kLevelWarps + warp;
                if (it < ns) {
                    SmallPre p;
                    small_load(a, v.sml_begin + it, blocks + kWarpFloats * warp, lane, p);
                    if (fwd) fwd_small_run(a, p, blocks + kWarpFloats * warp, vec + 32 * warp, lane);
                    else bwd_small_run(a, p, blocks + kWarpFloats * warp, lane);
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
// never wait on each other.  What bounds a body is the chain of its items: a batch
// has two bodies an SM (32 registers and a few spilled; 4,096 of 4^3 take 3.7 ms a
// step of ten iterations, 9.5 with one), a single body all the registers that the
// eight entries a lane has on the way want (58; with the 46 that the compiler
// stopped at, 10^3 took 982 us instead of 802).
template <int kPerSm>
__global__ void __launch_bounds__(kCtaSolveThreads, kPerSm) k_chol_solve_cta(CholArgs a) {
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
    if (nbodies == 1) k_chol_solve_cta<1><<<1, kCtaSolveThreads, 0, s>>>(a);
    else if (nbodies > 1) k_chol_solve_cta<2><<<nbodies, kCtaSolveThreads, 0, s>>>(a);
}

// ---- one body per thread-block cluster: the cluster's warps stride over
// the items of a level, with a cluster barrier between levels.  The barrier
// (arrive with release, wait with acquire semantics at cluster scope) makes
// the level's global writes and atomics of every CTA of the cluster visible
// to all of them.  All CTAs of a cluster run the same level loops, so every
// thread arrives at every barrier; the hardware co-schedules the cluster.
// Without a bound on the CTAs an SM the compiler keeps to 40 registers, too few
// for the eight entries a lane has on the way: with two an SM (58 registers) a
// 16^3, a 28^3 and a dense 10^3 body take 1,272, 7,265 and 565 us a step instead
// of 1,645, 9,300 and 726.
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterSolveThreads, 2)
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

// ---- iterative refinement.  The three kernels are links of the same chain of
// dependent launches as the levels (pdl.cuh).
__global__ void __launch_bounds__(256) k_copy_rhs(int nv, const float4* __restrict__ b, float4* bsave,
                                                  const int* done) {
    pdl_wait();
    pdl_trigger();
    if (done && *done) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nv) bsave[i] = b[i];
}

// r = bsave - K x0 accumulated in double over the row's nonzeros (7 to 27 on
// a tet mesh), kRowLanes lanes a row.  FP64 runs at two lanes a clock and SM
// whether they hold a value or not: with a warp a row, most of its adds were
// of the reduction and of idle lanes (12.5 us on 5,760 rows).  Row bounds,
// indices and values are read before the wait.
constexpr int kRowLanes = 4;
constexpr int kRowPre = 4;  // entries a lane holds before the wait
__global__ void __launch_bounds__(128) k_refine_residual(RefineArgs a) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = t / kRowLanes, lane = t % kRowLanes;
    const bool live = row < a.nv;
    const int e0 = live ? __ldg(&a.rowptr[row]) + lane : 0, e1 = live ? __ldg(&a.rowptr[row + 1]) : 0;
    double kv[kRowPre];
    int ci[kRowPre];
#pragma unroll
    for (int q = 0; q < kRowPre; ++q) {
        const int e = e0 + kRowLanes * q;
        kv[q] = e < e1 ? __ldg(&a.val[e]) : 0.0;
        ci[q] = e < e1 ? __ldg(&a.colind[e]) : -1;
    }
    pdl_wait();
    pdl_trigger();
    if (a.done && *a.done) return;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    auto add = [&](double k, const float4& x) {
        sx = fma(k, (double)x.x, sx);
        sy = fma(k, (double)x.y, sy);
        sz = fma(k, (double)x.z, sz);
    };
    float4 xv[kRowPre];
#pragma unroll
    for (int q = 0; q < kRowPre; ++q) xv[q] = ci[q] >= 0 ? __ldcg(&a.x0[ci[q]]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < kRowPre; ++q)
        if (ci[q] >= 0) add(kv[q], xv[q]);
    for (int e = e0 + kRowLanes * kRowPre; e < e1; e += kRowLanes) add(__ldg(&a.val[e]), __ldcg(&a.x0[__ldg(&a.colind[e])]));
#pragma unroll
    for (int off = kRowLanes / 2; off > 0; off >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, off);
        sy += __shfl_xor_sync(0xffffffffu, sy, off);
        sz += __shfl_xor_sync(0xffffffffu, sz, off);
    }
    if (live && lane == 0) {
        const float4 b = a.bsave[row];
        a.b[row] = make_float4((float)((double)b.x - sx), (float)((double)b.y - sy), (float)((double)b.z - sz), 0.f);
        a.y[row] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__global__ void __launch_bounds__(256) k_refine_update(RefineArgs a) {
    pdl_wait();
    pdl_trigger();
    if (a.done && *a.done) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nv) return;
    const float4 x = a.x[i], d = a.dx[i];
    a.x[i] = make_float4(x.x + d.x, x.y + d.y, x.z + d.z, 0.f);
}

void launch_copy_rhs(int nv, const float4* b, float4* bsave, const int* done, cudaStream_t s) {
    if (nv > 0) launch_pdl(k_copy_rhs, (nv + 255) / 256, 256, 0, s, nv, b, bsave, done);
}
void launch_refine_residual(const RefineArgs& a, cudaStream_t s) {
    constexpr int kRows = 128 / kRowLanes;
    if (a.nv > 0) launch_pdl(k_refine_residual, (a.nv + kRows - 1) / kRows, 128, 0, s, a);
}
void launch_refine_update(const RefineArgs& a, cudaStream_t s) {
    if (a.nv > 0) launch_pdl(k_refine_update, (a.nv + 255) / 256, 256, 0, s, a);
}

void launch_chol_vertex(const CholVertexArgs& a, cudaStream_t s) {
    const int blocks = (a.nv + 255) / 256;
    if (blocks) k_chol_vertex<<<blocks, 256, 0, s>>>(a);
}

void launch_chol_finish(const CholVertexArgs& a, cudaStream_t s) {
    const int blocks = (a.nv + 255) / 256;
    if (blocks) k_chol_finish<<<blocks, 256, 0, s>>>(a);
}

// The kernels between two local steps of a chain all ask for one split of L1 and
// shared memory (19 x 11 x 23 refined twice, two steps: 930 -> 882 us); the
// local step gains more from its L1 (10^3: 186 us as it is, 197 with the rest).
void configure_chol_kernels() {
    PDGB_CUDA_TRY(cudaFuncSetAttribute(k_chol_root, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)root_smem(kRootCols)));
    prefer_shared(k_chol_root);
    prefer_shared(k_chol_fwd_level);
    prefer_shared(k_chol_bwd_level);
    prefer_shared(k_copy_rhs);
    prefer_shared(k_refine_residual);
    prefer_shared(k_refine_update);
    prefer_shared(k_chol_vertex);
    prefer_shared(k_chol_finish);
}

}  // namespace pdgb
