// FP64 numeric factorisation of the PD system on the GPU (supernodal,
// multifrontal), run once per system matrix.
//
// The reference factors A = K (x) I_3 on the GPU with cuSOLVER's low-level
// sparse Cholesky in FP32 (cusolverSpScsrcholFactor, cholesky.cu:152-157).
// Here the scalar K is factored in FP64 with the engine's own dense kernels,
// level by level of the supernodal elimination tree (leaves first; all
// bodies of a batch together), and the result is stored as the FP32 blocks
// M_s = [L_ss^-1 ; L_os L_ss^-1] that the triangular solves use (solve.cu).
//
// Per level:
//   k_fz     zero the level's fronts (memory of finished fronts is reused)
//   k_fk     entries of K in the pivot columns of each front
//   k_fea    extend-add: the children's Schur complements into the front
//   per panel of 32 pivot columns:
//     k_panel  the diagonal block's factor and inverse, the panel's rows of L
//              and of M_s
//     k_trail  trailing update of the front's lower triangle and of M_s
// A non-positive pivot is recorded in a status word; the host raises
// PDGB_ERR_NOT_SPD after the last level.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "cholesky.h"
#include "engine.h"
#include "panel.h"
#include "pdl.cuh"

namespace pdgb {
namespace {

constexpr int kNB = 32;           // panel width and tile size
constexpr int kFillCtas = 304;    // two CTAs an SM: launches with fewer are split further
constexpr int kZeroChunk = 1 << 16;

struct FDev {
    double* pool;
    const int64_t* foff;
    const int* sk;
    const int* sm;
    const int64_t* moff;
    float* mval;
    const int* child_ptr;
    const int* child;
    const int* rel_ptr;
    const int* rel;
    const int* kptr;
    const int* kpos;
    const double* kval;
    int* status;
};

__device__ __forceinline__ int lower_bound_dev(const int* a, int n, int x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Zeroes the front and M_s block of list[blockIdx.x], kZeroChunk doubles per CTA.
__global__ void __launch_bounds__(256) k_fz(FDev d, const int* __restrict__ list) {
    const int s = list[blockIdx.x];
    const int64_t m = d.sm[s], k = d.sk[s];
    const int64_t tot = m * m + m * k;
    const int64_t b0 = (int64_t)blockIdx.y * kZeroChunk;
    if (b0 >= tot) return;
    const int64_t b1 = b0 + kZeroChunk < tot ? b0 + kZeroChunk : tot;
    double* F = d.pool + d.foff[s];
    for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) F[i] = 0.0;
}

// Entries of K in the pivot columns (positions are distinct within a front).
__global__ void __launch_bounds__(256) k_fk(FDev d, const int* __restrict__ list) {
    const int s = list[blockIdx.x];
    double* F = d.pool + d.foff[s];
    for (int i = d.kptr[s] + threadIdx.x; i < d.kptr[s + 1]; i += blockDim.x) F[d.kpos[i]] += d.kval[i];
}

// Extend-add of the children's Schur complements (lower triangles) into the
// front, parent columns [32 y, 32 y + 32) per CTA, children one after the
// other: no two threads ever add into the same entry at once.
__global__ void __launch_bounds__(256) k_fea(FDev d, const int* __restrict__ list) {
    const int s = list[blockIdx.x];
    const int mp = d.sm[s];
    const int j0 = blockIdx.y * kNB;
    if (j0 >= mp) return;
    const int j1 = min(mp, j0 + kNB);
    double* Fp = d.pool + d.foff[s];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int ci = d.child_ptr[s]; ci < d.child_ptr[s + 1]; ++ci) {
        const int c = d.child[ci];
        const int kc = d.sk[c], mc = d.sm[c], uc = mc - kc;
        const int* rc = d.rel + d.rel_ptr[c];  // ascending positions in the parent's rows
        const double* Fc = d.pool + d.foff[c];
        const int b0 = lower_bound_dev(rc, uc, j0), b1 = lower_bound_dev(rc, uc, j1);
        for (int b = b0 + warp; b < b1; b += nw) {
            double* dst = Fp + (int64_t)rc[b] * mp;
            const double* src = Fc + (int64_t)(kc + b) * mc + kc;
            for (int a = b + lane; a < uc; a += 32) dst[rc[a]] += src[a];
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ panels
// One panel of kNB pivot columns of every front of a level, two launches:
//
//   k_panel  each CTA factors the panel's diagonal block A_JJ = L_JJ L_JJ^T
//            and inverts it, W = L_JJ^-1, in shared memory (the same few
//            thousand multiply-adds in every CTA, instead of a launch that
//            all the others wait for), then takes its share of
//              L[i, J] = A[i, J] W^T          rows i below the panel
//              X[J, c] = W X[J, c]            columns c left of the panel
//   k_trail  rows i below the panel, 32-row tiles:
//              A[i, c] -= L[i, J] L[c, J]^T   columns c past the panel, c <= i
//              X[i, c] -= L[i, J] X[J, c]     columns c up to the panel's last
//
// X, the m x k block after the front, starts as [I ; 0] (the identity is
// implicit: X[J, J] = W) and ends as [L_ss^-1 ; -L_os L_ss^-1]: M_s comes out
// of the same elimination, with the whole GPU on every panel, and its rows go
// to mval as they become final.
//
// FP64 runs at two multiply-adds a clock and SM here, so a 32-cubed tile takes
// 16 k clocks (8 us) and a chain of small steps on one warp a multiple of
// that: what counts is to spread each panel's work over the SMs.  A tile's
// columns are therefore split over 2 or 4 CTAs where a launch has few tiles.
constexpr int kPanelThreads = 256;

// A launch's fronts: front i has the CTAs from fronts[i].first to the next
// one's; hint[b] is the front of CTA 64 b, the last hint the last front.
struct FrontRef {
    int s, first;
};
constexpr int kHintStep = 64;

__device__ __forceinline__ int find_front(const FrontRef* f, const int* hint, int block) {
    int lo = hint[block / kHintStep];
    int hi = hint[block / kHintStep + 1];
    while (lo < hi) {  // the last front that begins at or before the block
        const int mid = (lo + hi + 1) >> 1;
        if (f[mid].first <= block) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Lower triangle of the nb x nb block D -> its Cholesky factor, W -> the
// factor's inverse (both lower, row-major in shared memory).  The pivots are a
// chain of 32 reciprocal square roots, each some eight dependent FP64
// operations of 64 clocks or more; everything else is kept out of it.  Eight
// columns at a time, warp 0 (lane = row) factors the columns in registers while
// the other warps bring W up to date with the eight before:
//   rows J of W   W[J, c] = L_JJ^-1 W[J, c]
//   rows below    W[r, c] -= L[r, J] W[J, c]
// then all warps take the columns out of the rest of D.  One column a step with
// two barriers, all warps on each, took 50 us a block; this takes 22.
constexpr int kSub = 8;

struct PanelShared {
    double D[kNB][kNB + 1], W[kNB][kNB + 1], T[kNB][kNB + 1];
    double inv[kNB];  // 1 / L_jj
};

// Warp 0: columns c0 .. c0 + 8 of D.  With y the single precision value of
// 1 / sqrt(d) and e = 1 - d y^2 (about 2^-22), 1 / sqrt(d) is y (1 - e)^(-1/2) =
// y (1 + e / 2 + 3 e^2 / 8 + O(e^3)), the rest below the rounding of double.
// Outside the range of float the library's function.
__device__ __forceinline__ void factor_columns(PanelShared& S, int c0, int nb, bool& bad) {
    const int lane = threadIdx.x;
    double a[kSub];
#pragma unroll
    for (int c = 0; c < kSub; ++c) a[c] = S.D[lane][c0 + c];
#pragma unroll
    for (int c = 0; c < kSub; ++c) {
        if (c0 + c >= nb) break;
        double d = __shfl_sync(0xffffffffu, a[c], c0 + c);
        if (!(d > 0.0) || !isfinite(d)) {
            bad = true;
            d = 1.0;
            if (lane == c0 + c) a[c] = 1.0;
        }
        double inv;
        if (d > 1e-30 && d < 1e30) {
            const double y = (double)rsqrtf((float)d);
            const double e = fma(-d * y, y, 1.0);
            const double ay = a[c] * y;
            const double q = e * fma(0.375, e, 0.5);
            a[c] = fma(ay, q, ay);
            inv = fma(y, q, y);
        } else {
            inv = rsqrt(d);
            a[c] *= inv;
        }
        if (lane == 0) S.inv[c0 + c] = inv;
#pragma unroll
        for (int k = c + 1; k < kSub; ++k) a[k] = fma(-a[c], __shfl_sync(0xffffffffu, a[c], c0 + k), a[k]);
    }
#pragma unroll
    for (int c = 0; c < kSub; ++c)
        if (lane >= c0 + c) S.D[lane][c0 + c] = a[c];
}

// Warps 1 .. 7: W after the columns c0 .. c0 + 8 of L.
__device__ __forceinline__ void update_inverse(PanelShared& S, int c0, int nb) {
    const int t = threadIdx.x - 32;
    const int n = min(nb, c0 + kSub);  // rows of W that end here, and its columns so far
    if (t < n) {
        double w[kSub];
#pragma unroll
        for (int i = 0; i < kSub; ++i) {
            w[i] = 0.0;
            if (c0 + i >= nb) continue;
            double v = S.W[c0 + i][t];
#pragma unroll
            for (int q = 0; q < i; ++q) v = fma(-S.D[c0 + i][c0 + q], w[q], v);
            w[i] = t <= c0 + i ? v * S.inv[c0 + i] : 0.0;
            S.W[c0 + i][t] = w[i];
        }
    }
    asm volatile("bar.sync 1, 224;" ::: "memory");
    const int rows = nb - n;
    for (int e = t; e < rows * n; e += kPanelThreads - 32) {
        const int r = n + e / n, c = e % n;
        double v = S.W[r][c];
#pragma unroll
        for (int q = 0; q < kSub; ++q) v = fma(-S.D[r][c0 + q], S.W[c0 + q][c], v);
        S.W[r][c] = v;
    }
}

__device__ __forceinline__ void factor_block(PanelShared& S, int nb, bool& bad) {
    static_assert(kPanelThreads == 256, "warps 1 to 7 share barrier 1");
    for (int e = threadIdx.x; e < kNB * kNB; e += kPanelThreads) S.W[e / kNB][e % kNB] = e / kNB == e % kNB ? 1.0 : 0.0;
    __syncthreads();
    int c0 = 0;
    for (; c0 < nb; c0 += kSub) {
        if (threadIdx.x < 32) factor_columns(S, c0, nb, bad);
        else if (c0 > 0) update_inverse(S, c0 - kSub, nb);
        __syncthreads();
        const int r0 = c0 + kSub, entries = trailing_entries(nb, r0);
        for (int e = threadIdx.x; e < entries; e += kPanelThreads) {
            const auto [r, c] = trailing_entry(nb, r0, e);
            if (c > r) continue;
            double v = S.D[r][c];
#pragma unroll
            for (int q = 0; q < kSub; ++q) v = fma(-S.D[r][c0 + q], S.D[c][c0 + q], v);
            S.D[r][c] = v;
        }
        __syncthreads();
    }
    if (threadIdx.x >= 32) update_inverse(S, c0 - kSub, nb);
    __syncthreads();
}

__global__ void __launch_bounds__(kPanelThreads) k_panel(FDev d, const FrontRef* __restrict__ fronts,
                                                         const int* __restrict__ hint, int j0, int chunk) {
    __shared__ PanelShared S;
    auto& W = S.W;
    auto& T = S.T;
    pdl_trigger();
    const int fi = find_front(fronts, hint, blockIdx.x);
    const int s = fronts[fi].s, part = blockIdx.x - fronts[fi].first;
    const int k = d.sk[s], m = d.sm[s];
    const int nb = min(kNB, k - j0), j1 = j0 + nb;
    const int64_t ld = m_stride(m, k);
    double* F = d.pool + d.foff[s];
    double* X = F + (int64_t)m * m;
    float* M = d.mval + d.moff[s];
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < kNB * kNB; e += kPanelThreads) {
        const int r = e % kNB, c = e / kNB;
        S.D[r][c] = (r < nb && c <= r) ? F[(int64_t)(j0 + c) * m + j0 + r] : 0.0;
    }
    __syncthreads();
    bool bad = false;
    factor_block(S, nb, bad);
    const int nrow = max(1, (m - j1 + chunk - 1) / chunk);
    if (part == 0) {
        if (bad) atomicCAS(d.status, 0, s + 1);
        for (int e = threadIdx.x; e < nb * kNB; e += kPanelThreads) {
            const int r = e % kNB, c = e / kNB;
            if (r >= nb || c > r) continue;
            X[(int64_t)(j0 + c) * m + j0 + r] = W[r][c];
            M[(int64_t)(j0 + c) * ld + j0 + r] = (float)W[r][c];
        }
    }
    if (part < nrow) {  // (nothing reads L_JJ any more: the diagonal block of F stays as it is)
        for (int r0 = j1 + part * chunk; r0 < min(m, j1 + (part + 1) * chunk); r0 += kNB) {
            __syncthreads();
            for (int e = threadIdx.x; e < kNB * kNB; e += kPanelThreads) {
                const int r = e % kNB, q = e / kNB;
                T[r][q] = (q < nb && r0 + r < m) ? F[(int64_t)(j0 + q) * m + r0 + r] : 0.0;
            }
            __syncthreads();
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            for (int q = 0; q < nb; ++q) {
                const double t = T[lane][q];
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[u] = fma(t, W[warp + 8 * u][q], acc[u]);  // zero for q > j
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = warp + 8 * u;
                if (j < nb && r0 + lane < m) F[(int64_t)(j0 + j) * m + r0 + lane] = acc[u];
            }
        }
        return;
    }
    // X[J, c] = W X[J, c]: column block of the left part
    const int c0 = (part - nrow) * chunk;
    for (int cb = c0; cb < min(j0, c0 + chunk); cb += kNB) {
        __syncthreads();
        for (int e = threadIdx.x; e < kNB * kNB; e += kPanelThreads) {
            const int r = e % kNB, c = e / kNB;
            T[r][c] = (r < nb && cb + c < j0) ? X[(int64_t)(cb + c) * m + j0 + r] : 0.0;
        }
        __syncthreads();
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int q = 0; q < nb; ++q) {
            const double w = W[lane][q];
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] = fma(w, T[q][warp + 8 * u], acc[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = cb + warp + 8 * u;
            if (c < j0 && lane < nb) {
                X[(int64_t)c * m + j0 + lane] = acc[u];
                M[(int64_t)c * ld + j0 + lane] = (float)acc[u];
            }
        }
    }
}

// Tiles of a panel's trailing update: 32 rows from j1 + 32 ti, and kCols
// columns of A (the tile column tj <= ti) or of X.
template <int kCols>
__global__ void __launch_bounds__(kPanelThreads) k_trail(FDev d, const FrontRef* __restrict__ fronts,
                                                         const int* __restrict__ hint, int j0) {
    __shared__ double Lr[kNB][kNB + 1], Lc[kCols][kNB + 1];
    pdl_trigger();
    constexpr int kSplit = kNB / kCols;
    constexpr int kPer = kCols / 8;  // outputs a thread: 8 warps
    const int fi = find_front(fronts, hint, blockIdx.x);
    const int s = fronts[fi].s;
    int t = blockIdx.x - fronts[fi].first;
    const int k = d.sk[s], m = d.sm[s];
    const int nb = min(kNB, k - j0), j1 = j0 + nb;
    const int sub = t % kSplit;
    t /= kSplit;
    const int T = (m - j1 + kNB - 1) / kNB;
    const int ta = T * (T + 1) / 2;
    const bool in_x = t >= ta;
    int ti, tj;
    if (in_x) {
        const int nc = (j1 + kNB - 1) / kNB;
        ti = (t - ta) / nc;
        tj = (t - ta) % nc;
    } else {
        ti = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
        while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
        while (ti * (ti + 1) / 2 > t) --ti;
        tj = t - ti * (ti + 1) / 2;
    }
    const int r0 = j1 + kNB * ti, c0 = (in_x ? 0 : j1) + kNB * tj + kCols * sub;
    const int cend = in_x ? j1 : m;
    double* F = d.pool + d.foff[s];
    double* X = F + (int64_t)m * m;
    pdl_wait();
    for (int e = threadIdx.x; e < kNB * kNB; e += kPanelThreads) {
        const int r = e % kNB, q = e / kNB;
        Lr[r][q] = (q < nb && r0 + r < m) ? F[(int64_t)(j0 + q) * m + r0 + r] : 0.0;
    }
    if (in_x) {
        for (int e = threadIdx.x; e < kCols * kNB; e += kPanelThreads) {
            const int q = e % kNB, c = e / kNB;
            Lc[c][q] = (q < nb && c0 + c < cend) ? X[(int64_t)(c0 + c) * m + j0 + q] : 0.0;
        }
    } else {
        for (int e = threadIdx.x; e < kCols * kNB; e += kPanelThreads) {
            const int c = e % kCols, q = e / kCols;
            Lc[c][q] = (q < nb && c0 + c < cend) ? F[(int64_t)(j0 + q) * m + c0 + c] : 0.0;
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = r0 + lane;
    double* out = in_x ? X : F;
    double acc[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int col = c0 + warp + 8 * u;
        acc[u] = row < m && col < cend && (in_x || col <= row) ? out[(int64_t)col * m + row] : 0.0;
    }
#pragma unroll 8
    for (int q = 0; q < kNB; ++q) {
        const double a = -Lr[lane][q];
#pragma unroll
        for (int u = 0; u < kPer; ++u) acc[u] = fma(a, Lc[warp + 8 * u][q], acc[u]);
    }
    if (row >= m) return;
    const int64_t ld = m_stride(m, k);
    float* M = d.mval + d.moff[s];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int col = c0 + warp + 8 * u;
        if (col >= cend || (!in_x && col > row)) continue;
        out[(int64_t)col * m + row] = acc[u];
        if (in_x && j1 == k) M[col * ld + row] = (float)-acc[u];  // the last panel: rows past the pivots are final
    }
}

// The root's inverse S = L^-T L^-1 from X = L^-1 (k x k, lower, column major):
// S[i][j] is the product of columns i and j of X from row max(i, j) on, 32 x 32
// entries a CTA (column blocks bi >= bj), written to both triangles.
__global__ void __launch_bounds__(256) k_root_inverse(const double* __restrict__ X, int k, float* S, int ld) {
    __shared__ double A[kNB][kNB + 1], B[kNB][kNB + 1];
    int bi = (int)((sqrtf(8.0f * (float)blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while ((bi + 1) * (bi + 2) / 2 <= (int)blockIdx.x) ++bi;
    while (bi * (bi + 1) / 2 > (int)blockIdx.x) --bi;
    const int bj = (int)blockIdx.x - bi * (bi + 1) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q0 = kNB * bi; q0 < k; q0 += kNB) {
        __syncthreads();
        for (int e = threadIdx.x; e < kNB * kNB; e += 256) {
            const int q = e % kNB, c = e / kNB;
            const int ci = kNB * bi + c, cj = kNB * bj + c;
            // zero above the diagonal, where X is not written
            A[c][q] = q0 + q < k && ci < k && q0 + q >= ci ? X[(int64_t)ci * k + q0 + q] : 0.0;
            B[c][q] = q0 + q < k && cj < k && q0 + q >= cj ? X[(int64_t)cj * k + q0 + q] : 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int q = 0; q < kNB; ++q) {
            const double a = A[lane][q];
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] = fma(a, B[warp + 8 * u][q], acc[u]);
        }
    }
    const int i = kNB * bi + lane;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int j = kNB * bj + warp + 8 * u;
        if (i >= k || j >= k) continue;
        S[(int64_t)j * ld + i] = (float)acc[u];
        S[(int64_t)i * ld + j] = (float)acc[u];
    }
}

template <class T> void put(DBuf<T>& b, const std::vector<T>& h, cudaStream_t s) {
    b.alloc(std::max<size_t>(h.size(), 1));
    if (!h.empty()) PDGB_CUDA_TRY(cudaMemcpyAsync(b.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s));
}

}  // namespace

double gpu_factor(const CholFactor& f, float* mval, void* stream) {
    const FrontPlan& P = f.fp;
    if (!P.on) throw Error{PDGB_ERR_INVALID_ARGUMENT, "gpu_factor: no front plan"};
    cudaStream_t s = (cudaStream_t)stream;
    const int ns = f.nsuper;
    const int nl = (int)P.lvl_ptr.size() - 1;
    // ---- launch lists, built on the host and uploaded at once
    struct Launch {
        int kind;        // 0 level start (zero / K / extend-add), 1 panel, 2 trailing update
        int level;
        int j0;
        size_t front0, hint0;
        int ctas;
        int size;        // panel: rows or columns a CTA; trailing update: columns a CTA
        int ychunks, ycols;
    };
    std::vector<Launch> plan;
    std::vector<FrontRef> fronts;
    std::vector<int> hints;
    // a launch over the fronts of a level with more than j0 pivots, count(k, m)
    // CTAs each
    auto launch = [&](int kind, int L, int j0, int size, auto&& count) {
        Launch l{kind, L, j0, fronts.size(), hints.size(), 0, size, 0, 0};
        int nf = 0;
        for (int q = P.lvl_ptr[L]; q < P.lvl_ptr[L + 1]; ++q) {
            const int sn = P.lvl_sn[q];
            if (f.sk[sn] <= j0) continue;
            const int64_t c = count(f.sk[sn], f.sm[sn]);
            if (c == 0) continue;
            if (l.ctas + c > INT32_MAX) throw Error{PDGB_ERR_UNSUPPORTED, "factorisation: too many tiles in one launch"};
            for (; (int64_t)hints.size() - (int64_t)l.hint0 < (l.ctas + c + kHintStep - 1) / kHintStep;) hints.push_back(nf);
            fronts.push_back(FrontRef{sn, l.ctas});
            l.ctas += (int)c;
            ++nf;
        }
        if (nf == 0) return;
        hints.push_back(nf - 1);
        plan.push_back(l);
    };
    auto blocks = [](int n, int size) { return (int64_t)((n + size - 1) / size); };
    for (int L = 0; L < nl; ++L) {
        const int a = P.lvl_ptr[L], b = P.lvl_ptr[L + 1];
        int64_t max_tot = 0;
        int max_m = 0, max_k = 0;
        for (int q = a; q < b; ++q) {
            const int sn = P.lvl_sn[q];
            max_tot = std::max<int64_t>(max_tot, front_doubles(f, sn));
            max_m = std::max(max_m, f.sm[sn]);
            max_k = std::max(max_k, f.sk[sn]);
        }
        plan.push_back(Launch{0, L, 0, 0, 0, 0, 0, (int)((max_tot + kZeroChunk - 1) / kZeroChunk), (max_m + kNB - 1) / kNB});
        for (int j0 = 0; j0 < max_k; j0 += kNB) {
            auto panel_ctas = [&](int size) {
                return [=](int k, int m) {
                    const int j1 = j0 + std::min(kNB, k - j0);
                    return std::max<int64_t>(1, blocks(m - j1, size)) + blocks(j0, size);
                };
            };
            auto tiles = [&](int k, int m) {
                const int j1 = j0 + std::min(kNB, k - j0);
                const int64_t T = blocks(m - j1, kNB);
                return T * (T + 1) / 2 + T * blocks(j1, kNB);
            };
            int64_t np = 0, nt = 0;
            for (int q = a; q < b; ++q) {
                const int sn = P.lvl_sn[q];
                if (f.sk[sn] <= j0) continue;
                np += panel_ctas(kNB)(f.sk[sn], f.sm[sn]);
                nt += tiles(f.sk[sn], f.sm[sn]);
            }
            // every panel CTA factors the diagonal block anew: a few rows each
            // while the SMs are not full, more of them past that
            const int size = np <= kFillCtas ? kNB : 4 * kNB;
            launch(1, L, j0, size, panel_ctas(size));
            const int cols = nt * 4 <= kFillCtas ? kNB / 4 : nt * 2 <= kFillCtas ? kNB / 2 : kNB;
            launch(2, L, j0, cols, [&](int k, int m) { return tiles(k, m) * (kNB / cols); });
        }
    }
    // ---- device data
    DBuf<double> pool, kval;
    DBuf<int64_t> foff, moff;
    DBuf<int> sk, sm, cptr, child, rptr, rel, kptr, kpos, lvl, status;
    DBuf<FrontRef> dfronts;
    DBuf<int> dhints;
    pool.alloc((size_t)std::max<int64_t>(P.pool, 1));
    put(foff, P.foff, s);
    put(moff, std::vector<int64_t>(f.moff.begin(), f.moff.begin() + ns), s);
    put(sk, f.sk, s);
    put(sm, f.sm, s);
    put(cptr, P.child_ptr, s);
    put(child, P.child, s);
    put(rptr, P.rel_ptr, s);
    put(rel, P.rel, s);
    put(kptr, P.kptr, s);
    put(kpos, P.kpos, s);
    put(kval, P.kval, s);
    put(lvl, P.lvl_sn, s);
    put(dfronts, fronts, s);
    put(dhints, hints, s);
    status.alloc(1);
    PDGB_CUDA_TRY(cudaMemsetAsync(status.p, 0, sizeof(int), s));
    PDGB_CUDA_TRY(cudaMemsetAsync(mval, 0, (size_t)f.mval_total * sizeof(float), s));
    FDev d{pool.p, foff.p, sk.p, sm.p, moff.p, mval, cptr.p, child.p, rptr.p, rel.p, kptr.p, kpos.p, kval.p, status.p};
    cudaEvent_t ev[2];
    PDGB_CUDA_TRY(cudaEventCreate(&ev[0]));
    PDGB_CUDA_TRY(cudaEventCreate(&ev[1]));
    float ms = 0.f;
    cudaError_t err = cudaEventRecord(ev[0], s);
    for (const Launch& l : plan) {
        if (err != cudaSuccess) break;
        const int a = P.lvl_ptr[l.level], nf = P.lvl_ptr[l.level + 1] - a;
        const int* list = lvl.p + a;
        if (l.kind == 0) {
            k_fz<<<dim3(nf, l.ychunks), 256, 0, s>>>(d, list);
            k_fk<<<nf, 256, 0, s>>>(d, list);
            k_fea<<<dim3(nf, l.ycols), 256, 0, s>>>(d, list);
        } else {
            const FrontRef* fr = dfronts.p + l.front0;
            const int* hint = dhints.p + l.hint0;
            if (l.kind == 1) launch_pdl(k_panel, l.ctas, kPanelThreads, 0, s, d, fr, hint, l.j0, l.size);
            else if (l.size == kNB) launch_pdl(k_trail<kNB>, l.ctas, kPanelThreads, 0, s, d, fr, hint, l.j0);
            else if (l.size == kNB / 2) launch_pdl(k_trail<kNB / 2>, l.ctas, kPanelThreads, 0, s, d, fr, hint, l.j0);
            else launch_pdl(k_trail<kNB / 4>, l.ctas, kPanelThreads, 0, s, d, fr, hint, l.j0);
        }
        err = cudaGetLastError();
    }
    if (err == cudaSuccess && f.root >= 0) {
        const int k = f.sk[f.root], nb = (k + kNB - 1) / kNB;
        k_root_inverse<<<nb * (nb + 1) / 2, 256, 0, s>>>(pool.p + P.foff[f.root] + (int64_t)k * k, k, mval + f.root_off,
                                                         m_stride(k, k));
        err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaEventRecord(ev[1], s);
    if (err == cudaSuccess) err = cudaEventSynchronize(ev[1]);
    if (err == cudaSuccess) err = cudaEventElapsedTime(&ms, ev[0], ev[1]);
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    PDGB_CUDA_TRY(err);
    int bad = 0;
    PDGB_CUDA_TRY(cudaMemcpy(&bad, status.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (bad)
        throw Error{PDGB_ERR_NOT_SPD, "system matrix is not positive definite (supernode " + std::to_string(bad - 1) + ")"};
    return (double)ms;
}

}  // namespace pdgb
