// pdgb_step_noalloc: PD time steps (Jacobi + Chebyshev global solve) that
// allocate no memory at all.
//
// Who needs this.  Some callers cannot call cudaMalloc (or any allocating
// routine) at the point where they want to advance a soft body:
//   - a host application whose device-memory allocator owns the GPU's memory
//     (a game engine or renderer with its own pools) and forbids plugins to
//     allocate behind its back;
//   - code running inside a frame loop with a hard latency budget, where a
//     cudaMalloc/cudaFree can synchronise the whole device;
//   - plugins that receive only device pointers to the simulation arrays
//     (the way the reference's SolverData is handed to its solvers) and have
//     no place to keep per-body allocations between calls.
// pdgb_create/pdgb_step allocate the engine's buffers once; this entry point
// instead keeps its scratch in one fixed, file-scope device array that every
// GPU loading the library holds until the process exits.
//
// Limits and sharing rules (also stated in include/pdgb.h):
//   - at most kNaMaxVerts vertices and kNaMaxTets tets per call;
//   - every call uses the same scratch array, so calls that overlap on the
//     GPU (on different streams, or from several host threads) race and
//     corrupt each other's results; serialise them;
//   - the scratch keeps the previous call's contents; everything a call
//     needs is recomputed or cleared by that call;
//   - the first call on a device looks up the array's device address
//     (cudaGetSymbolAddress) once for that device.  The address is kept for
//     the life of the process, so a cudaDeviceReset between calls is not
//     supported;
//   - every call waits for its stream once, before it returns, so no call can
//     be captured into a CUDA graph;
//   - the mesh is checked on the device (tet indices, rest volumes, weights)
//     before any step: a bad mesh returns PDGB_ERR_BAD_MESH with X and V
//     untouched.
//
// All steps of a call are one cooperative launch: the iterations of a small
// body are a few microseconds of work each, less than two launches of one
// (a call of two 20-iteration steps on 5,400 tets took 81 of them).
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "../../include/pdgb.h"
#include "relax.cuh"
#include "rotation.cuh"

namespace pdgb {
namespace {

constexpr int kNaMaxVerts = 32768;
constexpr int kNaMaxTets = 131072;
constexpr int kNaMaxDevices = 64;

// Scratch layout (bytes):
//   tet part   : per tet 10 floats (DmInv row-major, V0 * mu)       [kNaMaxTets]
//   vertex part: float4 sn, prev, b, base, coef {M/h^2, diag, pin, m} [kNaMaxVerts]
//                float  diag accumulator                            [kNaMaxVerts]
//   flags      : NaFlags (256 bytes reserved)
// 5.2 MB + 2.6 MB + 0.1 MB = about 8 MB in total.
constexpr size_t kNaTetBytes = (size_t)kNaMaxTets * 10 * sizeof(float);
constexpr size_t kNaVecBytes = (size_t)kNaMaxVerts * sizeof(float4);
constexpr size_t kNaDiagBytes = (size_t)kNaMaxVerts * sizeof(float);
constexpr size_t kNaScratchBytes = kNaTetBytes + 5 * kNaVecBytes + kNaDiagBytes + 256;

static __device__ __align__(256) unsigned char g_na_scratch[kNaScratchBytes];

// Cleared by each call with the diagonal before them.
struct NaFlags {
    int bad;                // set when a tet has an out-of-range index, no float-representable
                            // DmInv (zero or nearly zero rest volume) or a negative or
                            // non-finite weight
    int timeout;            // a barrier wait ran out
    unsigned arrived;       // CTAs that have arrived at the grid barriers so far
};

struct NaScratch {
    float* geo;     // [10][kNaMaxTets] SoA
    float4* sn;
    float4* prev;
    float4* b;
    float4* base;
    float4* coef;
    float* diag;
    NaFlags* flags;
};

NaScratch carve(unsigned char* base) {
    NaScratch s;
    s.geo = reinterpret_cast<float*>(base);
    unsigned char* p = base + kNaTetBytes;
    s.sn = reinterpret_cast<float4*>(p);
    s.prev = reinterpret_cast<float4*>(p + kNaVecBytes);
    s.b = reinterpret_cast<float4*>(p + 2 * kNaVecBytes);
    s.base = reinterpret_cast<float4*>(p + 3 * kNaVecBytes);
    s.coef = reinterpret_cast<float4*>(p + 4 * kNaVecBytes);
    s.diag = reinterpret_cast<float*>(p + 5 * kNaVecBytes);
    s.flags = reinterpret_cast<NaFlags*>(p + 5 * kNaVecBytes + kNaDiagBytes);
    return s;
}

// Per-tet DmInv and V0 * mu from the rest shape (solverUtil.cuh:108-138) and
// the stiffness diagonal sum_t c_t (B_t^T B_t)_jj (pdUtil.cu:21-24).
__global__ void na_tets(int nv, int nt, const uint32_t* __restrict__ tets, const float* __restrict__ X0,
                        const float* __restrict__ mu, NaScratch s) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const uint32_t i0 = tets[4 * t], i1 = tets[4 * t + 1], i2 = tets[4 * t + 2], i3 = tets[4 * t + 3];
    if (i0 >= (uint32_t)nv || i1 >= (uint32_t)nv || i2 >= (uint32_t)nv || i3 >= (uint32_t)nv) {
        atomicExch(&s.flags->bad, 1);
        return;
    }
    double D[3][3];
    const uint32_t id[3] = {i1, i2, i3};
    for (int c = 0; c < 3; ++c)
        for (int r = 0; r < 3; ++r) D[r][c] = (double)X0[3 * id[c] + r] - (double)X0[3 * i0 + r];
    const double det = D[0][0] * (D[1][1] * D[2][2] - D[1][2] * D[2][1]) - D[0][1] * (D[1][0] * D[2][2] - D[1][2] * D[2][0]) +
                       D[0][2] * (D[1][0] * D[2][1] - D[1][1] * D[2][0]);
    const float w = mu[t];
    if (!(det != 0.0) || !isfinite(det) || !(w >= 0.f) || !isfinite(w)) {
        atomicExch(&s.flags->bad, 1);
        return;
    }
    const double rdet = 1.0 / det;  // FP64 divides are slow here: one, not nine
    double inv[9];
    inv[0] = (D[1][1] * D[2][2] - D[1][2] * D[2][1]) * rdet;
    inv[1] = (D[0][2] * D[2][1] - D[0][1] * D[2][2]) * rdet;
    inv[2] = (D[0][1] * D[1][2] - D[0][2] * D[1][1]) * rdet;
    inv[3] = (D[1][2] * D[2][0] - D[1][0] * D[2][2]) * rdet;
    inv[4] = (D[0][0] * D[2][2] - D[0][2] * D[2][0]) * rdet;
    inv[5] = (D[0][2] * D[1][0] - D[0][0] * D[1][2]) * rdet;
    inv[6] = (D[1][0] * D[2][1] - D[1][1] * D[2][0]) * rdet;
    inv[7] = (D[0][1] * D[2][0] - D[0][0] * D[2][1]) * rdet;
    inv[8] = (D[0][0] * D[1][1] - D[0][1] * D[1][0]) * rdet;
    const double coef = fabs(det) / 6.0 * (double)w;
    // a nearly flat tet has a finite double inverse that overflows float:
    // rejected like a flat one (the layout of pdgb_create does the same)
    bool finite = isfinite((float)coef);
    for (int k = 0; k < 9; ++k) finite = finite && isfinite((float)inv[k]);
    if (!finite) {
        atomicExch(&s.flags->bad, 1);
        return;
    }
    for (int k = 0; k < 9; ++k) s.geo[(size_t)k * kNaMaxTets + t] = (float)inv[k];
    s.geo[(size_t)9 * kNaMaxTets + t] = (float)coef;
    const uint32_t corner[4] = {i0, i1, i2, i3};
    for (int j = 0; j < 4; ++j) {
        double bx, by, bz;  // column j of B = DmInv^T G
        if (j == 0) {
            bx = -(inv[0] + inv[3] + inv[6]);
            by = -(inv[1] + inv[4] + inv[7]);
            bz = -(inv[2] + inv[5] + inv[8]);
        } else {
            bx = inv[3 * (j - 1)];
            by = inv[3 * (j - 1) + 1];
            bz = inv[3 * (j - 1) + 2];
        }
        atomicAdd(&s.diag[corner[j]], (float)(coef * (bx * bx + by * by + bz * bz)));
    }
}

// Grid barrier of a cooperative launch: the n-th barrier is passed once
// n gridDim.x CTAs have arrived.  A wait is bounded (kNaSpins: some seconds);
// past it the timeout word ends every CTA at its next barrier.  A check makes it
// wait for `missing` more arrivals than there are CTAs.
constexpr unsigned kNaSpins = 1u << 22;
struct NaWait {
    unsigned spins, missing;
};
__device__ __forceinline__ bool na_barrier(NaFlags* f, unsigned& target, const NaWait& w) {
    __shared__ int ok;
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) {
        // released with the CTA's writes and atomics before the barrier above,
        // acquired before those after the one below
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&f->arrived) : "memory");
        bool there = false;
        for (unsigned n = 0; n < w.spins && !there; ++n) {
            unsigned seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&f->arrived) : "memory");
            there = (int)(seen - target - w.missing) >= 0;  // the count may wrap
            if (n % 1024 == 1023 && *reinterpret_cast<volatile int*>(&f->timeout)) break;
        }
        if (!there) atomicExch(&f->timeout, 1);
        ok = there;
    }
    __syncthreads();
    return ok;
}

struct NaTet {
    uint32_t id[4];
    float D[9], c;
};
__device__ __forceinline__ NaTet na_tet(const uint32_t* tets, const NaScratch& s, int t) {
    const uint4 q = make_uint4(tets[4 * t], tets[4 * t + 1], tets[4 * t + 2], tets[4 * t + 3]);
    NaTet r{{q.x, q.y, q.z, q.w}, {}, s.geo[(size_t)9 * kNaMaxTets + t]};
#pragma unroll
    for (int k = 0; k < 9; ++k) r.D[k] = s.geo[(size_t)k * kNaMaxTets + t];
    return r;
}

// Local step of one tet, residual form c (R - F) B, float4 atomics into the
// scratch b (pinned vertices ignore b).
__device__ __forceinline__ void na_local(const NaTet& q, const NaScratch& s) {
    const float* D = q.D;
    const float4 p0 = __ldcg(&s.sn[q.id[0]]), p1 = __ldcg(&s.sn[q.id[1]]), p2 = __ldcg(&s.sn[q.id[2]]),
                 p3 = __ldcg(&s.sn[q.id[3]]);
    const float e[3][3] = {{p1.x - p0.x, p2.x - p0.x, p3.x - p0.x},
                           {p1.y - p0.y, p2.y - p0.y, p3.y - p0.y},
                           {p1.z - p0.z, p2.z - p0.z, p3.z - p0.z}};
    float F[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) F[3 * r + cc] = e[r][0] * D[cc] + e[r][1] * D[3 + cc] + e[r][2] * D[6 + cc];
    float R[9];
    closest_rotation_quat(F, R);
#pragma unroll
    for (int k = 0; k < 9; ++k) R[k] -= F[k];
    float M[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int cc = 0; cc < 3; ++cc)
            M[3 * r + cc] = q.c * (R[3 * r] * D[3 * cc] + R[3 * r + 1] * D[3 * cc + 1] + R[3 * r + 2] * D[3 * cc + 2]);
    atomicAdd(&s.b[q.id[0]], make_float4(-(M[0] + M[1] + M[2]), -(M[3] + M[4] + M[5]), -(M[6] + M[7] + M[8]), 0.f));
    atomicAdd(&s.b[q.id[1]], make_float4(M[0], M[3], M[6], 0.f));
    atomicAdd(&s.b[q.id[2]], make_float4(M[1], M[4], M[7], 0.f));
    atomicAdd(&s.b[q.id[3]], make_float4(M[2], M[5], M[8], 0.f));
}

struct NaParams {
    float dt, dt_inv, gravity, pw, wpin, rho;
    int iters, steps;
    NaWait wait;
};

// One vertex: its mass terms, pin right-hand side, state and iterates.
struct NaVertex {
    float cm, md, m;
    bool pinned;
    float3 pin, x, v, sn, prev, base;
};

__device__ __forceinline__ float3 na_load3(const float* a, int i) { return make_float3(a[3 * i], a[3 * i + 1], a[3 * i + 2]); }
__device__ __forceinline__ void na_store3(float* a, int i, float3 v) {
    a[3 * i] = v.x;
    a[3 * i + 1] = v.y;
    a[3 * i + 2] = v.z;
}
__device__ __forceinline__ float4 na_f4(float3 v) { return make_float4(v.x, v.y, v.z, 0.f); }

__device__ __forceinline__ NaVertex na_vertex(const float* X0, const float* mass, const float* dbc, const float* X,
                                              const float* V, const NaParams& p, const NaScratch& s, int i) {
    NaVertex q{};
    const float pin = dbc ? dbc[i] : 0.f;
    q.m = mass[i];
    q.cm = (q.m + pin * p.pw) / (p.dt * p.dt);
    q.md = s.diag[i];
    q.pinned = pin > 0.f;
    const float3 x0 = na_load3(X0, i);
    q.pin = make_float3(x0.x * p.wpin, x0.y * p.wpin, x0.z * p.wpin);
    q.x = na_load3(X, i);
    q.v = na_load3(V, i);
    return q;
}

// s = x + h v + f / (M/h^2); base = b = (M/h^2) s.
__device__ __forceinline__ void na_begin(NaVertex& q, const NaParams& p, const NaScratch& s, int i) {
    const float dt2_m_1 = 1.0f / q.cm;
    const float fy = -p.gravity * q.m;
    q.sn = make_float3(q.x.x + p.dt * q.v.x, q.x.y + p.dt * q.v.y + dt2_m_1 * fy, q.x.z + p.dt * q.v.z);
    q.base = make_float3(q.cm * q.sn.x, q.cm * q.sn.y, q.cm * q.sn.z);
    s.sn[i] = na_f4(q.sn);
    s.b[i] = na_f4(q.base);
}

// Jacobi update + 0.9 relaxation + Chebyshev blend (pdUtil.cu:195-226) with
// the pin RHS x0 * w / h^2 (pdUtil.cu:147-166); the last iteration makes V and
// X (pdUtil.cu:180-193).
__device__ __forceinline__ void na_update(NaVertex& q, float omega, int iter, const NaParams& p, const NaScratch& s,
                                          int i) {
    const float4 b4 = __ldcg(&s.b[i]);
    const float3 bb = q.pinned ? q.pin : make_float3(b4.x, b4.y, b4.z);
    const float den = q.cm + q.md;
    float3 n = make_float3(relax09((bb.x - q.cm * q.sn.x) / den + q.sn.x, q.sn.x),
                           relax09((bb.y - q.cm * q.sn.y) / den + q.sn.y, q.sn.y),
                           relax09((bb.z - q.cm * q.sn.z) / den + q.sn.z, q.sn.z));
    if (iter >= 11)
        n = make_float3((n.x - q.prev.x) * omega + q.prev.x, (n.y - q.prev.y) * omega + q.prev.y,
                        (n.z - q.prev.z) * omega + q.prev.z);
    q.prev = q.sn;
    if (iter + 1 == p.iters) {
        q.v = make_float3((n.x - q.x.x) * p.dt_inv, (n.y - q.x.y) * p.dt_inv, (n.z - q.x.z) * p.dt_inv);
        q.x = n;
    } else {
        q.sn = n;
        s.sn[i] = na_f4(n);
        s.b[i] = na_f4(q.base);
    }
}

__device__ __forceinline__ float na_omega(float omega, int iter, float rho) {
    return iter <= 10 ? 1.f : iter == 11 ? 2 / (2 - rho * rho) : 4 / (4 - rho * rho * omega);
}

// Every step of the call.  A thread owns one tet, whose geometry stays in its
// registers, and one vertex, whose state and iterates do: what goes through L2
// is the iterate (published, gathered by the tets) and the sums b.  With fewer
// threads than tets or vertices (kOwn false: 1,024 a CTA on fewer than 128 SMs)
// they are walked in strides, the vertex data in the scratch and X, V.
template <bool kOwn, int kThreads>
__global__ void __launch_bounds__(kThreads, 1)
    na_run(int nv, int nt, const uint32_t* __restrict__ tets, const float* __restrict__ X0,
           const float* __restrict__ mass, const float* __restrict__ dbc, NaParams p, float* X, float* V, NaScratch s,
           unsigned target) {
    if (s.flags->bad || s.flags->timeout) return;  // set before this launch: the same for every CTA
    const int g = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;
    if (kOwn) {
        NaTet tet{};
        NaVertex q{};
        if (g < nt) tet = na_tet(tets, s, g);
        if (g < nv) q = na_vertex(X0, mass, dbc, X, V, p, s, g);
        for (int step = 0; step < p.steps; ++step) {
            if (g < nv) na_begin(q, p, s, g);
            float omega = 1.f;
            for (int i = 0; i < p.iters; ++i) {
                if (!na_barrier(s.flags, target, p.wait)) return;
                if (g < nt) na_local(tet, s);
                omega = na_omega(omega, i, p.rho);
                if (!na_barrier(s.flags, target, p.wait)) return;
                if (g < nv) na_update(q, omega, i, p, s, g);
            }
        }
        if (g < nv) {
            na_store3(X, g, q.x);
            na_store3(V, g, q.v);
        }
        return;
    }
    for (int step = 0; !kOwn && step < p.steps; ++step) {
        for (int i = g; i < nv; i += all) {
            NaVertex q = na_vertex(X0, mass, dbc, X, V, p, s, i);
            na_begin(q, p, s, i);
            s.base[i] = na_f4(q.base);
            s.prev[i] = na_f4(q.sn);
        }
        float omega = 1.f;
        for (int it = 0; it < p.iters; ++it) {
            if (!na_barrier(s.flags, target, p.wait)) return;
            for (int t = g; t < nt; t += all) na_local(na_tet(tets, s, t), s);
            omega = na_omega(omega, it, p.rho);
            if (!na_barrier(s.flags, target, p.wait)) return;
            for (int i = g; i < nv; i += all) {
                NaVertex q = na_vertex(X0, mass, dbc, X, V, p, s, i);
                const float4 sn = s.sn[i], pr = s.prev[i], ba = s.base[i];
                q.sn = make_float3(sn.x, sn.y, sn.z);
                q.prev = make_float3(pr.x, pr.y, pr.z);
                q.base = make_float3(ba.x, ba.y, ba.z);
                na_update(q, omega, it, p, s, i);
                s.prev[i] = na_f4(q.prev);
                if (it + 1 == p.iters) {
                    na_store3(X, i, q.x);
                    na_store3(V, i, q.v);
                }
            }
        }
    }
}

// Threads per CTA: as few CTAs as hold a tet and a vertex a thread (a barrier
// costs by the CTA: 22 x 256 threads pass it in 1.3 us), as many as the SMs
// once 256 threads each are not enough.
constexpr int kNaLaunchIters = 8192;  // iterations of one launch, a fraction of a second at the most
int na_threads(int n, int sms) { return n <= 256 * sms ? 256 : n <= 512 * sms ? 512 : 1024; }

std::mutex g_na_mutex;
unsigned char* g_na_ptr[kNaMaxDevices] = {};

}  // namespace
}  // namespace pdgb

using namespace pdgb;

namespace {
// max_ctas: most CTAs of the launch (0: as many as the SMs).
int step_noalloc(const pdgb_noalloc_mesh* mesh, const pdgb_params* p, float* X, float* V, int nsteps, void* stream,
                 int max_ctas, NaWait wait) {
    if (!mesh || !p || !X || !V || !mesh->tets || !mesh->X0 || !mesh->mass || !mesh->mu || nsteps < 0)
        return PDGB_ERR_INVALID_ARGUMENT;
    if (mesh->num_verts <= 0 || mesh->num_tets <= 0) return PDGB_ERR_INVALID_ARGUMENT;
    if (mesh->num_verts > kNaMaxVerts || mesh->num_tets > kNaMaxTets) return PDGB_ERR_UNSUPPORTED;
    if (!(p->dt > 0.f) || p->num_iterations < 1 || p->num_iterations > 4096) return PDGB_ERR_INVALID_ARGUMENT;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNaMaxDevices) return PDGB_ERR_CUDA;
    unsigned char* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_na_mutex);
        if (!g_na_ptr[dev]) {
            void* ptr = nullptr;
            if (cudaGetSymbolAddress(&ptr, g_na_scratch) != cudaSuccess || !ptr) return PDGB_ERR_CUDA;
            g_na_ptr[dev] = static_cast<unsigned char*>(ptr);
        }
        base = g_na_ptr[dev];
    }
    const NaScratch s = carve(base);
    cudaStream_t st = (cudaStream_t)stream;
    const int nv = mesh->num_verts, nt = mesh->num_tets;
    if (cudaMemsetAsync(s.diag, 0, kNaDiagBytes + sizeof(NaFlags), st) != cudaSuccess) return PDGB_ERR_CUDA;
    na_tets<<<(nt + 255) / 256, 256, 0, st>>>(nv, nt, mesh->tets, mesh->X0, mesh->mu, s);
    if (cudaGetLastError() != cudaSuccess) return PDGB_ERR_CUDA;
    if (nsteps > 0) {
        int most = 0;
        if (cudaDeviceGetAttribute(&most, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return PDGB_ERR_CUDA;
        if (max_ctas > 0 && max_ctas < most) most = max_ctas;
        const int n = nv > nt ? nv : nt, threads = na_threads(n, most);
        const int want = (n + threads - 1) / threads, grid = want < most ? want : most;
        const bool own = grid == want;  // else 1,024 threads
        const auto kernel = !own ? na_run<false, 1024>
                            : threads == 256 ? na_run<true, 256>
                            : threads == 512 ? na_run<true, 512>
                                             : na_run<true, 1024>;
        const float dt_inv = 1.0f / p->dt;
        NaParams np{p->dt, dt_inv, p->gravity, p->positional_weight, p->positional_weight * (dt_inv * dt_inv),
                    p->rho, p->num_iterations, 0, wait};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const int at_once = p->num_iterations >= kNaLaunchIters ? 1 : kNaLaunchIters / p->num_iterations;
        unsigned arrived = 0;
        for (int done = 0; done < nsteps; done += np.steps) {
            np.steps = nsteps - done < at_once ? nsteps - done : at_once;
            if (cudaLaunchKernelEx(&cfg, kernel, nv, nt, mesh->tets, mesh->X0, mesh->mass, mesh->dbc, np, X, V, s,
                                   arrived) != cudaSuccess)
                return PDGB_ERR_CUDA;
            arrived += 2u * (unsigned)np.iters * (unsigned)np.steps * (unsigned)grid;
        }
    }
    NaFlags flags{};
    if (cudaMemcpyAsync(&flags, s.flags, sizeof(flags), cudaMemcpyDeviceToHost, st) != cudaSuccess) return PDGB_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return PDGB_ERR_CUDA;
    if (flags.bad) return PDGB_ERR_BAD_MESH;
    if (flags.timeout) return PDGB_ERR_TIMEOUT;
    return PDGB_OK;
}
}  // namespace

extern "C" int pdgb_step_noalloc(const pdgb_noalloc_mesh* mesh, const pdgb_params* p, float* X, float* V, int nsteps,
                                 void* stream) {
    return step_noalloc(mesh, p, X, V, nsteps, stream, 0, NaWait{kNaSpins, 0u});
}

extern "C" int pdgb_noalloc_check(const pdgb_noalloc_mesh* mesh, const pdgb_params* p, float* X, float* V, int nsteps,
                                  void* stream, int max_ctas, int missing, int spin_limit) {
    if (max_ctas < 0 || missing < 0 || spin_limit < 1) return PDGB_ERR_INVALID_ARGUMENT;
    return step_noalloc(mesh, p, X, V, nsteps, stream, max_ctas, NaWait{(unsigned)spin_limit, (unsigned)missing});
}
