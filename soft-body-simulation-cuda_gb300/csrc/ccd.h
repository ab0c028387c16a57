// Continuous collision between bodies (internal to the engine).
//
// The reference runs, after every PD step with collision handling on
// (PdSolver::Update, pdSolver.cu:218-224), CollisionDetection::DetectCollision
// (src/collision/bvh.cu:153-165: LBVH over the surface triangles' swept
// boxes, candidate pairs of triangles of different bodies, point-face and
// edge-edge continuous tests, earliest contact per vertex / edge) and then
// CCDKernel (collisionUtil.cu:50-70).  CcdContext is the GPU form of both.
#pragma once
#include <memory>
#include <vector>

#include "engine.h"

namespace pdgb {

// Surface of a collision system, in the engine's vertex order.  Triangle t
// keeps its caller index t (face queries break contact-time ties by it);
// its vertices are stored in ascending caller id (the reference sorts a
// face query's face vertices), edges likewise, edge ids follow the
// lexicographic order of (smaller, larger) caller id.
struct CcdSurface {
    int nv = 0, ntris = 0, nedges = 0;
    std::vector<uint4> tri;        // x, y, z: internal vertex ids; w: body
    std::vector<uint4> tri_edges;  // x, y, z: edge ids of the triangle
    std::vector<uint2> edges;      // internal vertex ids (ascending caller id)
    std::vector<int> order;        // tree position -> triangle
};

// tris: [3 ntris] caller vertex ids; tri_body: [ntris]; viperm: caller ->
// internal vertex (null: identity); x: [nv] positions, internal order, that the
// triangles' tree order follows; now: those of the detection to come.  Throws Error
// on bad input.
CcdSurface build_ccd_surface(int nv, int ntris, const uint32_t* tris, const int* tri_body, const int* viperm,
                             const float4* x, bool now);

// A device list that grows, and the capacity its kernels get: never more than it
// holds, also after an allocation that failed (which leaves no list).
struct CcdList {
    DBuf<int2> items;
    int cap = 0;
    int least = 1;  // what it starts with

    void grow(long long count) {
        cap = 0;
        items.alloc((size_t)count);
        cap = (int)count;
    }
    void ensure() {
        if (cap == 0) grow(least);
    }
};

struct CcdStats {
    long long pairs = 0;        // candidate triangle pairs of the last detection
    int marked = 0;             // vertices with tI < 1
    int regrows = 0;            // candidate buffer enlargements so far
    double ms = 0.0;            // device time of the last detection
};

// CCDKernel + the fixed-body correction of XTilde and v (the reference
// applies it after the collision response, pdSolver.cu:228-231).
struct CcdResponse {
    float4* x;
    float4* v;
    SceneArgs sc;
};

class CcdContext {
public:
    // vcaller: device array internal -> caller vertex id (null: identity),
    // kept by the caller for the context's lifetime.  once: for one detection.
    CcdContext(const CcdSurface& s, const int* vcaller, cudaStream_t stream, bool once = false);
    ~CcdContext();
    CcdContext(const CcdContext&) = delete;
    CcdContext& operator=(const CcdContext&) = delete;

    // Detection between x (start, internal order) and xt (end): fills tI and
    // normals (device, internal order), and does the response if there is one to
    // do.  Waits for the stream once, behind both: the counts decide whether the
    // lists were long enough.
    void detect(const float4* x, const float4* xt, const CcdResponse* response = nullptr);

    const float* tI() const;
    const float4* normals() const;
    const CcdStats& stats() const { return stats_; }
    int nv() const { return nv_; }

private:
    void upload_order(const std::vector<uint4>& tri, const std::vector<int>& order);
    void keep_order(const float4* x);

    struct Buffers;
    std::unique_ptr<Buffers> b_;
    int nv_ = 0, ntris_ = 0, nedges_ = 0;
    const int* vcaller_ = nullptr;
    cudaStream_t stream_ = nullptr;
    CcdStats stats_;
};

}  // namespace pdgb
