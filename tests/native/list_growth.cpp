// A collision list whose allocation fails, against stand-ins for the CUDA calls:
// kernels never get a capacity that no memory stands behind.
#include <cstdio>
#include <cstdlib>

#include "ccd.h"

static int g_fail = 0;  // allocations that fail from now on
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    if (g_fail > 0) {
        --g_fail;
        return g_last = cudaErrorMemoryAllocation;
    }
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return ""; }
}

static void expect(bool ok, const char* what) {
    if (ok) return;
    std::printf("failed: %s\n", what);
    std::exit(1);
}

static bool throws(pdgb::CcdList& l, long long n) {
    try {
        n ? l.grow(n) : l.ensure();
    } catch (const pdgb::Error& e) {
        return e.status == PDGB_ERR_OUT_OF_MEMORY;
    }
    return false;
}

static bool backed(const pdgb::CcdList& l) { return l.cap == 0 || (l.items.p && l.items.n >= (size_t)l.cap); }

int main() {
    pdgb::CcdList l;
    l.least = 64;
    l.ensure();
    expect(l.cap == 64 && backed(l), "the first allocation");
    g_fail = 1;
    expect(throws(l, 1000), "a failure is reported");
    expect(backed(l), "capacity after a failure");
    expect(cudaGetLastError() == cudaSuccess, "the error is not left behind");
    g_fail = 1;
    expect(throws(l, 0) && backed(l), "a second failure");
    l.ensure();
    expect(l.cap == 64 && backed(l), "the next detection has its first list again");
    l.grow(1000);
    l.ensure();
    expect(l.cap == 1000 && backed(l), "growth");
    std::puts("ok");
    return 0;
}
