// build_layout of a mesh large enough for several threads, with the n-th
// allocation failing, for every n: it throws, and never ends the program.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>

#include "engine.h"

static std::atomic<long> g_left{-1};  // allocations until one fails; < 0: none does
static std::atomic<long> g_count{0};

void* operator new(std::size_t n) {
    g_count++;
    if (g_left.load() >= 0 && g_left.fetch_sub(1) == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

namespace pdgb {
void set_last_error(int, const std::string&) {}
}  // namespace pdgb

int main() {
    // a row of 33,000 cells of 2 tets each: 66,000 tets, four parts
    const int cells = 33000, nv = 3 * (cells + 1), nt = 2 * cells;
    std::vector<float> X(3 * (size_t)nv), mass(nv, 1.f), mu(nt, 1.f);
    std::vector<uint32_t> tets;
    for (int i = 0; i <= cells; ++i)
        for (int c = 0; c < 3; ++c) {
            X[9 * (size_t)i + 3 * c] = 0.01f * i;
            X[9 * (size_t)i + 3 * c + 1] = c == 1;
            X[9 * (size_t)i + 3 * c + 2] = c == 2;
        }
    for (int i = 0; i < cells; ++i) {
        const uint32_t a = 3 * i;
        for (uint32_t v : {a, a + 1, a + 2, a + 3, a + 1, a + 2, a + 3, a + 4}) tets.push_back(v);
    }
    pdgb_params prm{};
    prm.dt = 0.01f;
    prm.num_iterations = 1;
    auto run = [&](long fail) {  // allocations made, or -1 where one failed
        g_count = 0;
        g_left = fail;
        long made = -1;
        try {
            pdgb::HostLayout L;
            pdgb::build_layout(nv, nt, X.data(), tets.data(), mass.data(), mu.data(), nullptr, prm, L);
            made = g_count;
        } catch (const std::bad_alloc&) {
        }
        g_left = -1;
        return made;
    };
    const long all = run(-1);
    // the allocations of the tile cut are many and alike: the last of them, and all before
    long failed = 0;
    for (long n = 0; n < all && n < 100; ++n) failed += run(n) < 0;
    std::printf("ok %d\n", failed > 20);
    return 0;
}
