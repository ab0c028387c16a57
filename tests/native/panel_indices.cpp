// Walks the entries that the diagonal block's trailing update touches, for every
// block size, as factor.cu does: prints the first bad size, or "ok".
#include <cstdio>
#include <vector>

#include "panel.h"

int main() {
    constexpr int kNB = 32, kSub = 8;
    for (int nb = 1; nb <= kNB; ++nb)
        for (int c0 = 0; c0 < nb; c0 += kSub) {
            const int r0 = c0 + kSub, n = pdgb::trailing_entries(nb, r0);
            std::vector<int> seen(kNB * kNB, 0);
            for (int e = 0; e < n; ++e) {
                const pdgb::BlockEntry q = pdgb::trailing_entry(nb, r0, e);
                if (q.r < r0 || q.r >= nb || q.c < r0 || q.c >= nb) {
                    std::printf("block of %d past column %d: entry (%d, %d)\n", nb, r0, q.r, q.c);
                    return 1;
                }
                seen[kNB * q.r + q.c]++;
            }
            for (int r = r0; r < nb; ++r)
                for (int c = r0; c < nb; ++c)
                    if (seen[kNB * r + c] != 1) {
                        std::printf("block of %d past column %d: (%d, %d) taken %d times\n", nb, r0, r, c, seen[kNB * r + c]);
                        return 1;
                    }
        }
    std::puts("ok");
    return 0;
}
