// Index arithmetic of a panel's diagonal block (factor.cu), for host and device.
#pragma once

#ifdef __CUDACC__
#define PDGB_PANEL_HD __host__ __device__
#else
#define PDGB_PANEL_HD
#endif

namespace pdgb {

// Entries of the nb x nb block past its first r0 rows and columns: none once r0
// reaches nb, which it passes by up to seven where nb is not a multiple of the
// eight columns of a step.
PDGB_PANEL_HD inline int trailing_entries(int nb, int r0) { return r0 < nb ? (nb - r0) * (nb - r0) : 0; }

struct BlockEntry {
    int r, c;
};
// Entry e < trailing_entries(nb, r0) of them, row after row.
PDGB_PANEL_HD inline BlockEntry trailing_entry(int nb, int r0, int e) {
    return {r0 + e / (nb - r0), r0 + e % (nb - r0)};
}

}  // namespace pdgb
