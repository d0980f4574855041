// mxf4_tiles.cuh -- the output tiles of a launch of the SM-pair 4-bit kernels.
#pragma once

#include <cuda_runtime.h>

namespace qld {

// Tiles of 256 A rows x bn B rows over B rows [b0, b1), numbered B rows
// first.  Tile row t holds B rows [b0 + t bn, ...); its A tiles start at a0(t)
// and follow one another every 256 rows: from row 0 for two regions, from the
// 256-row boundary below the diagonal for a single region, and for a band
// right at the band's first row (1 <= a - b <= band), which the TMA loads allow
// (only their inner coordinate has an alignment rule).  Starting a band's
// tiles on the 256-row grid instead covers the W + bn - 1 rows a tile row
// needs with (W + bn + 255) / 256 tiles on average: 5.84 against 5 for
// W = 1,000 (50,000 SNPs x 10,001 samples: 285 against 222 us), 21.46 against
// 21 for W = 5,000 (24,000 x 100,000: 3.39 against 3.29 ms).
struct RowTiles {
    static constexpr int BM = 256;
    int m, b0, b1, bn, symmetric, band;

    __host__ __device__ __forceinline__ int rows() const { return (b1 - b0 + bn - 1) / bn; }
    __host__ __device__ __forceinline__ int b(int t) const { return b0 + t * bn; }
    __host__ __device__ __forceinline__ int a0(int t) const {
        return band > 0 ? b(t) + 1 : symmetric ? (b(t) & ~255) : 0;
    }
    // A tiles of tile row t
    __host__ __device__ __forceinline__ int width(int t) const {
        int end = m;
        if (band > 0) {
            const int last = (b1 - b(t) < bn ? b1 : b(t) + bn) - 1;   // its last B row
            if (band < m - 1 - last) end = last + band + 1;
        }
        const int w = end - a0(t);
        return w > 0 ? (w + (BM - 1)) / BM : 0;
    }
    __host__ __device__ __forceinline__ int count() const {
        int n = 0;
        for (int t = 0; t < rows(); ++t) n += width(t);
        return n;
    }
    // First A and B row of tile idx, for a caller whose indices never
    // decrease (a persistent CTA walking its tiles): the walk over tile rows
    // resumes at (t, base), the tile row and the count of tiles before it
    // where the previous call stopped, so a call costs the tile rows stepped
    // over instead of all of them.
    __device__ __forceinline__ void decode_from(int idx, int &a, int &brow, int &t,
                                                int &base) const {
        const int nt = rows();
        for (; t < nt; ++t) {
            const int w = width(t);
            if (idx < base + w) {
                a = a0(t) + (idx - base) * BM;
                brow = b(t);
                return;
            }
            base += w;
        }
        a = brow = 0;
    }
};

}  // namespace qld
