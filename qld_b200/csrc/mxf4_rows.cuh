// mxf4_rows.cuh -- the bit -> E2M1 unpack of the SM-pair 4-bit kernels
// (ld_mxf4_pair.cu, ld_mxf4_split.cu, ld_batch.cu), one packed row at a time.
#pragma once

#include <stdint.h>

#include "tcgen05.cuh"

namespace qld {
namespace mxf4rows {

template <int T>
__device__ __forceinline__ uint4 spread4(const uint4 &w) {
    return make_uint4(tc::spread_e2m1<T>(w.x), tc::spread_e2m1<T>(w.y), tc::spread_e2m1<T>(w.z),
                      tc::spread_e2m1<T>(w.w));
}

// A packed stage holds the CTA's 128 A rows and then its B rows, 64 bytes
// each (64-byte swizzle); an unpacked stage the same rows in the same order,
// 128 bytes each (128-byte swizzle).  A thread of a group of GT takes rows
// row0, row0 + GT, ...: GT is a multiple of 8, so all of them have row0's
// swizzle phases and one set of offsets serves every row.  A quarter-warp
// covers 8 consecutive rows, so its 16-byte loads and stores touch all 32
// banks once.
template <int GT>
struct RowLane {
    static_assert(GT % 8 == 0, "rows of a thread share their swizzle phase");
    int row0;
    uint32_t xr;         // 64-byte swizzle phase
    uint32_t off[8];     // destination of chunk 0..7 in row0
    __device__ __forceinline__ explicit RowLane(int r) : row0(r), xr((uint32_t)(r >> 1) & 3u) {
#pragma unroll
        for (int c = 0; c < 8; ++c) off[c] = (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4));
    }
};

// Sub-stage `sub` (0 or 1: 256 of the 512 samples) of a packed stage into an
// unpacked stage: every word's bits spread over four E2M1 words
// (spread_e2m1).  Up to TASKS rows per thread of the stage's nrows, two rows'
// loads in flight at a time.
template <int GT, int TASKS>
__device__ __forceinline__ void unpack_rows(const RowLane<GT> &l, int nrows, const uint8_t *packed,
                                            uint8_t *unpacked, int sub) {
#pragma unroll
    for (int j0 = 0; j0 < TASKS; j0 += 2) {
        uint4 w[2][2];
#pragma unroll
        for (int j = j0; j < j0 + 2 && j < TASKS; ++j)
            if (l.row0 + j * GT < nrows) {
                const uint8_t *row = packed + (l.row0 + j * GT) * 64;
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    w[j - j0][h] = *reinterpret_cast<const uint4 *>(
                        row + ((((uint32_t)sub * 2 + h) ^ l.xr) << 4));
            }
#pragma unroll
        for (int j = j0; j < j0 + 2 && j < TASKS; ++j) {
            if (l.row0 + j * GT >= nrows) continue;
            uint8_t *dst = unpacked + j * GT * 128;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 &x = w[j - j0][h];
                *reinterpret_cast<uint4 *>(dst + l.off[h * 4 + 0]) = spread4<0>(x);
                *reinterpret_cast<uint4 *>(dst + l.off[h * 4 + 1]) = spread4<1>(x);
                *reinterpret_cast<uint4 *>(dst + l.off[h * 4 + 2]) = spread4<2>(x);
                *reinterpret_cast<uint4 *>(dst + l.off[h * 4 + 3]) = spread4<3>(x);
            }
        }
    }
}

}  // namespace mxf4rows
}  // namespace qld
