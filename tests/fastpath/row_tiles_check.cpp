// CPU check of RowTiles (qld_b200/csrc/mxf4_tiles.cuh): over random tasks, row
// ranges and tile heights, every entry the launch owes is in exactly one
// tile, and every tile starts inside the table.
#include <cstdio>
#include <cstdlib>
#include <vector>

#define __host__
#define __device__
#define __forceinline__ inline
#include "mxf4_tiles.cuh"

int main() {
    srand(7);
    long long tiles = 0;
    for (int trial = 0; trial < 4000; ++trial) {
        const int kind = rand() % 3;   // two regions, single region, band
        const int m = 1 + rand() % 900, n = kind ? m : 1 + rand() % 900;
        const int band = kind == 2 ? 1 + rand() % 500 : 0;
        const int bn = 16 * (1 + rand() % 15);
        const int b0 = rand() % 2 ? 0 : rand() % n / 16 * 16, b1 = b0 + 1 + rand() % (n - b0);
        const qld::RowTiles tl{m, b0, b1, bn, kind != 0, band};
        std::vector<unsigned char> hit((size_t)n * m, 0);
        int t = 0, base = 0;
        const int count = tl.count();
        for (int idx = 0; idx < count; ++idx, ++tiles) {
            int a, b;
            tl.decode_from(idx, a, b, t, base);
            if (a < 0 || a >= m || b < b0 || b >= b1) return printf("tile outside\n"), 1;
            for (int i = b; i < b + bn && i < b1; ++i)
                for (int j = a; j < a + tl.BM && j < m; ++j) ++hit[(size_t)i * m + j];
        }
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < m; ++j) {
                const bool owed = i >= b0 && i < b1 &&
                                  (band ? j > i && j - i <= band : kind == 1 ? j >= i : true);
                if (hit[(size_t)i * m + j] > 1 || (owed && !hit[(size_t)i * m + j]))
                    return printf("entry %d %d covered %d times\n", i, j, hit[(size_t)i * m + j]), 1;
            }
    }
    printf("ok %lld tiles\n", tiles);
    return 0;
}
