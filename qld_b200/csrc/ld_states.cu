// ld_states.cu -- qLD's COUNTSTATES mode on the CUDA cores.
//
// countStates_mode (src/correlator/src/correlate_IO.c:472-516) gives every
// (A row, B row) pair a state value st: st = 0, then for each 64-bit word k
// the states present among the word's 64 bit pairs (bit bitA*2 + bitB) are
// ORed into st and st becomes the popcount of the result; the next word
// starts from that count read as a bit set.  The reference's per-bit loop
// (with its early exit once st == 15, which cannot change the popcount)
// reduces per word to
//     st = popc(st | S_k),  S_k bit 0: ~a & ~b != 0   bit 1: ~a & b != 0
//                           bit 2:  a & ~b != 0   bit 3:  a & b != 0
// Every word 0..K-1 counts, the zero tail bits of the last one included (they
// are state 00, as in the reference); words past K do not.
//
// A word maps the four values st can have after any word (1..4) to fewer:
// S = {00,01,10} makes it 3 and all four states make it 4 whatever came
// before, and most pairs of other words leave one value as well (f_S of 1..4
// for S = 1, 3, 5, 7, 15: 1,2,2,2 / 2,2,2,3 / 2,3,3,2 / 3,3,3,3 / 4,4,4,4).
// So the fold is evaluated from the END of the rows: F, four bytes, holds the
// final state for each value st may have before the words seen so far, and
// the word before them makes it F o f_S -- one byte permutation of F, whose
// selector is a sum of four terms (below).  A pair whose four bytes have
// become one value is finished, however long its rows are.  A tile takes
//   1. the last 4 words of all its pairs;
//   2. the remaining pairs (of founder haplotypes with 1 % noise, 1.3 %), up to
//      1,024, one by one towards the start, up to 64 words each, spread over
//      the threads;
//   3. for what remains (rows that are zero almost everywhere), one pass over
//      the remaining words of its 256 rows: if neither row has a bit there,
//      the state before the words seen is 1; if one has but every word still
//      contains state 00 (the largest word popcounts add up to less than 64),
//      it is 2, 3 or 4, which often suffices;
//   4. the next 16 words of all pairs, then 64, and so on to the start.
// Word 0 is entered with st = 0, so its map gives every byte F(popc(S)) and
// settles every pair.  The results are the same for any input, and rows that
// defeat every shortcut cost one walk over all their words.
//
// Bound by integer issue: 13 instructions per pair and word (two LOP3 per joint
// state, the second setting the predicate of an addition, and a permutation),
// 6.8-8.0 us per word of a 4,001-SNP single region, over 4 words instead of K.
// With compares and selects between them, 19 instructions, tables of up to
// seven words and rows that defeat every shortcut took longer than the forward
// fold (one POPC per pair and word, over all words).  In us, forward fold / 19
// instructions / 13: 200 SNPs x 300 samples (K = 5) 17.3 / 19.0 / 15.3; 64 SNPs
// of K = 2 8.1 / 10.5 / 8.0; 4,001 SNPs x 16,622 samples (K = 260) all ones
// 2,368 / 2,531 / 2,089, 24 founder haplotypes with 1 % noise 2,365 / 61 / 54, one
// bit per row 2,367 / 209 / 202, dense random rows 2,367 / 49 / 42.
//
// One CTA per 128 x 128 tile, 256 threads: lane l holds A rows l + 32 i, warp
// w B rows 16 w + j, a thread 4 x 16 pairs, so a store writes 32 consecutive
// bytes.  Output: one byte per pair, st[(b - out_row0) * lds + a], inside the
// diagonal window (single region: a >= b).
#include "qld_device.cuh"
#include "qld_kernels.h"

namespace qld {

namespace {

constexpr int BM = 128, BN = 128;
constexpr int THREADS = 256;
constexpr int NI = 4, NJ = 16;           // A and B rows of a thread
constexpr int W = 4;                     // words per chunk, and of the first walk
constexpr int SHORT = 5;
constexpr int LIST = 1024;               // remaining pairs walked one by one
constexpr int LIST_WORDS = 64;           // words each of them may take
constexpr uint32_t START = 0x04030201u;  // F before any word

// F o f_S for one word pair (32-bit halves).  Byte i of the result is byte
// f_S(i + 1) - 1 of F, and f_S(v) = popc(v | S): as a permutation selector, a
// nibble for each v = 1..4, state 00 adds 1 to those of v = 2 and 4 if present,
// 01 to v = 1 and 4, 10 to v = 1, 2 and 3, 11 to all, and v = 3 starts from 1.
// Before word 0 st is 0: every state adds 1 to every nibble, and they start
// from -1.
struct Terms {
    uint32_t base, c00, c01, c10;
    __device__ __forceinline__ explicit Terms(bool word0)
        : base(word0 ? 0u - 0x1111u : 0x0100u), c00(word0 ? 0x1111u : 0x1010u),
          c01(word0 ? 0x1111u : 0x1001u), c10(word0 ? 0x1111u : 0x0111u) {}
};
// x += c if LUT(t, u, v) has a bit: the LOP3's own predicate, without a compare.
template <int LUT>
__device__ __forceinline__ void add_if(uint32_t &x, uint32_t t, uint32_t u, uint32_t v, uint32_t c) {
    asm("{\n\t.reg .pred p, f;\n\t.reg .b32 d;\n\t"
        "setp.ne.u32 f, 0, 0;\n\t"
        "lop3.or.b32 d|p, %1, %2, %3, %5, f;\n\t"
        "@p add.u32 %0, %0, %4;\n\t}"
        : "+r"(x) : "r"(t), "r"(u), "r"(v), "r"(c), "n"(LUT));
}
__device__ __forceinline__ uint32_t before(uint32_t F, uint2 a, uint2 b, const Terms &t) {
    uint32_t sel = t.base;
    add_if<0xF8>(sel, a.x & b.x, a.y, b.y, 0x1111u);
    add_if<0xF4>(sel, a.x & ~b.x, a.y, b.y, t.c10);
    add_if<0xF2>(sel, ~a.x & b.x, a.y, b.y, t.c01);
    add_if<0x1F>(sel, a.x | b.x, a.y, b.y, t.c00);
    return __byte_perm(F, F, sel);
}

// The state if it does not depend on the words before (1..4), else 0.
__device__ __forceinline__ uint32_t settled(uint32_t F) {
    const uint32_t v = F & 255u;
    return F == v * 0x01010101u ? v : 0u;
}

__device__ __forceinline__ uint2 load_word(const uint64_t *p) {
    return *reinterpret_cast<const uint2 *>(p);
}

// One pair's words s0 - 1, s0 - 2, ... put before those of F, until its state is
// settled; 0 if it is not after LIST_WORDS words.  Eight words' loads are in
// flight at once.
__device__ __noinline__ uint32_t walk_back(const uint64_t *a, const uint64_t *b, int s0,
                                           uint32_t F) {
    const int stop = s0 > LIST_WORDS ? s0 - LIST_WORDS : 0;
    for (int k0 = s0; k0 > stop; k0 -= 8) {
        uint2 wa[8], wb[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (k0 - 1 - q >= stop) {
                wa[q] = load_word(a + k0 - 1 - q);
                wb[q] = load_word(b + k0 - 1 - q);
            }
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (k0 - 1 - q >= stop) F = before(F, wa[q], wb[q], Terms(k0 - 1 - q == 0));
        const uint32_t v = settled(F);
        if (v) return v;
    }
    return 0u;
}

__global__ void __launch_bounds__(THREADS, 2) k_states(const StatesParams p) {
    __shared__ uint2 sA[W][BM], sB[W][BN];
    __shared__ uint32_t row_info[BM + BN];   // largest word popcount of the remaining words
    __shared__ uint32_t list_pair[LIST], list_x[LIST];
    __shared__ uint32_t not_done[THREADS][2];
    __shared__ int listed;

    int ta = blockIdx.x, tb = blockIdx.y;    // the tile, tb from tb0
    if (p.symmetric) {
        // the grid is the triangle's tiles in a row: tile row y starts at first(y)
        const int wide = (p.m + BM - 1) / BM - p.tb0, at = blockIdx.x;
        auto first = [wide](int y) { return (long long)y * wide - (long long)y * (y - 1) / 2; };
        const float w2 = 2.0f * (float)wide + 1.0f;
        tb = (int)((w2 - sqrtf(fmaxf(w2 * w2 - 8.0f * (float)at, 0.0f))) * 0.5f);
        while (first(tb + 1) <= at) ++tb;
        while (first(tb) > at) --tb;
        ta = p.tb0 + tb + (int)(at - first(tb));
    }
    const int a0 = ta * BM, b0 = (p.tb0 + tb) * BN;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int my_a = a0 + lane, my_b = b0 + warp * NJ;
    // the row this thread loads: A rows first
    const bool is_a = tid < BM;
    const int row = is_a ? a0 + tid : b0 + tid - BM;
    const bool row_ok = row < (is_a ? p.m : p.n);
    const uint64_t *row_words =
        is_a ? p.A + (long long)row * p.lda : p.B + (long long)row * p.ldb;
    uint2 *row_smem = is_a ? &sA[0][tid] : &sB[0][tid - BM];

    // pairs the task does not have count as finished (0.5 us of a small table's
    // time when asked pair by pair)
    static_assert(NI == 4 && NI * NJ == 64, "a bit per pair");
    uint64_t done = ~0ull;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int a = my_a + 32 * i;
        int n = (p.symmetric && a + 1 < p.n ? a + 1 : p.n) - my_b;   // my first n B rows count
        n = a < p.m && n > 0 ? (n < NJ ? n : NJ) : 0;
        const uint64_t mine = n == NJ ? ~0ull : (1ull << (NI * n)) - 1ull;
        done &= ~(mine & 0x1111111111111111ull << i);
    }
    auto put = [&](int j, int i, uint32_t st) {
        p.out[(long long)(my_b + j - p.out_row0) * p.lds + my_a + 32 * i] = (uint8_t)st;
        done |= 1ull << (j * NI + i);
    };

    uint32_t x[NJ][NI];                      // F of every pair
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < NI; ++i) x[j][i] = START;

    // up to SHORT words at once: what follows the first four costs more than one
    // word does (200 SNPs x 300 samples 17.4 -> 15.3 us; all of K = 8 17.4 -> 21.2)
    long long len = p.K <= SHORT ? p.K : W;
    for (int end = p.K;; len *= 4) {
        const int s0 = end > len ? (int)(end - len) : 0;
        const bool busy = __any_sync(0xffffffffu, ~done != 0ull);
        for (int e = end; e > s0; e -= W) {  // words [e - W, e), last first
            __syncthreads();
#pragma unroll
            for (int w = 0; w < W; ++w)
                row_smem[w * BM] = row_ok && e - 1 - w >= s0 ? load_word(row_words + e - 1 - w)
                                                             : make_uint2(0u, 0u);
            __syncthreads();
            if (!busy) continue;
            const int words = e - s0 < W ? e - s0 : W;
#pragma unroll 1
            for (int w = 0; w < words; ++w) {
                const Terms terms(e - 1 - w == 0);
                uint2 a[NI];
#pragma unroll
                for (int i = 0; i < NI; ++i) a[i] = sA[w][lane + 32 * i];
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const uint2 b = sB[w][warp * NJ + j];
#pragma unroll
                    for (int i = 0; i < NI; ++i) x[j][i] = before(x[j][i], a[i], b, terms);
                }
            }
        }
        end = s0;
        // 1. the settled pairs; the others are listed
        if (tid == 0) listed = 0;
        not_done[tid][0] = not_done[tid][1] = 0u;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int k = j * NI + i;
                if ((done >> k) & 1ull) continue;
                const uint32_t v = settled(x[j][i]);
                if (v) {
                    put(j, i, v);
                    continue;
                }
                const int at = atomicAdd(&listed, 1);
                if (at < LIST) {                 // its walker finishes it, or says so
                    list_pair[at] = (uint32_t)(tid << 8 | k);
                    list_x[at] = x[j][i];
                    done |= 1ull << k;
                }
            }
        __syncthreads();
        const int entries = listed < LIST ? listed : LIST;
        if (listed == 0) break;
        // 2. one by one, spread over the threads
        for (int e = tid; e < entries; e += THREADS) {
            const int k = (int)(list_pair[e] & 255u), owner = (int)(list_pair[e] >> 8);
            const int a = a0 + (owner & 31) + 32 * (k % NI), b = b0 + (owner >> 5) * NJ + k / NI;
            const uint32_t v = walk_back(p.A + (long long)a * p.lda, p.B + (long long)b * p.ldb,
                                         s0, list_x[e]);
            if (v) p.out[(long long)(b - p.out_row0) * p.lds + a] = (uint8_t)v;
            else atomicOr(&not_done[owner][k >> 5], 1u << (k & 31));
        }
        __syncthreads();
        done &= ~((uint64_t)not_done[tid][1] << 32 | not_done[tid][0]);
        if (!__syncthreads_or(~done != 0ull)) break;
        // 3. what the words before s0 hold, row by row
        uint32_t most = 0;
        if (row_ok) {
#pragma unroll 8
            for (int k = 0; k < s0; ++k) {
                const uint2 v = load_word(row_words + k);
                const uint32_t c = (uint32_t)(__popc(v.x) + __popc(v.y));
                most = c > most ? c : most;
            }
        }
        row_info[tid] = most;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                if ((done >> (j * NI + i)) & 1ull) continue;
                const uint32_t ca = row_info[lane + 32 * i], cb = row_info[BM + warp * NJ + j];
                const uint32_t F = x[j][i], v = (F >> 8) & 255u;
                if (ca + cb == 0u) put(j, i, F & 255u);
                else if (ca + cb < 64u && F >> 8 == v * 0x010101u) put(j, i, v);
            }
        if (!__syncthreads_or(~done != 0ull)) break;
    }
}

}  // namespace

cudaError_t launch_states(const StatesParams &p, int tiles_b, cudaStream_t st) {
    if (tiles_b <= 0 || p.m <= 0) return cudaSuccess;
    dim3 grid((p.m + BM - 1) / BM, tiles_b);
    if (p.symmetric) {
        // Only the tiles at or above the diagonal: blocks that return at once let
        // two of the others share an SM while a third of the SMs is idle
        const long long wide = (long long)grid.x - p.tb0, rows = wide < tiles_b ? wide : tiles_b;
        if (rows <= 0) return cudaSuccess;
        grid = dim3((unsigned)(rows * wide - rows * (rows - 1) / 2));
    }
    k_states<<<grid, THREADS, 0, st>>>(p);
    return cudaGetLastError();
}

const int kStatesRows = BN;

}  // namespace qld
