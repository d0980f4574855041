// ld_mxf4_pair.cu -- counts kernel, variant (c) on SM pairs: the 4-bit
// tensor-core path of ld_mxf4.cu (bits spread to E2M1 with normalising
// UE8M0 scale factors, tcgen05.mma.kind::mxf4 into F32 accumulators, exact
// below 2^24, FP32 r^2 epilogue)
// with every 256 x 240 output tile computed by a cluster of two CTAs on two
// SMs through tcgen05.mma.cta_group::2.
//
// Why pairs: one SM computing a 256 x 240 tile needs two 240-column
// accumulators, which with the scale factors fill its 512 TMEM columns, so
// the r^2 epilogue of a tile cannot overlap the MMAs of the next; and each
// of its two 128-row MMAs reads all 240 unpacked B rows.  Split over a pair,
// each SM holds 128 A rows and 120 B rows, one 128 x 240 accumulator per
// tile, and TMEM room for two of them: the epilogue warps drain one while
// the MMAs fill the other, and each SM's shared memory supplies every
// unpacked row once per MMA.
//
// Roles (both CTAs of a pair, 576 or 608 threads):
//   warp 0       TMA producer: the CTA's 128 A rows and 120 B rows, 8 packed
//                words (512 samples) per stage, 64-byte swizzle.
//   warp 1       TMEM allocation for the pair (cta_group::2); in rank 0 the
//                MMA issuer: per unpacked stage (256 samples) 4 MMAs of
//                256 x 240 x 64, then one commit that arrives on the stage's
//                "empty" barrier in both CTAs.  The whole warp runs the issue
//                loop (tcgen05.cuh, elect_one): single region 2.39 -> 2.375
//                ms, band of 5,000 over 24,000 x 100,000 3.45 -> 3.39 ms.
//   warps 2-9    unpack (w -> four words of nibbles, mxf4_rows.cuh) into the
//                CTA's stage; they arrive on rank 0's "full" barrier.  Four
//                groups of two warps take the unpacked stages in turn.  A
//                group's steps for a stage are one serial chain (wait for the
//                packed data and for the free buffer, load, spread, store,
//                proxy fence, arrive: ~1,250 cycles by clock64), so two groups
//                (of five warps) handed a stage over only every ~650 cycles,
//                whatever the tensor cores and shared memory allowed; with
//                four a stage takes ~580, where the MMAs alone take 523 (565 at
//                the rate they keep up back to back).  Single region 2.36 -> 2.12 ms (first 100
//                launches; 2.41 -> 2.21 in a power-capped loop), 5,000-wide
//                band 3.26 -> 2.80 ms, 9,001 x 7,003 x 16,622 reference mode
//                with counts 403 -> 349 us.  Three groups of three: 2.16 ms /
//                2.85 / 367; four of three (80 registers): 2.13 / 2.82 / 359.
//   warps 10-17  epilogue: warp w reads TMEM lane quarter w % 4 of the
//                accumulator buffer the tile used, every other one of its
//                fifteen 16-column chunks, applies the r^2 epilogue (gemm_cpu.c:343-404) and
//                stores; they arrive on rank 0's "accumulator empty" barrier.
//                The next tile's bit counts load meanwhile: loading them and
//                dividing at the tile's start cost 2,600-4,600 of the 12,000-
//                23,000 cycles a tile's epilogue took.  Twelve epilogue warps
//                (80 registers): band of 1,000 210 us against 199, reference
//                mode 347 against 341.
//   warp 18      (FW) the column factors, a tile or two ahead: the epilogue
//                warps then neither divide for columns nor meet at a barrier,
//                and each runs ahead of the others by up to a tile.  Where it
//                pays: factor_warp() below.
// Every wait on an mbarrier is bounded.  No thread returns early: both CTAs meet
// at the cluster barriers at start and end on every path, including after a
// timeout, and the TMEM is released only after the last MMA has completed.  Those
// barriers and the epilogue warps' named one (!FW) have no limit: after a failed
// wait an epilogue warp goes on through its tiles, meeting the others once in each.
#include "epilogue.cuh"
#include "launch_util.h"
#include "mxf4_rows.cuh"
#include "mxf4_tiles.cuh"
#include "qld_kernels.h"
#include "tcgen05.cuh"

namespace qld {

namespace {

using namespace tc;

constexpr int BM = RowTiles::BM, BN = 240;        // output tile of a pair
constexpr int HM = 128, HN = 120;        // A and B rows held by each CTA
constexpr int PW = 8;                    // packed words per row per packed stage
constexpr int SUB = 2;                   // unpacked stages (256 samples) per packed stage
constexpr int SW = PW / SUB;             // words per row per unpacked stage
constexpr int UST = 4;                   // one unpacked stage per unpack group
constexpr int PA_BYTES = HM * PW * 8;    // 8 KB
constexpr int P_MAX = (HM + HN) * PW * 8;   // up to 15.5 KB delivered per stage
constexpr int P_BYTES = 15872;           // stage stride: A rows, then B rows (a multiple of 512)
constexpr int UA_BYTES = HM * 128;       // 16 KB: 256 E2M1 per row
constexpr int U_BYTES = (HM + HN) * 128; // 31 KB: A rows, then B rows
constexpr int GROUPS = 4, GROUP_WARPS = 2;
constexpr int UNPACK_WARPS = GROUPS * GROUP_WARPS, EPI_WARPS = 8;
constexpr int FIRST_UNPACK_WARP = 2;
constexpr int FIRST_EPI_WARP = FIRST_UNPACK_WARP + UNPACK_WARPS;
constexpr int FACTOR_WARP = FIRST_EPI_WARP + EPI_WARPS;
constexpr int threads(bool fw) { return (FACTOR_WARP + fw) * 32; }   // 576 or 608
constexpr int GROUP_THREADS = GROUP_WARPS * 32;              // unpackers per stage
constexpr int TASKS = (HM + HN + GROUP_THREADS - 1) / GROUP_THREADS;   // rows per thread
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t ACC_STRIDE = 256;     // accumulator buffers at columns 0 and 256
constexpr uint32_t SF_COL = 496;         // 16 columns of scale factors
constexpr int COLS_N = 256;              // epilogue column factors (BN used)
constexpr uint16_t BOTH = 0x3;           // CTA mask of a commit to both ranks

// Shared-memory layout per r^2 mode.  R2_EXACT needs 8 bytes of column
// factors per column (epi::ColsF), R2_REFERENCE 16 (epi::ColsR2); both leave
// room for six packed stages (more TMA lookahead than five: 2.576 -> 2.562
// ms on the single region).
template <int MODE>
struct Smem {
    static constexpr int PST = 6;                          // packed stages in flight
    static constexpr int OFF_U = 0;
    static constexpr int OFF_P = OFF_U + UST * U_BYTES;
    static constexpr int OFF_ROWS = OFF_P + PST * P_BYTES;
    static constexpr int ROWS_BYTES = COLS_N * (MODE == R2_EXACT ? 8 : epi::COLR_BYTES);
    static constexpr int OFF_BAR = OFF_ROWS + 2 * ROWS_BYTES;   // this tile's and the next one's
    static constexpr int NBARS = 2 * PST + 2 * UST + 2 + 2 + 1 + 2 + 2;
    static constexpr int OFF_TMEM = OFF_BAR + NBARS * 8;        // and the halves' special flags
    static constexpr int BYTES = OFF_TMEM + 16 + 1024;
    static_assert(BYTES <= 232448, "shared memory budget");
    static_assert(U_BYTES % 1024 == 0 && UA_BYTES % 1024 == 0 && OFF_P % 1024 == 0 &&
                      P_BYTES % 512 == 0 && P_MAX <= P_BYTES,
                  "swizzled stages must start on whole swizzle atoms");
    // a group sees every (GROUPS / 2)-th packed stage or so: a slot must
    // always belong to the same groups for its phase bit to be enough
    static_assert(PST * SUB % GROUPS == 0 && GROUPS == UST && GROUPS % SUB == 0, "stage rings");
};
static_assert(ACC_STRIDE + BN <= SF_COL && SF_COL + 16 <= TMEM_COLS, "TMEM map");
static_assert(SUB == 2 && EPI_WARPS * 32 == COLS_N && EPI_WARPS == 8, "work split");

// BAND: a band's launch (its window and tiles); otherwise two regions or a
// single region.  One kernel for both ran the other two 1.2 % slower.
// FULL: 240-row tiles, else tl.bn (a multiple of 16).
// PLAIN: a launch without counts (p.counts null; in reference mode R2_PLAIN_S <=
// S <= 2^24) whose tiles without special rows or columns take the epilogue
// without the rare cases' votes, flags and per-chunk addresses: 4,001 SNPs x
// 1,920 samples 22.0 -> 18.0 us, 12,000 x 5,120 155 -> 141, band of 1,000 over
// 50,000 x 10,001 199 -> 192, in reference mode 241 -> 222.  A branch in one
// kernel cost the launches with counts 1 %.
// FW: a warp of its own stores the column factors (otherwise the epilogue warps
// do, after a tile's chunks; factor_warp chooses).
template <int MODE, bool BAND, bool FULL, bool PLAIN, bool FW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(threads(FW), 1)
k_ld_mxf4_pair(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const LdParams p, const RowTiles all, const int ntiles) {
    using L = Smem<MODE>;
    constexpr int PST = L::PST;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::OFF_BAR);
    uint64_t *pfull = bars, *pempty = bars + PST;
    uint64_t *ufull = bars + 2 * PST, *uempty = bars + 2 * PST + UST;
    uint64_t *accfull = bars + 2 * PST + 2 * UST;
    uint64_t *accempty = accfull + 2;
    uint64_t *mma_done = accempty + 2;
    uint64_t *facfull = mma_done + 1, *facempty = facfull + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L::OFF_TMEM);
    volatile uint32_t *col_flag = tmem_slot + 1;     // a column of the half is special

    const uint32_t rank = cluster_rank();
    const int pair = (int)cluster_id_x(), npairs = (int)cluster_count_x();
    RowTiles tl = all;
    if (!BAND) tl.band = 0;
    if (FULL) tl.bn = BN;
    const int bn = tl.bn, hn = bn / 2;
    const int dlo = diag_lo(p.symmetric, tl.band), dhi = diag_hi(tl.band);
    const int my_tiles = pair < ntiles ? (ntiles - pair + npairs - 1) / npairs : 0;

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int np = (p.K + PW - 1) / PW;
    const int nu = np * SUB;
    // Stages that hold samples: a tile's last one is all padding if K mod 8 is 1
    // to 4, and is neither unpacked nor multiplied (29,817 SNPs, K = 260: 1,986 ->
    // 1,975 us; 9,001 x 7,003 in reference mode with counts 336 -> 333).  Tiles of
    // up to six stages keep it: they wait for their results' stores, which take
    // turns of their own (9,001 x 7,003, K = 18: 77 -> 83 us without it, but
    // 9,000 x 7,000 75 -> 73).
    const int nu_k = np > 3 ? (p.K + SW - 1) / SW : nu;

    if (tid == 0) {
        for (int s = 0; s < PST; ++s) {
            mbar_init(smem_u32(&pfull[s]), 1);
            mbar_init(smem_u32(&pempty[s]), SUB * GROUP_WARPS);
        }
        for (int s = 0; s < UST; ++s) {
            mbar_init(smem_u32(&ufull[s]), 2 * GROUP_WARPS);   // one group in each CTA
            mbar_init(smem_u32(&uempty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&accfull[b]), 1);
            mbar_init(smem_u32(&accempty[b]), 2 * EPI_WARPS);   // both CTAs' epilogues
            mbar_init(smem_u32(&facfull[b]), 1);
            mbar_init(smem_u32(&facempty[b]), EPI_WARPS);
        }
        mbar_init(smem_u32(mma_done), 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc<2>(smem_u32(tmem_slot), TMEM_COLS);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // The spread's scale factors (kSpreadScales) in columns SF_COL.. of every
    // lane, in both CTAs; warps 2-5 cover the four TMEM lane quarters.
    if (warp >= FIRST_UNPACK_WARP && warp < FIRST_UNPACK_WARP + 4)
        tc_st_32x32b_x16_fill(tmem + ((uint32_t)((warp & 3) * 32) << 16) + SF_COL, kSpreadScales);
    tc_fence_before();
    // barrier initialisation and both CTAs' scale factors, cluster-wide
    cluster_sync_all();
    tc_fence_after();
    griddep_launch();
    griddep_wait();

    if (warp == 0) {
        // ------------------------------------------------------- producer --
        if (lane == 0) {
            prefetch_tmap(&tmA);
            prefetch_tmap(&tmB);
            int gp = 0, cur_t = 0, cur_base = 0;
            bool ok = true;
            for (int i = 0; i < my_tiles && ok; ++i) {
                int a_row, b_row;
                tl.decode_from(pair + i * npairs, a_row, b_row, cur_t, cur_base);
                const int ra = a_row + (int)rank * HM, rb = b_row + (int)rank * hn;
                for (int kp = 0; kp < np; ++kp, ++gp) {
                    const int s = gp % PST;
                    if (gp >= PST && !mbar_wait(smem_u32(&pempty[s]), ((gp / PST) - 1) & 1,
                                                p.timeout_cycles, p.status)) {
                        flag_error(p.status, ST_TIMEOUT_EMPTY);
                        ok = false;
                        break;
                    }
                    const uint32_t fb = smem_u32(&pfull[s]);
                    const uint32_t dst = smem_u32(smem + L::OFF_P + s * P_BYTES);
                    mbar_arrive_expect_tx(fb, PA_BYTES + (uint32_t)(hn * PW * 8));
                    tma_load_2d(dst, &tmA, kp * PW, ra, fb);
                    tma_load_2d(dst + PA_BYTES, &tmB, kp * PW, rb, fb);
                }
            }
            for (int g = gp > PST ? gp - PST : 0; g < gp; ++g)
                if (!mbar_wait(smem_u32(&pfull[g % PST]), (g / PST) & 1, kDrainCycles,
                               nullptr)) {
                    flag_error(p.status, ST_TIMEOUT_DRAIN);
                    break;
                }
        }
    } else if (warp == 1) {
        // ------------------------------------------- MMA issuer (rank 0) --
        if (rank == 0) {
            const uint32_t sf = tmem + SF_COL;
            const uint32_t even = idesc_mxf4_sf(BM, bn, 0);   // k-steps 0, 2: scale bytes 0-1
            const uint32_t odd = idesc_mxf4_sf(BM, bn, 2);    // k-steps 1, 3: scale bytes 2-3
            const uint32_t a_lo = sw128_desc_lo(smem_u32(smem + L::OFF_U));
            uint32_t s = 0, ph = 0;      // unpacked stage and its phase
            bool ok = true;
            for (int it = 0; it < my_tiles && ok; ++it) {
                const int ab = it & 1;
                if (it >= 2) {
                    const bool free = mbar_wait(smem_u32(&accempty[ab]), ((it >> 1) - 1) & 1,
                                                p.timeout_cycles, p.status);
                    if (!__all_sync(0xffffffffu, free)) {
                        if (lane == 0) flag_error(p.status, ST_TIMEOUT_MMA);
                        break;
                    }
                }
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)ab * ACC_STRIDE;
                for (int u = 0; u < nu; ++u) {
                    const bool full = mbar_wait(smem_u32(&ufull[s]), ph, p.timeout_cycles,
                                                p.status);
                    if (!__all_sync(0xffffffffu, full)) {
                        if (lane == 0) flag_error(p.status, ST_TIMEOUT_UNPACK);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t da = a_lo + s * (U_BYTES >> 4), db = da + (UA_BYTES >> 4);
                    if (elect_one()) {
                        if (u < nu_k) {
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                tc_mma_mxf4_pair_lo(d, da + kk * 2, db + kk * 2,
                                                    (kk & 1) ? odd : even,
                                                    (u > 0 || kk > 0) ? 1u : 0u, sf, sf);
                        }
                        tc_commit_pair(smem_u32(&uempty[s]), BOTH);
                    }
                    __syncwarp();
                    if (++s == UST) s = 0, ph ^= 1;
                }
                if (elect_one()) tc_commit_pair(smem_u32(&accfull[ab]), BOTH);
                __syncwarp();
            }
            if (elect_one()) tc_commit_pair(smem_u32(mma_done), BOTH);
            __syncwarp();
        }
    } else if (warp < FIRST_EPI_WARP) {
        // --------------------------------------------------------- unpack --
        // Group g takes the unpacked stages gu = g, g + GROUPS, ...: always buffer
        // g and the same half of every other packed slot, so slot and phases
        // are counted up rather than divided out of gu and one vote serves
        // both waits (9,001 x 7,003 in reference mode with counts 340 -> 336 us,
        // 3,300 SNPs at K = 200 34.5 -> 33.1, single region 1,991 -> 1,986).
        const int grp = (warp - FIRST_UNPACK_WARP) / GROUP_WARPS;
        const mxf4rows::RowLane<GROUP_THREADS> rows(
            ((warp - FIRST_UNPACK_WARP) % GROUP_WARPS) * 32 + lane);
        const int total_u = my_tiles * nu;
        uint8_t *const dst = smem + L::OFF_U + grp * U_BYTES;
        const uint32_t uf = smem_u32(&ufull[grp]), ue = smem_u32(&uempty[grp]);
        int ps = grp / SUB, u = grp % nu;    // packed slot; the stage's place in its tile
        uint32_t ph = 0, eh = 1;             // phases of the packed slot and of the unpacked stage
        for (int gu = grp; gu < total_u; gu += GROUPS) {
            const bool got = mbar_wait(smem_u32(&pfull[ps]), ph, p.timeout_cycles, p.status);
            const bool freed = got && (gu < UST || mbar_wait(ue, eh, p.timeout_cycles, p.status));
            if (!__all_sync(0xffffffffu, freed)) {
                if (lane == 0) flag_error(p.status, got ? ST_TIMEOUT_MMA : ST_TIMEOUT_FULL);
                break;
            }
            if (u < nu_k)
                mxf4rows::unpack_rows<GROUP_THREADS, TASKS>(
                    rows, HM + hn, smem + L::OFF_P + ps * P_BYTES, dst, grp % SUB);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_rank(uf, 0);
                mbar_arrive(smem_u32(&pempty[ps]));     // one group per sub-stage
            }
            eh ^= 1;
            for (u += GROUPS; u >= nu;) u -= nu;
            if ((ps += GROUPS / SUB) >= PST) ps -= PST, ph ^= 1;
        }
    } else if (FW && warp == FACTOR_WARP) {
        // ------------------------------------------------- column factors --
        int cur_t = 0, cur_base = 0;
        for (int it = 0; it < my_tiles; ++it) {
            const int ab = it & 1;
            int a_row, b_row;
            tl.decode_from(pair + it * npairs, a_row, b_row, cur_t, cur_base);
            // every column factor the chunks read; 0 past the tile and the task
            uint32_t cb[COLS_N / 32];
#pragma unroll
            for (int i = 0; i < COLS_N / 32; ++i) {
                const int e = i * 32 + lane;
                cb[i] = e < bn && b_row + e < p.n ? p.bcB[b_row + e] : 0u;
            }
            const bool free = it < 2 || mbar_wait(smem_u32(&facempty[ab]), ((it >> 1) - 1) & 1,
                                                  p.timeout_cycles, p.status);
            if (!__all_sync(0xffffffffu, free)) {
                if (lane == 0) flag_error(p.status, ST_TIMEOUT_EMPTY);
                break;
            }
            uint8_t *base = smem + L::OFF_ROWS + ab * L::ROWS_BYTES;
            bool special = false;
#pragma unroll
            for (int i = 0; i < COLS_N / 32; ++i) {
                if constexpr (MODE == R2_EXACT)
                    special |= epi::store_col_f32(epi::ColsF(base, COLS_N), i * 32 + lane, cb[i], p.S);
                else
                    special |= epi::store_col_ref(epi::ColsR2(base, COLS_N), i * 32 + lane, cb[i],
                                                  p.S);
            }
            special = __any_sync(0xffffffffu, special);
            __syncwarp();                // every lane's factors are stored: a vote does not order them
            if (lane == 0) {
                col_flag[ab] = special;
                mbar_arrive(smem_u32(&facfull[ab]));
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------- epilogue --
        // The bit counts of the next tile's rows are loaded while this tile is
        // worked on, and (!FW) its factors stored in the other half of the buffer.
        const int et = tid - FIRST_EPI_WARP * 32;
        const int ew = warp - FIRST_EPI_WARP;
        const int q = warp & 3;                 // TMEM lane quarter
        int cur_t = 0, cur_base = 0, a_row = 0, b_row = 0;
        uint32_t ca = 0, cb = 0;                // bit counts of my row and column
        auto load_counts = [&](int it) {
            tl.decode_from(pair + it * npairs, a_row, b_row, cur_t, cur_base);
            const int a = a_row + (int)rank * HM + q * 32 + lane, b = b_row + et;
            ca = a < p.m ? p.bcA[a] : 0u;
            // every column factor the chunks read; 0 past the tile and the task
            if (!FW) cb = et < bn && b < p.n ? p.bcB[b] : 0u;
        };
        bool failed = false, special = false;
        epi::ARowR ra{};
        epi::ARowF raf{};
        auto store_factors = [&](int it) {
            uint8_t *base = smem + L::OFF_ROWS + (it & 1) * L::ROWS_BYTES;
            if constexpr (MODE == R2_EXACT) {
                raf = epi::make_arow_f32(ca, p.S);
                if (!FW) special = epi::store_col_f32(epi::ColsF(base, COLS_N), et, cb, p.S);
            } else {
                ra = epi::make_arow_ref(ca, p.S);
                if (!FW) special = epi::store_col_ref(epi::ColsR2(base, COLS_N), et, cb, p.S);
            }
        };
        if (my_tiles > 0) {
            load_counts(0);
            store_factors(0);
        }
        for (int it = 0; it < my_tiles; ++it) {
            const int ab = it & 1;
            // chunks colh, colh + 2, ... of the 15: without a barrier, 8 and 7 in turn
            const int colh = (ew >> 2) ^ (FW ? ab : 0);
            const int a = a_row + (int)rank * HM + q * 32 + lane, b_tile = b_row;
            const bool a_ok = a < p.m;
            // this tile's factors are stored, and (!FW) the other half is free
            bool cols_special = false;
            if constexpr (!FW) cols_special = named_bar_or(1, EPI_WARPS * 32, special);
            if (it + 1 < my_tiles) load_counts(it + 1);
            bool ready = !failed &&
                         (!FW || mbar_wait(smem_u32(&facfull[ab]), (it >> 1) & 1,
                                           p.timeout_cycles, p.status)) &&
                         mbar_wait(smem_u32(&accfull[ab]), (it >> 1) & 1, p.timeout_cycles,
                                   p.status);
            ready = __all_sync(0xffffffffu, ready);
            if (!ready && !failed) {            // (!FW: keep meeting the others at the barrier)
                if (lane == 0) flag_error(p.status, ST_TIMEOUT_MMA);
                failed = true;
            }
            if constexpr (FW) {
                if (!ready) break;
                cols_special = col_flag[ab] != 0u;
            }
            if (ready) {
                __syncwarp();
                tc_fence_after();
                uint8_t *base = smem + L::OFF_ROWS + ab * L::ROWS_BYTES;
                const uint32_t tbase =
                    tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)ab * ACC_STRIDE;
                const int n_tile = b_tile + bn < p.n ? b_tile + bn : p.n;
                // Chunks of 16 columns, in reference mode of 8: their packed
                // arithmetic keeps more values live (16 columns spill: band of
                // 1,000 in reference mode 244 us against 241).
                constexpr int CW = MODE == R2_EXACT ? 16 : 8;
                bool full = true;                // chunks with the rare cases' bookkeeping
                if constexpr (PLAIN) {
                    full = cols_special ||
                           __any_sync(0xffffffffu, MODE == R2_EXACT ? raf.special : ra.k.y != ra.k.y);
                    const long long step = (long long)(CW * EPI_WARPS / 4) * p.ldr;
                    float *o = p.r2 + (long long)(b_tile + colh * CW - p.out_row0) * p.ldr + a;
                    float rmax = 0.0f;
#pragma unroll 1
                    for (int c = colh; !full && c < bn / CW; c += EPI_WARPS / 4, o += step) {
                        const uint32_t taddr = tbase + (uint32_t)(c * CW);
                        uint32_t v[CW];
                        __syncwarp();
                        tc_ld_32x32b<CW>(taddr, v);
                        if constexpr (MODE == R2_EXACT)
                            epi::chunk_f32_plain<CW>(v, raf, epi::ColsF(base, COLS_N), c * CW,
                                                     b_tile + c * CW, a, a_ok, n_tile, dlo, dhi, o,
                                                     p.ldr, (float)p.S, rmax);
                        else
                            epi::chunk_ref_plain<CW>(
                                v, ra, epi::ColsR2(base, COLS_N), c * CW, b_tile + c * CW, a, a_ok,
                                n_tile, dlo, dhi, p.r2, o, p.ldr, p.out_row0, p.S,
                                [&](uint32_t (&w)[CW]) { tc_ld_32x32b<CW>(taddr, w); });
                    }
                    if (MODE == R2_EXACT && __any_sync(0xffffffffu, rmax > epi::R2_RECHECK))
                        full = true;
                }
#pragma unroll 1
                for (int c = colh; full && c < bn / CW; c += EPI_WARPS / 4) {
                    uint32_t v[CW];
                    __syncwarp();
                    tc_ld_32x32b<CW>(tbase + (uint32_t)(c * CW), v);
                    if constexpr (MODE == R2_EXACT) {
                        epi::chunk_f32<CW, true>(v, tbase + (uint32_t)(c * CW), raf,
                                           epi::ColsF(base, COLS_N), cols_special, c * CW,
                                           b_tile + c * CW, a, a_ok, n_tile, dlo, dhi, p.r2, p.ldr,
                                           p.counts, p.ldc, p.out_row0, p.S);
                    } else {
                        // the F32 accumulators hold the counts as floats
                        epi::chunk_ref<0, true, CW>(v, ra, epi::ColsR2(base, COLS_N), c * CW,
                                                    b_tile + c * CW, a, a_ok, n_tile, dlo, dhi,
                                                    p.r2, p.ldr, p.counts, p.ldc, p.out_row0,
                                                    p.S);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_rank(smem_u32(&accempty[ab]), 0);
                    if (FW) mbar_arrive(smem_u32(&facempty[ab]));
                }
            }
            if (it + 1 < my_tiles) store_factors(it + 1);
        }
    }

    // Teardown: the last commit of rank 0 arrives on mma_done in both CTAs;
    // neither CTA releases the pair's TMEM or exits while the other may
    // still touch its shared memory.
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (!mbar_wait(smem_u32(mma_done), 0, kDrainCycles, nullptr))
            flag_error(p.status, ST_TIMEOUT_MMA);
        __syncwarp();
    }
    tc_fence_before();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<2>(tmem, TMEM_COLS);
    }
}

// Clusters that run at once, asked of the driver once.
int max_pairs() {
    static std::atomic<int> known;
    int n = known.load(std::memory_order_relaxed);
    if (n > 0) return n;
    auto kern = k_ld_mxf4_pair<R2_EXACT, false, true, true, true>;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (sms / 2), 1, 1);
    cfg.blockDim = dim3(threads(true), 1, 1);
    cfg.dynamicSmemBytes = Smem<R2_EXACT>::BYTES;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Smem<R2_EXACT>::BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
        (void)cudaGetLastError();
        n = sms / 2;
    }
    known.store(n, std::memory_order_relaxed);
    return n;
}

template <int MODE, bool BAND, bool FULL, bool PLAIN, bool FW>
cudaError_t launch_mode(const CUtensorMap &tmA, const CUtensorMap &tmB, const LdParams &p,
                        const RowTiles &tl, cudaStream_t st) {
    auto kern = k_ld_mxf4_pair<MODE, BAND, FULL, PLAIN, FW>;
    static std::atomic<unsigned long long> allowed;
    cudaError_t e = allow_smem(kern, Smem<MODE>::BYTES, allowed);
    if (e != cudaSuccess) return e;
    const int ntiles = tl.count(), most = max_pairs();
    if (ntiles == 0) return cudaSuccess;
    const int pairs = ntiles < most ? ntiles : most;
    cudaLaunchAttribute at = overlap_attr();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
    cfg.blockDim = dim3(threads(FW), 1, 1);
    cfg.dynamicSmemBytes = Smem<MODE>::BYTES;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p, tl, ntiles);
}

template <int MODE, bool PLAIN, bool FW>
cudaError_t launch_tiles(const CUtensorMap &tmA, const CUtensorMap &tmB, const LdParams &p,
                         const RowTiles &tl, cudaStream_t st) {
    if (tl.band > 0)
        return tl.bn == BN ? launch_mode<MODE, true, true, PLAIN, FW>(tmA, tmB, p, tl, st)
                           : launch_mode<MODE, true, false, PLAIN, FW>(tmA, tmB, p, tl, st);
    return tl.bn == BN ? launch_mode<MODE, false, true, PLAIN, FW>(tmA, tmB, p, tl, st)
                       : launch_mode<MODE, false, false, PLAIN, FW>(tmA, tmB, p, tl, st);
}

template <int MODE, bool PLAIN>
cudaError_t launch_rule(bool fw, const CUtensorMap &tmA, const CUtensorMap &tmB, const LdParams &p,
                        const RowTiles &tl, cudaStream_t st) {
    return fw ? launch_tiles<MODE, PLAIN, true>(tmA, tmB, p, tl, st)
              : launch_tiles<MODE, PLAIN, false>(tmA, tmB, p, tl, st);
}

}  // namespace

const KernelShape kMxf4PairShape = {BM, BN, PW, HM, HN, 64};

// B rows per tile of a launch.  240 rows make the most of the MMAs, but a
// launch of few tiles ends on a wave that few SM pairs work in: 90 tiles on 74
// pairs take as long as 148.  Lower tiles fill that wave at a little more work
// per entry, so up to sixteen waves the height with the least estimated time
// is taken, if it saves 5 %.  The estimate (us, fitted to a sweep of 60
// launches of 2,700 to 9,001 SNPs and K = 16, 80, 260 on a B200): waves times
// the longer of a tile's MMAs (0.31 per 256-sample stage at 240 rows, 0.20 +
// 0.00053 bn at fewer, 0.21 + 0.00034 bn up to 128, whose unpack takes a row
// less per thread) and its epilogue (1.1 + 0.02 bn, reference mode 0.0405),
// plus what the shorter adds beside it.  3,000 SNPs: K = 80 24.5 -> 20.9 us,
// reference mode 33.2 -> 24.9; 5,286: 43.4 -> 39.5, 60.8 -> 53.8; 6,001: 52.7
// -> 50.1, 72.6 -> 68.9; 7.5 % on average over the sweep.
int pair_tile_rows(const RowTiles &tl, int K, int r2_mode) {
    RowTiles t = tl;
    t.bn = BN;
    const int most = max_pairs();
    if (t.rows() > 64 || t.count() > 16 * most) return BN;
    const double stages = (double)((K + PW - 1) / PW * SUB);
    auto estimate = [&](int bn) {
        t.bn = bn;
        const int waves = (t.count() + most - 1) / most;
        const double mma = stages * (bn == BN    ? 0.31
                                     : bn > 128 ? 0.20 + 0.00053 * bn
                                                : 0.21 + 0.00034 * bn);
        const double epi = 1.1 + (r2_mode == R2_REFERENCE ? 0.0405 : 0.02) * bn;
        const double a = mma > epi ? mma : epi, b = mma > epi ? epi : mma;
        return waves * (a + 0.42 * b * b / a);
    };
    double best = 0.95 * estimate(BN);
    int bn = BN;
    for (int x = BN - 16; x >= 80; x -= 16) {
        const double us = estimate(x);
        if (us < best) {
            best = us;
            bn = x;
        }
    }
    return bn;
}

// Whether the column factors get a warp of their own.  The epilogue warps pay
// ~2,000 cycles a tile for loading and dividing them and meeting at a barrier,
// which is the launch's time where its epilogues are (few stages per tile) and
// hidden behind the MMAs elsewhere; there the extra warp costs 1-4 % (whatever
// warps it shares a scheduler with unpack later, and a stage waits for both
// CTAs' slowest).  Exact mode, K = 60 / 80 / 100 / 120 / 140: 9,001 x 7,003
// 114 -> 102, 128 -> 117, 147 -> 144, 161 -> 161, 185 -> 188 us; reference
// mode, K = 80 / 120 / 160 / 200 / 260: 195 -> 164, 210 -> 184, 231 -> 221,
// 265 -> 266, 327 -> 339; 12,000 SNPs, K = 80: 144 -> 132, 222 -> 187.
// A launch of one or two waves gains less than the first tile's factors, all
// from one warp, cost it: 3,300 SNPs, exact mode, K = 60 17.6 -> 17.8.
// In rows that do not start on 32-byte sectors (`odd_rows`) warps that run apart
// write the two parts of a sector at distant times, and a launch bound by its
// stores pays for it: with counts beside r^2, and without in exact mode where
// the output is several times the L2.  Without / with the extra warp, counts,
// exact mode: 11,734 x 10,140 K = 3 214 / 359, K = 40 278 / 331, 8,547 x 4,813 K = 7
// 87 / 116, 9,001 x 7,003 K = 80 185 / 175; reference mode: 10,501 SNPs K = 3 295 /
// 329, K = 20 333 / 378, K = 80 389 / 345, 7,001 x 6,999 K = 20 159 / 156; no counts,
// exact mode: 29,817 SNPs K = 4 524 / 665, K = 20 560 / 606, K = 30 643 / 542, 20,001 x
// 9,000 K = 4 211 / 246, 9,001 x 7,003 K = 8 80 / 73.  In whole sectors the extra warp
// pays: counts, 11,776 x 10,140 K = 3 183 / 167, 12,000 SNPs K = 20 in reference mode
// 425 / 384; no counts, 29,824 SNPs K = 4 468 / 400.
bool factor_warp(const RowTiles &tl, const LdParams &p, int r2_mode) {
    const bool exact = r2_mode != R2_REFERENCE;
    auto odd = [](const void *base, long long ld) {
        return ld % 8 != 0 || (reinterpret_cast<uintptr_t>(base) & 31) != 0;
    };
    const int tiles = tl.count(), most = max_pairs();
    if (odd(p.r2, p.ldr) || (p.counts && odd(p.counts, p.ldc))) {
        if (p.counts && (exact || p.K < 40)) return false;
        if (!p.counts && exact && p.K < 24 && tiles > 30 * most) return false;
    }
    return p.K <= (exact ? 100 : 160) && tiles > 2 * most;
}

cudaError_t launch_mxf4_pair(const CUtensorMap &tmA, const CUtensorMap &tmB, const LdParams &p,
                             const RowTiles &tl, int r2_mode, cudaStream_t st) {
    const bool fw = factor_warp(tl, p, r2_mode);
    if (r2_mode == R2_REFERENCE)
        return !p.counts && p.S >= epi::R2_PLAIN_S && p.S <= (1 << 24)
                   ? launch_rule<R2_REFERENCE, true>(fw, tmA, tmB, p, tl, st)
                   : launch_rule<R2_REFERENCE, false>(fw, tmA, tmB, p, tl, st);
    return !p.counts ? launch_rule<R2_EXACT, true>(fw, tmA, tmB, p, tl, st)
                     : launch_rule<R2_EXACT, false>(fw, tmA, tmB, p, tl, st);
}

}  // namespace qld
