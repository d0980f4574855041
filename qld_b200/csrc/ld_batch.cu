// ld_batch.cu -- many independent LD tasks (region pairs of uneven SNP and
// sample counts) in one persistent launch fed by a device work queue.
//
// Per-task arithmetic is that of the 4-bit kernels on SM pairs
// (ld_mxf4_pair.cu): bits spread to E2M1 with normalising UE8M0 scale
// factors (tcgen05.cuh: spread_e2m1), tcgen05.mma.cta_group::2.kind::mxf4
// into F32 TMEM accumulators that hold the counts exactly (K * 64 <= 2^24),
// fused r^2 epilogue of qLD gemm_cpu.c:343-404 (R2_EXACT in FP32 from the
// exact counts, epilogue.cuh: chunk_f32).  qLD itself runs such task lists
// one task at a time (-inputList, src/correlator/src/input_list.c:205-323
// and correlate_function.c:59-83).  Here every output tile of every task is a
// work item, computed by a cluster of two CTAs: 256 A rows and as many B rows
// bn (a multiple of 16 up to 240) as spread the task's rows evenly over its
// tile rows (batch_tile_rows); rank r holds A rows 128 r.. and B rows bn/2 r..
// of the tile.  The device job table holds per task its tensor maps, sizes and
// output, and the item prefix offsets; items are numbered task by task (tasks
// sorted by cost on the host, most expensive first).
//
// Work queue: rank 0's queue warp runs ahead of the others, claims the next
// item with an atomic ticket on a global counter, decodes it into (task, A row,
// B row) and writes it into the 4-slot item ring of both CTAs (the peer's copy
// through st.shared::cluster, published by a cluster-scope release arrive).  In
// each CTA the TMA thread, the unpack warps and the epilogue warps (and in rank
// 0 the MMA warp) pop the same items in the same order, and each releases the
// slot on rank 0's barrier when done with its item.  A ticket past the last
// item pushes an end marker.  With the TMA thread claiming and decoding its
// items itself (an atomic and a binary search, ~4 us) and 240-row tiles
// throughout, the 300 tasks took 567 us against 533 (reference mode 647 /
// 614).
//
// Roles per CTA (640 threads): warp 0 TMA of the CTA's rows, warp 1 TMEM and
// (rank 0) the MMAs, warps 2-9 unpack in four groups taking the 256-sample
// stages in turn (each thread whole rows), warps 10-17 epilogue, two per TMEM
// lane quarter, warp 18 (rank 0) the queue, warp 19 the column factors, an item
// ahead of the epilogue.  With the factors loaded, divided and handed over at
// two barriers by the epilogue warps themselves, which items of few stages or
// rows pay in full, the 300 tasks took 488 us against 472 (reference mode, then
// with twelve epilogue warps, 588 against 549).  TMEM: two accumulators
// (columns 0 and 256), so a tile's epilogue overlaps the next tile's MMAs,
// and the scale factors at columns 496-511.  Every wait on an mbarrier is bounded
// and no thread returns early: both CTAs meet at the cluster barriers, which have
// no limit, at start and end on every path.
// The times here and below are of 300 tasks of 64-2,048 SNPs, as a replayed plan,
// with and without the one change on the kernel of that day; it takes 457 us now,
// 540 in reference mode.
#include "epilogue.cuh"
#include "mxf4_rows.cuh"
#include "mxf4_tiles.cuh"
#include "qld_kernels.h"
#include "tcgen05.cuh"

namespace qld {

namespace {

using namespace tc;

constexpr int BM = RowTiles::BM, BN = 240;  // work item: output tile of a pair (up to)
constexpr int HM = 128, HN = 120;           // A and B rows held by each CTA
constexpr int PW = 8;                       // packed words per row per packed stage
constexpr int SUB = 2;                      // unpacked stages (256 samples) per packed stage
constexpr int SW = PW / SUB;                // words per row per unpacked stage
constexpr int UST = 4;                      // one unpacked stage per unpack group
constexpr int PA_BYTES = HM * PW * 8;       // 8 KB
constexpr int P_MAX = (HM + HN) * PW * 8;   // up to 15.5 KB delivered per stage
constexpr int P_BYTES = 15872;              // stage stride: A rows, then B rows (a multiple of 512)
constexpr int UA_BYTES = HM * 128;          // 16 KB: 256 E2M1 per row
constexpr int U_BYTES = (HM + HN) * 128;    // 31 KB: A rows, then B rows
constexpr int GROUPS = 4, GROUP_WARPS = 2;  // as ld_mxf4_pair.cu
constexpr int UNPACK_WARPS = GROUPS * GROUP_WARPS;
constexpr int GROUP_THREADS = GROUP_WARPS * 32;
constexpr int FIRST_UNPACK_WARP = 2;
constexpr int FIRST_EPI_WARP = FIRST_UNPACK_WARP + UNPACK_WARPS;
// Twelve epilogue warps (at 80 registers): 300-task mix 492 us against 472,
// reference mode 552 against 549.
constexpr int EPI_WARPS = 8;
constexpr int QUEUE_WARP = FIRST_EPI_WARP + EPI_WARPS;
constexpr int FACTOR_WARP = QUEUE_WARP + 1;
constexpr int THREADS = (FACTOR_WARP + 1) * 32;              // 640
constexpr int TASKS = (HM + HN + GROUP_THREADS - 1) / GROUP_THREADS;   // rows per thread
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t ACC_STRIDE = 256;
constexpr uint32_t SF_COL = 496;
constexpr int COLS_N = 256;                                  // epilogue column factors (BN used)
constexpr uint16_t BOTH = 0x3;                               // CTA mask of a commit to both ranks
constexpr int QSLOTS = 4;                                    // item ring depth
// arrivals on rank 0's slot-free barrier per item: rank 0's MMA warp; both
// CTAs' TMA threads, unpack, epilogue and factor warps
constexpr int ITEM_USERS = 2 * (1 + UNPACK_WARPS + EPI_WARPS + 1) + 1;

// Shared-memory layout per r^2 mode: R2_EXACT needs 8 bytes of column
// factors per column (epi::ColsF), R2_REFERENCE 16 (epi::ColsR2); both leave
// room for six packed stages (more TMA lookahead than five).
template <int MODE>
struct Smem {
    static constexpr int PST = 6;                          // packed stages in flight
    static constexpr int OFF_U = 0;
    static constexpr int OFF_P = OFF_U + UST * U_BYTES;
    static constexpr int OFF_ROWS = OFF_P + PST * P_BYTES;
    static constexpr int ROWS_BYTES = COLS_N * (MODE == R2_EXACT ? 8 : epi::COLR_BYTES);
    static constexpr int OFF_ITEMS = OFF_ROWS + 2 * ROWS_BYTES;   // two items' factors
    static constexpr int OFF_BAR = OFF_ITEMS + QSLOTS * 16;
    static constexpr int NBARS = 2 * PST + 2 * UST + 2 + 2 + 1 + 2 * QSLOTS + 2 + 2;
    static constexpr int OFF_TMEM = OFF_BAR + NBARS * 8;        // and the halves' special flags
    static constexpr int BYTES = OFF_TMEM + 16 + 1024;
    static_assert(BYTES <= 232448, "shared memory budget");
    static_assert(U_BYTES % 1024 == 0 && UA_BYTES % 1024 == 0 && OFF_P % 1024 == 0 &&
                      P_BYTES % 512 == 0 && P_MAX <= P_BYTES && OFF_ITEMS % 16 == 0,
                  "swizzled stages must start on whole swizzle atoms");
    // group g takes sub-stage g % 2 of packed stages g / 2, g / 2 + 2, ...: a
    // slot always belongs to the same two groups
    static_assert(PST % 2 == 0 && GROUPS == 2 * SUB && GROUPS == UST, "stage rings");
};
static_assert(ACC_STRIDE + BN <= SF_COL && SF_COL + 16 <= TMEM_COLS, "TMEM map");
static_assert(SUB == 2 && EPI_WARPS % 4 == 0, "work split");

// A work item: task (< 0: end of the queue), its tile's first A and B row, and
// the words per row (low 24 bits) and tile rows / 16 (high 8) of the task.
struct Item {
    int job, a_row, b_row, shape;
    __device__ __forceinline__ int words() const { return shape & 0xFFFFFF; }
    __device__ __forceinline__ int np() const { return (words() + PW - 1) / PW; }
    // stages that hold samples, as ld_mxf4_pair.cu's nu_k
    __device__ __forceinline__ int nu_k() const {
        return np() > 3 ? (words() + SW - 1) / SW : np() * SUB;
    }
    __device__ __forceinline__ int bn() const { return (shape >> 24) * 16; }
};
static_assert(sizeof(Item) == 16, "an item is one 16-byte record");

// Global item g, found by the whole warp: a 32-way search of the item prefix
// (two or three rounds of loads instead of log2(njobs)), then the job's own
// B-tile-row-first tile list.
__device__ __forceinline__ Item decode_item(const BatchJob *jobs, int njobs, long long g,
                                            int lane) {
    int lo = 0, n = njobs;                   // the job is in [lo, lo + n)
    while (n > 1) {
        const int step = (n + 31) / 32, at = lo + lane * step;
        const bool below = at < lo + n && jobs[at].item0 <= g;
        const int k = __popc(__ballot_sync(0xffffffffu, below)) - 1;   // lane 0 is always below
        n = min(step, n - k * step);
        lo += k * step;
    }
    const BatchJob &J = jobs[lo];
    const RowTiles tl{J.m, 0, J.n, J.bn, J.symmetric, 0};
    Item it;
    it.job = lo;
    int t = 0, base = 0;
    tl.decode_from((int)(g - J.item0), it.a_row, it.b_row, t, base);
    it.shape = J.K | (J.bn / 16) << 24;
    return it;
}

// What the epilogue needs of a task, in registers: read through the table, the
// fields come from memory again after every store to the task's outputs
// (300-task batch 533 against 504 us).
struct JobFields {
    const uint32_t *bcA, *bcB;
    float *r2;
    uint32_t *counts;
    long long ldr, ldc;
    int m, n, S, symmetric;
    float threshold;
    BatchSummary *summary;
    __device__ __forceinline__ explicit JobFields(const BatchJob &J)
        : bcA(J.bcA), bcB(J.bcB), r2(J.r2), counts(J.counts), ldr(J.ldr), ldc(J.ldc), m(J.m),
          n(J.n), S(J.S), symmetric(J.symmetric), threshold(J.threshold), summary(J.summary) {}
};

// PLAIN: no task has counts or a summary (in reference mode: every S within
// R2_PLAIN_S..2^24), as ld_mxf4_pair.cu's.
template <int MODE, bool PLAIN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
k_ld_batch(const BatchParams bp) {
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
    uint64_t *ifull = mma_done + 1, *iempty = ifull + QSLOTS;
    uint64_t *facfull = iempty + QSLOTS, *facempty = facfull + 2;
    Item *items = reinterpret_cast<Item *>(smem + L::OFF_ITEMS);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L::OFF_TMEM);
    volatile uint32_t *col_flag = tmem_slot + 1;     // a column of the half is special

    const uint32_t rank = cluster_rank();
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const long long limit = bp.timeout_cycles;
    // the item ring is written by rank 0; rank 1 reads it under cluster-scope acquire
    auto wait_item = [&](int qi) {
        const uint32_t b = smem_u32(&ifull[qi % QSLOTS]);
        const uint32_t par = (uint32_t)(qi / QSLOTS) & 1u;
        return rank == 0 ? mbar_wait(b, par, limit, bp.status)
                         : mbar_wait_acq_cluster(b, par, limit, bp.status);
    };
    auto release_item = [&](int qi) { mbar_arrive_rank(smem_u32(&iempty[qi % QSLOTS]), 0); };

    if (tid == 0) {
        for (int s = 0; s < PST; ++s) {
            mbar_init(smem_u32(&pfull[s]), 1);
            mbar_init(smem_u32(&pempty[s]), SUB * GROUP_WARPS);   // one group per sub-stage
        }
        for (int s = 0; s < UST; ++s) {
            mbar_init(smem_u32(&ufull[s]), 2 * GROUP_WARPS);      // one group in each CTA
            mbar_init(smem_u32(&uempty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&accfull[s]), 1);
            mbar_init(smem_u32(&accempty[s]), 2 * EPI_WARPS);   // both CTAs' epilogues
            mbar_init(smem_u32(&facfull[s]), 1);
            mbar_init(smem_u32(&facempty[s]), EPI_WARPS);
        }
        mbar_init(smem_u32(mma_done), 1);
        for (int s = 0; s < QSLOTS; ++s) {
            mbar_init(smem_u32(&ifull[s]), 1);
            mbar_init(smem_u32(&iempty[s]), ITEM_USERS);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc<2>(smem_u32(tmem_slot), TMEM_COLS);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // the spread's scale factors in columns SF_COL.. of every lane, in both
    // CTAs (warps 2-5 cover the four TMEM lane quarters)
    if (warp >= FIRST_UNPACK_WARP && warp < FIRST_UNPACK_WARP + 4)
        tc_st_32x32b_x16_fill(tmem + ((uint32_t)((warp & 3) * 32) << 16) + SF_COL, kSpreadScales);
    tc_fence_before();
    // barrier initialisation and both CTAs' scale factors, cluster-wide
    cluster_sync_all();
    tc_fence_after();

    if (warp == QUEUE_WARP) {
        // ------------------------------------------- work queue (rank 0) --
        if (rank == 0) {
            bool ok = true;
            for (int qi = 0;; ++qi) {
                const int slot = qi % QSLOTS;
                if (qi >= QSLOTS) {
                    const bool free = mbar_wait_acq_cluster(smem_u32(&iempty[slot]),
                                                            ((qi / QSLOTS) - 1) & 1, limit,
                                                            bp.status);
                    if (!__all_sync(0xffffffffu, free)) {
                        if (lane == 0) flag_error(bp.status, ST_TIMEOUT_EMPTY);
                        ok = false;
                    }
                }
                long long g = (long long)bp.nitems;
                if (ok && lane == 0) g = (long long)atomicAdd(bp.queue, 1ull);
                g = __shfl_sync(0xffffffffu, g, 0);
                Item it{-1, 0, 0, 0};
                if (g < bp.nitems) it = decode_item(bp.jobs, bp.njobs, g, lane);
                if (lane == 0) {
                    items[slot] = it;
                    mbar_arrive(smem_u32(&ifull[slot]));   // release: the item is visible
                    st_rank_and_arrive(smem_u32(&items[slot]),
                                       make_int4(it.job, it.a_row, it.b_row, it.shape),
                                       smem_u32(&ifull[slot]), 1);
                }
                __syncwarp();
                if (it.job < 0) break;
            }
        }
    } else if (warp == 0) {
        // --------------------------------------------------- TMA producer --
        if (lane == 0) {
            int gp = 0;
            bool ok = true;
            for (int qi = 0; ok; ++qi) {
                if (!wait_item(qi)) {
                    flag_error(bp.status, ST_TIMEOUT_FULL);
                    break;
                }
                const Item it = items[qi % QSLOTS];
                if (it.job < 0) break;
                const BatchJob &J = bp.jobs[it.job];
                const int hn = it.bn() / 2, np = it.np();
                const int ra = it.a_row + (int)rank * HM, rb = it.b_row + (int)rank * hn;
                for (int kp = 0; kp < np; ++kp, ++gp) {
                    const int s = gp % PST;
                    if (gp >= PST && !mbar_wait(smem_u32(&pempty[s]), ((gp / PST) - 1) & 1,
                                                limit, bp.status)) {
                        flag_error(bp.status, ST_TIMEOUT_EMPTY);
                        ok = false;
                        break;
                    }
                    const uint32_t fb = smem_u32(&pfull[s]);
                    const uint32_t dst = smem_u32(smem + L::OFF_P + s * P_BYTES);
                    mbar_arrive_expect_tx(fb, PA_BYTES + (uint32_t)(hn * PW * 8));
                    tma_load_2d(dst, &J.tmA, kp * PW, ra, fb);
                    tma_load_2d(dst + PA_BYTES, &J.tmB, kp * PW, rb, fb);
                }
                release_item(qi);
            }
            for (int g = gp > PST ? gp - PST : 0; g < gp; ++g)
                if (!mbar_wait(smem_u32(&pfull[g % PST]), (g / PST) & 1, kDrainCycles, nullptr)) {
                    flag_error(bp.status, ST_TIMEOUT_DRAIN);
                    break;
                }
        }
    } else if (warp == 1) {
        // ------------------------------------------- MMA issuer (rank 0) --
        if (rank == 0) {
            const uint32_t sf = tmem + SF_COL;
            const uint32_t a_lo = sw128_desc_lo(smem_u32(smem + L::OFF_U));
            uint32_t s = 0, ph = 0;      // unpacked stage and its phase
            int it_n = 0;
            bool ok = true;
            for (int qi = 0; ok; ++qi, ++it_n) {
                const int slot = qi % QSLOTS;
                if (!__all_sync(0xffffffffu, wait_item(qi))) {
                    if (lane == 0) flag_error(bp.status, ST_TIMEOUT_UNPACK);
                    break;
                }
                const Item it = items[slot];
                if (it.job < 0) break;
                const uint32_t even = idesc_mxf4_sf(BM, it.bn(), 0);   // k-steps 0, 2: scale bytes 0-1
                const uint32_t odd = idesc_mxf4_sf(BM, it.bn(), 2);    // k-steps 1, 3: scale bytes 2-3
                const int nu = it.np() * SUB, nu_k = it.nu_k();
                const int ab = it_n & 1;
                if (it_n >= 2) {
                    const bool free = mbar_wait(smem_u32(&accempty[ab]), ((it_n >> 1) - 1) & 1,
                                                limit, bp.status);
                    if (!__all_sync(0xffffffffu, free)) {
                        if (lane == 0) flag_error(bp.status, ST_TIMEOUT_MMA);
                        break;
                    }
                }
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)ab * ACC_STRIDE;
                for (int u = 0; u < nu; ++u) {
                    const bool full = mbar_wait(smem_u32(&ufull[s]), ph, limit, bp.status);
                    if (!__all_sync(0xffffffffu, full)) {
                        if (lane == 0) flag_error(bp.status, ST_TIMEOUT_UNPACK);
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
                if (elect_one()) {
                    tc_commit_pair(smem_u32(&accfull[ab]), BOTH);
                    release_item(qi);
                }
                __syncwarp();
            }
            if (elect_one()) tc_commit_pair(smem_u32(mma_done), BOTH);
            __syncwarp();
        }
    } else if (warp < FIRST_EPI_WARP) {
        // --------------------------------------------------------- unpack --
        const int grp = (warp - FIRST_UNPACK_WARP) / GROUP_WARPS;
        const mxf4rows::RowLane<GROUP_THREADS> rows(
            ((warp - FIRST_UNPACK_WARP) % GROUP_WARPS) * 32 + lane);
        // slot and phases counted up, as in ld_mxf4_pair.cu: the group's stages are
        // buffer grp and the same half of every other packed slot
        uint8_t *const dst = smem + L::OFF_U + grp * U_BYTES;
        const uint32_t uf = smem_u32(&ufull[grp]), ue = smem_u32(&uempty[grp]);
        int ps = grp / SUB, kp = grp / SUB;  // packed slot; the stage's place in the item
        uint32_t ph = 0, eh = 1;             // phases of the packed slot and of the unpacked stage
        bool ok = true, first = true;
        for (int qi = 0; ok; ++qi) {
            const bool got_item = wait_item(qi);
            if (!__all_sync(0xffffffffu, got_item)) {
                if (lane == 0) flag_error(bp.status, ST_TIMEOUT_FULL);
                break;
            }
            const Item it = items[qi % QSLOTS];
            if (it.job < 0) break;
            const int np = it.np(), nu_k = it.nu_k(), nrows = HM + it.bn() / 2;
            for (; kp < np; kp += GROUPS / SUB) {
                const bool got = mbar_wait(smem_u32(&pfull[ps]), ph, limit, bp.status);
                const bool freed = got && (first || mbar_wait(ue, eh, limit, bp.status));
                if (!__all_sync(0xffffffffu, freed)) {
                    if (lane == 0) flag_error(bp.status, got ? ST_TIMEOUT_MMA : ST_TIMEOUT_FULL);
                    ok = false;
                    break;
                }
                if (kp * SUB + grp % SUB < nu_k)
                    mxf4rows::unpack_rows<GROUP_THREADS, TASKS>(
                        rows, nrows, smem + L::OFF_P + ps * P_BYTES, dst, grp % SUB);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_rank(uf, 0);
                    mbar_arrive(smem_u32(&pempty[ps]));
                }
                first = false;
                eh ^= 1;
                if ((ps += GROUPS / SUB) >= PST) ps -= PST, ph ^= 1;
            }
            kp -= np;                        // its first stage of the next item
            __syncwarp();
            if (lane == 0) release_item(qi);
        }
    } else if (warp == FACTOR_WARP) {
        // ------------------------------------------------- column factors --
        for (int qi = 0;; ++qi) {
            const int ab = qi & 1;
            if (!__all_sync(0xffffffffu, wait_item(qi))) {
                if (lane == 0) flag_error(bp.status, ST_TIMEOUT_FULL);
                break;
            }
            const Item it = items[qi % QSLOTS];
            if (it.job < 0) break;
            const BatchJob &J = bp.jobs[it.job];
            const int n = J.n, S = J.S;
            // every column factor the chunks read; 0 past the tile and the task
            uint32_t cb[COLS_N / 32];
#pragma unroll
            for (int i = 0; i < COLS_N / 32; ++i) {
                const int e = i * 32 + lane;
                cb[i] = e < it.bn() && it.b_row + e < n ? J.bcB[it.b_row + e] : 0u;
            }
            const bool free = qi < 2 || mbar_wait(smem_u32(&facempty[ab]), ((qi >> 1) - 1) & 1,
                                                  limit, bp.status);
            if (!__all_sync(0xffffffffu, free)) {
                if (lane == 0) flag_error(bp.status, ST_TIMEOUT_EMPTY);
                break;
            }
            uint8_t *base = smem + L::OFF_ROWS + ab * L::ROWS_BYTES;
            bool special = false;
#pragma unroll
            for (int i = 0; i < COLS_N / 32; ++i) {
                if constexpr (MODE == R2_EXACT)
                    special |= epi::store_col_f32(epi::ColsF(base, COLS_N), i * 32 + lane, cb[i], S);
                else
                    special |= epi::store_col_ref(epi::ColsR2(base, COLS_N), i * 32 + lane, cb[i], S);
            }
            special = __any_sync(0xffffffffu, special);
            __syncwarp();                // every lane's factors are stored: a vote does not order them
            if (lane == 0) {
                col_flag[ab] = special;
                mbar_arrive(smem_u32(&facfull[ab]));
                release_item(qi);
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------- epilogue --
        const int ew = warp - FIRST_EPI_WARP;
        const int q = warp & 3;             // TMEM lane quarter
        for (int qi = 0;; ++qi) {
            if (!__all_sync(0xffffffffu, wait_item(qi))) {
                if (lane == 0) flag_error(bp.status, ST_TIMEOUT_FULL);
                break;
            }
            const Item it = items[qi % QSLOTS];
            if (it.job < 0) break;
            const JobFields J(bp.jobs[it.job]);
            const int ab = qi & 1;
            // chunks colh, colh + EPI_WARPS / 4, ...: the longer shares in turn
            const int colh = ((ew >> 2) + qi) % (EPI_WARPS / 4);
            const int a = it.a_row + (int)rank * HM + q * 32 + lane;
            const bool a_ok = a < J.m;
            const uint32_t ca = a_ok ? J.bcA[a] : 0u;
            const epi::ARowR ra = epi::make_arow_ref(ca, J.S);
            const epi::ARowF raf = epi::make_arow_f32(ca, J.S);
            const bool ready = mbar_wait(smem_u32(&facfull[ab]), (qi >> 1) & 1, limit, bp.status) &&
                               mbar_wait(smem_u32(&accfull[ab]), (qi >> 1) & 1, limit, bp.status);
            if (!__all_sync(0xffffffffu, ready)) {
                if (lane == 0) flag_error(bp.status, ST_TIMEOUT_MMA);
                break;
            }
            const bool cols_special = col_flag[ab] != 0u;
            const epi::ColsR2 colsr(smem + L::OFF_ROWS + ab * L::ROWS_BYTES, COLS_N);
            const epi::ColsF colsf(smem + L::OFF_ROWS + ab * L::ROWS_BYTES, COLS_N);
            __syncwarp();
            tc_fence_after();
            const uint32_t tbase =
                tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)ab * ACC_STRIDE;
            const int n_tile = it.b_row + it.bn() < J.n ? it.b_row + it.bn() : J.n;
            const int dlo = diag_lo(J.symmetric, 0), dhi = diag_hi(0);
            uint32_t *const counts = PLAIN ? nullptr : J.counts;
            BatchSummary *const summary = PLAIN ? nullptr : J.summary;
            epi::SumAcc acc;
            // Chunks of 16 columns, in reference mode of 8 (more columns spill:
            // 32 in exact mode 620 us against 566 on 300 tasks, 16 in
            // reference mode 668 against 647)
            constexpr int CW = MODE == R2_EXACT ? 16 : 8;
            bool full = true;                // chunks with the rare cases' bookkeeping
            if constexpr (PLAIN) {
                full = cols_special ||
                       __any_sync(0xffffffffu, MODE == R2_EXACT ? raf.special : ra.k.y != ra.k.y);
                const long long step = (long long)(CW * EPI_WARPS / 4) * J.ldr;
                float *o = J.r2 + (long long)(it.b_row + colh * CW) * J.ldr + a;
                float rmax = 0.0f;
#pragma unroll 1
                for (int c = colh; !full && c < it.bn() / CW; c += EPI_WARPS / 4, o += step) {
                    const uint32_t taddr = tbase + (uint32_t)(c * CW);
                    uint32_t v[CW];
                    __syncwarp();
                    tc_ld_32x32b<CW>(taddr, v);
                    if constexpr (MODE == R2_EXACT)
                        epi::chunk_f32_plain<CW>(v, raf, colsf, c * CW, it.b_row + c * CW, a,
                                                 a_ok, n_tile, dlo, dhi, o, J.ldr, (float)J.S,
                                                 rmax);
                    else
                        epi::chunk_ref_plain<CW>(
                            v, ra, colsr, c * CW, it.b_row + c * CW, a, a_ok, n_tile, dlo, dhi,
                            J.r2, o, J.ldr, 0, J.S,
                            [&](uint32_t (&w)[CW]) { tc_ld_32x32b<CW>(taddr, w); });
                }
                if (MODE == R2_EXACT && __any_sync(0xffffffffu, rmax > epi::R2_RECHECK))
                    full = true;
            }
#pragma unroll 1
            for (int c = colh; full && c < it.bn() / CW; c += EPI_WARPS / 4) {   // the tile's chunks
                uint32_t v[CW];
                __syncwarp();
                tc_ld_32x32b<CW>(tbase + (uint32_t)(c * CW), v);
                if constexpr (MODE == R2_EXACT) {
                    epi::chunk_f32<CW, true>(v, tbase + (uint32_t)(c * CW), raf, colsf, cols_special,
                                       c * CW, it.b_row + c * CW, a, a_ok, n_tile, dlo, dhi, J.r2,
                                       J.ldr, counts, J.ldc, 0, J.S);
                    if (summary)
                        acc.fold(v, it.b_row + c * CW, a, a_ok, J.n, J.symmetric,
                                 J.threshold);
                } else {
                    // the F32 accumulators hold the counts as floats
                    epi::chunk_ref<0, true, CW>(v, ra, colsr, c * CW, it.b_row + c * CW, a,
                                                a_ok, n_tile, dlo, dhi, J.r2, J.ldr,
                                                counts, J.ldc, 0, J.S);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_rank(smem_u32(&accempty[ab]), 0);
                mbar_arrive(smem_u32(&facempty[ab]));
                release_item(qi);
            }
            if (MODE == R2_EXACT && summary) acc.flush(summary);
            __syncwarp();
        }
    }

    // Teardown: rank 0's last commit arrives on mma_done in both CTAs;
    // neither CTA frees the pair's TMEM or exits while the other may still
    // touch its shared memory.
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (!mbar_wait(smem_u32(mma_done), 0, kDrainCycles, nullptr))
            flag_error(bp.status, ST_TIMEOUT_MMA);
        __syncwarp();
    }
    tc_fence_before();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<2>(tmem, TMEM_COLS);
    }
}

int g_max_pairs = 0;

template <int MODE, bool PLAIN>
cudaError_t launch_mode(const BatchParams &bp, int max_ctas, cudaStream_t st) {
    auto kern = k_ld_batch<MODE, PLAIN>;
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<MODE>::BYTES);
    if (e != cudaSuccess) return e;
    if (g_max_pairs == 0) {
        int dev = 0, sms = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) !=
            cudaSuccess)
            return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * (sms / 2), 1, 1);
        cfg.blockDim = dim3(THREADS, 1, 1);
        cfg.dynamicSmemBytes = Smem<MODE>::BYTES;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            n = sms / 2;
        }
        g_max_pairs = n;
    }
    long long pairs = bp.nitems < g_max_pairs ? bp.nitems : g_max_pairs;
    if (max_ctas > 0 && 2 * pairs > max_ctas) pairs = max_ctas / 2;
    if (pairs <= 0) return cudaSuccess;
    kern<<<(int)(2 * pairs), THREADS, Smem<MODE>::BYTES, st>>>(bp);
    return cudaGetLastError();
}

}  // namespace

const KernelShape kBatchShape = {BM, BN, PW, HM, HN, 64};
const int kBatchMaxSamples = 1 << 24;

bool batch_job_plain(const BatchJob &j, int r2_mode) {
    return !j.counts && !j.summary &&
           (r2_mode != R2_REFERENCE || (j.S >= epi::R2_PLAIN_S && j.S <= (1 << 24)));
}

// As few tile rows as 240-row tiles need, of (nearly) equal height: 250 B rows
// are two tiles of 128, not 240 + 10, and 64 are one of 64, so padding rows are
// not unpacked, multiplied or run through the epilogue.
int batch_tile_rows(int n) {
    const int rows = (n + BN - 1) / BN;
    return rows < 1 ? 16 : ((n + rows - 1) / rows + 15) / 16 * 16;
}
long long batch_tiles(int m, int n, int symmetric) {
    return RowTiles{m, 0, n, batch_tile_rows(n), symmetric, 0}.count();
}

cudaError_t launch_batch(const BatchParams &bp, int r2_mode, int max_ctas, cudaStream_t st) {
    if (r2_mode == R2_REFERENCE)
        return bp.plain ? launch_mode<R2_REFERENCE, true>(bp, max_ctas, st)
                        : launch_mode<R2_REFERENCE, false>(bp, max_ctas, st);
    return bp.plain ? launch_mode<R2_EXACT, true>(bp, max_ctas, st)
                    : launch_mode<R2_EXACT, false>(bp, max_ctas, st);
}

}  // namespace qld
