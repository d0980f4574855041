// ld_mxf4_split.cu -- counts kernel, variant (c) on SM pairs for tasks whose
// tiles all run at once: one output tile per cluster, its samples split over
// the cluster's SM pairs.
//
// The arithmetic is ld_mxf4_pair.cu's (bits spread to E2M1,
// tcgen05.mma.cta_group::2.kind::mxf4 into F32 accumulators exact below 2^24,
// the fused r^2 epilogue of qLD gemm_cpu.c:343-404); what differs is the
// division of a small task.  The persistent kernel gives a task of up to one
// tile per SM pair whole 256 x 240 tiles: most pairs stay idle, one pair
// walks all K words, and eight of its warps then run an epilogue that nothing
// overlaps.  Measured, persistent against this kernel (us per launch
// in a CUDA graph, SNPs x samples): single region 200 x 1,000 8.0 / 5.9,
// 2,048 x 4,096 12.1 / 11.3, 64 x 50,000 58 / 17.7; two regions 731 x 530 x
// 5,008 in reference mode 17.0 / 10.4.  A launch of one part per pair is bound
// by the latency of its steps: launch and setup, the first TMA, 0.235 us per
// 256-sample stage (the handshakes; the MMAs take 0.12), the epilogue.  Here
//   * the tile is 256 x bn with bn (16..240, a multiple of 16) chosen per
//     task, so that the tiles spread over the SMs;
//   * a cluster of 2 ks CTAs (ks = 1, 2, 4 SM pairs) computes one tile: pair s
//     takes the s-th part of the packed words, and the pairs exchange partial
//     counts through distributed shared memory: 16-column chunk c of the tile
//     belongs to pair c % ks, which receives the others' counts of it and
//     runs its epilogue.  Partial counts are integers below 2^24, so the F32
//     sums are exact in any order;
//   * all sixteen worker warps unpack, then run the epilogue.  Four groups of
//     four warps take the stages in turn: the stages are short and their
//     latency counts (two groups of eight: 10 % slower on long tables; eight
//     unpacked stages instead of four: no faster);
//   * the per-row and per-column factors are computed before the first data
//     arrives.
// Roles (18 warps): warp 0 TMA producer, warp 1 TMEM and (rank 0 of each pair)
// the MMAs, warps 2-17 workers, each thread up to two packed rows of every
// fourth 256-sample stage.
//
// Every wait on an mbarrier is bounded and no thread returns early.  The named
// barrier of the workers and the cluster barriers have no limit: every worker
// warp meets the one once, and every warp of every CTA the others, on every path,
// a failed wait included.
#include <atomic>

#include "epilogue.cuh"
#include "launch_util.h"
#include "mxf4_rows.cuh"
#include "mxf4_tiles.cuh"
#include "qld_kernels.h"
#include "tcgen05.cuh"

namespace qld {

namespace {

using namespace tc;

constexpr int BM = 256;
constexpr int HM = 128;                  // A rows held by each CTA
constexpr int MAX_BN = 240;
constexpr int PW = 8;                    // packed words per row per packed stage
constexpr int SUB = 2;                   // unpacked stages (256 samples) per packed stage
constexpr int UST = 4;
constexpr int MAX_PST = 6;
constexpr int PA_BYTES = HM * PW * 8;    // 8 KB
constexpr int UA_BYTES = HM * 128;       // 16 KB
constexpr int FIRST_WORKER = 2, WORKER_WARPS = 16;
constexpr int WORKERS = WORKER_WARPS * 32;
constexpr int GROUPS = 4, GROUP_WARPS = WORKER_WARPS / GROUPS;
constexpr int TASKS = 2;                 // packed rows per thread and stage (up to 248 rows)
constexpr int THREADS = (FIRST_WORKER + WORKER_WARPS) * 32;   // 576
constexpr int CH = 16;                   // epilogue chunk: columns
constexpr int SLOT_BYTES = CH * HM * 4;  // a chunk's partial counts of one CTA: 8 KB
constexpr uint32_t TMEM_COLS = 256;
constexpr uint32_t SF_COL = 240;         // 16 columns of scale factors
constexpr int COLS_BYTES = MAX_BN * 16;
constexpr int NBARS = 2 * MAX_PST + 2 * UST + 1;
constexpr int MAX_SMEM = 232448;

// Shared-memory layout of a launch.
struct Layout {
    int u, p, pst, push, cols, bars, bytes;     // stage strides, then offsets
    __host__ __device__ Layout(int bn, int ks, int pst_) {
        const int hn = bn / 2;
        u = (HM + hn) * 128;                        // hn is a multiple of 8
        p = ((HM + hn) * PW * 8 + 1023) / 1024 * 1024;
        pst = pst_;
        push = UST * u + pst * p;
        const int chunks = bn / CH;
        cols = push + (ks - 1) * ((chunks + ks - 1) / ks) * SLOT_BYTES;
        bars = cols + COLS_BYTES;
        bytes = bars + NBARS * 8 + 16 + 1024;
    }
};

__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// PLAIN: as ld_mxf4_pair.cu's.
template <int MODE, bool PLAIN>
__global__ void __launch_bounds__(THREADS, 1)
k_ld_mxf4_split(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const LdParams p, const RowTiles tl, const int ks, const int pst) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int bn = tl.bn, hn = bn / 2;
    const Layout L(bn, ks, pst);
    uint8_t *unpacked = smem, *packed = smem + UST * L.u;   // A rows, then B rows, per stage
    const float *push = reinterpret_cast<const float *>(smem + L.push);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bars);
    uint64_t *pfull = bars, *pempty = pfull + MAX_PST;
    uint64_t *ufull = pempty + MAX_PST, *uempty = ufull + UST;
    uint64_t *accfull = uempty + UST;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L.bars + NBARS * 8);
    const epi::ColsR2 colsr(smem + L.cols, MAX_BN);
    const epi::ColsF colsf(smem + L.cols, MAX_BN);

    const uint32_t crank = cluster_rank();
    const int split = (int)(crank >> 1);           // SM pair of the cluster
    const uint32_t rank = crank & 1u, leader = crank & ~1u;
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int s = 0; s < MAX_PST; ++s) {
            mbar_init(smem_u32(&pfull[s]), 1);
            mbar_init(smem_u32(&pempty[s]), 2 * GROUP_WARPS);
        }
        for (int s = 0; s < UST; ++s) {
            mbar_init(smem_u32(&ufull[s]), 2 * GROUP_WARPS);   // one group in each CTA
            mbar_init(smem_u32(&uempty[s]), 1);
        }
        mbar_init(smem_u32(accfull), 1);
        fence_barrier_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
    }
    if (warp == 1) tmem_alloc<2>(smem_u32(tmem_slot), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (warp >= FIRST_WORKER && warp < FIRST_WORKER + 4)
        tc_st_32x32b_x16_fill(tmem + ((uint32_t)((warp & 3) * 32) << 16) + SF_COL, kSpreadScales);
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    griddep_launch();
    griddep_wait();

    // the cluster's tile, and the pair's part of the packed words
    int a_row, b_row, t0 = 0, base = 0;
    tl.decode_from((int)cluster_id_x(), a_row, b_row, t0, base);
    const int np_all = (p.K + PW - 1) / PW;
    const int kp0 = np_all * split / ks, kp1 = np_all * (split + 1) / ks;
    const int k_end = kp1 * PW < p.K ? kp1 * PW : p.K;
    const int np = kp1 - kp0;
    const int nu = (k_end - kp0 * PW + PW / SUB - 1) / (PW / SUB);   // 256-sample stages

    const int q = warp & 3;                        // worker: TMEM lane quarter
    const int cg = (warp - FIRST_WORKER) >> 2;     // worker: chunk group 0..3
    const int a = a_row + (int)rank * HM + q * 32 + lane;
    const bool a_ok = a < p.m;
    const int chunks = bn / CH;
    const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16);
    epi::ARowR ra{};
    epi::ARowF raf{};
    bool ready = false, cols_special = false;

    if (warp == 0) {
        // ------------------------------------------------------- producer --
        if (lane == 0) {
            const int rowa = a_row + (int)rank * HM, rowb = b_row + (int)rank * hn;
            int gp = 0;
            for (; gp < np; ++gp) {
                const int s = gp % pst;
                if (gp >= pst && !mbar_wait(smem_u32(&pempty[s]), ((gp / pst) - 1) & 1,
                                            p.timeout_cycles, p.status)) {
                    flag_error(p.status, ST_TIMEOUT_EMPTY);
                    break;
                }
                const uint32_t fb = smem_u32(&pfull[s]);
                const uint32_t dst = smem_u32(packed + s * L.p);
                mbar_arrive_expect_tx(fb, PA_BYTES + (uint32_t)(hn * PW * 8));
                tma_load_2d(dst, &tmA, (kp0 + gp) * PW, rowa, fb);
                tma_load_2d(dst + PA_BYTES, &tmB, (kp0 + gp) * PW, rowb, fb);
            }
            for (int g = gp > pst ? gp - pst : 0; g < gp; ++g)
                if (!mbar_wait(smem_u32(&pfull[g % pst]), (g / pst) & 1, kDrainCycles, nullptr)) {
                    flag_error(p.status, ST_TIMEOUT_DRAIN);
                    break;
                }
        }
        __syncwarp();
    } else if (warp == 1) {
        // -------------------------------- MMA issuer (rank 0 of the pair) --
        if (rank == 0) {
            const uint32_t sf = tmem + SF_COL;
            const uint32_t even = idesc_mxf4_sf(BM, bn, 0), odd = idesc_mxf4_sf(BM, bn, 2);
            const uint16_t both = (uint16_t)(0x3u << leader);
            const uint32_t a_lo = sw128_desc_lo(smem_u32(unpacked));
            const uint32_t step = (uint32_t)L.u >> 4;
            for (int u = 0; u < nu; ++u) {
                const uint32_t s = (uint32_t)u % UST;
                const bool full = mbar_wait(smem_u32(&ufull[s]), (u / UST) & 1, p.timeout_cycles,
                                            p.status);
                if (!__all_sync(0xffffffffu, full)) {
                    if (lane == 0) flag_error(p.status, ST_TIMEOUT_UNPACK);
                    break;
                }
                tc_fence_after();
                const uint32_t da = a_lo + s * step, db = da + (UA_BYTES >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        tc_mma_mxf4_pair_lo(tmem, da + kk * 2, db + kk * 2, (kk & 1) ? odd : even,
                                            (u > 0 || kk > 0) ? 1u : 0u, sf, sf);
                    tc_commit_pair(smem_u32(&uempty[s]), both);
                }
                __syncwarp();
            }
            if (elect_one()) tc_commit_pair(smem_u32(accfull), both);   // also after a failed wait
            __syncwarp();
        }
        __syncwarp();
    } else {
        // --------------------------------------------------------- unpack --
        const int wt = tid - FIRST_WORKER * 32;
        bool special = false;
        if (wt < bn) {
            const int b = b_row + wt;
            const uint32_t cb = b < p.n ? p.bcB[b] : 0u;
            if constexpr (MODE == R2_EXACT) special = epi::store_col_f32(colsf, wt, cb, p.S);
            else special = epi::store_col_ref(colsr, wt, cb, p.S);
        }
        const uint32_t ca = a_ok ? p.bcA[a] : 0u;
        if constexpr (MODE == R2_EXACT) raf = epi::make_arow_f32(ca, p.S);
        else ra = epi::make_arow_ref(ca, p.S);

        const int grp = (warp - FIRST_WORKER) / GROUP_WARPS;
        const mxf4rows::RowLane<GROUP_WARPS * 32> rows(
            ((warp - FIRST_WORKER) % GROUP_WARPS) * 32 + lane);
        bool ok = true;
        int gp = 0, ps = 0, pph = 0;               // packed stage: index, slot, phase
        for (int u = grp; u < nu; u += GROUPS) {
            const int us = u % UST;
            for (; gp < u / SUB; ++gp)
                if (++ps == pst) ps = 0, pph ^= 1;
            const bool got = mbar_wait(smem_u32(&pfull[ps]), pph, p.timeout_cycles, p.status);
            if (!__all_sync(0xffffffffu, got)) {
                if (lane == 0) flag_error(p.status, ST_TIMEOUT_FULL);
                ok = false;
                break;
            }
            const bool freed = u < UST || mbar_wait(smem_u32(&uempty[us]), ((u / UST) - 1) & 1,
                                                    p.timeout_cycles, p.status);
            if (!__all_sync(0xffffffffu, freed)) {
                if (lane == 0) flag_error(p.status, ST_TIMEOUT_MMA);
                ok = false;
                break;
            }
            mxf4rows::unpack_rows<GROUP_WARPS * 32, TASKS>(rows, HM + hn, packed + ps * L.p,
                                                           unpacked + us * L.u, u & 1);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_rank(smem_u32(&ufull[us]), leader);
                mbar_arrive(smem_u32(&pempty[ps]));
            }
        }
        cols_special = named_bar_or(1, WORKERS, special);   // the column factors are stored
        // the accumulators; on a failed wait the drain wait still keeps the
        // CTA until its MMAs are done
        ready = mbar_wait(smem_u32(accfull), 0, ok ? p.timeout_cycles : 1, p.status);
        ready = __all_sync(0xffffffffu, ready && ok);
        if (!ready && ok && lane == 0) flag_error(p.status, ST_TIMEOUT_MMA);
        __syncwarp();
        tc_fence_after();
        if (ready && ks > 1) {
            // ------------------------ partial counts to the chunks' owners --
#pragma unroll 1
            for (int c = cg; c < chunks; c += 4) {
                const int owner = c % ks;
                if (owner == split) continue;
                uint32_t v[CH];
                __syncwarp();
                tc_ld_32x32b_x16(tbase + (uint32_t)(c * CH), v);
                const int slot = (split < owner ? split : split - 1) * ((chunks + ks - 1) / ks) + c / ks;
                const uint32_t dst = mapa(smem_u32(smem + L.push + slot * SLOT_BYTES) +
                                              (uint32_t)(q * 32 + lane) * 4u,
                                          (uint32_t)owner * 2u + rank);
#pragma unroll
                for (int t = 0; t < CH; ++t) st_cluster(dst + (uint32_t)(t * HM * 4), v[t]);
            }
        }
    }
    if (ks > 1) cluster_sync_all();                // every part has been delivered

    if (warp >= FIRST_WORKER && ready) {
        // ------------------------------------------------------- epilogue --
        const int dlo = diag_lo(p.symmetric, p.band), dhi = diag_hi(p.band);
        const int n_tile = b_row + bn < p.n ? b_row + bn : p.n;
        const int per = (chunks + ks - 1) / ks;
        const bool full = !PLAIN || cols_special ||
                          __any_sync(0xffffffffu, MODE == R2_EXACT ? raf.special : ra.k.y != ra.k.y);
#pragma unroll 1
        for (int i = cg; i * ks + split < chunks; i += 4) {
            const int c = i * ks + split;
            // in reference mode in halves, whose packed arithmetic does not spill
            constexpr int CW = MODE == R2_EXACT ? CH : CH / 2;
#pragma unroll 1
            for (int h = 0; h < CH; h += CW) {
                const int col = c * CH + h;
                const uint32_t taddr = tbase + (uint32_t)col;
                uint32_t v[CW];
                __syncwarp();
                tc_ld_32x32b<CW>(taddr, v);
                if (ks > 1) {
                    for (int o = 0; o < ks - 1; ++o) {
                        const float *part = push + (o * per + i) * (SLOT_BYTES / 4) + h * HM +
                                            q * 32 + lane;
#pragma unroll
                        for (int t = 0; t < CW; ++t)
                            v[t] = __float_as_uint(__uint_as_float(v[t]) + part[t * HM]);
                    }
                    // the rare pairs evaluated again are read again
                    tc_st_32x32b<CW>(taddr, v);
                }
                if constexpr (PLAIN) {
                    if (!full) {
                        float *o = p.r2 + (long long)(b_row + col - p.out_row0) * p.ldr + a;
                        if constexpr (MODE == R2_EXACT) {
                            float rmax = 0.0f;
                            epi::chunk_f32_plain<CW>(v, raf, colsf, col, b_row + col, a, a_ok,
                                                     n_tile, dlo, dhi, o, p.ldr, (float)p.S, rmax);
                            if (!__any_sync(0xffffffffu, rmax > epi::R2_RECHECK)) continue;
                            tc_ld_32x32b<CW>(taddr, v);
                        } else {
                            epi::chunk_ref_plain<CW>(
                                v, ra, colsr, col, b_row + col, a, a_ok, n_tile, dlo, dhi, p.r2, o,
                                p.ldr, p.out_row0, p.S,
                                [&](uint32_t (&w)[CW]) { tc_ld_32x32b<CW>(taddr, w); });
                            continue;
                        }
                    }
                }
                if constexpr (MODE == R2_EXACT)
                    epi::chunk_f32<CW, true>(v, taddr, raf, colsf, cols_special, col, b_row + col, a,
                                       a_ok, n_tile, dlo, dhi, p.r2, p.ldr, p.counts, p.ldc,
                                       p.out_row0, p.S);
                else
                    epi::chunk_ref<0, true, CW>(v, ra, colsr, col, b_row + col, a, a_ok, n_tile,
                                                dlo, dhi, p.r2, p.ldr, p.counts, p.ldc,
                                                p.out_row0, p.S);
            }
        }
    }

    // Teardown: no CTA frees its pair's TMEM or exits before the pair's last
    // commit has arrived in both CTAs and every peer is done with its memory.
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (!mbar_wait(smem_u32(accfull), 0, kDrainCycles, nullptr))
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


// Packed stages that fit beside the rest: an even number (an unpack group sees
// every other packed stage, so a slot must always belong to the same groups
// for its phase bit to be enough), or 0.
int packed_stages(int bn, int ks) {
    struct Table {
        signed char pst[MAX_BN / CH][3];
        Table() {
            for (int b = CH; b <= MAX_BN; b += CH)
                for (int k = 1; k <= 4; k *= 2) {
                    int n = MAX_PST;
                    while (n > 0 && Layout(b, k, n).bytes > MAX_SMEM) n -= 2;
                    pst[b / CH - 1][k >> 1] = (signed char)n;
                }
        }
    };
    static const Table table;
    return table.pst[bn / CH - 1][ks >> 1];
}

// Clusters of 2 ks CTAs that run at once, asked of the driver once per ks.
int max_clusters(int ks) {
    static std::atomic<int> known[3];
    std::atomic<int> &slot = known[ks >> 1];
    int n = slot.load(std::memory_order_relaxed);
    if (n > 0) return n;
    auto kern = k_ld_mxf4_split<R2_EXACT, true>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM) !=
        cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * ks) * 64, 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = MAX_SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)(2 * ks);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 0) {
        (void)cudaGetLastError();
        n = 0;
    }
    slot.store(n, std::memory_order_relaxed);
    return n;
}

template <int MODE, bool PLAIN>
cudaError_t launch_mode(const CUtensorMap &tmA, const CUtensorMap &tmB, const LdParams &p,
                        const RowTiles &tl, int ks, cudaStream_t st) {
    auto kern = k_ld_mxf4_split<MODE, PLAIN>;
    const int tiles = tl.count(), pst = packed_stages(tl.bn, ks);
    if (tiles == 0) return cudaSuccess;
    if (pst < 2) return cudaErrorInvalidConfiguration;
    static std::atomic<unsigned long long> allowed;
    cudaError_t e = allow_smem(kern, MAX_SMEM, allowed);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * 2 * ks), 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = (size_t)Layout(tl.bn, ks, pst).bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)(2 * ks);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1] = overlap_attr();
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p, tl, ks, pst);
}

}  // namespace

// The launch runs at once if its 256 x 240 tiles do, one per SM pair; the
// persistent kernel takes the others, where its epilogue overlaps the next
// tile's MMAs.  Among the (bn, ks) whose clusters all run at once the one
// with the least estimated time is taken (us, fitted to a sweep of bn and ks
// over sixteen shapes from 64 x 64 to 2,500 x 2,500 SNPs and 300 to 50,000
// samples on a B200; the choice was within 4 % of the sweep's best on each):
// 0.235 per 256-sample stage of a pair's part (a little more for long B
// tiles, half as much again when only two packed stages fit), 0.019 (exact)
// or 0.034 (reference) per column of a CTA's epilogue, and for a split 0.5
// plus 0.008 per column delivered to another pair; 0.01 per CTA.
bool plan_split(const RowTiles &tl, int K, int r2_mode, SplitPlan *plan) {
    const int np = (K + PW - 1) / PW, nu = (K + PW / SUB - 1) / (PW / SUB);
    const int most[3] = {max_clusters(1), max_clusters(2),
                         max_clusters(4)};
    const double per_col = r2_mode == R2_REFERENCE ? 0.034 : 0.019;
    double best = 0.0;
    bool found = false;
    for (int bn = MAX_BN; bn >= CH; bn -= CH) {
        RowTiles t = tl;
        t.bn = bn;
        if (t.rows() > most[0]) break;                  // every tile row has a tile
        const int tiles = t.count(), chunks = bn / CH;
        if (tiles > most[0]) break;
        for (int ks = 1; ks <= 4 && ks <= np; ks *= 2) {
            const int pst = packed_stages(bn, ks);
            if (tiles > most[ks >> 1] || pst < 2) continue;
            const double stage = (0.235 + (bn > 128 ? 0.0003 * (bn - 128) : 0.0)) *
                                 (pst < 4 && np > 2 * ks ? 1.5 : 1.0);
            const int own = (chunks + ks - 1) / ks * CH;
            const double us = stage * ((nu + ks - 1) / ks) + per_col * own +
                              (ks > 1 ? 0.5 + 0.008 * (bn - own) : 0.0) + 0.01 * (2 * tiles * ks);
            if (!found || us < best) {
                best = us;
                *plan = SplitPlan{bn, ks};
                found = true;
            }
        }
    }
    return found;
}

cudaError_t launch_mxf4_split(const CUtensorMap &tmA, const CUtensorMap &tmB, const LdParams &p,
                              const RowTiles &tl, int ks, int r2_mode, cudaStream_t st) {
    if (r2_mode == R2_REFERENCE)
        return !p.counts && p.S >= epi::R2_PLAIN_S && p.S <= (1 << 24)
                   ? launch_mode<R2_REFERENCE, true>(tmA, tmB, p, tl, ks, st)
                   : launch_mode<R2_REFERENCE, false>(tmA, tmB, p, tl, ks, st);
    return !p.counts ? launch_mode<R2_EXACT, true>(tmA, tmB, p, tl, ks, st)
                     : launch_mode<R2_EXACT, false>(tmA, tmB, p, tl, ks, st);
}

}  // namespace qld
