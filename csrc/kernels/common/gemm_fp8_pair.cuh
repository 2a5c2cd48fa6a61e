// The block-scaled fp8 product of gemm_fp8.cuh (same contract, same two-level accumulation) in the two forms that the plain
// GEMM uses: on CTA pairs, and split along K over a cluster.
//
// Pairs (tcgen05 cta_group::2, 256 x 256 tiles). A single CTA's 128 x 256 x 128 block is 512 cycles of tensor pipe, but
// its operands are 48 KB that are written into shared memory once and read once, 768 cycles at 128 bytes each: with all of the
// promotion work left out the single-CTA kernel still took 540 us for 8192^3, with it 648. In a pair each CTA
// holds half of B, 32 KB per block. Both CTAs keep a 128 x 256 partial of their own rows in TMEM (two partials of 256 columns,
// or up to eight of a narrower tile), and eight promotion warps per CTA read it, multiply by sa * sb and add into
// registers: one thread owns one row and half of the tile's columns. The read of the next 32 columns is in flight while the
// current 32 are added (64 registers beside the 128 accumulators), a partial is handed back as soon as its last read has
// landed, and the first read of the next one is issued before the last additions when that partial is ready. That is more
// than the 168 registers that 12 warps may have at launch: the promotion warpgroups take over what the producer's
// warpgroup gives back (setmaxnreg). A K block now takes 650 cycles, 512 of them MMA, as long as the clock holds; what is left is the
// power limit: 8192 x 3584 x 8192 309 -> 283 us, 4096 x 4096 x 7168 148 -> 127-139 us, 8192^3 level at 600-610 us (1.8 PFLOP/s).
// The tiles left over after the last full round of the grid are cut into 2, 4 or 8 column parts of a pair each.
//
// Split along K (128 x 256 tiles, cluster of 2, 4 or 8 CTAs): for products with fewer tiles than a quarter of the SMs. Each CTA of
// a cluster takes an equal run of K blocks and leaves its sums in its shared memory; then each adds one slice of
// the columns over the cluster, in the order of K, through distributed shared memory, and stores it. Narrower tiles
// instead have all CTAs read the same rows of A: 72 x 4096 x 7168 took 27 us on 128 CTAs with tiles of 32 columns, and
// leaving the promotion out changed nothing. Of the 14 us that 72 rows take in the kernel, 6 are the K blocks and 8 the exchange of
// the sums. 72 x 4096 x 7168 38.9 -> 21 us, 33 x 2048 x 8192 41 -> 16.4 us, 500 x 2048 x 7168 39 -> 25-29 us.
#pragma once

#include "cluster_sum.cuh"
#include "gemm_fp8.cuh"

namespace slime {
namespace gemm {

constexpr int kF8pPromoWarps = 8;
constexpr int kF8pCtlWarps   = 4;
constexpr int kF8pThreads    = (kF8pCtlWarps + kF8pPromoWarps) * 32;
// 128 * 40 + 256 * 232 = 384 * 168, the registers a 384-thread block is launched with
constexpr int kF8pRegsCtl   = 40;
constexpr int kF8pRegsPromo = 232;
static_assert(kF8pCtlWarps * kF8pRegsCtl + kF8pPromoWarps * kF8pRegsPromo <= (kF8pCtlWarps + kF8pPromoWarps) * 168, "register split");
constexpr int kF8pNarrowBox = 16;  // B rows per TMA box of a narrow tile (half of the narrowest)
constexpr int kF8pMaxStages = 8;
constexpr int kF8pMaxParts  = 8;
constexpr int kF8pABytes    = kBM * kF8BK;
constexpr int kF8pRingBytes = 6 * (kF8pABytes + kF8BN / 2 * kF8BK);  // stages * stage_bytes is at most this
constexpr int kF8pBarBytes  = (2 * kF8pMaxStages + 2 * kF8pMaxParts) * 8 + 16;
constexpr int kF8pEpiBytes  = kF8pPromoWarps * 32 * kEpiRowPitch;  // results leave through one 128-byte slot per row and warp
constexpr int kF8pSmem      = kF8pRingBytes + kF8pEpiBytes + kF8pBarBytes + 1024;
static_assert(kF8pSmem <= kSmemLimit, "shared memory budget");

struct F8PairArgs {
    int M, N, K;
    __nv_bfloat16* C;
    long long      ldc;
    const float*   sa;          // [M, K/128]
    const float*   sb;          // [ceil(N/128), K/128]
    int            full_tiles;  // pairs: leading tiles that are 256 wide (a multiple of the pairs, or all)
    int            split;       // pairs: column parts (1, 2, 4 or 8) that every later tile is cut into; split along K: CTAs per cluster
    int            stages;      // pipeline stages, and the bytes of one
    int            stage_bytes;
    KernelStatus*  status;
    unsigned long long wait_ns;
};

struct F8Tile {
    int row0;   // of the tile (256 rows on pairs)
    int col0;
    int width;  // 256, 128, 64 or 32
    // TMEM partials of this width and the columns between two of them
    __device__ int parts() const { return width == 256 ? 2 : width == 128 ? 4 : kF8pMaxParts; }
    __device__ int part_stride() const { return 512 / parts(); }
};

// Tile sequence of one pair, m fastest. The full tiles come first; the remaining ones are cut into `split` column parts,
// part fastest, so that neighbouring pairs share the A rows.
struct F8PairWalker {
    const F8PairArgs& f;
    int               mtiles, total, t, step;
    __device__ F8PairWalker(const F8PairArgs& args): f(args)
    {
        mtiles           = (f.M + 2 * kBM - 1) / (2 * kBM);
        const int ntiles = (f.N + kF8BN - 1) / kF8BN;
        total            = f.full_tiles + (mtiles * ntiles - f.full_tiles) * f.split;
        t                = blockIdx.x >> 1;
        step             = gridDim.x >> 1;
    }
    __device__ bool next(F8Tile& c)
    {
        while (t < total) {
            int lt = t, sub = 0;
            c.width = kF8BN;
            if (t >= f.full_tiles) {
                lt      = f.full_tiles + (t - f.full_tiles) / f.split;
                sub     = (t - f.full_tiles) % f.split;
                c.width = kF8BN / f.split;
            }
            t += step;
            c.row0 = lt % mtiles * 2 * kBM;
            c.col0 = lt / mtiles * kF8BN + sub * c.width;
            if (c.col0 < f.N) return true;  // the last tile column may have parts past the end
        }
        return false;
    }
};

// Position in the ring of TMEM partials. The number of partials changes with the tile width, so every partial has a
// phase bit of its own.
struct F8Parts {
    int      part   = 0;
    uint32_t phases = 0;
    __device__ uint32_t phase() const { return (phases >> part) & 1u; }
    __device__ void     advance(int parts)
    {
        phases ^= 1u << part;
        if (++part >= parts) part = 0;
    }
};

// acc += s * v for 32 columns, as packed pairs (each half is one IEEE fused multiply-add).
__device__ __forceinline__ void f8_promote32(unsigned long long* acc, float s, const uint32_t (&v)[32])
{
    unsigned long long s2;
    asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        unsigned long long v2;
        asm("mov.b64 %0, {%1, %2};" : "=l"(v2) : "r"(v[2 * i]), "r"(v[2 * i + 1]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i]) : "l"(s2), "l"(v2));
    }
}

// Arrives on an mbarrier of the cluster with the default (CTA-scope) release. What it hands back are TMEM reads, which
// tcgen05.wait::ld and the tcgen05 fence have ordered; a release at cluster scope would also wait for the
// thread's loads in flight, about 1000 cycles per K block here.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// The promotion of `kblocks` K blocks of one tile by one thread: NCH chunks of 32 columns per K block. Narrow tiles read a
// whole chunk where only 16 columns are the thread's; the rest lies inside the partial's stride and is never stored.
// pempty: shared::cluster addresses of the barriers that the MMA issuer waits for.
template<int NCH>
__device__ __forceinline__ bool f8_accumulate(unsigned long long (&acc)[NCH * 16], F8Parts& pp, int parts, int stride, uint64_t* pfull_bar,
                                              uint32_t pempty, uint32_t tcol, const float* sa_row, const float* sb_row, int kblocks,
                                              KernelStatus* st, unsigned long long lim)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < NCH * 16; ++i) acc[i] = 0ull;
    // The row scales are fetched four K blocks ahead: one in eight of them comes from L2 or beyond. The weight scales
    // are the same for the whole warp: each lane keeps one of the next 32.
    float sa_q[4], sb_lane = 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) sa_q[u] = sa_row[u < kblocks ? u : kblocks - 1];
    uint32_t v[2][32];
    if (!__all_sync(0xffffffffu, mbar_wait(&pfull_bar[pp.part], pp.phase(), st, 4, pp.part, lim))) return false;
    tc_fence_after_sync();
    tmem_ld_32x32b_x32(tcol + pp.part * stride, v[0]);
    for (int kb0 = 0; kb0 < kblocks; kb0 += 4) {
        if ((kb0 & 31) == 0) sb_lane = sb_row[kb0 + lane < kblocks ? kb0 + lane : kblocks - 1];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int kb = kb0 + u;
            if (kb >= kblocks) break;
            const float s = sa_q[u] * __shfl_sync(0xffffffffu, sb_lane, kb & 31);
            sa_q[u]       = sa_row[kb + 4 < kblocks ? kb + 4 : kblocks - 1];
            bool early    = true;
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const int b = (c + ((NCH & 1) ? u : 0)) & 1;  // an odd chunk count moves the first buffer of every other K block
                tmem_ld_wait_x32(v[b]);
                if (c + 1 < NCH) {
                    tmem_ld_32x32b_x32(tcol + pp.part * stride + (c + 1) * 32, v[b ^ 1]);
                }
                else {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(pempty + pp.part * 8);
                    pp.advance(parts);
                    if (kb + 1 < kblocks) {
                        early = __all_sync(0xffffffffu, mbar_test_wait(&pfull_bar[pp.part], pp.phase()));
                        if (early) {
                            tc_fence_after_sync();
                            tmem_ld_32x32b_x32(tcol + pp.part * stride, v[b ^ 1]);
                        }
                    }
                }
                f8_promote32(acc + c * 16, s, v[b]);
                if (c + 1 == NCH && !early) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&pfull_bar[pp.part], pp.phase(), st, 4, pp.part, lim))) return false;
                    tc_fence_after_sync();
                    tmem_ld_32x32b_x32(tcol + pp.part * stride, v[b ^ 1]);
                }
            }
        }
    }
    return true;
}

// One tile of the pair kernel by one thread: promotion, then its `cols` columns of its row.
template<int NCH>
__device__ __forceinline__ bool f8_pair_tile(const F8PairArgs& f, const F8Tile& tc, F8Parts& pp, uint64_t* pfull_bar, uint32_t pempty,
                                             uint32_t taddr_lane, int grp, int row, int kblocks, uint8_t* warp_slots,
                                             unsigned long long lim)
{
    const bool   valid = row < f.M;
    const int    cols  = tc.width / 2;
    const int    col0  = tc.col0 + grp * cols;
    const int    nblk  = col0 / 128, nblk_last = (f.N + 127) / 128 - 1;  // a thread's columns never straddle a scale block
    const float* sb_row = f.sb + static_cast<long long>(nblk < nblk_last ? nblk : nblk_last) * kblocks;
    const float* sa_row = f.sa + static_cast<long long>(valid ? row : f.M - 1) * kblocks;
    unsigned long long acc[NCH * 16];
    if (!f8_accumulate<NCH>(acc, pp, tc.parts(), tc.part_stride(), pfull_bar, pempty, taddr_lane + grp * cols, sa_row, sb_row, kblocks, f.status, lim))
        return false;
    // whole 128-byte lines leave the SM (see epi_store_piece); 64 columns at a time, 32 for the narrow tiles
    int left = f.N - col0;  // a multiple of 8 (N % 32 == 0)
    if (left > cols) left = cols;
    const unsigned long long dst = reinterpret_cast<unsigned long long>(f.C + static_cast<long long>(row) * f.ldc + col0);
#pragma unroll
    for (int i = 0; i < NCH; i += 2) {
        uint32_t o[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const int q = i * 16 + j;
            o[j]        = q < NCH * 16 ? pack_bf16(__uint_as_float(static_cast<uint32_t>(acc[q < NCH * 16 ? q : 0])),
                                                   __uint_as_float(static_cast<uint32_t>(acc[q < NCH * 16 ? q : 0] >> 32))) : 0u;
        }
        epi_store_piece(warp_slots + (threadIdx.x & 31) * kEpiRowPitch, warp_slots, o, dst + static_cast<unsigned long long>(i) * 64, valid,
                        min(64, left - i * 32), threadIdx.x & 31);
    }
    return true;
}

__device__ __forceinline__ void umma_f8f6f4_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

static __global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kF8pThreads, 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmBn, const __grid_constant__ F8PairArgs f)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    uint8_t*  epi_smem   = smem + kF8pRingBytes;
    uint64_t* full_bar   = reinterpret_cast<uint64_t*>(epi_smem + kF8pEpiBytes);  // used in the leader only
    uint64_t* empty_bar  = full_bar + kF8pMaxStages;                           // one set per CTA
    uint64_t* pfull_bar  = empty_bar + kF8pMaxStages;                          // one set per CTA
    uint64_t* pempty_bar = pfull_bar + kF8pMaxParts;                           // used in the leader only
    uint32_t* tmem_slot  = reinterpret_cast<uint32_t*>(pempty_bar + kF8pMaxParts);
    volatile uint32_t* fail_slot = tmem_slot + 1;

    const int          warp    = threadIdx.x >> 5;
    const int          lane    = threadIdx.x & 31;
    const uint32_t     crank   = cluster_ctarank();  // 0 = leader
    const int          kblocks = f.K / kF8BK;
    const int          stages  = f.stages;
    KernelStatus*      st      = f.status;
    const unsigned long long lim = f.wait_ns ? f.wait_ns : kDefaultWaitNs;

    if (threadIdx.x == 0) {
        *fail_slot = 0;
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 1);   // the leader's producer arrives once and expects the bytes of both CTAs
            mbar_init(&empty_bar[s], 1);  // one commit
        }
        for (int s = 0; s < kF8pMaxParts; ++s) {
            mbar_init(&pfull_bar[s], 1);
            mbar_init(&pempty_bar[s], 2 * kF8pPromoWarps);  // the promotion warps of both CTAs
        }
        fence_mbar_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        tma_prefetch_desc(&tmBn);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 512);
        tmem_relinquish_pair();
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers exist before anything is sent to them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    griddep_wait();  // launched while the kernel in front of it drains
    griddep_launch_dependents();

    if (warp < kF8pCtlWarps) {
        setmaxnreg_dec<kF8pRegsCtl>();
        if (warp == 0) {
            // ------------------------------ TMA producer (both CTAs) ------------------------------
            F8PairWalker walk(f);
            F8Tile       tc;
            int          stage = 0;
            uint32_t     phase = 0;
            bool         ok    = true;
            fence_proxy_async();  // the operands may have been written by the kernel in front of this one
            while (ok && walk.next(tc)) {
                const int arow = tc.row0 + static_cast<int>(crank) * kBM;
                const int half = tc.width / 2;
                const int brow = tc.col0 + static_cast<int>(crank) * half;
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1, st, 1, stage, lim))) {
                        ok = false;
                        break;
                    }
                    uint8_t* sa = smem + stage * f.stage_bytes;
                    uint8_t* sb = sa + kF8pABytes;
                    const uint32_t leader_full = mapa_u32(&full_bar[stage], 0);
                    if (elect_one()) {
                        if (crank == 0) mbar_arrive_expect_tx(&full_bar[stage], 2 * (kF8pABytes + half * kF8BK));
                        tma_load_2d_pair(sa, &tmA, leader_full, kb * kF8BK, arow);
                        if (tc.width == kF8BN)
                            tma_load_2d_pair(sb, &tmB, leader_full, kb * kF8BK, brow);
                        else
                            for (int r = 0; r < half; r += kF8pNarrowBox) tma_load_2d_pair(sb + r * kF8BK, &tmBn, leader_full, kb * kF8BK, brow + r);
                    }
                    __syncwarp();
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) *fail_slot = 1;
        }
        else if (warp == 1 && crank == 0) {
            // ------------------------------ MMA issuer (leader only) ------------------------------
            F8PairWalker walk(f);
            F8Tile       tc;
            F8Parts      pp;
            int          stage = 0, width = 0;
            uint32_t     phase = 0;
            bool         ok = true;
            while (ok && walk.next(tc)) {
                const int parts = tc.parts(), stride = tc.part_stride();
                if (width != 0 && width != tc.width) {
                    // another cut of the TMEM columns: every partial of the old one has to be consumed first
                    for (int p = 0; p < kF8pMaxParts && ok; ++p)
                        ok = __all_sync(0xffffffffu, mbar_wait(&pempty_bar[p], ((pp.phases >> p) & 1u) ^ 1u, st, 2, p, lim));
                    if (!ok) break;
                    pp.part = 0;
                }
                width = tc.width;
                const uint32_t idesc = make_idesc(kFmtE4M3, kFmtE4M3, 2 * kBM, static_cast<uint32_t>(tc.width));
                for (int kb = 0; kb < kblocks && ok; ++kb) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&pempty_bar[pp.part], pp.phase() ^ 1u, st, 2, pp.part, lim)
                                                     && mbar_wait(&full_bar[stage], phase, st, 3, stage, lim))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t tmem_d = tmem_base + pp.part * stride;
                    const uint32_t sa = smem_u32(smem + stage * f.stage_bytes);
                    const uint64_t da = make_kmajor_sw128_desc(sa);
                    const uint64_t db = make_kmajor_sw128_desc(sa + kF8pABytes);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < kF8BK / 32; ++k) umma_f8f6f4_pair(tmem_d, da + 2 * k, db + 2 * k, idesc, k != 0);
                        umma_commit_pair(&empty_bar[stage], 3);     // frees the stage in both CTAs
                        umma_commit_pair(&pfull_bar[pp.part], 3);   // the partials of both CTAs are complete
                    }
                    __syncwarp();
                    pp.advance(parts);
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) *fail_slot = 1;
        }
        __syncwarp();
    }
    else {
        // ------------------------------ promotion + epilogue (both CTAs, own rows) ------------------------------
        setmaxnreg_inc<kF8pRegsPromo>();
        const int      quad   = warp & 3;
        const int      grp    = (warp - kF8pCtlWarps) >> 2;  // which half of the tile's columns
        const uint32_t pempty = mapa_u32(pempty_bar, 0);
        const uint32_t taddr  = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        uint8_t*       warp_slots = epi_smem + (warp - kF8pCtlWarps) * 32 * kEpiRowPitch;
        F8PairWalker   walk(f);
        F8Tile         tc;
        F8Parts        pp;
        int            width = 0;
        bool           ok = true;
        while (ok && walk.next(tc)) {
            const int row = tc.row0 + static_cast<int>(crank) * kBM + quad * 32 + lane;
            if (width != 0 && width != tc.width) pp.part = 0;  // as the MMA issuer does
            width = tc.width;
            if (tc.width == 256)
                ok = f8_pair_tile<4>(f, tc, pp, pfull_bar, pempty, taddr, grp, row, kblocks, warp_slots, lim);
            else if (tc.width == 128)
                ok = f8_pair_tile<2>(f, tc, pp, pfull_bar, pempty, taddr, grp, row, kblocks, warp_slots, lim);
            else
                ok = f8_pair_tile<1>(f, tc, pp, pfull_bar, pempty, taddr, grp, row, kblocks, warp_slots, lim);
        }
        if (!ok) *fail_slot = 1;
    }

    // teardown: both CTAs meet (no CTA may leave while its peer still reads its shared memory or signals its
    // barriers), then the allocating warps free TMEM
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        if (*fail_slot != 0) settle_copies();
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

constexpr int kF8kStages     = 4;
constexpr int kF8kStageBytes = kBM * kF8BK + kF8BN * kF8BK;
static_assert(kF8BN == kSumCols && kF8kStages * kF8kStageBytes >= kSumPitch * kBM * 4, "the ring holds the sums of the tile afterwards");
static_assert(kF8kStages * kF8kStageBytes <= kF8pRingBytes, "same shared memory as the pair kernel");

// One 128 x 256 tile per cluster of f.split CTAs, each with its run of K blocks.
static __global__ void __launch_bounds__(kF8pThreads, 1)
gemm_fp8_ksplit_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ F8PairArgs f)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    uint64_t* full_bar   = reinterpret_cast<uint64_t*>(smem + kF8pRingBytes + kF8pEpiBytes);
    uint64_t* empty_bar  = full_bar + kF8pMaxStages;
    uint64_t* pfull_bar  = empty_bar + kF8pMaxStages;
    uint64_t* pempty_bar = pfull_bar + kF8pMaxParts;
    uint32_t* tmem_slot  = reinterpret_cast<uint32_t*>(pempty_bar + kF8pMaxParts);
    volatile uint32_t* fail_slot = tmem_slot + 1;

    const int          warp    = threadIdx.x >> 5;
    const int          lane    = threadIdx.x & 31;
    const int          crank   = static_cast<int>(cluster_ctarank());
    const int          total   = f.K / kF8BK;
    const int          kb0     = static_cast<int>(static_cast<long long>(crank) * total / f.split);
    const int          kblocks = static_cast<int>(static_cast<long long>(crank + 1) * total / f.split) - kb0;  // at least one
    const int          mtiles  = (f.M + kBM - 1) / kBM;
    const int          tile    = blockIdx.x / f.split;
    const int          row0    = tile % mtiles * kBM;
    const int          col0    = tile / mtiles * kF8BN;
    KernelStatus*      st      = f.status;
    const unsigned long long lim = f.wait_ns ? f.wait_ns : kDefaultWaitNs;

    if (threadIdx.x == 0) {
        *fail_slot = 0;
        for (int s = 0; s < kF8kStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&pfull_bar[s], 1);
            mbar_init(&pempty_bar[s], kF8pPromoWarps);
        }
        fence_mbar_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    griddep_wait();
    griddep_launch_dependents();

    float* sums = reinterpret_cast<float*>(smem);  // [128 rows][kSumPitch], once the ring has been consumed
    if (warp < kF8pCtlWarps) {
        setmaxnreg_dec<kF8pRegsCtl>();
        if (warp == 0) {
            // ------------------------------ TMA producer ------------------------------
            fence_proxy_async();
            for (int i = 0; i < kblocks; ++i) {
                const int stage = i % kF8kStages;
                if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], ((i / kF8kStages) & 1) ^ 1, st, 1, stage, lim))) {
                    *fail_slot = 1;
                    break;
                }
                uint8_t* sa = smem + stage * kF8kStageBytes;
                uint8_t* sb = sa + kBM * kF8BK;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&full_bar[stage], kF8kStageBytes);
                    tma_load_2d(sa, &tmA, &full_bar[stage], (kb0 + i) * kF8BK, row0);
                    tma_load_2d(sb, &tmB, &full_bar[stage], (kb0 + i) * kF8BK, col0);
                    tma_load_2d(sb + kF8BN / 2 * kF8BK, &tmB, &full_bar[stage], (kb0 + i) * kF8BK, col0 + kF8BN / 2);
                }
                __syncwarp();
            }
        }
        else if (warp == 1) {
            // ------------------------------ MMA issuer ------------------------------
            constexpr uint32_t idesc = make_idesc(kFmtE4M3, kFmtE4M3, kBM, kF8BN);
            for (int i = 0; i < kblocks; ++i) {
                const int stage = i % kF8kStages, part = i & 1;
                if (!__all_sync(0xffffffffu, mbar_wait(&pempty_bar[part], ((i >> 1) & 1) ^ 1, st, 2, part, lim)
                                                 && mbar_wait(&full_bar[stage], (i / kF8kStages) & 1, st, 3, stage, lim))) {
                    *fail_slot = 1;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t sa = smem_u32(smem + stage * kF8kStageBytes);
                const uint64_t da = make_kmajor_sw128_desc(sa);
                const uint64_t db = make_kmajor_sw128_desc(sa + kBM * kF8BK);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < kF8BK / 32; ++k) umma_f8f6f4(tmem_base + part * kF8BN, da + 2 * k, db + 2 * k, idesc, k != 0);
                    umma_commit(&empty_bar[stage]);
                    umma_commit(&pfull_bar[part]);
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
    else {
        // ------------------------------ promotion ------------------------------
        setmaxnreg_inc<kF8pRegsPromo>();
        const int    quad = warp & 3, grp = (warp - kF8pCtlWarps) >> 2;
        const int    trow = quad * 32 + lane;
        const int    row  = row0 + trow;
        const int    nblk = (col0 + grp * 128) / 128, nblk_last = (f.N + 127) / 128 - 1;
        const float* sa_row = f.sa + static_cast<long long>(row < f.M ? row : f.M - 1) * total + kb0;
        const float* sb_row = f.sb + static_cast<long long>(nblk < nblk_last ? nblk : nblk_last) * total + kb0;
        F8Parts      pp;
        unsigned long long acc[64];
        const bool ok = f8_accumulate<4>(acc, pp, 2, kF8BN, pfull_bar, mapa_u32(pempty_bar, static_cast<uint32_t>(crank)),
                                         tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + grp * 128, sa_row, sb_row, kblocks, st, lim);
        if (!ok) *fail_slot = 1;
        // Every block of this CTA has gone through the tensor core, so the ring is free. (After a wait that ran out copies may
        // still land there: nothing is left in it, and nobody stores.)
        if (ok && row < f.M) {
            float4* dst = reinterpret_cast<float4*>(sums + trow * kSumPitch + grp * 128);
#pragma unroll
            for (int i = 0; i < 32; ++i)
                dst[i] = make_float4(__uint_as_float(static_cast<uint32_t>(acc[2 * i])), __uint_as_float(static_cast<uint32_t>(acc[2 * i] >> 32)),
                                     __uint_as_float(static_cast<uint32_t>(acc[2 * i + 1])), __uint_as_float(static_cast<uint32_t>(acc[2 * i + 1] >> 32)));
        }
    }

    cluster_add_store(sums, fail_slot, crank, f.split, row0, col0, f.M, f.N, f.C, f.ldc);

    // teardown: no CTA may leave while another one still reads its sums
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        if (*fail_slot != 0) settle_copies();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace gemm
}  // namespace slime
