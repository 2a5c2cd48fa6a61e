// bf16 product with few output tiles: one 128 x 256 tile per cluster of 2, 4 or 8 CTAs that share its K.
//
// A product with a small M has N / 256 tiles, 2 to 32 of them, and one CTA per tile leaves most of the chip idle while each
// CTA pulls its weights through one SM (about 70 GB/s from HBM). Here every CTA of a cluster takes an equal run of K blocks,
// leaves its sums in its shared memory, and then adds one slice of the columns over the cluster, in the order of K, through
// distributed shared memory. 16 x 4096 x 4096 23.6 -> 15.3 us, 72 x 4096 x 7168 35.8 -> 21.3 us, 129 x 2048 x 8192 39.9 -> 23.7 us,
// 500 x 2048 x 7168 35.8 (on CTA pairs) -> 25.5 us.
#pragma once

#include "cluster_sum.cuh"

namespace slime {
namespace gemm {

constexpr int kKsStages     = 4;
constexpr int kKsBN         = kSumCols;
constexpr int kKsStageBytes = (kBM + kKsBN) * kBK * 2;
constexpr int kKsSmem       = kKsStages * kKsStageBytes + (2 * kKsStages + 1) * 8 + 16 + 1024;
static_assert(kKsStages * kKsStageBytes >= kSumPitch * kBM * 4, "the ring holds the sums of the tile afterwards");

static __global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_ksplit_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ Args args, int split)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    uint64_t* full_bar  = reinterpret_cast<uint64_t*>(smem + kKsStages * kKsStageBytes);
    uint64_t* empty_bar = full_bar + kKsStages;
    uint64_t* done_bar  = empty_bar + kKsStages;  // every MMA of this CTA has retired
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
    volatile uint32_t* fail_slot = tmem_slot + 1;

    const int          warp    = threadIdx.x >> 5;
    const int          lane    = threadIdx.x & 31;
    const int          crank   = static_cast<int>(cluster_ctarank());
    const int          total   = (args.K + kBK - 1) / kBK;
    const int          kb0     = static_cast<int>(static_cast<long long>(crank) * total / split);
    const int          kblocks = static_cast<int>(static_cast<long long>(crank + 1) * total / split) - kb0;  // at least one
    const int          mtiles  = (args.M_total + kBM - 1) / kBM;
    const int          tile    = blockIdx.x / split;
    const int          row0    = tile % mtiles * kBM;
    const int          col0    = tile / mtiles * kKsBN;
    KernelStatus*      st      = args.status;
    const unsigned long long lim = args.wait_ns ? args.wait_ns : kDefaultWaitNs;

    if (threadIdx.x == 0) {
        *fail_slot = 0;
        for (int s = 0; s < kKsStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(done_bar, 1);
        fence_mbar_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 256);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    float* sums = reinterpret_cast<float*>(smem);  // [128 rows][kSumPitch], once the ring has been consumed
    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        for (int i = 0; i < kblocks; ++i) {
            const int stage = i % kKsStages;
            if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], ((i / kKsStages) & 1) ^ 1, st, 1, stage, lim))) {
                *fail_slot = 1;
                break;
            }
            uint8_t* sa = smem + stage * kKsStageBytes;
            uint8_t* sb = sa + kBM * kBK * 2;
            if (elect_one()) {
                mbar_arrive_expect_tx(&full_bar[stage], kKsStageBytes);
                tma_load_2d(sa, &tmA, &full_bar[stage], (kb0 + i) * kBK, row0);
                tma_load_2d(sb, &tmB, &full_bar[stage], (kb0 + i) * kBK, col0);
                tma_load_2d(sb + kKsBN / 2 * kBK * 2, &tmB, &full_bar[stage], (kb0 + i) * kBK, col0 + kKsBN / 2);
            }
            __syncwarp();
        }
    }
    else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------
        constexpr uint32_t idesc = make_idesc(kFmtBF16, kFmtBF16, kBM, kKsBN);
        bool               ok    = true;
        for (int i = 0; i < kblocks && ok; ++i) {
            const int stage = i % kKsStages;
            ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[stage], (i / kKsStages) & 1, st, 3, stage, lim));
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t sa = smem_u32(smem + stage * kKsStageBytes);
            const uint64_t da = make_kmajor_sw128_desc(sa);
            const uint64_t db = make_kmajor_sw128_desc(sa + kBM * kBK * 2);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) umma_f16(tmem_base, da + 2 * k, db + 2 * k, idesc, (i | k) != 0);
                umma_commit(&empty_bar[stage]);
                if (i == kblocks - 1) umma_commit(done_bar);
            }
            __syncwarp();
        }
        if (!ok) *fail_slot = 1;
    }
    else {
        // ------------------------------ accumulator -> shared memory --------------
        const int quad = warp & 3;
        const int trow = quad * 32 + lane;
        if (!__all_sync(0xffffffffu, mbar_wait(done_bar, 0, st, 4, 0, lim))) {
            *fail_slot = 1;
        }
        else if (row0 + quad * 32 < args.M_total) {
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
            for (int c = 0; c < kKsBN; c += 32) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(taddr + c, v);
                tmem_ld_wait();
                uint4* dst = reinterpret_cast<uint4*>(sums + trow * kSumPitch + c);
#pragma unroll
                for (int i = 0; i < 8; ++i) dst[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        }
    }

    cluster_add_store(sums, fail_slot, crank, split, row0, col0, args.M_total, args.N, args.C, args.ldc);

    // teardown: no CTA may leave while another one still reads its sums
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        if (*fail_slot != 0) settle_copies();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 256);
    }
}

}  // namespace gemm
}  // namespace slime
