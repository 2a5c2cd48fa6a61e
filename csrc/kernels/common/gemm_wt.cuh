// The grouped expert GEMM for launches that stream weights from HBM (up to a few hundred rows per group): one CTA per
// SM, weights on the M side of the MMA, the tokens of a group on the N side.
//
//   C[g] (rows of group g, N) = A[g] (rows of group g, K) * B[g] (N, K)^T      (the contract of gemm_tc.cuh)
//
// A tile is 256 weight rows (two M = 128 blocks: 256 output features, or 128 gate rows and the 128 up rows of the same
// features) by ALL tokens of the group, up to PTOK, rounded up to 16. Larger groups are cut into equal parts.
//
// What bounds such a launch, and why this shape: every weight byte is read from HBM once (6.9-7.0 TB/s for a bare TMA
// stream with 96-128 KB in flight per SM), but it also has to get into the SM beside the tokens, at 64 bytes per clock, and at
// full load the power limit holds the SM clock at 1.1-1.4 GHz. With tokens on the M side a group of 128 +- 11 rows is one or two
// 128-row tiles, so a 64-deep K block of 256 weight rows costs 48 KB per row tile, 70 KB on average, and 1.47 times the
// rows that exist go through the tensor core. Here it costs 32 KB + 128 bytes per token, 50 KB, and the MMAs
// are as wide as the group. Whole one-rank steps, hidden 7168, intermediate 2048, replayed from graphs in turn with the row-tiled
// kernel in the same step: 128 experts x 128 rows 2426 -> 2183 us, x 160 rows 3009 -> 2341, x 192 rows 3166 -> 2970, x 256 rows
// 3690 -> 4204: there a group is two parts whose accumulators leave no room for a second buffer, and the row tiles waste little.
// When it came in: 64 x 97 rows 1125 -> 1082 us, 32 x 32 rows 559 -> 514 us, 19 x 1 354 -> 339 us.
//
// The accumulator is transposed: tensor-memory lanes are features, columns are tokens. Eight epilogue warps (two per lane
// quadrant, taking 32-token chunks in turn) round to bf16, turn a 32-token x 128-feature block around in shared memory
// and write 256 contiguous bytes per token. Gate and up of a feature sit in the same lane of the two blocks.
// Tiles of up to 128 tokens double-buffer the accumulator (two blocks x 128 columns x 2); larger ones take all 512 columns.
#pragma once

#include "gemm_tc.cuh"

namespace slime {
namespace gemm {

constexpr int kWtEpiWarps = 8;
constexpr int kWtThreads  = 64 + 32 * kWtEpiWarps;
constexpr int kWtGroups   = 256;  // group prefixes up to this length are kept in shared memory

template<int PTOK>
struct SmemWt {
    static constexpr int kStages     = PTOK > 128 ? 3 : 4;  // 96 or 128 KB of weights in flight
    static constexpr int kWBytes     = 256 * kBK * 2;
    static constexpr int kXBytes     = PTOK * kBK * 2;
    static constexpr int kStageBytes = kWBytes + kXBytes;
    static constexpr int kBlockBytes = 32 * 128 * 2;        // one staged block: 32 tokens x 128 features, bf16
    static constexpr int kEpiBytes   = 2 * 2 * kBlockBytes;  // two buffers per half of the epilogue warps
    static constexpr int kBarBytes   = (2 * kStages + 4) * 8 + 16;
    static constexpr int kOffBytes   = (kWtGroups + 1) * 4;
    static constexpr int kTotal      = kStages * kStageBytes + kEpiBytes + kBarBytes + kOffBytes + 1024;
    static_assert(kTotal <= kSmemLimit, "shared memory budget");
};

struct WtTile {
    int group;
    int tok0;     // first token row of the tile
    int tok_end;  // one past its last valid token row
    int ntok;     // N of the MMAs: the valid tokens rounded up to 16
    int nt;       // feature tile
};

// Tiles of a group: ceil(rows / PTOK) equal parts (rounded up to 16 tokens), part fastest, then the feature tile, so that CTAs
// running at the same time share the tokens and, where a group has several parts, the weights.
template<int PTOK>
struct WtWalker {
    const Args& a;
    const int*  offs;
    int         ntiles_n, t, g, cum, g_begin, g_end, g_parts, g_part_rows;
    __device__ WtWalker(const Args& args, const int* offsets, int feat_out): a(args), offs(offsets)
    {
        ntiles_n = (a.N + feat_out - 1) / feat_out;
        t        = blockIdx.x;
        g        = -1;
        cum      = 0;
        g_begin = g_end = g_parts = g_part_rows = 0;
        advance_group();
    }
    __device__ void advance_group()
    {
        ++g;
        if (g < a.num_groups) {
            g_end   = min(offs[g + 1], a.M_total);
            g_begin = min(offs[g], g_end);
            const int rows = g_end - g_begin;
            g_parts        = (rows + PTOK - 1) / PTOK;
            g_part_rows    = g_parts ? (((rows + g_parts - 1) / g_parts + 15) & ~15) : 0;  // <= PTOK
        }
    }
    __device__ bool next(WtTile& c)
    {
        while (g < a.num_groups) {
            const int tiles_g = g_parts * ntiles_n;
            if (t < cum + tiles_g) {
                const int local = t - cum;
                c.group   = g;
                c.nt      = local / g_parts;
                c.tok0    = min(g_begin + (local % g_parts) * g_part_rows, g_end);
                c.tok_end = min(c.tok0 + g_part_rows, g_end);
                c.ntok    = max(16, (c.tok_end - c.tok0 + 15) & ~15);  // a part may be empty after the rounding: nothing is stored
                t += gridDim.x;
                return true;
            }
            cum += tiles_g;
            advance_group();
        }
        return false;
    }
};

template<int PTOK, int EPI>
__global__ void __launch_bounds__(kWtThreads, 1)
gemm_bf16_wt_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX32,
                    const __grid_constant__ CUtensorMap tmX16, const __grid_constant__ Args args)
{
    using S = SmemWt<PTOK>;
    constexpr int kStages  = S::kStages;
    constexpr int kFeatOut = EPI == kEpiSwiGLU ? 128 : 256;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    uint8_t*  epi_smem   = smem + kStages * S::kStageBytes;
    uint64_t* full_bar   = reinterpret_cast<uint64_t*>(epi_smem + S::kEpiBytes);
    uint64_t* empty_bar  = full_bar + kStages;
    uint64_t* tfull_bar  = empty_bar + kStages;  // [2] accumulator half ready
    uint64_t* tempty_bar = tfull_bar + 2;        // [2] accumulator half drained
    uint32_t* tmem_slot  = reinterpret_cast<uint32_t*>(tempty_bar + 2);
    volatile uint32_t* fail_slot = tmem_slot + 1;
    volatile uint32_t* epi_fail  = tmem_slot + 2;  // [2] written by the epilogue warps of one half only, read after their named barrier
    int*      s_offs     = reinterpret_cast<int*>(tmem_slot + 4);

    const int          warp    = threadIdx.x >> 5;
    const int          lane    = threadIdx.x & 31;
    const int          kblocks = (args.K + kBK - 1) / kBK;
    KernelStatus*      st      = args.status;
    const unsigned long long lim = args.wait_ns ? args.wait_ns : kDefaultWaitNs;

    if (threadIdx.x == 0) {
        *fail_slot  = 0;
        epi_fail[0] = 0;
        epi_fail[1] = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tfull_bar[s], 1);
            mbar_init(&tempty_bar[s], kWtEpiWarps);
        }
        fence_mbar_init();
        tma_prefetch_desc(&tmW);
        tma_prefetch_desc(&tmX32);
        tma_prefetch_desc(&tmX16);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    const bool held = args.num_groups <= kWtGroups;  // the group prefix fits in shared memory
    // chained == 2: the group prefix and the weights are older than the kernel in front of this one, so the first weight
    // boxes are fetched while that kernel drains; everything else waits for it (griddep_wait is a no-op in an ordinary launch)
    const bool ahead = args.chained == 2 && held;
    if (!ahead) griddep_wait();
    griddep_launch_dependents();
    if (held)  // read past L1: with `ahead` this kernel may have begun before the one in front of it was done
        for (int g = threadIdx.x; g <= args.num_groups; g += blockDim.x) s_offs[g] = __ldcg(args.group_offsets + g);
    const int* offs = held ? s_offs : args.group_offsets;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    if (ahead && warp != 0) griddep_wait();

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        {
            WtWalker<PTOK> walk(args, offs, kFeatOut);
            WtTile   tc;
            int      stage = 0;
            uint32_t phase = 0;
            bool     ok    = true;
            bool     have  = walk.next(tc);
            int      early = 0;  // stages whose weights are on their way already
            auto load_w = [&](int s, int kb) {
                uint8_t*  sw = smem + s * S::kStageBytes;
                const int y  = tc.group * args.rowsB + tc.nt * kFeatOut;
                mbar_arrive_expect_tx(&full_bar[s], S::kWBytes + tc.ntok * kBK * 2);
                tma_load_2d(sw, &tmW, &full_bar[s], kb * kBK, y);
                tma_load_2d(sw + S::kWBytes / 2, &tmW, &full_bar[s], kb * kBK, y + (EPI == kEpiSwiGLU ? args.N : 128));
            };
            if (ahead) {
                if (have && elect_one())
                    for (int i = 0; i < kStages && i < kblocks; ++i) load_w(i, i);
                __syncwarp();
                early = have ? min(kStages, kblocks) : 0;
                griddep_wait();
            }
            if (args.chained) fence_proxy_async();  // the tokens were written by the kernel in front of this one
            for (; ok && have; have = walk.next(tc)) {
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1, st, 1, stage, lim))) {
                        ok = false;
                        break;
                    }
                    if (elect_one()) {
                        if (early == 0) load_w(stage, kb);
                        uint8_t* sx = smem + stage * S::kStageBytes + S::kWBytes;
                        int      r  = 0;
                        for (; r + 32 <= tc.ntok; r += 32) tma_load_2d(sx + r * kBK * 2, &tmX32, &full_bar[stage], kb * kBK, tc.tok0 + r);
                        if (r < tc.ntok) tma_load_2d(sx + r * kBK * 2, &tmX16, &full_bar[stage], kb * kBK, tc.tok0 + r);
                    }
                    __syncwarp();
                    if (early > 0) --early;
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) *fail_slot = 1;
        }
    }
    else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------
        {
            WtWalker<PTOK> walk(args, offs, kFeatOut);
            WtTile   tc;
            int      stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase[2] = {0, 0};
            bool     ok = true;
            while (ok && walk.next(tc)) {
                const bool large = tc.ntok > 128;
                if (large) acc = 0;
                ok = __all_sync(0xffffffffu, mbar_wait(&tempty_bar[acc], acc_phase[acc] ^ 1, st, 2, acc, lim)
                                                 && (!large || mbar_wait(&tempty_bar[1], acc_phase[1] ^ 1, st, 2, 1, lim)));
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t idesc  = make_idesc(kFmtBF16, kFmtBF16, 128, static_cast<uint32_t>(tc.ntok));
                const uint32_t tmem_d = tmem_base + acc * 256;
                const uint32_t block1 = large ? 256 : 128;
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, st, 3, stage, lim))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t sw = smem_u32(smem + stage * S::kStageBytes);
                    const uint64_t d0 = make_kmajor_sw128_desc(sw);
                    const uint64_t d1 = make_kmajor_sw128_desc(sw + S::kWBytes / 2);
                    const uint64_t dx = make_kmajor_sw128_desc(sw + S::kWBytes);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < kBK / 16; ++k) {
                            umma_f16(tmem_d, d0 + 2 * k, dx + 2 * k, idesc, (kb | k) != 0);
                            umma_f16(tmem_d + block1, d1 + 2 * k, dx + 2 * k, idesc, (kb | k) != 0);
                        }
                        umma_commit(&empty_bar[stage]);
                    }
                    __syncwarp();
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                if (elect_one()) {
                    umma_commit(&tfull_bar[acc]);
                    if (large) umma_commit(&tfull_bar[1]);
                }
                __syncwarp();
                acc_phase[acc] ^= 1;
                if (large) {
                    acc_phase[1] ^= 1;
                }
                else {
                    acc ^= 1;
                }
            }
            if (!ok) *fail_slot = 1;
        }
    }
    else {
        // ------------------------------ epilogue ----------------------------------
        const int quad = warp & 3;         // TMEM lane quadrant
        const int half = (warp - 2) >> 2;  // which of the 32-token chunks: even or odd ones
        const int w4   = (warp - 2) & 3;   // warp inside the half
        const int bar  = 1 + half;
        WtWalker<PTOK> walk(args, offs, kFeatOut);
        WtTile         tc;
        int            acc = 0;
        uint32_t       acc_phase[2] = {0, 0};
        unsigned int   block_no = 0;
        while (walk.next(tc)) {
            const bool large = tc.ntok > 128;
            if (large) acc = 0;
            if (!mbar_wait_relaxed(&tfull_bar[acc], acc_phase[acc], st, 4, acc, lim)
                || (large && !mbar_wait_relaxed(&tfull_bar[1], acc_phase[1], st, 4, 1, lim))) {
                *fail_slot     = 1;
                epi_fail[half] = 1;
            }
            // The warps of a half meet at named barriers below, which have no time limit: they leave the loop together or not
            // at all. A thread whose wait ran out says so before this barrier and everyone reads the word after it.
            asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
            if (epi_fail[half] != 0) break;
            tc_fence_after_sync();
            const uint32_t taddr  = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * 256;
            const uint32_t block1 = large ? 256 : 128;
#pragma unroll 1
            for (int c = half * 32; c < tc.ntok; c += 64) {
                // this lane stores 16 bytes of tokens c + w4 * 8 + 2 * j + (lane >> 4), j = 0..3
                unsigned long long drow[4];
                bool               store[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int row = tc.tok0 + c + w4 * 8 + 2 * j + (lane >> 4);
                    store[j]      = row < tc.tok_end;
                    if (EPI == kEpiScatterRows) {
                        const unsigned long long inf    = store[j] ? args.row_info[row] : ~0ull;
                        const unsigned int       region = static_cast<unsigned int>(inf >> 48);
                        const unsigned long long slot   = inf & 0xffffffffffffull;
                        const unsigned long long base   = region < 8 ? args.scatter_base[region] : 0ull;
                        store[j] = store[j] && base != 0ull && slot < args.scatter_slots;
                        drow[j]  = base + slot * args.scatter_row_bytes;
                    }
                    else {
                        drow[j] = reinterpret_cast<unsigned long long>(args.C + static_cast<long long>(row) * args.ldc);
                    }
                }
                float scale = 1.0f;  // of token c + lane
                if (EPI == kEpiScatterRows && args.row_scale && tc.tok0 + c + lane < tc.tok_end) scale = args.row_scale[tc.tok0 + c + lane];
#pragma unroll
                for (int b = 0; b < (EPI == kEpiSwiGLU ? 1 : 2); ++b) {
                    __nv_bfloat16* blk = reinterpret_cast<__nv_bfloat16*>(epi_smem + (half * 2 + (block_no & 1u)) * S::kBlockBytes);
                    ++block_no;
                    uint32_t v[32];
                    tmem_ld_32x32b_x32(taddr + b * block1 + c, v);
                    if (EPI == kEpiSwiGLU) {
                        uint32_t u[32];
                        tmem_ld_32x32b_x32(taddr + block1 + c, u);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(silu(__uint_as_float(v[i])) * __uint_as_float(u[i]));
                    }
                    else {
                        tmem_ld_wait();
                        if (EPI == kEpiScatterRows && args.row_scale) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * __shfl_sync(0xffffffffu, scale, i));
                        }
                    }
                    // lane = feature quad * 32 + lane of the block, v[i] = token c + i
#pragma unroll
                    for (int i = 0; i < 32; ++i) blk[i * 128 + quad * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[i]));
                    asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
                    const int col = tc.nt * kFeatOut + b * 128 + (lane & 15) * 8;
                    if (col < args.N) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint4 x = *reinterpret_cast<const uint4*>(blk + (w4 * 8 + 2 * j + (lane >> 4)) * 128 + (lane & 15) * 8);
                            if (store[j]) *reinterpret_cast<uint4*>(drow[j] + static_cast<unsigned long long>(col) * 2) = x;
                        }
                    }
                    // no second barrier: the next block goes to the other buffer, and a thread writes into this buffer again
                    // only after the next block's barrier, which every thread passes after it has finished reading here
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&tempty_bar[acc]);
                if (large) mbar_arrive(&tempty_bar[1]);
            }
            acc_phase[acc] ^= 1;
            if (large)
                acc_phase[1] ^= 1;
            else
                acc ^= 1;
        }
    }

    // teardown: everyone meets, then the allocating warp frees TMEM
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        if (*fail_slot != 0) {
            // a wait ran out somewhere: give copies still in flight a bounded moment to land
            settle_copies();
        }
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace gemm
}  // namespace slime
