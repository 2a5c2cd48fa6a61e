// Entry points of the block-scaled fp8 GEMM (common/gemm_fp8.cuh): the plain product and the
// all-gather -> GEMM built on it (fp8 payload and scales cross NVLink, half the bytes of the bf16 form).
#include "common/gemm_fp8_pair.cuh"
#include "common/host_utils.h"
#include "slime_cuda.h"

using namespace slime;
using namespace slime::gemm;

namespace {

// Push-only kernel of the all-gather form (single-GPU replay of multi-rank runs, and the unfused baseline).
__global__ void __launch_bounds__(32) ag_push_only_f8_kernel(const F8Args f)
{
    __shared__ __align__(128) uint8_t bufs[4 * kAgChunkBytes];
    __shared__ uint64_t               bars[4];
    if (threadIdx.x == 0) {
        for (int s = 0; s < 4; ++s) mbar_init(&bars[s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0 && !ag_push_bulk_f8(f, bufs, bars, 4, blockIdx.x, gridDim.x, f.ag.status, f.ag.wait_ns ? f.ag.wait_ns : kDefaultWaitNs))
        settle_copies();
}

template<bool AG>
int launch_f8(const void* Aq, const void* Bq, const void* A_local, const F8Args& f, long long lda, long long ldb, cudaStream_t stream)
{
    using S = SmemF8<AG>;
    CUtensorMap tmA, tmB, tmAL;
    if (make_tmap_2d(&tmA, Aq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, f.M, f.K, lda, kBM, kF8BK)) return -1;
    if (make_tmap_2d(&tmB, Bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, f.N, f.K, ldb, kF8BN / 2, kF8BK)) return -1;
    if (A_local) {
        if (make_tmap_2d(&tmAL, A_local, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, f.ag.ag_rows, f.K, f.K, kBM, kF8BK)) return -1;
    }
    else {
        tmAL = tmA;
    }
    auto kern = gemm_fp8_blockscaled_kernel<AG>;
    static bool configured[64] = {};
    SLIME_CUDA_OK(allow_dynamic_smem(kern, S::kTotal, configured));
    const long tiles = static_cast<long>((f.M + kBM - 1) / kBM) * ((f.N + kF8BN - 1) / kF8BN);
    int        grid  = sm_count();
    if (!AG && tiles < grid) grid = static_cast<int>(tiles);
    kern<<<grid, kF8Threads + (AG ? kAgThreads : 0), S::kTotal, stream>>>(tmA, tmB, tmAL, f);
    SLIME_CUDA_OK(cudaGetLastError());
    return 0;
}

int ksplit_clusters(int size)
{
    static int cached[64][3] = {};
    return max_active_clusters(gemm_fp8_ksplit_kernel, size, kF8pThreads, kF8pSmem, cached);
}

// Which form a plain product takes. Fewer 128 x 256 tiles than a quarter of the SMs: one cluster per tile, split along K over as
// many CTAs as still run at the same time, if that shortens each CTA's run by 14 blocks: meeting twice and adding the sums
// costs about 6 us (2000 x 544 x 1024: 20.5 us in clusters, 14.3 without). Else, with more than one row tile, CTA pairs: the r tiles that are left over after
// the last full round are cut into the most column parts (2, 4 or 8) that still have a pair each, since a last round of few
// wide tiles would take as long as a full one. Where there is nothing to cut, single CTAs have as many rounds as pairs, and for a few
// rounds of a deep product they are the faster ones: 1024 x 4096 x 7168 (one round) 38.1 us against 40.2 on pairs, x 4096 25.2 / 25.4,
// 1500 x 8192 x 7168 (three rounds) 111 / 116, x 4096 71 / 70; with 3.9 rounds 153 / 153. One row tile and all-gathered
// operands, whose order and pace are set by the arriving shards, stay on single CTAs too.
int launch_plain_f8(const void* Aq, const void* Bq, const F8Args& g, long long lda, long long ldb, cudaStream_t stream)
{
    F8PairArgs f{};
    f.M = g.M, f.N = g.N, f.K = g.K, f.C = g.C, f.ldc = g.ldc, f.sa = g.sa, f.sb = g.sb, f.status = g.ag.status, f.wait_ns = g.ag.wait_ns;
    const int  sms     = sm_count();
    const long ntiles  = (f.N + kF8BN - 1) / kF8BN;
    const long tiles   = static_cast<long>((f.M + kBM - 1) / kBM) * ntiles;
    const int  kblocks = f.K / kF8BK;
    const int  pairs   = sms / 2;
    const long pair_tiles = static_cast<long>((f.M + 2 * kBM - 1) / (2 * kBM)) * ntiles;
    const long rest       = pair_tiles % pairs;
    int split = 1, parts = 1;
    if (4 * tiles <= sms) {
        static bool configured[64] = {};
        SLIME_CUDA_OK(allow_dynamic_smem(gemm_fp8_ksplit_kernel, kF8pSmem, configured));
        for (int c : {2, 4, 8})
            if (kblocks - kblocks / c >= 14 && tiles <= ksplit_clusters(c)) split = c;
    }
    while (parts < 8 && rest > 0 && rest * parts * 2 <= pairs) parts *= 2;
    if (split == 1) {
        if (reinterpret_cast<unsigned long long>(f.C) % 16 != 0) return fail("fp8 gemm: the output must be 16-byte aligned (%p)", static_cast<void*>(f.C));
        const bool few_rounds = parts == 1 && (pair_tiles <= pairs ? kblocks >= 36 : pair_tiles <= 3 * pairs && kblocks >= 44);
        if (f.M <= kBM || few_rounds) return launch_f8<false>(Aq, Bq, nullptr, g, lda, ldb, stream);
    }
    CUtensorMap tmA, tmB, tmBn;
    if (make_tmap_2d(&tmA, Aq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, f.M, f.K, lda, kBM, kF8BK)) return -1;
    if (make_tmap_2d(&tmB, Bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, f.N, f.K, ldb, kF8BN / 2, kF8BK)) return -1;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim         = dim3(kF8pThreads);
    cfg.dynamicSmemBytes = kF8pSmem;
    cfg.stream           = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs                                          = attr;
    cfg.numAttrs                                       = 1;
    if (split > 1) {
        f.split                  = split;
        cfg.gridDim              = dim3(static_cast<unsigned>(tiles * split));
        attr[1].id               = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = split;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        cfg.numAttrs             = 2;
        SLIME_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_fp8_ksplit_kernel, tmA, tmB, f));
        return 0;
    }
    static bool configured[64] = {};
    SLIME_CUDA_OK(allow_dynamic_smem(gemm_fp8_pair_kernel, kF8pSmem, configured));
    f.split      = parts;
    f.full_tiles = static_cast<int>(parts > 1 ? pair_tiles - rest : pair_tiles);
    const int widest = f.full_tiles > 0 ? kF8BN : kF8BN / f.split;
    f.stage_bytes    = kF8pABytes + widest / 2 * kF8BK;
    f.stages         = kF8pRingBytes / f.stage_bytes < kF8pMaxStages ? kF8pRingBytes / f.stage_bytes : kF8pMaxStages;
    tmBn             = tmB;
    if (f.split > 1 && make_tmap_2d(&tmBn, Bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, f.N, f.K, ldb, kF8pNarrowBox, kF8BK)) return -1;
    const long units = f.full_tiles + (pair_tiles - f.full_tiles) * f.split;
    cfg.gridDim      = dim3(static_cast<unsigned>(2 * (units < pairs ? units : pairs)));
    SLIME_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_fp8_pair_kernel, tmA, tmB, tmBn, f));
    return 0;
}

int check_f8(const void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int out_align = 16)
{
    if (M <= 0 || N <= 0 || K <= 0) return fail("fp8 gemm: M, N, K must be positive (got %d, %d, %d)", M, N, K);
    if (K % kF8BK != 0) return fail("fp8 gemm: K (%d) must be a multiple of %d (one scale block)", K, kF8BK);
    if (lda % 16 != 0 || ldb % 16 != 0) return fail("fp8 gemm: lda and ldb must be multiples of 16 bytes");
    if (N % 32 != 0 || ldc % 8 != 0) return fail("fp8 gemm: N must be a multiple of 32 and ldc of 8");
    if (reinterpret_cast<unsigned long long>(C) % out_align != 0) return fail("fp8 gemm: the output must be %d-byte aligned (%p)", out_align, C);
    return 0;
}

}  // namespace

extern "C" {

// C[M, N] (bf16) = dequant(Aq, sa) * dequant(Bq, sb)^T with 1x128 scales for A and 128x128 scales for B.
int slime_gemm_fp8_blockscaled(const void* Aq, const float* sa, const void* Bq, const float* sb, void* C, int M, int N, int K,
                               long long lda, long long ldb, long long ldc, void* status, void* stream)
{
    if (check_f8(C, M, N, K, lda, ldb, ldc, 8)) return -1;  // 16 where the form stores 16 bytes at a time, see launch_plain_f8
    F8Args f{};
    f.M = M;
    f.N = N;
    f.K = K;
    f.C = static_cast<__nv_bfloat16*>(C);
    f.ldc = ldc;
    f.sa = sa;
    f.sb = sb;
    f.ag.status = static_cast<KernelStatus*>(status);
    return launch_plain_f8(Aq, Bq, f, lda, ldb, static_cast<cudaStream_t>(stream));
}

// All-gather -> GEMM in fp8. xq_local / sx_local: this rank's quantised shard [rows_local, K] and its scales
// [rows_local, K/128]; aq_full / sa_full: this rank's gathered matrices inside its symmetric region; dst8 / sdst8 /
// flags8: the addresses of those two matrices and of the arrival counters on every rank.
// mode 0: push only; 1: GEMM only, gated on the counters; 2: one fused kernel.
int slime_ag_gemm_fp8(int mode, const void* xq_local, const float* sx_local, const void* aq_full, const float* sa_full,
                      const void* Bq, const float* sb, void* C, int rows_local, int N, int K, long long ldb, long long ldc, int rank,
                      int world, const unsigned long long* dst8, const unsigned long long* sdst8, const unsigned long long* flags8,
                      unsigned long long step, int push_blocks, void* status, void* stream)
{
    if (world < 1 || world > 8 || rank < 0 || rank >= world) return fail("ag_gemm_fp8: bad rank/world");
    if (rows_local <= 0 || rows_local % kBM != 0) return fail("ag_gemm_fp8: rows per rank (%d) must be a multiple of %d", rows_local, kBM);
    if (K % kF8BK != 0) return fail("ag_gemm_fp8: K must be a multiple of %d", kF8BK);
    F8Args f{};
    f.M = rows_local * world;
    f.N = N;
    f.K = K;
    f.C = static_cast<__nv_bfloat16*>(C);
    f.ldc = ldc;
    f.sa = sa_full;
    f.sa_local = sx_local;
    f.sb = sb;
    f.ag.status   = static_cast<KernelStatus*>(status);
    f.ag.ag_rows  = rows_local;
    f.ag.ag_rank  = rank;
    f.ag.ag_world = world;
    for (int i = 0; i < 8; ++i) {
        f.ag.ag_dst[i]     = i < world ? dst8[i] : 0;
        f.ag.ag_flags[i]   = i < world ? flags8[i] : 0;
        f.ag_dst_scales[i] = i < world ? sdst8[i] : 0;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (mode == 0 || mode == 2) {
        if ((reinterpret_cast<unsigned long long>(xq_local) & 15) != 0 || (reinterpret_cast<unsigned long long>(sx_local) & 15) != 0)
            return fail("ag_gemm_fp8: local shard and scales must be 16-byte aligned");
        f.ag.ag_src      = static_cast<const uint4*>(xq_local);
        f.ag_src_scales  = reinterpret_cast<const uint8_t*>(sx_local);
    }
    if (mode == 0) {
        ag_push_only_f8_kernel<<<push_blocks > 0 ? push_blocks : 64, 32, 0, s>>>(f);
        SLIME_CUDA_OK(cudaGetLastError());
        return 0;
    }
    if (check_f8(C, f.M, N, K, K, ldb, ldc)) return -1;
    f.ag.a_ready        = reinterpret_cast<const unsigned long long*>(flags8[rank]);
    f.ag.a_ready_rows   = kBM;
    f.ag.a_ready_target = step * (kBM / kAgSliceRows);
    f.ag.ag_shard_order = 1;
    if (mode == 1) return launch_f8<false>(aq_full, Bq, nullptr, f, K, ldb, s);
    if (mode == 2) {
        f.ag.ag_local_direct = 1;
        return launch_f8<true>(aq_full, Bq, xq_local, f, K, ldb, s);
    }
    return fail("ag_gemm_fp8: unknown mode %d", mode);
}

}  // extern "C"
