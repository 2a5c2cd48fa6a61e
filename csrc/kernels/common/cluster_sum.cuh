// The last step of a product that a cluster has split along K: every CTA's fp32 sums of the same 128 x 256 tile lie in its own
// shared memory; each CTA adds one slice of the columns over the cluster, in the order of K, through distributed shared
// memory, rounds and stores it.
#pragma once

#include "gemm_tc.cuh"

namespace slime {
namespace gemm {

constexpr int kSumCols  = 256;
constexpr int kSumPitch = kSumCols + 4;  // floats per row of the sums: 16-byte accesses of eight rows hit all banks

// Called by all threads of all `split` (2, 4 or 8) CTAs of the cluster after they have written their sums [kBM][kSumPitch]. Contains
// the barrier in front of the exchange; the caller keeps every CTA until the others have read. If a wait ran out in any CTA
// of the cluster (its *fail_slot is set), nobody stores: the slices need the sums of all.
__device__ __forceinline__ void cluster_add_store(float* sums, volatile uint32_t* fail_slot, int crank, int split, int row0, int col0, int M,
                                                  int N, __nv_bfloat16* C, long long ldc)
{
    __syncwarp();  // rows past the end of A have split the last warp: an aligned barrier is for whole warps
    cluster_sync_all();
    const int      lane   = threadIdx.x & 31;
    const uint32_t failed = lane < split ? ld_cluster_u32(mapa_u32(const_cast<const uint32_t*>(fail_slot), static_cast<uint32_t>(lane))) : 0u;
    if (__any_sync(0xffffffffu, failed != 0)) return;
    // four columns at a time: N is a multiple of 32, so they exist together or not at all
    const int quads = kSumCols / split / 4;
    const int rows  = min(kBM, M - row0);
    for (int i = threadIdx.x; i < rows * quads; i += blockDim.x) {
        const int r = i / quads;
        const int c = (crank * quads + i % quads) * 4;
        if (col0 + c >= N) continue;
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j < split) v[j] = ld_cluster_f32x4(mapa_u32(sums + r * kSumPitch + c, static_cast<uint32_t>(j)));
        float4 a = v[0];
#pragma unroll
        for (int j = 1; j < 8; ++j)
            if (j < split) a = make_float4(a.x + v[j].x, a.y + v[j].y, a.z + v[j].z, a.w + v[j].w);
        *reinterpret_cast<uint2*>(C + static_cast<long long>(row0 + r) * ldc + col0 + c) = make_uint2(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
    }
}

}  // namespace gemm
}  // namespace slime
