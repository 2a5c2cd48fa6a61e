// Paged KV-cache movement: prefill -> decode page transfer fused with the paged
// scatter, and the local pack / unpack between contiguous and paged layouts.
//
// A KV plane (K or V of one layer) is addressed in two ways:
//   token-major   [tokens][row_bytes]                      (row = all local heads of one token)
//   paged         [blocks][page_tokens][row_bytes]         (block table decides where a page lives)
// A task moves up to page_tokens consecutive rows between "token offset tok_off[p]" on one
// side and "block blk[p]" on the other; the token-major side may itself be a paged cache,
// in which case tok_off = src_block * page_tokens. With to_paged the token-major side is the
// source (pack, or prefill -> decode transfer when the paged side is a peer's cache);
// otherwise the paged side is the source (unpack).
//
// One launch moves K and V of one layer for the whole batch, through registers (warps walk 4 KB slices of the (task, plane)
// pages) or, for pages of 16 KB and more, through the bulk-copy engine (kv_bulk_kernel).
// The last CTA to finish publishes `done_value` at `done_flag` (release, system scope), typically a per-layer
// word in the decode rank's memory, so the consumer can start attention on layer l while
// layer l+1 is still in flight.
//
// Register form. Its CTAs take no shared memory, so they fit beside a GEMM's, and a transfer that runs beside the prefill
// GEMMs gets few of them (32 by default): its rate is the bytes that those keep in flight over the memory latency. Every warp has a slice being stored, the next one on
// its way and the page header of the one after that, whatever the page size. (With one page per CTA at a time, its
// header fetched when the CTA came to it, nothing was in flight between two pages: 30 MB per layer, 32 CTAs, 64-token pages of 512-byte
// rows took 55 us a layer where this takes 42 us, and 4 KB pages left most of a CTA idle. With 148 CTAs it is 20 us,
// 2.9 TB/s read and written.)
#include "common/host_utils.h"
#include "common/ptx.cuh"
#include "slime_cuda.h"

#include <atomic>

using namespace slime;

namespace {

struct KvArgs {
    unsigned long long tok_k, tok_v;    // token-major planes (base addresses)
    unsigned long long page_k, page_v;  // paged planes (base addresses; may be peer memory)
    const int*         tok_off;         // [n_tasks] first token row of the task on the token-major side
    const int*         blk;             // [n_tasks] block index on the paged side
    const int*         ntok;            // [n_tasks] rows to move (<= page_tokens), or nullptr for full pages
    int                n_tasks;
    int                page_tokens;
    unsigned long long row_bytes;
    unsigned long long tok_rows;     // rows available on the token-major side (range check)
    unsigned long long page_blocks;  // blocks available on the paged side (range check)
    int                to_paged;
    unsigned long long* done_flag;
    unsigned long long  done_value;
    unsigned int*       block_counter;
    KernelStatus*       status;
};

constexpr int kSliceVecs = 8;                      // 16-byte vectors per lane and slice
constexpr int kSliceSpan = 32 * kSliceVecs;        // vectors of a slice: 4 KB

// One slice of one page: where it lies and how many of this lane's vectors exist.
struct KvSlice {
    const uint4* src;
    uint4*       dst;
    int          left;  // vectors from this lane's first one to the end of the page; lane's j-th exists if 32 * j < left
};

struct KvHeader {
    int toff, blk, n;
};

__device__ __forceinline__ KvHeader kv_header(const KvArgs& a, int p)
{
    return {a.tok_off[p], a.blk[p], a.ntok ? a.ntok[p] : a.page_tokens};
}

// Resolves item -> slice. An item of a short page that lies past the page's end, or whose task is out of range (reported
// once), moves nothing.
__device__ __forceinline__ KvSlice kv_slice(const KvArgs& a, KvHeader h, long long item, int slices, int lane)
{
    const long long u     = item / slices;
    const int       slice = static_cast<int>(item - u * slices);
    const int       p     = static_cast<int>(u >> 1);
    const int       plane = static_cast<int>(u & 1);
    KvSlice         s{nullptr, nullptr, 0};
    if (h.n > a.page_tokens) h.n = a.page_tokens;
    if (h.n <= 0) return s;
    if (h.toff < 0 || static_cast<unsigned long long>(h.toff) + h.n > a.tok_rows || h.blk < 0
        || static_cast<unsigned long long>(h.blk) >= a.page_blocks) {
        if (lane == 0 && slice == 0) report_status(a.status, K_BAD_INDEX, 80, p, a.page_blocks, static_cast<unsigned long long>(h.blk));
        return s;
    }
    const unsigned long long tok_addr  = (plane ? a.tok_v : a.tok_k) + static_cast<unsigned long long>(h.toff) * a.row_bytes;
    const unsigned long long page_addr = (plane ? a.page_v : a.page_k) + static_cast<unsigned long long>(h.blk) * a.page_tokens * a.row_bytes;
    const long long          first     = static_cast<long long>(slice) * kSliceSpan + lane;
    const long long          left      = static_cast<long long>(static_cast<unsigned long long>(h.n) * a.row_bytes / 16) - first;
    s.src  = reinterpret_cast<const uint4*>(a.to_paged ? tok_addr : page_addr) + first;
    s.dst  = reinterpret_cast<uint4*>(a.to_paged ? page_addr : tok_addr) + first;
    s.left = left <= 0 ? 0 : left > kSliceSpan ? kSliceSpan : static_cast<int>(left);
    return s;
}

__device__ __forceinline__ void kv_load(const KvSlice& s, uint4 (&v)[kSliceVecs])
{
#pragma unroll
    for (int j = 0; j < kSliceVecs; ++j)
        if (32 * j < s.left) v[j] = s.src[32 * j];
}

__device__ __forceinline__ void kv_store(const KvSlice& s, const uint4 (&v)[kSliceVecs])
{
#pragma unroll
    for (int j = 0; j < kSliceVecs; ++j)
        if (32 * j < s.left) s.dst[32 * j] = v[j];
}

__global__ void __launch_bounds__(256) kv_transfer_kernel(KvArgs a)
{
    const int       lane   = threadIdx.x & 31;
    const int       warps  = blockDim.x >> 5;
    const int       slices = static_cast<int>((a.page_tokens * a.row_bytes / 16 + kSliceSpan - 1) / kSliceSpan);
    const long long items  = 2ll * a.n_tasks * slices;
    const long long step   = static_cast<long long>(gridDim.x) * warps;
    long long       item   = static_cast<long long>(blockIdx.x) * warps + (threadIdx.x >> 5);
    // Two slices per warp are in flight at any time, and the page header of the one after them.
    auto header = [&](long long i) { return i < items ? kv_header(a, static_cast<int>(i / slices >> 1)) : KvHeader{0, 0, 0}; };
    auto resolve = [&](const KvHeader& h, long long i) { return i < items ? kv_slice(a, h, i, slices, lane) : KvSlice{nullptr, nullptr, 0}; };
    uint4    v0[kSliceVecs], v1[kSliceVecs];
    KvHeader h0 = header(item), h1 = header(item + step);
    KvSlice  s0 = resolve(h0, item), s1;
    kv_load(s0, v0);
    while (item < items) {
        h0 = header(item + 2 * step);
        s1 = resolve(h1, item + step);
        kv_load(s1, v1);
        kv_store(s0, v0);
        h1 = header(item + 3 * step);
        s0 = resolve(h0, item + 2 * step);
        kv_load(s0, v0);
        kv_store(s1, v1);
        item += 2 * step;
    }
    if (a.done_flag != nullptr) {
        __shared__ bool is_last;
        __syncthreads();
        if (threadIdx.x == 0) {
            fence_acq_rel_sys();
            is_last = atomicAdd(a.block_counter, 1u) == gridDim.x - 1;
            if (is_last) {
                fence_acq_rel_sys();
                st_release_sys(a.done_flag, a.done_value);
                *a.block_counter = 0;
            }
        }
    }
}

// The same move through the bulk-copy engine, one warp per CTA: global -> shared bulk loads run ahead of the shared -> global
// bulk stores by a ring of 192 KB, so that a CTA keeps more than the bytes of the register form in flight, without a break
// between pages. The page headers of 32 chunks are resolved at a time, one per lane, and those of the
// next 32 are on their way meanwhile. Layers replayed back to back from a graph, register form -> this: five prompts, 32 KB pages
// (30 MB) on 32 CTAs 43.6 -> 29.8 us, 31 GB/s in and 31 out per SM, on 148 CTAs 21.0 -> 19.2 us; 16 prompts, 64 KB pages (167 MB)
// on 32 CTAs 199 -> 119 us, on 148 72.5 -> 63.4 us, 5.3 TB/s read and written. Which of an SM's two directions stops a CTA is not
// known. Smaller chunks cost more issue than they carry: 8 KB pages take 44.1 us through registers, 45.6 here (32 CTAs).
constexpr int kKvRingBytes = 192 * 1024;
constexpr int kKvChunk     = 16 * 1024;
constexpr int kKvSlots     = kKvRingBytes / kKvChunk;
constexpr int kKvLag       = 2;          // stores that may still be reading their slots when the next load is issued

__global__ void __launch_bounds__(32) kv_bulk_kernel(const __grid_constant__ KvArgs a)
{
    constexpr int chunk = kKvChunk, slots = kKvSlots;
    extern __shared__ __align__(128) unsigned char kv_ring[];
    __shared__ uint64_t           full[kKvSlots];
    __shared__ unsigned long long s_dst[kKvSlots];
    __shared__ uint32_t           s_bytes[kKvSlots];
    const int lane = threadIdx.x;
    if (lane == 0) {
        for (int i = 0; i < slots; ++i) mbar_init(&full[i], 1);
        fence_mbar_init();
    }
    __syncwarp();
    const unsigned long long page_bytes = static_cast<unsigned long long>(a.page_tokens) * a.row_bytes;
    const long long          per_page   = static_cast<long long>((page_bytes + chunk - 1) / chunk);
    const long long          items      = 2ll * a.n_tasks * per_page;
    auto header = [&](long long i) {
        return i < items ? KvHeader{a.tok_off[i / per_page >> 1], a.blk[i / per_page >> 1], a.ntok ? a.ntok[i / per_page >> 1] : a.page_tokens}
                         : KvHeader{0, 0, 0};
    };
    int  n_ld = 0, n_st = 0;
    bool ok   = true;
    auto store_next = [&]() {  // by lane 0
        const int s = n_st % slots;
        if (!mbar_wait(&full[s], static_cast<uint32_t>((n_st / slots) & 1), a.status, 81, s)) {
            ok = false;  // the load never landed: stop issuing, leave through the common exit
            return;
        }
        bulk_store_s2g(reinterpret_cast<void*>(s_dst[s]), kv_ring + s * chunk, s_bytes[s]);
        tma_store_commit();
        ++n_st;
    };
    long long base = blockIdx.x;  // this CTA's items: base + j * gridDim.x
    KvHeader  next = header(base + static_cast<long long>(lane) * gridDim.x);
    for (; base < items; base += 32ll * gridDim.x) {
        const long long i = base + static_cast<long long>(lane) * gridDim.x;
        KvHeader        h = next;
        next              = header(i + 32ll * gridDim.x);
        unsigned long long src = 0, dst = 0;
        uint32_t           bytes = 0;
        if (i < items) {
            const int p     = static_cast<int>(i / per_page >> 1);
            const int plane = static_cast<int>(i / per_page & 1);
            const unsigned long long off = static_cast<unsigned long long>(i % per_page) * chunk;
            if (h.n > a.page_tokens) h.n = a.page_tokens;
            if (h.n > 0) {
                if (h.toff < 0 || static_cast<unsigned long long>(h.toff) + h.n > a.tok_rows || h.blk < 0
                    || static_cast<unsigned long long>(h.blk) >= a.page_blocks) {
                    if (off == 0) report_status(a.status, K_BAD_INDEX, 80, p, a.page_blocks, static_cast<unsigned long long>(h.blk));
                }
                else {
                    const unsigned long long total = static_cast<unsigned long long>(h.n) * a.row_bytes;
                    const unsigned long long tok   = (plane ? a.tok_v : a.tok_k) + static_cast<unsigned long long>(h.toff) * a.row_bytes + off;
                    const unsigned long long page  = (plane ? a.page_v : a.page_k) + static_cast<unsigned long long>(h.blk) * page_bytes + off;
                    src   = a.to_paged ? tok : page;
                    dst   = a.to_paged ? page : tok;
                    bytes = total > off ? static_cast<uint32_t>(min(total - off, static_cast<unsigned long long>(chunk))) : 0u;
                }
            }
        }
        for (unsigned int todo = __ballot_sync(0xffffffffu, bytes != 0); todo != 0; todo &= todo - 1) {
            const int                from = __ffs(todo) - 1;
            const unsigned long long gs   = __shfl_sync(0xffffffffu, src, from);
            const unsigned long long gd   = __shfl_sync(0xffffffffu, dst, from);
            const uint32_t           n    = __shfl_sync(0xffffffffu, bytes, from);
            if (lane == 0 && ok) {
                if (n_ld - n_st > slots - 2 - kKvLag) store_next();
                const int s = n_ld % slots;
                // the slot was read by store number n_ld - slots, which is more than kKvLag stores back
                if (n_ld >= slots) tma_store_wait_read<kKvLag>();
                if (ok) {
                    s_dst[s]   = gd;
                    s_bytes[s] = n;
                    mbar_arrive_expect_tx(&full[s], n);
                    bulk_load_g2s(kv_ring + s * chunk, reinterpret_cast<const void*>(gs), n, &full[s]);
                    ++n_ld;
                }
            }
        }
    }
    if (lane == 0) {
        while (ok && n_st < n_ld) store_next();
        if (!ok) settle_copies();
        tma_store_wait<0>();  // every byte has been written before the CTA reports in
        fence_proxy_async();
        if (a.done_flag != nullptr) {
            fence_acq_rel_sys();
            // a CTA whose wait ran out leaves a mark before it counts itself in: then the bytes are not announced
            constexpr unsigned int kMark = 1u << 31;
            if (!ok) atomicOr(a.block_counter, kMark);
            const unsigned int old = atomicAdd(a.block_counter, 1u);
            if ((old & (kMark - 1)) == gridDim.x - 1) {
                fence_acq_rel_sys();
                if ((old & kMark) == 0) st_release_sys(a.done_flag, a.done_value);
                *a.block_counter = 0;
            }
        }
    }
}

std::atomic<int> g_kv_threads{256};

int check_threads(int threads)
{
    if (threads < 32 || threads > 256 || threads % 32 != 0) return fail("kv transfer: %d threads per CTA not in [32, 256] or not a multiple of 32", threads);
    return 0;
}

}  // namespace

extern "C" {

// Threads per CTA of the register form (32 .. 256, a multiple of 32; default 256) where a call names none, for the whole
// process. A transfer that runs beside a GEMM is best spread thin: one small CTA on every SM slows every GEMM CTA a
// little, a few large CTAs slow a few GEMM CTAs a lot, and the GEMM ends with its slowest CTA.
int slime_kv_tune(int threads)
{
    if (check_threads(threads)) return -1;
    g_kv_threads = threads;
    return 0;
}

int slime_kv_transfer(unsigned long long tok_k, unsigned long long tok_v, unsigned long long page_k,
                      unsigned long long page_v, const int* tok_off, const int* blk, const int* ntok, int n_tasks,
                      int page_tokens, unsigned long long row_bytes, unsigned long long tok_rows,
                      unsigned long long page_blocks, int to_paged, void* done_flag, unsigned long long done_value,
                      unsigned int* block_counter, int max_blocks, void* status, void* stream)
{
    return slime_kv_transfer_form(tok_k, tok_v, page_k, page_v, tok_off, blk, ntok, n_tasks, page_tokens, row_bytes, tok_rows, page_blocks,
                                  to_paged, done_flag, done_value, block_counter, max_blocks, SLIME_KV_AUTO, 0, status, stream);
}

// The same with the form and (register form) the threads per CTA of this call; threads 0: what slime_kv_tune set.
// SLIME_KV_AUTO takes bulk copies for pages of 16 KB and more, unless this call or the process asks for other CTAs than the
// register form's 256 threads. Bulk copies hold 192 KB of shared memory per CTA, so they never share an SM with a GEMM's CTA: a
// caller whose transfer runs under compute for long names SLIME_KV_REGISTERS.
int slime_kv_transfer_form(unsigned long long tok_k, unsigned long long tok_v, unsigned long long page_k,
                           unsigned long long page_v, const int* tok_off, const int* blk, const int* ntok, int n_tasks,
                           int page_tokens, unsigned long long row_bytes, unsigned long long tok_rows,
                           unsigned long long page_blocks, int to_paged, void* done_flag, unsigned long long done_value,
                           unsigned int* block_counter, int max_blocks, int form, int threads, void* status, void* stream)
{
    if (form < SLIME_KV_AUTO || form > SLIME_KV_BULK) return fail("kv transfer: unknown form %d", form);
    if (threads == 0) threads = g_kv_threads;
    else if (check_threads(threads)) return -1;
    if (n_tasks < 0 || page_tokens <= 0) return fail("kv transfer: bad task count or page size");
    if (row_bytes == 0 || row_bytes % 16 != 0) return fail("kv transfer: row_bytes (%llu) must be a positive multiple of 16", row_bytes);
    if (((tok_k | tok_v | page_k | page_v) & 15) != 0) return fail("kv transfer: plane addresses must be 16-byte aligned");
    if (done_flag != nullptr && block_counter == nullptr) return fail("kv transfer: a completion flag needs a block counter");
    KvArgs a{};
    a.tok_k = tok_k, a.tok_v = tok_v, a.page_k = page_k, a.page_v = page_v;
    a.tok_off = tok_off, a.blk = blk, a.ntok = ntok;
    a.n_tasks = n_tasks, a.page_tokens = page_tokens, a.row_bytes = row_bytes;
    a.tok_rows = tok_rows, a.page_blocks = page_blocks, a.to_paged = to_paged;
    a.done_flag     = static_cast<unsigned long long*>(done_flag);
    a.done_value    = done_value;
    a.block_counter = block_counter;
    a.status        = static_cast<KernelStatus*>(status);
    if (form == SLIME_KV_BULK || (form == SLIME_KV_AUTO && threads == 256 && static_cast<unsigned long long>(page_tokens) * row_bytes >= kKvChunk)) {
        const unsigned long long page  = static_cast<unsigned long long>(page_tokens) * row_bytes;
        const long long          items = 2ll * n_tasks * static_cast<long long>((page + kKvChunk - 1) / kKvChunk);
        long long                ctas  = max_blocks > 0 ? max_blocks : sm_count();
        if (ctas > items) ctas = items;
        if (ctas < 1) ctas = 1;
        static bool configured[64] = {};
        SLIME_CUDA_OK(allow_dynamic_smem(kv_bulk_kernel, kKvRingBytes, configured));
        kv_bulk_kernel<<<static_cast<int>(ctas), 32, kKvRingBytes, static_cast<cudaStream_t>(stream)>>>(a);
        SLIME_CUDA_OK(cudaGetLastError());
        return 0;
    }
    const unsigned long long slices = (static_cast<unsigned long long>(page_tokens) * row_bytes / 16 + kSliceSpan - 1) / kSliceSpan;
    if (slices > 0x7fffffffull) return fail("kv transfer: a page of %d rows of %llu bytes is too large", page_tokens, row_bytes);
    const long long warps = threads / 32;
    long long       grid  = (2ll * n_tasks * static_cast<long long>(slices) + warps - 1) / warps;
    const long long cap = max_blocks > 0 ? max_blocks : sm_count() * 4;
    if (grid > cap) grid = cap;
    if (grid < 1) grid = 1;
    static bool carveout[64] = {false};  // runs beside the prefill GEMMs: see prefer_max_shared_carveout
    SLIME_CUDA_OK(prefer_max_shared_carveout(kv_transfer_kernel, carveout));
    kv_transfer_kernel<<<static_cast<int>(grid), threads, 0, static_cast<cudaStream_t>(stream)>>>(a);
    SLIME_CUDA_OK(cudaGetLastError());
    return 0;
}

}  // extern "C"
