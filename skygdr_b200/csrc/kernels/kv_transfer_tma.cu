// Paged KV transfer by the SM's copy hardware: the gather, the token-major -> head-major conversion and the peer write are TMA
// loads and bulk stores. Three forms, one CTA per SM each:
//
//   bf16, head-major   one thread drives it. Load: 3-D tensor map over the source pool viewed as [token][head][dim]; one box
//                      {128 dims, 1 head, 16 tokens} per head lands that head's [16][128] tile at head*4 KB of a
//                      shared-memory slot, so the slot holds the page in destination order. Store: cp.async.bulk shared ->
//                      global of the slot (32 KB, or one piece per destination when heads are scattered or the page is
//                      replicated) straight into the peer's pool: long contiguous writes for NVLink.
//   bf16, source order the same thread, with one untiled bulk load per page (offload to mapped host memory).
//   fp8                the same loads by one warp; eight warps pack the page (16384 elements, an e4m3 byte each and a scale byte per
//                      32) from its input slot into an output slot in destination order; a third role stores the output slot,
//                      2 KB and 64 bytes per head, in one bulk store each per destination.
//
// Loads run ahead of stores in a ring; a slot is reused once the store that read it has finished reading (bulk-group
// accounting). Credit, cursor, accounting and the end of a launch are those of kv_transfer.cuh, shared with the register engine
// (kv_transfer.cu), which remains for multicast destinations and for layouts these forms do not cover.
//
// Bound: HBM when source and destination share a GPU, the link otherwise. On one B200,
// with a credit page that does not limit the flow, whole calls through ops.KvTransferFlow (transfer and result): 64k tokens
// 2.87 ms (6.7 TB/s of reads and writes, 104 % of a plain copy's rate), 4096 tokens 233 us, 17 tokens 35 us; fp8 to four
// destinations, 9001 tokens, 392 us (5.1 TB/s; 2.77 ms by the register engine, whose loads, packing and stores take turns);
// 1500 tokens to pinned host memory 4.25 ms (52 GB/s of the link; 5.06 ms by the register engine).
//
// Same reference counterpart: one contiguous cudaMemcpyPeerAsync per request
// (llm_problem_analysis/kv_nvlink_transfer.cu:109-122, llm_problem_analysis/kv_nvlink_transfer_trace.cu:378-393).
#include <cuda.h>

#include "kv_transfer.cuh"

namespace sky {
namespace {

constexpr int SLOTS = 6;
constexpr int LOOKAHEAD = 3;
constexpr int SLOT_BYTES = 32768;                 // 8 heads x 16 tokens x 128 x bf16
constexpr int TMA_THREADS = 32;

__device__ __forceinline__ void bulk_s2g(void* gdst, const void* smem_src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_u32(smem_src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// One page of the work list: where it is, where it goes. False for a block id outside its pool (reported, nothing is moved).
__device__ __forceinline__ bool locate_page(const KvTransferParams& p, const KvUnits& u, long long pg, long long& src_elem, long long& dst_elem) {
    const int pair = (int)(pg / u.pages_per_pair);
    const int rem = (int)(pg - (long long)pair * u.pages_per_pair);
    const int layer = rem >> 1, kv = rem & 1;
    const int sb = __ldg(p.src_blocks + pair), db = __ldg(p.dst_blocks + pair);
    if ((p.src_num_blocks && (unsigned)sb >= (unsigned)p.src_num_blocks) || (p.dst_num_blocks && (unsigned)db >= (unsigned)p.dst_num_blocks)) {
        set_status(p.status, SKY_STATUS_BAD_INDEX, (unsigned)pair);
        return false;
    }
    src_elem = (long long)sb * p.src_block_stride + (long long)layer * p.src_layer_stride + (long long)kv * p.src_kv_stride;
    dst_elem = (long long)db * p.dst_block_stride + (long long)layer * p.dst_layer_stride + (long long)kv * p.dst_kv_stride;
    return true;
}

// KEEP: pages stay in the source's order.
template <bool KEEP>
__global__ void __launch_bounds__(TMA_THREADS) kv_transfer_tma_kernel(const __grid_constant__ CUtensorMap tmap, const KvTransferParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full[SLOTS];
    __shared__ long long dst_off[SLOTS], slot_unit[SLOTS];      // destination element offset and unit of the page in each slot
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    if (threadIdx.x != 0) return;                  // one thread drives the copy hardware

    const KvUnits units(p);
    const uint32_t page_bytes = (uint32_t)p.heads * p.block_tokens * p.head_dim * 2;
    const unsigned long long page_link_bytes = (unsigned long long)page_bytes * (p.replicate ? p.n_dst : 1);
    const uint32_t piece = p.replicate || KEEP ? page_bytes : (uint32_t)p.heads_per_dst * p.block_tokens * p.head_dim * 2;

    for (int s = 0; s < SLOTS; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
    if (!KEEP) tma_prefetch_desc(&tmap);
    atomicMin(&p.status->t_start_ns, globaltimer_ns());

    KvCredit credit;
    long long granted_unit = -1;                  // unit whose credit this CTA has
    long long issued = 0, stored = 0;             // pages of this CTA whose loads / stores have been issued
    bool good = true;

    // The j-th page of this CTA: credit for its unit (asked for here and not before the loads, so that the first round trip to the
    // page in host memory overlaps the first loads), wait for its loads, write it out.
    auto store_page = [&](long long j) -> bool {
        const int s = (int)(j % SLOTS);
        if (slot_unit[s] != granted_unit) {
            if (!credit.acquire(p, units, slot_unit[s], page_link_bytes)) return false;
            granted_unit = slot_unit[s];
        }
        if (!mbar_wait(&full[s], (uint32_t)(j / SLOTS) & 1)) { set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 21); return false; }
        const unsigned char* slot = smem + s * SLOT_BYTES;
        for (int g = 0; g < p.n_dst; ++g)
            bulk_s2g((__nv_bfloat16*)p.dst[g] + dst_off[s], slot + (p.replicate ? 0 : (size_t)g * piece), piece);
        bulk_commit();
        return true;
    };

    for (long long unit = (long long)p.first_chunk * p.subs + blockIdx.x; good && unit < units.n_units;) {
        const long long next = kv_next_unit(p, units);          // in flight while this unit is moved
        long long page0, page1;
        units.pages_of(p, unit, page0, page1);
        for (long long pg = page0; pg < page1 && good; ++pg) {
            long long src_elem, dst_elem;
            if (!locate_page(p, units, pg, src_elem, dst_elem)) continue;
            // the slot about to be loaded was last read by the store of page (issued - SLOTS)
            bulk_wait_read<SLOTS - LOOKAHEAD - 1>();
            const int s = (int)(issued % SLOTS);
            dst_off[s] = dst_elem;
            slot_unit[s] = unit;
            mbar_expect_tx(&full[s], page_bytes);
            if (KEEP) {
                bulk_g2s(smem + s * SLOT_BYTES, p.src_pool + src_elem, page_bytes, &full[s]);
            } else {
                const int tok_row = (int)(src_elem / ((long long)p.heads * p.head_dim));       // global token row of the page's first token
                for (int h = 0; h < p.heads; ++h)
                    tma_load_3d(smem + s * SLOT_BYTES + h * (p.block_tokens * p.head_dim * 2), &tmap, 0, h, tok_row, &full[s]);
            }
            ++issued;
            if (issued - stored > LOOKAHEAD) { good = store_page(stored); stored += good; }
        }
        unit = next;
    }
    while (good && stored < issued) { good = store_page(stored); stored += good; }
    // loads still in flight must land before this CTA's shared memory goes away (bounded)
    for (long long j = stored; j < issued; ++j) mbar_wait(&full[j % SLOTS], (uint32_t)(j / SLOTS) & 1, 1000000ull);
    bulk_wait_all();                               // every write of this CTA has completed
    asm volatile("fence.proxy.async;" ::: "memory");   // order the bulk writes (async proxy) before the generic-proxy signals of kv_finish
    kv_finish(p, credit);
}

// ---- fp8: load warp, eight packing warps, store warp ----
// A page costs an SM 32 KB in and 16.5 KB out, 1.1 us at the memory's rate; packing it is 64 elements per thread, about 0.4 us of
// issue slots, so one CTA keeps up as long as the three roles overlap.
constexpr int F8_IN = 4, F8_OUT = 4;
constexpr int F8_PACK_THREADS = 256;               // of one packing group
constexpr int F8_GROUPS = 2;                       // page j is packed by group j % 2: one waits and loads while the other converts
constexpr int F8_THREADS = 64 + F8_GROUPS * F8_PACK_THREADS;   // warp 0: loads, warp 1: stores, warps 2-17: packing
constexpr int F8_SCALES = 512;                     // 8 heads x 16 tokens x 4 scale bytes
constexpr int F8_OUT_BYTES = SLOT_BYTES / 2 + F8_SCALES;

__global__ void __launch_bounds__(F8_THREADS) kv_transfer_fp8_kernel(const __grid_constant__ CUtensorMap tmap, const KvTransferParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t in_full[F8_IN], in_empty[F8_IN], out_full[F8_OUT], out_empty[F8_OUT];
    __shared__ long long in_dst[F8_IN], out_dst[F8_OUT];        // destination element offset of the page in a slot; -1: no more pages
    unsigned char* in_sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    unsigned char* out_sm = in_sm + F8_IN * SLOT_BYTES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_vec = p.heads * 256;                            // 8-element vectors of a page
    const uint32_t page_bytes = (uint32_t)n_vec * 16;
    if (threadIdx.x == 0) {
        for (int s = 0; s < F8_IN; ++s) { mbar_init(&in_full[s], 1); mbar_init(&in_empty[s], F8_PACK_THREADS / 32); }
        for (int s = 0; s < F8_OUT; ++s) { mbar_init(&out_full[s], F8_PACK_THREADS / 32); mbar_init(&out_empty[s], 1); }
        fence_barrier_init();
        tma_prefetch_desc(&tmap);
        atomicMin(&p.status->t_start_ns, globaltimer_ns());
    }
    __syncthreads();
    // the packing and store roles outlast any wait of the load role for credit
    const unsigned long long patience = p.max_wait_ns + 1000000000ull;
    KvCredit credit;

    if (warp == 0) {
        if (lane == 0) {
            const KvUnits units(p);
            const unsigned long long page_link_bytes = ((unsigned long long)n_vec * 8ull + (unsigned long long)n_vec / 4ull) * (p.replicate ? p.n_dst : 1);
            long long j = 0;
            auto free_slot = [&]() {                            // the slot of page j, once the packing warps have read page j - F8_IN
                return j < F8_IN || mbar_wait(&in_empty[j % F8_IN], (uint32_t)(j / F8_IN - 1) & 1);
            };
            bool good = true;
            for (long long unit = (long long)p.first_chunk * p.subs + blockIdx.x; good && unit < units.n_units;) {
                const long long next = kv_next_unit(p, units);
                if (!credit.acquire(p, units, unit, page_link_bytes)) break;
                long long page0, page1;
                units.pages_of(p, unit, page0, page1);
                for (long long pg = page0; pg < page1; ++pg) {
                    long long src_elem, dst_elem;
                    if (!locate_page(p, units, pg, src_elem, dst_elem)) continue;
                    if (!free_slot()) { set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 22); good = false; break; }
                    const int s = (int)(j % F8_IN);
                    in_dst[s] = dst_elem;
                    mbar_expect_tx(&in_full[s], page_bytes);
                    const int tok_row = (int)(src_elem / ((long long)p.heads * p.head_dim));
                    for (int h = 0; h < p.heads; ++h) tma_load_3d(in_sm + s * SLOT_BYTES + h * 4096, &tmap, 0, h, tok_row, &in_full[s]);
                    ++j;
                }
                unit = next;
            }
            for (int e = 0; e < F8_GROUPS && good; ++e, ++j) {  // tell every group that there is no more
                if (!free_slot()) break;
                in_dst[j % F8_IN] = -1;
                mbar_arrive(&in_full[j % F8_IN]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            for (long long j = 0;; ++j) {
                const int s = (int)(j % F8_OUT);
                if (!mbar_wait(&out_full[s], (uint32_t)(j / F8_OUT) & 1, patience)) { set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 23); break; }
                const long long dst = out_dst[s];
                if (dst < 0) break;
                const unsigned char* q = out_sm + s * F8_OUT_BYTES;
                const int per = p.replicate ? p.heads : p.heads_per_dst;
                for (int g = 0; g < p.n_dst; ++g) {
                    const int h0 = p.replicate ? 0 : g * per;
                    bulk_s2g((unsigned char*)p.dst[g] + dst, q + h0 * 2048, (uint32_t)per * 2048);
                    bulk_s2g((unsigned char*)p.dst_scales[g] + (dst >> 5), q + SLOT_BYTES / 2 + h0 * 64, (uint32_t)per * 64);
                }
                bulk_commit();
                bulk_wait_read<1>();                            // page j - 1 has left its slot
                if (j > 0) mbar_arrive(&out_empty[(j - 1) % F8_OUT]);
            }
            bulk_wait_all();
        }
    } else {
        const int tid = (threadIdx.x - 64) % F8_PACK_THREADS;
        for (long long j = (threadIdx.x - 64) / F8_PACK_THREADS;; j += F8_GROUPS) {
            const int s = (int)(j % F8_IN), o = (int)(j % F8_OUT);
            bool ok = mbar_wait(&in_full[s], (uint32_t)(j / F8_IN) & 1, patience);
            const long long dst = ok ? in_dst[s] : -1;
            if (dst >= 0 && j >= F8_OUT) ok = mbar_wait(&out_empty[o], (uint32_t)(j / F8_OUT - 1) & 1, patience);
            if (!ok && lane == 0) set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 24);
            const bool last = !__all_sync(0xffffffffu, ok) || dst < 0;
            if (!last) {
                const uint4* src = reinterpret_cast<const uint4*>(in_sm + s * SLOT_BYTES);
                uint2* q = reinterpret_cast<uint2*>(out_sm + o * F8_OUT_BYTES);
                unsigned char* sc = out_sm + o * F8_OUT_BYTES + SLOT_BYTES / 2;
#pragma unroll 4
                for (int v = tid; v < n_vec; v += F8_PACK_THREADS) {       // n_vec is a multiple of the packing threads
                    unsigned char sb8;
                    q[v] = pack_fp8_mx(src[v], true, &sb8);
                    if ((lane & 3) == 0) sc[v >> 2] = sb8;
                }
            }
            if (tid == 0) out_dst[o] = last ? -1 : dst;
            fence_proxy_async();                                // the slot is read by bulk stores
            __syncwarp();
            if (lane == 0) {
                if (!last) mbar_arrive(&in_empty[s]);
                mbar_arrive(&out_full[o]);
            }
            if (last) break;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("fence.proxy.async;" ::: "memory");
        kv_finish(p, credit);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

}  // namespace

// The source pool must be one contiguous token-major allocation: page (block, layer, kv) at
// block*src_block_stride + layer*src_layer_stride + kv*src_kv_stride, each [16 tokens][heads][128].
bool kv_transfer_tma_takes(const KvTransferParams& p, long long pool_elems) {
    if (p.mc_dst || p.head_dim != 128 || p.block_tokens != 16 || p.heads < 1 || p.heads > 8) return false;
    if (p.n_dst < 1 || p.n_dst > KV_MAX_DST || p.pages_per_chunk < 1) return false;
    if (!p.replicate && p.heads_per_dst * p.n_dst != p.heads) return false;
    if (p.keep_layout && (p.fp8 || (p.n_dst > 1 && !p.replicate))) return false;
    const long long row = (long long)p.heads * p.head_dim;                   // elements per token row
    if (p.src_block_stride % row || p.src_layer_stride % row || p.src_kv_stride % row || pool_elems % row) return false;
    // bulk copies want 16-byte aligned addresses: of bf16 elements, of fp8 bytes and of their scale bytes (one per 32)
    const long long unit = p.fp8 ? 512 : 8;
    if (p.dst_block_stride % unit || p.dst_layer_stride % unit || p.dst_kv_stride % unit) return false;
    uintptr_t bits = reinterpret_cast<uintptr_t>(p.src_pool);
    for (int g = 0; g < p.n_dst; ++g) bits |= reinterpret_cast<uintptr_t>(p.dst[g]) | (p.fp8 ? reinterpret_cast<uintptr_t>(p.dst_scales[g]) : 0);
    return (bits & 15) == 0;
}

cudaError_t launch_kv_transfer_tma(const KvTransferParams& p, long long pool_elems, int ctas, cudaStream_t stream) {
    if (ctas < 1 || !kv_transfer_tma_takes(p, pool_elems)) return cudaErrorInvalidValue;
    KvTransferParams q = p;
    q.subs = kv_pick_subs(p, ctas);
    const long long chunks = (2LL * p.layers * p.n_pairs + p.pages_per_chunk - 1) / p.pages_per_chunk - (long long)p.first_chunk;
    ctas = (int)(chunks * q.subs < 1 ? 1 : chunks * q.subs < ctas ? chunks * q.subs : ctas);        // nobody without a unit of its own
    CUtensorMap tm = {};
    if (!p.keep_layout) {
        static const EncodeTiledFn fn = [] {
            void* ptr = nullptr;
            cudaDriverEntryPointQueryResult r;
            if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) ptr = nullptr;
            return reinterpret_cast<EncodeTiledFn>(ptr);
        }();
        if (!fn) return cudaErrorNotSupported;
        const long long row = (long long)p.heads * p.head_dim;
        const cuuint64_t dims[3] = {128, (cuuint64_t)p.heads, (cuuint64_t)(pool_elems / row)};
        const cuuint64_t strides[2] = {256, (cuuint64_t)row * 2};
        const cuuint32_t box[3] = {128, 1, 16};
        const cuuint32_t estr[3] = {1, 1, 1};
        if (fn(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(p.src_pool), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    constexpr int smem_bytes = SLOTS * SLOT_BYTES + 128;
    constexpr int fp8_smem_bytes = F8_IN * SLOT_BYTES + F8_OUT * F8_OUT_BYTES + 128;
    static unsigned long long attr_mask[3] = {0, 0, 0};
    const void* kern = p.fp8 ? (const void*)kv_transfer_fp8_kernel : p.keep_layout ? (const void*)kv_transfer_tma_kernel<true> : (const void*)kv_transfer_tma_kernel<false>;
    const int bytes = p.fp8 ? fp8_smem_bytes : smem_bytes;
    if (cudaError_t e = set_max_dynamic_smem_once(kern, bytes, &attr_mask[p.fp8 ? 2 : p.keep_layout ? 1 : 0]); e != cudaSuccess) return e;
    if (p.fp8) kv_transfer_fp8_kernel<<<ctas, F8_THREADS, fp8_smem_bytes, stream>>>(tm, q);
    else if (p.keep_layout) kv_transfer_tma_kernel<true><<<ctas, TMA_THREADS, smem_bytes, stream>>>(tm, q);
    else kv_transfer_tma_kernel<false><<<ctas, TMA_THREADS, smem_bytes, stream>>>(tm, q);
    return cudaGetLastError();
}

}  // namespace sky
