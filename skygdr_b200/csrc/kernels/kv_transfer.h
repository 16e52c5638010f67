// Host-visible parameters of the paged KV transfer kernel.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "credit_page.h"

namespace sky {

struct LaunchStatus;
struct SkyGrantCache;

constexpr int KV_MAX_DST = 8;

struct KvTransferParams {
    const __nv_bfloat16* src_pool;        // token-major pages on the source GPU
    void* dst[KV_MAX_DST];                // head-major pools (local or peer-mapped)
    void* mc_dst;                         // fan-out through NVSwitch: multicast address of the destinations' pools (bf16,
                                          // replicate only); stores go out once and land in every team member's copy
    void* dst_scales[KV_MAX_DST];         // fp8 mode: one byte per 32 elements, same indexing / 32
    unsigned int* done_flag[KV_MAX_DST];  // optional: set to done_value (release, system scope) when all pages landed
    const int* src_blocks;                // [n_pairs] block ids in the source pool
    const int* dst_blocks;                // [n_pairs] block ids in the destination pool(s)
    int n_pairs, layers, heads, block_tokens, head_dim;
    int src_num_blocks, dst_num_blocks;   // pool sizes for the index check (0 = unchecked): a block id outside its pool
                                          // is skipped and reported as SKY_STATUS_BAD_INDEX with the pair's position
    long long src_block_stride, src_layer_stride, src_kv_stride;  // in source elements
    long long dst_block_stride, dst_layer_stride, dst_kv_stride;  // in destination elements
    int n_dst, heads_per_dst, replicate, fp8;
    int keep_layout;                      // 1: destination pages keep the source's token-major order (offload to host)
    int pages_per_chunk;                  // granularity of credit, cursor and accounting
    int subs;                             // scheduling units per chunk (set by the launchers)
    unsigned int done_value;
    const SkyCreditPage* page;            // grant half is read here; nullptr = ungated
    SkyCreditPage* usage;                 // usage half is written here at the end; may be nullptr
    unsigned long long consumed_base;     // flow's cumulative bytes before this launch
    unsigned long long max_wait_ns;       // credit wait per chunk before the kernel yields
    unsigned long long first_chunk;       // resume cursor
    // Working block (FlowWork) in its "unset" state before the launch; the last CTA hands the outcome to `result` and to its host copy
    // `mirror` (mapped memory, readable once the launch has ended) and resets the block, so a flow needs no reset between launches.
    LaunchStatus* status;
    SkyGrantCache* grant;
    LaunchStatus* result;
    LaunchStatus* mirror;
};

// Units per chunk: about 32 per CTA, so that a short transfer reaches every CTA and a long one ends evenly (a unit of 8 pages is 12 us
// of a CTA's time at full rate).
inline int kv_pick_subs(const KvTransferParams& p, int ctas) {
    const long long n_chunks = (2LL * p.layers * p.n_pairs + p.pages_per_chunk - 1) / p.pages_per_chunk;
    const long long want = (32LL * ctas + n_chunks - 1) / (n_chunks > 0 ? n_chunks : 1);
    const int subs = (int)(want < 1 ? 1 : want > p.pages_per_chunk ? p.pages_per_chunk : want);
    const int per = (p.pages_per_chunk + subs - 1) / subs;
    return (p.pages_per_chunk + per - 1) / per;         // no empty units
}

cudaError_t launch_kv_transfer(const KvTransferParams& p, int ctas, cudaStream_t stream);
// The engines that move pages with the SM's copy hardware (kv_transfer_tma.cu): bf16 pages, bf16 pages in the source's order, and fp8
// packing. pool_elems: elements of the whole source pool allocation. kv_transfer_tma_takes says whether the layout is one of theirs.
bool kv_transfer_tma_takes(const KvTransferParams& p, long long pool_elems);
cudaError_t launch_kv_transfer_tma(const KvTransferParams& p, long long pool_elems, int ctas, cudaStream_t stream);

}  // namespace sky
