// Paged KV transfer: gather pages named by a block table out of the prefill
// GPU's cache, convert the layout token-major -> head-major (optionally pack to
// block-scaled fp8), and store them straight into one or several decode GPUs'
// paged caches through peer mappings. Every chunk passes a credit gate, so
// pacing and cooperative yield happen inside the kernel.
//
// The reference moves KV with one contiguous cudaMemcpyPeerAsync per request on
// a destination-side stream (llm_problem_analysis/kv_nvlink_transfer.cu:109-122,
// llm_problem_analysis/kv_nvlink_transfer_trace.cu:378-393) and paces a flow by
// sleeping on the host between posts (src/cpu_client.cc:875-879). This kernel
// replaces both.
//
// Source page  (block b, layer l, K|V): [T tokens][H heads][D] bf16
// Destination page                    : [Hd heads][T tokens][D]  bf16, or e4m3 + one
//                                       power-of-two scale byte per 32 elements
// With n_dst > 1 the heads are either scattered (destination g receives heads
// [g*Hd, (g+1)*Hd): tensor-parallel decode ranks) or replicated (every
// destination receives all heads: fan-out). A fan-out can also go through an
// NVLink multicast address (`mc_dst`): one `multimem.st` per 16 bytes leaves
// this GPU and NVSwitch writes it into every destination, so the source's
// link carries the payload once instead of once per destination.
#include "kv_transfer.cuh"

namespace sky {

template <int UNROLL>
__global__ void __launch_bounds__(256) kv_transfer_kernel(const KvTransferParams p) {
    __shared__ long long s_unit;
    const int tid = threadIdx.x;
    const int vec_per_row = p.head_dim / 8;
    const int n_vec = p.block_tokens * p.heads * vec_per_row;
    const KvUnits units(p);
    const long long pages_per_pair = units.pages_per_pair;
    const unsigned long long page_link_bytes =
        (p.fp8 ? (unsigned long long)n_vec * 8ull + (unsigned long long)n_vec / 4ull : (unsigned long long)n_vec * 16ull) *
        (p.replicate && !p.mc_dst ? p.n_dst : 1);     // a multicast store leaves this GPU once

    KvCredit credit;
    long long unit = (long long)p.first_chunk * p.subs + blockIdx.x, ticket = 0;
    if (tid == 0) atomicMin(&p.status->t_start_ns, globaltimer_ns());

    for (;;) {
        if (tid == 0) {
            const bool go = unit < units.n_units && credit.acquire(p, units, unit, page_link_bytes);
            if (go) ticket = kv_next_unit(p, units);      // in flight while this unit is moved
            s_unit = go ? unit : -1;
        }
        __syncthreads();
        unit = s_unit;
        __syncthreads();
        if (unit < 0) break;

        long long page0, page1;
        units.pages_of(p, unit, page0, page1);
        for (long long pg = page0; pg < page1; ++pg) {
            const int pair = (int)(pg / pages_per_pair);
            const int rem = (int)(pg - (long long)pair * pages_per_pair);
            const int layer = rem >> 1, kv = rem & 1;
            const int sb = __ldg(p.src_blocks + pair), db = __ldg(p.dst_blocks + pair);
            if ((p.src_num_blocks && (unsigned)sb >= (unsigned)p.src_num_blocks) || (p.dst_num_blocks && (unsigned)db >= (unsigned)p.dst_num_blocks)) {
                if (tid == 0) set_status(p.status, SKY_STATUS_BAD_INDEX, (unsigned)pair);    // same decision in every thread
                continue;
            }
            const __nv_bfloat16* src = p.src_pool + (long long)sb * p.src_block_stride + (long long)layer * p.src_layer_stride +
                                       (long long)kv * p.src_kv_stride;
            const long long dst_off = (long long)db * p.dst_block_stride + (long long)layer * p.dst_layer_stride +
                                      (long long)kv * p.dst_kv_stride;
            for (int base = 0; base < n_vec; base += 256 * UNROLL) {
                uint4 v[UNROLL];
                int idx[UNROLL];
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    idx[u] = base + u * 256 + tid;
                    v[u] = idx[u] < n_vec ? ld_nc_v4(src + (long long)idx[u] * 8) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    const bool valid = idx[u] < n_vec;
                    const int row = idx[u] / vec_per_row, c = idx[u] - row * vec_per_row;
                    const int t = row / p.heads, h = row - t * p.heads;
                    const int g0 = p.replicate ? 0 : h / p.heads_per_dst;
                    const int hl = p.replicate ? h : h - g0 * p.heads_per_dst;
                    const long long e = p.keep_layout ? dst_off + (long long)idx[u] * 8
                                                      : dst_off + ((long long)hl * p.block_tokens + t) * p.head_dim + c * 8;
                    if (!p.fp8) {
                        if (valid) {
                            if (p.mc_dst) {
                                multimem_st_v4((__nv_bfloat16*)p.mc_dst + e, v[u]);
                            } else if (p.replicate) {
                                for (int g = 0; g < p.n_dst; ++g) st_v4((__nv_bfloat16*)p.dst[g] + e, v[u]);
                            } else {
                                st_v4((__nv_bfloat16*)p.dst[g0] + e, v[u]);
                            }
                        }
                    } else {
                        unsigned char sb8;
                        uint2 packed = pack_fp8_mx(v[u], valid, &sb8);
                        if (valid) {
                            const int ng = p.replicate ? p.n_dst : 1;
                            for (int gi = 0; gi < ng; ++gi) {
                                const int g = p.replicate ? gi : g0;
                                *reinterpret_cast<uint2*>((unsigned char*)p.dst[g] + e) = packed;
                                if ((c & 3) == 0) ((unsigned char*)p.dst_scales[g])[e >> 5] = sb8;
                            }
                        }
                    }
                }
            }
        }
        unit = ticket;                                     // thread 0's is the one that counts
    }

    __syncthreads();                                       // this CTA's payload stores are ordered before the counters
    if (tid == 0) kv_finish(p, credit);
}

cudaError_t launch_kv_transfer(const KvTransferParams& p, int ctas, cudaStream_t stream) {
    if (p.head_dim % 8 != 0 || p.n_dst < 1 || p.n_dst > KV_MAX_DST || p.pages_per_chunk < 1) return cudaErrorInvalidValue;
    if (!p.replicate && p.heads_per_dst * p.n_dst != p.heads) return cudaErrorInvalidValue;
    if (p.fp8 && (p.head_dim % 32 != 0)) return cudaErrorInvalidValue;
    if (p.mc_dst && (p.fp8 || !p.replicate)) return cudaErrorInvalidValue;   // multicast stores carry whole bf16 pages to every member
    KvTransferParams q = p;
    q.subs = kv_pick_subs(p, ctas);
    kv_transfer_kernel<8><<<ctas, 256, 0, stream>>>(q);
    return cudaGetLastError();
}

}  // namespace sky
