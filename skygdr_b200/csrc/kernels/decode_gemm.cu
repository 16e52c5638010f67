// Projections of a decode step on the 5th-generation tensor cores, each with the small ops around it.
//
// y[t][n] = sum_k x[t][k] w[n][k] for t < 256. Weight rows are the MMA's M (128 per tile), tokens its N: any multiple of 16, so a batch
// of 100 computes 112 columns. One CTA per (tile, K slice):
//   warp 0   : TMA producer. The weight tiles of the first stages are requested before the previous kernel has ended (weights are
//              constants), x after griddepcontrol.wait.
//   warp 1   : MMA issuer and TMEM owner.
//   warps 2-5: epilogue.
// The K slices of a tile are a thread-block cluster: each leaves its fp32 partial in its own shared memory, one cluster barrier,
// then CTA s takes the token columns [s ntok / splits, (s + 1) ntok / splits), with the loads of all partials in flight together.
//
// What bounds a decode layer is not the bytes alone: with every weight already in L2 a 4096 x 4096 projection of the general
// kernel (gemm_tcgen05.cu) took 8.5 us in a chain of launches, 9.8 us with cold weights (5.2 us of bytes). A launch boundary costs
// about 4 us whatever the kernel does, and RMSNorm and rotary embedding are launches that do nothing else. So the small ops live in
// the epilogues, on rows of 128 columns that are at hand there:
//   * the residual add, and RMSNorm split in two: the epilogue of O and down writes resid * gain and its tile's sums of squares per
//     row; the next projection multiplies the finished product by the row's 1 / rms (it is linear in x);
//   * QK-norm, rotary embedding and the append to the paged cache: a tile of the QKV projection is exactly one head.
// FIGURES
#include <cuda.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "decode_gemm.h"
#include "rope.cuh"

namespace sky {

bool make_tmap_bf16_2d(CUtensorMap* m, const void* base, long long rows, long long cols, long long ld, int box_rows);

namespace {

constexpr int DG_THREADS = 192;
constexpr int DG_BM = 128, DG_BK = 64;
constexpr int DG_W_BYTES = DG_BM * DG_BK * 2;
constexpr int DG_MAX_STAGES = 8;
constexpr int DG_PITCH = 132;                      // floats between staged rows of 128 values (16-byte rows, banks shifted)

struct DgShape {                                   // derived on the host once per launch
    int ntok, stages, stage_bytes, acc_cols, tmem_cols;
    int up_col;                                    // first TMEM column (and partial column) of the up accumulator
    int stage_off;                                 // where finished rows are staged, behind the partials
};

__device__ __forceinline__ uint32_t dg_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void dg_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void dg_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t dg_peer(uint32_t local, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
__device__ __forceinline__ float dg_ld_peer(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ void unpack4(uint2 v, float* f) {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
}
__device__ __forceinline__ uint2 pack4(const float* f) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ float silu_mul_f(float g, float u) { return g / (1.0f + __expf(-g)) * u; }

// One finished row of a tile: lane holds columns 4 lane .. 4 lane + 3 of the 128.
__device__ __forceinline__ void finish_row(const DecodeGemmParams& p, int tile, int t, int lane, float* v, int pos, int blk) {
    const int n0 = tile * DG_BM;
    if (p.mode == DG_STORE) {
        const int n = n0 + lane * 4;
        __nv_bfloat16* dst = p.y + (long long)t * p.ldy + n;
        if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) *reinterpret_cast<uint2*>(dst) = pack4(v);
        else
            for (int i = 0; i < 4 && n + i < p.N; ++i) dst[i] = __float2bfloat16(v[i]);
    } else if (p.mode == DG_RESID) {
        const long long at = (long long)t * p.N + n0 + lane * 4;
        float r[4], g[4];
        unpack4(*reinterpret_cast<const uint2*>(p.resid + at), r);
        unpack4(__ldg(reinterpret_cast<const uint2*>(p.gain + n0 + lane * 4)), g);
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] += v[i];
        const uint2 packed = pack4(r);
        *reinterpret_cast<uint2*>(p.resid + at) = packed;
        unpack4(packed, r);                        // the norm sees what was stored
        float ss = r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3];
#pragma unroll
        for (int i = 0; i < 4; ++i) g[i] *= r[i];
        *reinterpret_cast<uint2*>(p.xg + at) = pack4(g);
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) p.ss_out[(long long)tile * p.ss_pitch + t] = ss;
    } else {
        float cs[4], sn[4];
        rope_angles(pos, p.rope.inv_freq, lane, cs, sn);
        rope_append_row(p.rope, t, tile, lane, v, pos, blk, cs, sn);
    }
}

template <bool GATED>
__global__ void __launch_bounds__(DG_THREADS, 2) decode_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                                                                     const __grid_constant__ DecodeGemmParams p, const DgShape sh) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full_bar[DG_MAX_STAGES], empty_bar[DG_MAX_STAGES], acc_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ float s_inv[DECODE_GEMM_MAX_ROWS];
    __shared__ int s_pos[DECODE_GEMM_MAX_ROWS], s_blk[DECODE_GEMM_MAX_ROWS];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, split = blockIdx.z, splits = gridDim.z;
    const int n0 = tile * DG_BM;
    const int kb_total = p.K / DG_BK;
    const int kb0 = split * kb_total / splits, nkb = (split + 1) * kb_total / splits - kb0;
    constexpr int WB = GATED ? 2 : 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < sh.stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(&acc_bar, 1);
        fence_barrier_init();
        tma_prefetch_desc(&tmap_w);
        tma_prefetch_desc(&tmap_x);
        const int pre = min(nkb, sh.stages);
        for (int i = 0; i < pre; ++i) {            // constants: ahead of the previous kernel
            unsigned char* st = smem + i * sh.stage_bytes;
            mbar_expect_tx(&full_bar[i], (uint32_t)sh.stage_bytes);
            tma_load_2d(st, &tmap_w, (kb0 + i) * DG_BK, n0, &full_bar[i]);
            if (GATED) tma_load_2d(st + DG_W_BYTES, &tmap_w, (kb0 + i) * DG_BK, p.N + n0, &full_bar[i]);
        }
    }
    if (warp == 1) { tmem_alloc(&tmem_slot, (uint32_t)sh.tmem_cols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();                                 // with TMEM in hand: a CTA of the next kernel cannot take it first
    const uint32_t tmem_base = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            pdl_wait();
            const int pre = min(nkb, sh.stages);
            for (int i = 0; i < pre; ++i)
                tma_load_2d(smem + i * sh.stage_bytes + WB * DG_W_BYTES, &tmap_x, (kb0 + i) * DG_BK, 0, &full_bar[i]);
            // one thread runs at the latency of its own instructions: slot and phase are counted along, nothing is divided
            int slot = 0;
            uint32_t phase = 0;
            for (int i = pre; i < nkb; ++i) {
                if (!mbar_wait(&empty_bar[slot], phase)) { set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 81); break; }
                unsigned char* st = smem + slot * sh.stage_bytes;
                mbar_expect_tx(&full_bar[slot], (uint32_t)sh.stage_bytes);
                tma_load_2d(st, &tmap_w, (kb0 + i) * DG_BK, n0, &full_bar[slot]);
                if (GATED) tma_load_2d(st + DG_W_BYTES, &tmap_w, (kb0 + i) * DG_BK, p.N + n0, &full_bar[slot]);
                tma_load_2d(st + WB * DG_W_BYTES, &tmap_x, (kb0 + i) * DG_BK, 0, &full_bar[slot]);
                if (++slot == sh.stages) { slot = 0; phase ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16(DG_BM, 0) | ((uint32_t)(sh.ntok >> 3) << 17);
            pdl_wait();                            // bounded waits start when the previous kernel is done
            const uint64_t a0 = umma_desc_k_sw128(smem_u32(smem)), a1 = a0 + (DG_W_BYTES >> 4), b0 = a0 + (WB * DG_W_BYTES >> 4);
            const uint32_t step = (uint32_t)sh.stage_bytes >> 4, up = tmem_base + sh.up_col;       // descriptors count 16-byte units
            int slot = 0;
            uint32_t phase = 0, at = 0, accum = 0;
            for (int i = 0; i < nkb; ++i) {
                if (!mbar_wait(&full_bar[slot], phase)) { set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 82); break; }
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < DG_BK / 16; ++k) {
                    tc_mma_f16(tmem_base, a0 + at + 2 * k, b0 + at + 2 * k, idesc, k ? 1u : accum);
                    if (GATED) tc_mma_f16(up, a1 + at + 2 * k, b0 + at + 2 * k, idesc, k ? 1u : accum);
                }
                tc_commit(&empty_bar[slot]);
                accum = 1;
                at += step;
                if (++slot == sh.stages) { slot = 0; phase ^= 1u; at = 0; }
            }
            tc_commit(&acc_bar);
        }
        __syncwarp();
    }

    // ---- epilogue ----
    const int c_lo = split * sh.ntok / splits, c_hi = min((split + 1) * sh.ntok / splits, p.M);      // this CTA's token rows
    float* part = reinterpret_cast<float*>(smem);                        // [acc_cols][128], over the idle ring
    float* rows = reinterpret_cast<float*>(smem + sh.stage_off);         // [c_hi - c_lo][DG_PITCH]
    const int ew = warp - 2;                                             // 0..3; TMEM lanes 32 (warp % 4) ..
    const int r = (warp & 3) * 32 + lane;                                // weight row inside the tile
    const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    bool ok = true;
    if (warp >= 2) {
        pdl_wait();
        // what the rows need besides the product, while the product is being computed
        for (int t = c_lo + ew; t < c_hi; t += 4) {
            float inv = 1.0f;
            if (p.ss_in) {
                float ss = 0.f;
                for (int i = lane; i < p.n_ss; i += 32) ss += __ldcg(p.ss_in + (long long)i * p.ss_pitch + t);
                for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                inv = rsqrtf(ss / p.norm_dim + p.eps);
            }
            if (lane == 0) {
                s_inv[t] = inv;
                if (p.mode == DG_QKV) {
                    const int pos = p.rope.positions[t];
                    s_pos[t] = pos;
                    s_blk[t] = p.rope.block_table[(long long)(p.rope.seq_ids ? p.rope.seq_ids[t] : t) * p.rope.max_blocks + pos / p.rope.block_tokens];
                }
            }
        }
        if (nkb > 0) ok = mbar_wait(&acc_bar, 0);
        if (!ok && lane == 0) set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 83);
        tc_fence_after();
        if (splits > 1) {
            for (int c = 0; c < sh.acc_cols; c += 16) {
                uint32_t v[16];
                tmem_ld_x16(taddr + c, v);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) part[(c + i) * DG_BM + r] = ok ? __uint_as_float(v[i]) : 0.f;
            }
        } else {
            for (int c = 0; c < c_hi; c += 16) {
                uint32_t v[16], u[16];
                tmem_ld_x16(taddr + c, v);
                if (GATED) tmem_ld_x16(taddr + sh.up_col + c, u);
                tc_wait_ld();
                epi_bar();                                               // s_inv is written; and the staged rows of the last round have been read
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if (c + i >= c_hi) break;
                    const float inv = s_inv[c + i];
                    float val = __uint_as_float(v[i]) * inv;
                    if (GATED) val = silu_mul_f(val, __uint_as_float(u[i]) * inv);
                    rows[i * DG_PITCH + r] = ok ? val : 0.f;
                }
                epi_bar();
                for (int t = c + ew; t < min(c + 16, c_hi); t += 4) {
                    float4 q = *reinterpret_cast<const float4*>(rows + (t - c) * DG_PITCH + lane * 4);
                    finish_row(p, tile, t, lane, reinterpret_cast<float*>(&q), s_pos[t], s_blk[t]);
                }
            }
        }
    }
    if (splits > 1) {
        tc_fence_before();
        dg_cluster_arrive();
        dg_cluster_wait();                                               // every CTA's partial is in its shared memory
        if (warp >= 2) {
            uint32_t peer[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) peer[s] = s < splits ? dg_peer(smem_u32(smem), (uint32_t)s) + (uint32_t)r * 4u : 0u;
            constexpr int CH = 4;                                        // columns per round: 4 x splits loads in flight (gated: twice)
            for (int c = c_lo; c < c_hi; c += CH) {
                float g[CH] = {}, u[CH] = {};
#pragma unroll
                for (int half = 0; half < (GATED ? 2 : 1); ++half) {
                    float a[8][CH];
#pragma unroll
                    for (int s = 0; s < 8; ++s)
#pragma unroll
                        for (int i = 0; i < CH; ++i)
                            a[s][i] = (s < splits && c + i < c_hi) ? dg_ld_peer(peer[s] + (uint32_t)((half * sh.up_col + c + i) * DG_BM) * 4u) : 0.f;
#pragma unroll
                    for (int s = 0; s < 8; ++s)
#pragma unroll
                        for (int i = 0; i < CH; ++i) (half ? u : g)[i] += a[s][i];
                }
#pragma unroll
                for (int i = 0; i < CH; ++i)
                    if (c + i < c_hi) {
                        const float inv = s_inv[c + i];
                        rows[(c + i - c_lo) * DG_PITCH + r] = GATED ? silu_mul_f(g[i] * inv, u[i] * inv) : g[i] * inv;
                    }
            }
        }
        dg_cluster_arrive();                                             // this CTA has read its peers
        if (warp >= 2) {
            epi_bar();
            for (int t = c_lo + ew; t < c_hi; t += 4) {
                float4 q = *reinterpret_cast<const float4*>(rows + (t - c_lo) * DG_PITCH + lane * 4);
                finish_row(p, tile, t, lane, reinterpret_cast<float*>(&q), s_pos[t], s_blk[t]);
            }
        }
        __syncwarp();
        dg_cluster_wait();                                               // and nobody reads this one any more
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, (uint32_t)sh.tmem_cols);
}

}  // namespace

// Splits of K per tile: as many as bring the launch to about one CTA per SM (a CTA then leaves room for one of the next kernel, which
// streams its first weight tiles meanwhile), at most 8 (a portable cluster) and at least 4 k-blocks each.
int decode_gemm_splits(int M, int N, int K, bool gated, int sms) {
    const int tiles = (N + DG_BM - 1) / DG_BM, kb = K / DG_BK;
    int s = std::max(1, std::min({8, sms / tiles, kb / 4}));
    return s;
}

cudaError_t launch_decode_gemm(const DecodeGemmParams& p, cudaStream_t stream) {
    if (p.M < 1 || p.M > DECODE_GEMM_MAX_ROWS || p.N < 1 || p.K < DG_BK || p.K % DG_BK || p.splits < 1 || p.splits > 8 || p.splits > p.K / DG_BK) return cudaErrorInvalidValue;
    if (p.mode != DG_STORE && (p.N % DG_BM || p.gated)) return cudaErrorInvalidValue;
    if (p.mode == DG_QKV && p.N != (p.rope.q_heads + 2 * p.rope.kv_heads) * 128) return cudaErrorInvalidValue;
    DgShape sh;
    sh.ntok = (p.M + 15) / 16 * 16;
    sh.up_col = (sh.ntok + 31) / 32 * 32;
    sh.acc_cols = p.gated ? sh.up_col + sh.ntok : sh.ntok;
    sh.tmem_cols = 32;
    while (sh.tmem_cols < sh.acc_cols) sh.tmem_cols *= 2;
    sh.stage_bytes = DG_W_BYTES * (p.gated ? 2 : 1) + sh.ntok * DG_BK * 2;
    const int part = p.splits > 1 ? sh.acc_cols * DG_BM * 4 : 0;
    sh.stage_off = part;
    const int rows = (p.splits > 1 ? (sh.ntok + p.splits - 1) / p.splits + 1 : 16) * DG_PITCH * 4;
    // Two CTAs per SM (this kernel's and the next one's, or two of a launch with many tiles) where three stages fit in half of the
    // shared memory and half of TMEM is enough; one otherwise. With one, no second CTA can wait for TMEM that it will not get.
    const bool two = 3 * sh.stage_bytes <= 104 * 1024 && part + rows <= 104 * 1024 && sh.tmem_cols <= 256;
    const int budget = two ? 104 * 1024 : 200 * 1024;
    sh.stages = std::min(DG_MAX_STAGES, budget / sh.stage_bytes);
    int bytes = std::max(sh.stages * sh.stage_bytes, part + rows);
    if (!two) bytes = std::max(bytes, 116 * 1024);
    if (bytes > 226 * 1024 - 1024 - 8 * 1024 || sh.stages < 2) return cudaErrorInvalidValue;
    bytes += 1024;
    CUtensorMap tw, tx;
    if (!make_tmap_bf16_2d(&tw, p.w, p.gated ? 2LL * p.N : p.N, p.K, p.K, DG_BM)) return cudaErrorInvalidValue;
    if (!make_tmap_bf16_2d(&tx, p.x, p.M, p.K, p.K, sh.ntok)) return cudaErrorInvalidValue;
    static unsigned long long attr_mask[2] = {0, 0};
    auto kern = p.gated ? decode_gemm_kernel<true> : decode_gemm_kernel<false>;
    if (cudaError_t e = set_max_dynamic_smem_once(reinterpret_cast<const void*>(kern), 218 * 1024, &attr_mask[p.gated ? 1 : 0]); e != cudaSuccess) return e;
    return launch_pdl_cluster(kern, dim3((p.N + DG_BM - 1) / DG_BM, 1, p.splits), dim3(DG_THREADS), (size_t)bytes, stream, p.splits, tw, tx, p, sh);
}

namespace {
__global__ void __launch_bounds__(256) embed_norm_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table, int vocab, int hidden,
                                                          const __nv_bfloat16* __restrict__ gain, __nv_bfloat16* __restrict__ resid,
                                                          __nv_bfloat16* __restrict__ xg, float* __restrict__ ss_out) {
    __shared__ float red[8];
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    int id = ids[t];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    float ss = 0.f;
    for (int v = threadIdx.x; v < hidden / 4; v += 256) {
        const uint2 e = *reinterpret_cast<const uint2*>(table + (long long)id * hidden + v * 4);
        float x[4], g[4];
        unpack4(e, x);
        unpack4(*reinterpret_cast<const uint2*>(gain + v * 4), g);
        *reinterpret_cast<uint2*>(resid + (long long)t * hidden + v * 4) = e;
#pragma unroll
        for (int i = 0; i < 4; ++i) { ss += x[i] * x[i]; g[i] *= x[i]; }
        *reinterpret_cast<uint2*>(xg + (long long)t * hidden + v * 4) = pack4(g);
    }
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.f;
        for (int i = 0; i < 8; ++i) sum += red[i];
        ss_out[t] = sum;
    }
}
}  // namespace

cudaError_t launch_embed_norm(const int* ids, const __nv_bfloat16* table, int vocab, int hidden, int tokens, const __nv_bfloat16* gain, __nv_bfloat16* resid,
                              __nv_bfloat16* xg, float* ss, cudaStream_t stream) {
    if (hidden % 4 || tokens < 1) return cudaErrorInvalidValue;
    return launch_pdl(embed_norm_kernel, dim3(tokens), dim3(256), 0, stream, ids, table, vocab, hidden, gain, resid, xg, ss);
}

}  // namespace sky
