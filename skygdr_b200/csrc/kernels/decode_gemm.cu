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
// One B200, 8 layers of Qwen3-8B's widths, host token ids in and out, against separate kernels on the general projection: one sequence
// 1061 -> 954 us, 16 sequences of 2k to 16k tokens 1885 -> 1807 us, 32 of 1k to 32k 3049 -> 2626 us, 100 short ones with sampling
// 1964 -> 1869 us; prefill of 77 tokens 2174 -> 1118 us (with the passes driven from C++).
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

struct DgShape {                                   // derived on the host once per launch
    int ntok, stages, stage_bytes, acc_cols, tmem_cols;
    int up_col;                                    // first TMEM column (and partial column) of the up accumulator
};

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

// Finished rows t0, t0 + 4, ... (U of them, those below t_end) of a tile: lane holds columns 4 lane .. 4 lane + 3 of the 128. Several rows
// at once, because a row by itself is a chain of load, shuffles and store.
template <int MODE, int U>
__device__ __forceinline__ void finish_rows(const DecodeGemmParams& p, int tile, int t0, int t_end, int lane, float (*v)[4], const int* s_pos, const int* s_blk) {
    const int n0 = tile * DG_BM;
    if (MODE == DG_STORE) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = t0 + 4 * u, n = n0 + lane * 4;
            if (t >= t_end) break;
            __nv_bfloat16* dst = p.y + (long long)t * p.ldy + n;
            if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) *reinterpret_cast<uint2*>(dst) = pack4(v[u]);
            else
                for (int i = 0; i < 4 && n + i < p.N; ++i) dst[i] = __float2bfloat16(v[u][i]);
        }
    } else if (MODE == DG_RESID) {
        const long long at = (long long)t0 * p.N + n0 + lane * 4;
        uint2 res[U];
#pragma unroll
        for (int u = 0; u < U; ++u) res[u] = t0 + 4 * u < t_end ? *reinterpret_cast<const uint2*>(p.resid + at + 4LL * u * p.N) : make_uint2(0, 0);
        float g[4], ss[U];
        unpack4(__ldg(reinterpret_cast<const uint2*>(p.gain + n0 + lane * 4)), g);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float r[4];
            unpack4(res[u], r);
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] += v[u][i];
            const uint2 packed = pack4(r);
            unpack4(packed, r);                    // the norm sees what is stored
            ss[u] = r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3];
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] *= g[i];
            if (t0 + 4 * u < t_end) {
                *reinterpret_cast<uint2*>(p.resid + at + 4LL * u * p.N) = packed;
                *reinterpret_cast<uint2*>(p.xg + at + 4LL * u * p.N) = pack4(r);
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1)
#pragma unroll
            for (int u = 0; u < U; ++u) ss[u] += __shfl_xor_sync(0xffffffffu, ss[u], o);
        if (lane == 0)
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (t0 + 4 * u < t_end) p.ss_out[(long long)tile * p.ss_pitch + t0 + 4 * u] = ss[u];
    } else {
        if (p.round_product)
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < 4; ++i) v[u][i] = __bfloat162float(__float2bfloat16(v[u][i]));
        if (tile < p.rope.q_heads + p.rope.kv_heads) {
            const __nv_bfloat16* weight = tile < p.rope.q_heads ? p.rope.q_norm : p.rope.k_norm;
            if (weight) rope_norm_rows<U>(weight, p.rope.eps, lane, v);
            const float4 freqs = rope_freqs(p.rope.inv_freq, lane);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float cs[4], sn[4];
                rope_angles(t0 + 4 * u < t_end ? s_pos[t0 + 4 * u] : 0, freqs, cs, sn);
                rope_rotate(lane, v[u], cs, sn);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t0 + 4 * u < t_end) rope_store(p.rope, t0 + 4 * u, tile, lane, v[u], s_pos[t0 + 4 * u], s_blk[t0 + 4 * u]);
    }
}

template <bool GATED, int MODE>
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
                if (MODE == DG_QKV) {
                    const int pos = p.rope.positions[t];
                    s_pos[t] = pos;
                    s_blk[t] = p.rope.block_table[(long long)(p.rope.seq_ids ? p.rope.seq_ids[t] : t) * p.rope.max_blocks + pos / p.rope.block_tokens];
                }
            }
        }
        if (nkb > 0) ok = mbar_wait(&acc_bar, 0);
        if (!ok && lane == 0) set_status(p.status, SKY_STATUS_TIMEOUT_MBAR, 83);
        tc_fence_after();
        // the accumulator, token column by token column, to shared memory; a gated tile that is not split is finished on the way
        if (GATED && splits == 1) {
            epi_bar();                                                   // s_inv is written
            for (int c = 0; c < sh.ntok; c += 16) {
                uint32_t v[16], u[16];
                tmem_ld_x16(taddr + c, v);
                tmem_ld_x16(taddr + sh.up_col + c, u);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float inv = c + i < p.M ? s_inv[c + i] : 0.f;
                    part[(c + i) * DG_BM + r] = ok ? silu_mul_f(__uint_as_float(v[i]) * inv, __uint_as_float(u[i]) * inv) : 0.f;
                }
            }
        } else {
            int c = 0;
            for (; c + 32 <= sh.acc_cols; c += 32) {
                uint32_t v[32];
                tmem_ld_x32(taddr + c, v);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) part[(c + i) * DG_BM + r] = ok ? __uint_as_float(v[i]) : 0.f;
            }
            if (c < sh.acc_cols) {
                uint32_t v[16];
                tmem_ld_x16(taddr + c, v);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) part[(c + i) * DG_BM + r] = ok ? __uint_as_float(v[i]) : 0.f;
            }
        }
    }
    if (splits > 1) {
        tc_fence_before();
        cluster_arrive();
        cluster_wait();                                                  // every CTA's partial is in its shared memory
    }
    if (warp >= 2) {
        if (splits == 1) epi_bar();
        constexpr int U = GATED ? 2 : 4;                                 // rows at once: their loads from all slices are in flight together
        const uint32_t own = smem_u32(part) + (uint32_t)lane * 16u;
        for (int t0 = c_lo + ew; t0 < c_hi; t0 += 4 * U) {
            float v[U][4];
            if (splits == 1) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int t = t0 + 4 * u;
                    const float4 q = t < c_hi ? *reinterpret_cast<const float4*>(part + t * DG_BM + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float inv = GATED || t >= c_hi ? 1.0f : s_inv[t];
                    v[u][0] = q.x * inv; v[u][1] = q.y * inv; v[u][2] = q.z * inv; v[u][3] = q.w * inv;
                }
            } else {
                float up[U][4];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[u][i] = up[u][i] = 0.f;
                for (int s0 = 0; s0 < splits; s0 += 4) {
                    float4 a[4][U], b[4][U];
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        const uint32_t peer = dsmem_addr(own, (uint32_t)min(s0 + s, splits - 1));
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int t = t0 + 4 * u;
                            const bool in = s0 + s < splits && t < c_hi;
                            a[s][u] = in ? ld_dsmem_f32x4(peer + (uint32_t)(t * DG_BM) * 4u) : make_float4(0.f, 0.f, 0.f, 0.f);
                            if (GATED) b[s][u] = in ? ld_dsmem_f32x4(peer + (uint32_t)((sh.up_col + t) * DG_BM) * 4u) : make_float4(0.f, 0.f, 0.f, 0.f);
                        }
                    }
#pragma unroll
                    for (int s = 0; s < 4; ++s)
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            v[u][0] += a[s][u].x; v[u][1] += a[s][u].y; v[u][2] += a[s][u].z; v[u][3] += a[s][u].w;
                            if (GATED) { up[u][0] += b[s][u].x; up[u][1] += b[s][u].y; up[u][2] += b[s][u].z; up[u][3] += b[s][u].w; }
                        }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float inv = t0 + 4 * u < c_hi ? s_inv[t0 + 4 * u] : 1.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[u][i] = GATED ? silu_mul_f(v[u][i] * inv, up[u][i] * inv) : v[u][i] * inv;
                }
            }
            finish_rows<MODE, U>(p, tile, t0, c_hi, lane, v, s_pos, s_blk);
        }
    }
    if (splits > 1) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();                                                  // nobody reads this CTA's shared memory any more
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, (uint32_t)sh.tmem_cols);
}

// Token and accumulator columns of a launch.
DgShape dg_cols(int M, bool gated) {
    DgShape sh = {};
    sh.ntok = (M + 15) / 16 * 16;
    sh.up_col = (sh.ntok + 31) / 32 * 32;
    sh.acc_cols = gated ? sh.up_col + sh.ntok : sh.ntok;
    return sh;
}
// Shared memory of the finished or partial columns, over the ring.
int part_bytes(const DgShape& sh, int splits) { return (splits > 1 ? sh.acc_cols : sh.ntok) * DG_BM * 4; }
constexpr int DG_MAX_BYTES = 217 * 1024;           // of 227 KB, less the alignment of the ring and the static part

}  // namespace

// Splits of K per tile: as many as bring the launch to about one CTA per SM (a CTA then leaves room for one of the next kernel, which
// streams its first weight tiles meanwhile), at most 8 (a portable cluster) and at least 4 k-blocks each.
// Up to 16 tokens the partials are small, and two CTAs per SM, with twice the loads in flight, are the better use of the room; a gated
// tile, whose partial is twice as wide, stays at two slices. A step of 8 layers, all projections so, against one CTA per SM:
// 1 sequence 905 and 973 us, 16 sequences 985 and 1030 us, 64 sequences 1234 and 1133 us, 100 sequences 1500 and 1350 us (gate/up in
// three slices: 1011 us at 1, 1069 us at 16).
// The fp32 partials of a slice have to fit in shared memory: a gated tile of more than some 200 tokens does not split.
int decode_gemm_splits(int M, int N, int K, bool gated, int sms) {
    const int tiles = (N + DG_BM - 1) / DG_BM, kb = K / DG_BK;
    const int room = M <= 16 ? (gated ? std::min(2, 2 * sms / tiles) : 2 * sms / tiles) : sms / tiles;
    const int s = std::max(1, std::min({8, room, kb / 4}));
    return s > 1 && part_bytes(dg_cols(M, gated), s) > DG_MAX_BYTES ? 1 : s;
}

cudaError_t launch_decode_gemm(const DecodeGemmParams& p, cudaStream_t stream) {
    if (p.M < 1 || p.M > DECODE_GEMM_MAX_ROWS || p.N < 1 || p.K < DG_BK || p.K % DG_BK || p.splits < 1 || p.splits > 8 || p.splits > p.K / DG_BK) return cudaErrorInvalidValue;
    if (p.mode != DG_STORE && (p.N % DG_BM || p.gated)) return cudaErrorInvalidValue;
    if (p.mode == DG_QKV && p.N != (p.rope.q_heads + 2 * p.rope.kv_heads) * 128) return cudaErrorInvalidValue;
    DgShape sh = dg_cols(p.M, p.gated);
    sh.tmem_cols = 32;
    while (sh.tmem_cols < sh.acc_cols) sh.tmem_cols *= 2;
    sh.stage_bytes = DG_W_BYTES * (p.gated ? 2 : 1) + sh.ntok * DG_BK * 2;
    const int part = part_bytes(sh, p.splits);
    // Two CTAs per SM (this kernel's and the next one's, or two of a launch with many tiles) where three stages fit in half of the
    // shared memory and half of TMEM is enough; one otherwise. With one, no second CTA can wait for TMEM that it will not get.
    const bool two = 3 * sh.stage_bytes <= 104 * 1024 && part <= 104 * 1024 && sh.tmem_cols <= 256;
    const int budget = two ? 104 * 1024 : 200 * 1024;
    sh.stages = std::min(DG_MAX_STAGES, budget / sh.stage_bytes);
    int bytes = std::max(sh.stages * sh.stage_bytes, part);
    if (!two) bytes = std::max(bytes, 116 * 1024);
    if (bytes > DG_MAX_BYTES || sh.stages < 2) return cudaErrorInvalidValue;
    bytes += 1024;
    CUtensorMap tw, tx;
    if (!make_tmap_bf16_2d(&tw, p.w, p.gated ? 2LL * p.N : p.N, p.K, p.K, DG_BM)) return cudaErrorInvalidValue;
    if (!make_tmap_bf16_2d(&tx, p.x, p.M, p.K, p.K, sh.ntok)) return cudaErrorInvalidValue;
    static unsigned long long attr_mask[4] = {0, 0, 0, 0};
    const int form = p.gated ? 3 : p.mode;
    auto kern = p.gated ? decode_gemm_kernel<true, DG_STORE> : p.mode == DG_STORE ? decode_gemm_kernel<false, DG_STORE>
                        : p.mode == DG_RESID ? decode_gemm_kernel<false, DG_RESID> : decode_gemm_kernel<false, DG_QKV>;
    if (cudaError_t e = set_max_dynamic_smem_once(reinterpret_cast<const void*>(kern), 218 * 1024, &attr_mask[form]); e != cudaSuccess) return e;
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
