// Small fused decoder ops: RMSNorm (+ residual add), per-head QK-norm + RoPE +
// KV append into the paged cache, SiLU*mul, embedding gather, argmax.
//
// The reference's decode stressors only append raw K/V rows
// (llm_problem_analysis/decode_transformer_kvcache_stress.cu:360-391,
// llm_problem_analysis/decode_vllm_kvcache_hbm_stress.cu:284-328) and model the MLP
// as a streaming pass (decode_transformer_kvcache_stress.cu:323-356); these are the
// real ops of a Qwen3 decoder layer.
#include "common.cuh"
#include "fused_ops.h"
#include "rope.cuh"

namespace sky {

__device__ __forceinline__ void unpack8(uint4 v, float* f) {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
    f[4] = __uint_as_float(v.z << 16); f[5] = __uint_as_float(v.z & 0xffff0000u);
    f[6] = __uint_as_float(v.w << 16); f[7] = __uint_as_float(v.w & 0xffff0000u);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint4 pack8(const float* f) {
    return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}

__device__ __forceinline__ float block_sum(float v, float* red) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0) red[w] = v;
    __syncthreads();
    float t = 0.f;
    for (int i = 0; i < nw; ++i) t += red[i];
    __syncthreads();
    return t;
}

// One CTA per row; each thread owns up to 4 vectors of 8 elements (hidden <= 256*8*4 = 8192).
__device__ __forceinline__ void rmsnorm_row(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* residual, const __nv_bfloat16* __restrict__ w,
                                            __nv_bfloat16* __restrict__ y, int hidden, float eps, float* red) {
    const int nvec = hidden / 8;
    float vals[4][8];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int v = threadIdx.x + k * 256;
        if (v < nvec) {
            unpack8(*reinterpret_cast<const uint4*>(x + v * 8), vals[k]);
            if (residual) {
                float r[8];
                unpack8(*reinterpret_cast<const uint4*>(residual + v * 8), r);
#pragma unroll
                for (int i = 0; i < 8; ++i) vals[k][i] += r[i];
                uint4 packed = pack8(vals[k]);
                *reinterpret_cast<uint4*>(residual + v * 8) = packed;
                unpack8(packed, vals[k]);  // normalise what was stored (bf16-rounded), as a two-kernel version would
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += vals[k][i] * vals[k][i];
        }
    }
    ss = block_sum(ss, red);
    const float inv = rsqrtf(ss / hidden + eps);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int v = threadIdx.x + k * 256;
        if (v < nvec) {
            float g[8], o[8];
            unpack8(*reinterpret_cast<const uint4*>(w + v * 8), g);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = vals[k][i] * inv * g[i];
            *reinterpret_cast<uint4*>(y + v * 8) = pack8(o);
        }
    }
}

__global__ void __launch_bounds__(256) rmsnorm_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* residual,
                                                       const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                       int hidden, float eps) {
    __shared__ float red[8];
    pdl_trigger();
    pdl_wait();
    const long long at = (long long)blockIdx.x * hidden;
    rmsnorm_row(x + at, residual ? residual + at : nullptr, w, y + at, hidden, eps, red);
}

cudaError_t launch_rmsnorm(const __nv_bfloat16* x, __nv_bfloat16* residual, const __nv_bfloat16* w, __nv_bfloat16* y,
                           int rows, int hidden, float eps, cudaStream_t stream) {
    if (hidden % 8 || hidden > 8192 || rows <= 0) return cudaErrorInvalidValue;
    return launch_pdl(rmsnorm_kernel, dim3(rows), dim3(256), 0, stream, x, residual, w, y, hidden, eps);
}

__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* residual,
                                                            const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                            const __grid_constant__ RowMap rows, int hidden, float eps) {
    __shared__ float red[8];
    pdl_trigger();
    pdl_wait();
    const long long from = (long long)rows.src[blockIdx.x] * hidden, to = (long long)rows.dst[blockIdx.x] * hidden;
    rmsnorm_row(x + from, residual + from, w, y + to, hidden, eps, red);
}

cudaError_t launch_rmsnorm_rows(const __nv_bfloat16* x, __nv_bfloat16* residual, const __nv_bfloat16* w, __nv_bfloat16* y,
                                const RowMap& rows, int hidden, float eps, cudaStream_t stream) {
    if (hidden % 8 || hidden > 8192 || rows.n <= 0 || rows.n > ROW_MAP_MAX) return cudaErrorInvalidValue;
    return launch_pdl(rmsnorm_rows_kernel, dim3(rows.n), dim3(256), 0, stream, x, residual, w, y, rows, hidden, eps);
}

// One CTA per token of the pieces. Bound: the copy of the embedding rows (8 KB each at hidden 4096).
__global__ void __launch_bounds__(128) prefill_setup_kernel(const PrefillSetup p, const __grid_constant__ PrefillPieces pc) {
    pdl_trigger();
    pdl_wait();
    const int tok = pc.tok0[0] + blockIdx.x;
    int lo = 0, hi = pc.n - 1;                              // the piece that holds this token
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pc.tok0[mid] <= tok) lo = mid; else hi = mid - 1;
    }
    const int off = tok - pc.tok0[lo];
    const long long at = (long long)pc.src[lo] + off;
    int id = p.ids64 ? (int)reinterpret_cast<const long long*>(p.ids)[at] : reinterpret_cast<const int*>(p.ids)[at];
    id = id < 0 ? 0 : (id >= p.vocab ? p.vocab - 1 : id);
    if (threadIdx.x == 0) {
        p.positions[tok] = pc.pos0[lo] + off;
        p.tok_rows[tok] = pc.row[lo];
        if (off == 0) {
            p.seq_start[pc.first + lo] = tok;
            p.pos0[pc.first + lo] = pc.pos0[lo];
            p.rows[pc.first + lo] = pc.row[lo];
            if (lo == pc.n - 1) p.seq_start[pc.first + pc.n] = pc.tok0[pc.n];
        }
    }
    for (int v = threadIdx.x; v < p.hidden / 8; v += 128)
        *reinterpret_cast<uint4*>(p.resid + (long long)tok * p.hidden + v * 8) = *reinterpret_cast<const uint4*>(p.table + (long long)id * p.hidden + v * 8);
}

cudaError_t launch_prefill_setup(const PrefillSetup& p, const PrefillPieces& pieces, cudaStream_t stream) {
    if (pieces.n < 1 || pieces.n > PREFILL_PIECES_MAX || p.hidden % 8 || pieces.tok0[pieces.n] <= pieces.tok0[0]) return cudaErrorInvalidValue;
    return launch_pdl(prefill_setup_kernel, dim3(pieces.tok0[pieces.n] - pieces.tok0[0]), dim3(128), 0, stream, p, pieces);
}

// One warp per token and group of eight heads (q heads, then k heads, then v heads), 16 lanes per head: lane L of them has dims
// 4L .. 4L + 3 and the 64 + 4L .. that these rotate with, so the rotation needs no exchange, the norm four shuffles for two heads, and
// the angles are computed once for the group. Sums are formed in the order of rope_norm_rows.
// Bound: 2 bytes read and 2 written per element, with all loads of a group in flight; what it costs beyond that is the chain position ->
// angle -> norm -> store. For 4300 tokens of 48 heads (105 MB: 16 us of traffic): one warp per (token, head) with the angle reduced
// anew for every head in double precision took 67.7 us, one warp per four heads with 32 lanes on each 39.4 us, this 27.8 us (8192 tokens: 75 and 57 us).
constexpr int ROPE_HEADS = 8;
__global__ void __launch_bounds__(128) rope_append_kernel(const RopeAppendParams p, unsigned int groups) {
    pdl_trigger();
    pdl_wait();
    const int heads_total = p.q_heads + 2 * p.kv_heads;
    const unsigned int gw = blockIdx.x * 4u + (threadIdx.x >> 5);
    const int tok = (int)(gw / groups), h0 = (int)(gw % groups) * ROPE_HEADS;
    if (tok >= p.tokens) return;
    const int lane = threadIdx.x & 15, half = (threadIdx.x >> 4) & 1;
    constexpr int R = ROPE_HEADS / 2;                                    // heads per half warp: h0 + half, h0 + half + 2, ...
    const __nv_bfloat16* src = p.qkv + ((long long)tok * heads_total + h0 + half) * 128 + lane * 4;
    uint2 lo[R], hi[R];
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const bool in = h0 + half + 2 * u < heads_total;
        lo[u] = in ? *reinterpret_cast<const uint2*>(src + u * 256) : make_uint2(0, 0);
        hi[u] = in ? *reinterpret_cast<const uint2*>(src + u * 256 + 64) : make_uint2(0, 0);
    }
    const int pos = p.positions[tok];
    const int blk = p.block_table[(long long)(p.seq_ids ? p.seq_ids[tok] : tok) * p.max_blocks + pos / p.block_tokens];
    float cs[4], sn[4];
    if (h0 < p.q_heads + p.kv_heads) rope_angles(pos, rope_freqs(p.inv_freq, lane), cs, sn);
    float a[R][4], b[R][4], ss[R];
#pragma unroll
    for (int u = 0; u < R; ++u) {
        rope_unpack(lo[u], a[u]);
        rope_unpack(hi[u], b[u]);
        ss[u] = (a[u][0] * a[u][0] + a[u][1] * a[u][1] + a[u][2] * a[u][2] + a[u][3] * a[u][3]) +
                (b[u][0] * b[u][0] + b[u][1] * b[u][1] + b[u][2] * b[u][2] + b[u][3] * b[u][3]);
    }
#pragma unroll
    for (int o = 8; o; o >>= 1)
#pragma unroll
        for (int u = 0; u < R; ++u) ss[u] += __shfl_xor_sync(0xffffffffu, ss[u], o);
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int h = h0 + half + 2 * u;
        if (h >= heads_total) break;
        if (h < p.q_heads + p.kv_heads) {
            const __nv_bfloat16* weight = h < p.q_heads ? p.q_norm : p.k_norm;
            if (weight) {
                float ga[4], gb[4];
                rope_unpack(__ldg(reinterpret_cast<const uint2*>(weight + lane * 4)), ga);
                rope_unpack(__ldg(reinterpret_cast<const uint2*>(weight + lane * 4 + 64)), gb);
                const float inv = rsqrtf(ss[u] * (1.0f / 128.0f) + p.eps);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    a[u][i] = __bfloat162float(__float2bfloat16(a[u][i] * inv * ga[i]));
                    b[u][i] = __bfloat162float(__float2bfloat16(b[u][i] * inv * gb[i]));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float x = a[u][i], y = b[u][i];
                a[u][i] = x * cs[i] - y * sn[i];
                b[u][i] = y * cs[i] + x * sn[i];
            }
        }
        rope_store(p, tok, h, lane, a[u], pos, blk);
        rope_store(p, tok, h, lane + 16, b[u], pos, blk);
    }
}

cudaError_t launch_rope_append(const RopeAppendParams& p, cudaStream_t stream) {
    if (p.tokens <= 0) return cudaErrorInvalidValue;
    const int groups = (p.q_heads + 2 * p.kv_heads + ROPE_HEADS - 1) / ROPE_HEADS;
    const long long warps = (long long)p.tokens * groups;
    if (warps > 0x7fffffffLL) return cudaErrorInvalidValue;
    return launch_pdl(rope_append_kernel, dim3((unsigned)((warps + 3) / 4)), dim3(128), 0, stream, p, (unsigned)groups);
}

__global__ void __launch_bounds__(256) silu_mul_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                                        long long n_vec, int ffn_vec) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n_vec) return;
    const long long r = i / ffn_vec;
    const int c = (int)(i - r * ffn_vec);
    float g[8], u[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(gu + (r * 2 * ffn_vec + c) * 8), g);
    unpack8(*reinterpret_cast<const uint4*>(gu + (r * 2 * ffn_vec + ffn_vec + c) * 8), u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = g[k] / (1.0f + __expf(-g[k])) * u[k];
    *reinterpret_cast<uint4*>(out + i * 8) = pack8(o);
}

cudaError_t launch_silu_mul(const __nv_bfloat16* gate_up, __nv_bfloat16* out, int rows, int ffn, cudaStream_t stream) {
    if (ffn % 8 || rows <= 0) return cudaErrorInvalidValue;
    const long long n_vec = (long long)rows * (ffn / 8);
    silu_mul_kernel<<<(unsigned)((n_vec + 255) / 256), 256, 0, stream>>>(gate_up, out, n_vec, ffn / 8);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(128) embedding_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                                         __nv_bfloat16* __restrict__ out, int hidden, int vocab) {
    pdl_trigger();
    pdl_wait();
    const int tok = blockIdx.x;
    int id = ids[tok];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    for (int v = threadIdx.x; v < hidden / 8; v += 128)
        *reinterpret_cast<uint4*>(out + (long long)tok * hidden + v * 8) = *reinterpret_cast<const uint4*>(table + (long long)id * hidden + v * 8);
}

cudaError_t launch_embedding(const int* ids, const __nv_bfloat16* table, __nv_bfloat16* out, int tokens, int hidden, int vocab,
                             cudaStream_t stream) {
    if (hidden % 8 || tokens <= 0) return cudaErrorInvalidValue;
    return launch_pdl(embedding_kernel, dim3(tokens), dim3(128), 0, stream, ids, table, out, hidden, vocab);
}

// Temperature sampling without a normalisation pass (Gumbel-max): argmax_c (logit_c / T + g_c) with g_c = -log(-log(u_c)) and
// u_c uniform in (0, 1) picks column c with probability softmax(logits / T)_c. u_c comes from a counter-based hash of
// (seed, position of the row's sequence, row, column), so a replayed CUDA graph draws fresh noise every step (the position
// advances) and a given (seed, position) always draws the same token. The hash is restated in skygdr_b200/ops/small.py.
__device__ __forceinline__ unsigned int sample_hash(unsigned int seed, unsigned int pos, unsigned int row, unsigned int col) {
    unsigned int h = seed * 0x9E3779B1u ^ (pos + 0x7F4A7C15u) * 0x85EBCA77u ^ (row + 0x165667B1u) * 0xC2B2AE3Du ^ (col + 0x27D4EB2Fu) * 0x9E3779B1u;
    h ^= h >> 16; h *= 0x85EBCA6Bu; h ^= h >> 13; h *= 0xC2B2AE35u; h ^= h >> 16;      // murmur3 finaliser
    return h;
}

struct Pick { float v; int c; };
__device__ __forceinline__ void pick_better(Pick& best, float v, int c) {
    if (v > best.v || (v == best.v && c < best.c)) { best.v = v; best.c = c; }
}
__device__ __forceinline__ Pick warp_pick(Pick best) {
    for (int o = 16; o; o >>= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, best.v, o);
        const int c = __shfl_xor_sync(0xffffffffu, best.c, o);
        pick_better(best, v, c);
    }
    return best;
}

// Column of the largest value of each row (lowest index wins ties), greedy or with the sampling noise added. A row is shared by a
// cluster of gridDim.z CTAs, each scanning one contiguous span in 16-byte loads; the spans' winners meet in shared memory.
// Bound: at one row, the latency of the loads (300 KB of logits, just written, out of L2); at a hundred sampled rows the hash and the
// two logarithms of every column.
constexpr int PICK_THREADS = 512;
template <bool SAMPLE>
__global__ void __launch_bounds__(PICK_THREADS) pick_kernel(const __nv_bfloat16* __restrict__ logits, int* __restrict__ out, int vocab,
                                                            long long row_stride, float inv_temperature, unsigned int seed, const int* __restrict__ positions) {
    __shared__ Pick warp_best[PICK_THREADS / 32];
    __shared__ Pick cta_best;
    pdl_trigger();
    pdl_wait();
    const unsigned int row_id = blockIdx.x;
    const int splits = (int)gridDim.z, split = (int)blockIdx.z;
    const __nv_bfloat16* row = logits + (long long)row_id * row_stride;
    const unsigned int pos = SAMPLE && positions ? (unsigned int)positions[row_id] : 0u;
    Pick best = {-INFINITY, 0x7fffffff};
    auto take = [&](float x, int c) {
        if (SAMPLE) {
            const float u = ((float)(sample_hash(seed, pos, row_id, (unsigned int)c) >> 8) + 0.5f) * (1.0f / 16777216.0f);
            x = x * inv_temperature - logf(-logf(u));
        }
        pick_better(best, x, c);
    };
    if (((reinterpret_cast<uintptr_t>(logits) | (uintptr_t)(row_stride * 2)) & 15) == 0) {
        const int vecs = vocab / 8;
        const int lo = (int)((long long)vecs * split / splits), hi = (int)((long long)vecs * (split + 1) / splits);
        constexpr int DEPTH = SAMPLE ? 2 : 4;               // loads in flight per thread
        for (int v = lo + threadIdx.x; v < hi; v += DEPTH * PICK_THREADS) {
            uint4 raw[DEPTH];
#pragma unroll
            for (int d = 0; d < DEPTH; ++d)
                if (v + d * PICK_THREADS < hi) raw[d] = *reinterpret_cast<const uint4*>(row + (long long)(v + d * PICK_THREADS) * 8);
#pragma unroll
            for (int d = 0; d < DEPTH; ++d)
                if (v + d * PICK_THREADS < hi) {
                    float f[8];
                    unpack8(raw[d], f);
#pragma unroll
                    for (int i = 0; i < 8; ++i) take(f[i], (v + d * PICK_THREADS) * 8 + i);
                }
        }
        if (split == splits - 1)
            for (int c = vecs * 8 + threadIdx.x; c < vocab; c += PICK_THREADS) take(__bfloat162float(row[c]), c);
    } else {                                                // rows that start off a 16-byte boundary
        const int lo = (int)((long long)vocab * split / splits), hi = (int)((long long)vocab * (split + 1) / splits);
        for (int c = lo + threadIdx.x; c < hi; c += PICK_THREADS) take(__bfloat162float(row[c]), c);
    }
    best = warp_pick(best);
    if ((threadIdx.x & 31) == 0) warp_best[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x < 32) {
        best = warp_pick(threadIdx.x < PICK_THREADS / 32 ? warp_best[threadIdx.x] : Pick{-INFINITY, 0x7fffffff});
        if (threadIdx.x == 0) {
            if (splits == 1) out[row_id] = best.c; else cta_best = best;
        }
    }
    if (splits == 1) return;
    cluster_sync_all();
    if (split == 0 && threadIdx.x < 32) {
        Pick other = {-INFINITY, 0x7fffffff};
        if ((int)threadIdx.x < splits) {
            const uint32_t at = dsmem_addr(smem_u32(&cta_best), threadIdx.x);
            other.v = ld_dsmem_f32(at);
            other.c = __float_as_int(ld_dsmem_f32(at + 4));
        }
        other = warp_pick(other);
        if (threadIdx.x == 0) out[row_id] = other.c;
    }
    __syncwarp();
    cluster_sync_all();                                         // nobody leaves while CTA 0 reads
}

// CTAs per row: as many of 1, 2, 4, 8 as fit the GPU in one wave (four CTAs of 512 threads per SM), and at least 4096 columns each.
static int pick_splits(int rows, int vocab) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int s = 1;
    while (s < 8 && (long long)rows * s * 2 <= 4LL * sms && vocab / (s * 2) >= 4096) s *= 2;
    return s;
}

cudaError_t launch_sample(const __nv_bfloat16* logits, int* out, int rows, int vocab, long long row_stride, float temperature,
                          unsigned int seed, const int* positions, cudaStream_t stream) {
    if (rows <= 0 || vocab <= 0 || !(temperature > 0.f)) return cudaErrorInvalidValue;
    const int s = pick_splits(rows, vocab);
    return launch_pdl_cluster(pick_kernel<true>, dim3(rows, 1, s), dim3(PICK_THREADS), 0, stream, s, logits, out, vocab, row_stride, 1.0f / temperature, seed, positions);
}

cudaError_t launch_argmax(const __nv_bfloat16* logits, int* out, int rows, int vocab, long long row_stride, cudaStream_t stream) {
    if (rows <= 0 || vocab <= 0) return cudaErrorInvalidValue;
    const int s = pick_splits(rows, vocab);
    return launch_pdl_cluster(pick_kernel<false>, dim3(rows, 1, s), dim3(PICK_THREADS), 0, stream, s, logits, out, vocab, row_stride, 1.0f, 0u, (const int*)nullptr);
}

// The state of a decode batch between two steps: a few hundred bytes, so these are launches and nothing else; one each, where three
// element-wise kernels and two copies took 1.5 us apiece with gaps as long between them.
__global__ void __launch_bounds__(256) advance_kernel(const int* __restrict__ next_ids, int* ids, int* positions, int* ctx_lens, int n) {
    pdl_trigger();
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    ids[i] = next_ids[i];
    positions[i] += 1;
    ctx_lens[i] += 1;
}
cudaError_t launch_advance(const int* next_ids, int* ids, int* positions, int* ctx_lens, int n, cudaStream_t stream) {
    if (n < 1) return cudaErrorInvalidValue;
    return launch_pdl(advance_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, next_ids, ids, positions, ctx_lens, n);
}

__global__ void __launch_bounds__(256) ctx_from_positions_kernel(const int* __restrict__ positions, int* __restrict__ ctx_lens, int n) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) ctx_lens[i] = positions[i] + 1;
}
cudaError_t launch_step_inputs(const int* host_ids, const int* host_positions, int* ids, int* positions, int* ctx_lens, int n, cudaStream_t stream) {
    if (n < 1) return cudaErrorInvalidValue;
    if (cudaError_t e = cudaMemcpyAsync(ids, host_ids, (size_t)n * 4, cudaMemcpyHostToDevice, stream); e != cudaSuccess) return e;
    if (cudaError_t e = cudaMemcpyAsync(positions, host_positions, (size_t)n * 4, cudaMemcpyHostToDevice, stream); e != cudaSuccess) return e;
    ctx_from_positions_kernel<<<(n + 255) / 256, 256, 0, stream>>>(positions, ctx_lens, n);
    return cudaGetLastError();
}

}  // namespace sky
