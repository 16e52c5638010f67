// QK-norm + rotary embedding + append to the paged cache of one 128-wide head row, held by one warp: lane L has dims 4L .. 4L + 3.
#pragma once
#include "common.cuh"
#include "fused_ops.h"

namespace sky {

// cos and sin of position * inv_freq for the four dims of a lane. The angle is formed in fp32, as the usual eager implementation
// does, and reduced to [-pi, pi] by the two-constant method of Cody and Waite: 2 pi = hi + lo with hi the nearest float, so that
// angle - k hi is exact (a multiple of 2^-21 below 4 for angles into the millions) and the second step adds one rounding. The fast
// sincos is then in its accurate range.
__device__ __forceinline__ void rope_angles(int pos, float4 f, float* cs, float* sn) {
    const float fr[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float ang = __fmul_rn((float)pos, fr[i]);
        const float k = rintf(ang * 0.15915494309189535f);
        float a = __fmaf_rn(-k, 6.2831854820251465f, ang);
        a = __fmaf_rn(-k, -1.7484555e-7f, a);
        __sincosf(a, &sn[i], &cs[i]);
    }
}

__device__ __forceinline__ float4 rope_freqs(const float* inv_freq, int lane) {
    const float* f = inv_freq + (lane & 15) * 4;
    return make_float4(__ldg(f), __ldg(f + 1), __ldg(f + 2), __ldg(f + 3));
}

__device__ __forceinline__ void rope_unpack(uint2 v, float* f) {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
}

// RMSNorm of U head rows at once (their shuffles overlap); x[u]: the lane's four values. Rounded to bf16 like a separate norm kernel
// would, so results match a layer-by-layer reference.
template <int U>
__device__ __forceinline__ void rope_norm_rows(const __nv_bfloat16* weight, float eps, int lane, float (*x)[4]) {
    const uint2 wr = __ldg(reinterpret_cast<const uint2*>(weight + lane * 4));
    const float g[4] = {__uint_as_float(wr.x << 16), __uint_as_float(wr.x & 0xffff0000u), __uint_as_float(wr.y << 16), __uint_as_float(wr.y & 0xffff0000u)};
    float ss[U];
#pragma unroll
    for (int u = 0; u < U; ++u) ss[u] = x[u][0] * x[u][0] + x[u][1] * x[u][1] + x[u][2] * x[u][2] + x[u][3] * x[u][3];
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int u = 0; u < U; ++u) ss[u] += __shfl_xor_sync(0xffffffffu, ss[u], o);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const float inv = rsqrtf(ss[u] * (1.0f / 128.0f) + eps);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[u][i] = __bfloat162float(__float2bfloat16(x[u][i] * inv * g[i]));
    }
}

// Rotation pairs dim i with dim i + 64, i.e. lane L with lane L ^ 16.
__device__ __forceinline__ void rope_rotate(int lane, float* x, const float* cs, const float* sn) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, x[i], 16);
        x[i] = lane < 16 ? x[i] * cs[i] - other * sn[i] : x[i] * cs[i] + other * sn[i];
    }
}

// Head row h (q heads, then k heads, then v heads) of token tok at position pos, whose block is blk.
__device__ __forceinline__ void rope_store(const RopeAppendParams& p, int tok, int h, int lane, const float* x, int pos, int blk) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x[0], x[1]), b = __floats2bfloat162_rn(x[2], x[3]);
    const uint2 outv = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    if (h < p.q_heads) {
        *reinterpret_cast<uint2*>(p.q_out + ((long long)tok * p.q_heads + h) * 128 + lane * 4) = outv;
        return;
    }
    const bool is_k = h < p.q_heads + p.kv_heads;
    const int kvh = is_k ? h - p.q_heads : h - p.q_heads - p.kv_heads;
    __nv_bfloat16* dst = p.kv + (long long)blk * p.block_stride + (is_k ? 0 : p.kv_stride) + (long long)kvh * p.head_stride +
                         (long long)(pos % p.block_tokens) * p.tok_stride + lane * 4;
    *reinterpret_cast<uint2*>(dst) = outv;
}

}  // namespace sky
