// QK-norm + rotary embedding + append to the paged cache of one 128-wide head row, held by one warp: lane L has dims 4L .. 4L + 3.
#pragma once
#include "common.cuh"
#include "fused_ops.h"

namespace sky {

// cos and sin of position * inv_freq for the four dims of a lane. The angle is formed in fp32, as the usual eager implementation
// does, and reduced to [-pi, pi] by the two-constant method of Cody and Waite: 2 pi = hi + lo with hi the nearest float, so that
// angle - k hi is exact (a multiple of 2^-21 below 4 for angles into the millions) and the second step adds one rounding. The fast
// sincos is then in its accurate range.
__device__ __forceinline__ void rope_angles(int pos, const float* inv_freq, int lane, float* cs, float* sn) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(inv_freq) + (lane & 15));
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

// x: the lane's four values of head row `h` of token `tok` (q heads, then k heads, then v heads); blk: the block of its position.
// Rotation pairs dim i with dim i + 64, i.e. lane L with lane L ^ 16.
__device__ __forceinline__ void rope_append_row(const RopeAppendParams& p, int tok, int h, int lane, float* x, int pos, int blk,
                                                const float* cs, const float* sn) {
    const bool is_q = h < p.q_heads, is_k = !is_q && h < p.q_heads + p.kv_heads;
    if (is_q || is_k) {
        const __nv_bfloat16* nw = is_q ? p.q_norm : p.k_norm;
        if (nw) {
            const uint2 wr = __ldg(reinterpret_cast<const uint2*>(nw + lane * 4));
            float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
            for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float inv = rsqrtf(ss * (1.0f / 128.0f) + p.eps);
            const float g[4] = {__uint_as_float(wr.x << 16), __uint_as_float(wr.x & 0xffff0000u), __uint_as_float(wr.y << 16),
                                __uint_as_float(wr.y & 0xffff0000u)};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                // round to bf16 like a separate norm kernel would, so results match a layer-by-layer reference
                x[i] = __bfloat162float(__float2bfloat16(x[i] * inv * g[i]));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, x[i], 16);
            x[i] = lane < 16 ? x[i] * cs[i] - other * sn[i] : x[i] * cs[i] + other * sn[i];
        }
    }
    const __nv_bfloat162 a = __floats2bfloat162_rn(x[0], x[1]), b = __floats2bfloat162_rn(x[2], x[3]);
    const uint2 outv = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    if (is_q) {
        *reinterpret_cast<uint2*>(p.q_out + ((long long)tok * p.q_heads + h) * 128 + lane * 4) = outv;
    } else {
        const int kvh = is_k ? h - p.q_heads : h - p.q_heads - p.kv_heads;
        __nv_bfloat16* dst = p.kv + (long long)blk * p.block_stride + (is_k ? 0 : p.kv_stride) + (long long)kvh * p.head_stride +
                             (long long)(pos % p.block_tokens) * p.tok_stride + lane * 4;
        *reinterpret_cast<uint2*>(dst) = outv;
    }
}

}  // namespace sky
