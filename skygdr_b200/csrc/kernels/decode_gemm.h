// Host-visible interface of the decode projections (decode_gemm.cu): y = x w^T for up to 256 token rows, fused with what a decoder
// layer does next to a projection.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "fused_ops.h"

namespace sky {
struct LaunchStatus;

// What happens to the product of a tile.
enum DecodeGemmMode {
    DG_STORE = 0,      // y = product (gated: silu(gate) * up)
    DG_RESID = 1,      // resid += product; xg = resid * gain; ss_out = partial sums of squares of resid: the residual add and the RMSNorm that
                       // follow the O and down projections (the next projection divides by the root mean square, see ss_in)
    DG_QKV = 2,        // a tile is one head: QK-norm, rotary embedding, q -> q_out, k and v -> paged cache
};

struct DecodeGemmParams {
    const __nv_bfloat16* x;      // [M][K]
    const __nv_bfloat16* w;      // [N][K]; gated: [2N][K], gate rows then up rows
    int M, N, K;
    int gated, mode;
    int splits;                  // CTAs along K of a tile, one thread-block cluster (1-8)
    // RMSNorm of x, applied to the product: row t is multiplied by rsqrt(sum_i ss_in[i * ss_pitch + t] / norm_dim + eps)
    const float* ss_in;          // nullptr: x is taken as it is
    int n_ss, ss_pitch, norm_dim;
    float eps;
    // DG_STORE
    __nv_bfloat16* y;
    long long ldy;
    // DG_RESID ([M][N] rows, N % 128 == 0)
    __nv_bfloat16* resid;
    __nv_bfloat16* xg;
    const __nv_bfloat16* gain;
    float* ss_out;               // [N / 128][ss_pitch]
    // DG_QKV (N = (q_heads + 2 kv_heads) * 128)
    RopeAppendParams rope;       // qkv is not used
    int round_product;           // round the product to bf16 before the norm, as a projection that stores it would
    LaunchStatus* status;
};

constexpr int DECODE_GEMM_MAX_ROWS = 256;
// Splits for a shape (see the rule in decode_gemm.cu).
int decode_gemm_splits(int M, int N, int K, bool gated, int sms);
cudaError_t launch_decode_gemm(const DecodeGemmParams& p, cudaStream_t stream);

// The start of a decode step: resid = embed[ids], xg = resid * gain, ss[t] = sum of squares of row t (one partial per row).
cudaError_t launch_embed_norm(const int* ids, const __nv_bfloat16* table, int vocab, int hidden, int tokens, const __nv_bfloat16* gain, __nv_bfloat16* resid,
                              __nv_bfloat16* xg, float* ss, cudaStream_t stream);
}  // namespace sky
