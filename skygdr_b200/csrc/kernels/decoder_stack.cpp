// The layer stack of a decoder, driven from C++: one call per prefill instead of eight Python calls per layer.
//
// A prefill of a short prompt is a few dozen kernels of ten to forty microseconds; issued op by op from Python it left the GPU idle
// two thirds of the time (77 tokens, 8 layers of Qwen3-8B: 2240 us a pass for 760 us of kernels). Here a launch costs the host two
// to three microseconds, the pieces of a pass reach the GPU as kernel arguments, and nothing waits for the device.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "common_host.h"
#include "decode_gemm.h"
#include "fused_ops.h"
#include "gemm_tcgen05.h"
#include "paged_attn.h"
#include "prefill_attn.h"

namespace py = pybind11;
using namespace sky;

namespace {

#define STACK_CHECK(expr)                                                                       \
    do {                                                                                        \
        cudaError_t _e = (expr);                                                                \
        TORCH_CHECK(_e == cudaSuccess, #expr, " failed: ", cudaGetErrorString(_e));             \
    } while (0)

__nv_bfloat16* bf(const torch::Tensor& t) { return reinterpret_cast<__nv_bfloat16*>(t.data_ptr()); }

// How a projection runs: (token tile, splits, splits as a cluster, persistent form), as chosen by ops.gemm.
struct GemmChoice { int ntok, splits, cluster, persistent; };
using Choice = std::tuple<int, int, int, int>;

struct Layer { torch::Tensor qkv, o, gate_up, down, ln1, ln2, q_norm, k_norm; };

// One piece of a prompt in a pass: (sequence, first token, end token).
using Piece = std::tuple<int, int, int>;

class DecoderStack {
public:
    DecoderStack(std::vector<std::vector<torch::Tensor>> layers, torch::Tensor embed, torch::Tensor final_norm, torch::Tensor inv_freq, int q_heads,
                 int kv_heads, int ffn, double eps)
        : embed_(embed), final_norm_(final_norm), inv_freq_(inv_freq), q_heads_(q_heads), kv_heads_(kv_heads), ffn_(ffn), eps_((float)eps) {
        hidden_ = (int)embed.size(1);
        qkv_cols_ = (q_heads + 2 * kv_heads) * 128;
        for (auto& l : layers) {
            TORCH_CHECK(l.size() == 8, "qkv, o, gate_up, down, ln1, ln2, q_norm, k_norm");
            layers_.push_back({l[0], l[1], l[2], l[3], l[4], l[5], l[6], l[7]});
        }
    }

    // Whether the weights are what the kernels take: contiguous bf16 of the fused shapes, on one GPU. Asked before every pass, since a
    // tensor's storage and strides can be exchanged under its holder; 70 tensors take a microsecond.
    bool fits() const {
        if (!embed_.is_cuda() || embed_.dim() != 2) return false;
        auto ok = [&](const torch::Tensor& t, at::IntArrayRef shape) {
            return t.is_cuda() && t.device() == embed_.device() && t.scalar_type() == torch::kBFloat16 && t.is_contiguous() && t.sizes() == shape;
        };
        const int64_t h = hidden_, q = q_heads_ * 128LL, f = ffn_;
        bool all = ok(embed_, {embed_.size(0), h}) && ok(final_norm_, {h}) && inv_freq_.is_cuda() && inv_freq_.device() == embed_.device() &&
                   inv_freq_.scalar_type() == torch::kFloat32 && inv_freq_.is_contiguous() && inv_freq_.numel() == 64;
        for (auto& l : layers_)
            all = all && ok(l.qkv, {(int64_t)qkv_cols_, h}) && ok(l.o, {h, q}) && ok(l.gate_up, {2 * f, h}) && ok(l.down, {h, f}) && ok(l.ln1, {h}) &&
                  ok(l.ln2, {h}) && ok(l.q_norm, {128}) && ok(l.k_norm, {128});
        return all;
    }

    // Runs the passes and returns the normed hidden state of every prompt's last token, [sequences][hidden].
    //   starts: first token of each sequence in ids; lens: its length; passes: pieces, each pass with the choices of its four
    //   projections (QKV, O, gate/up, down); pool: the K/V pool, its base and element strides (block, layer, kv, head, token).
    torch::Tensor prefill(torch::Tensor ids, std::vector<int> starts, std::vector<int> lens, std::vector<std::vector<Piece>> passes,
                          std::vector<std::vector<Choice>> choices, torch::Tensor block_table, torch::Tensor pool, std::vector<int64_t> strides,
                          torch::Tensor workspace, torch::Tensor counters, torch::Tensor gemm_status, torch::Tensor attn_status) {
        c10::cuda::CUDAGuard guard(embed_.device());
        auto stream = at::cuda::getCurrentCUDAStream().stream();
        TORCH_CHECK(ids.is_cuda() && ids.is_contiguous() && (ids.scalar_type() == torch::kInt64 || ids.scalar_type() == torch::kInt32), "ids: contiguous CUDA int64 or int32");
        TORCH_CHECK(block_table.is_cuda() && block_table.is_contiguous() && block_table.scalar_type() == torch::kInt32 && block_table.dim() == 2 &&
                    block_table.size(0) >= (int64_t)lens.size(), "block_table: contiguous CUDA int32, a row per sequence");
        TORCH_CHECK(pool.is_cuda() && pool.scalar_type() == torch::kBFloat16 && strides.size() == 5 && passes.size() == choices.size(), "pool / passes");
        for (size_t s = 0; s < lens.size(); ++s) TORCH_CHECK(lens[s] >= 1 && starts[s] >= 0 && (int64_t)starts[s] + lens[s] <= ids.numel(), "prompts outside ids");
        auto opt = embed_.options();
        auto out = torch::empty({(int64_t)lens.size(), hidden_}, opt);
        int64_t most = 0, pieces_most = 0;
        for (auto& pass : passes) {
            int64_t t = 0;
            for (auto& [s, b, e] : pass) {
                TORCH_CHECK(s >= 0 && s < (int)lens.size() && b >= 0 && b < e && e <= lens[s], "piece outside its prompt");
                TORCH_CHECK((e + 15) / 16 <= block_table.size(1), "a block-table row does not cover the prompt");
                t += e - b;
            }
            most = std::max(most, t);
            pieces_most = std::max(pieces_most, (int64_t)pass.size());
        }
        auto resid = torch::empty({most, hidden_}, opt), xn = torch::empty({most, hidden_}, opt), h = torch::empty({most, hidden_}, opt);
        auto qkv = torch::empty({most, qkv_cols_}, opt), q = torch::empty({most, q_heads_ * 128}, opt), ao = torch::empty_like(q);
        auto act = torch::empty({most, ffn_}, opt);
        auto idx = torch::empty({2 * most + 3 * pieces_most + 1}, opt.dtype(torch::kInt32));
        int* positions = idx.data_ptr<int>();
        int* tok_rows = positions + most;
        int* seq_start = tok_rows + most;
        int* pos0 = seq_start + pieces_most + 1;
        int* rows = pos0 + pieces_most;
        const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
        PrefillSetup setup{ids.data_ptr(), ids.scalar_type() == torch::kInt64, bf(embed_), (int)embed_.size(0), hidden_, bf(resid), positions, tok_rows, seq_start, pos0, rows};

        for (size_t i = 0; i < passes.size(); ++i) {
            const auto& pass = passes[i];
            int T = 0, longest = 0;
            PrefillPieces pc;
            pc.n = 0; pc.first = 0;
            for (size_t k = 0; k < pass.size(); ++k) {
                auto [s, b, e] = pass[k];
                pc.tok0[pc.n] = T; pc.src[pc.n] = starts[s] + b; pc.pos0[pc.n] = b; pc.row[pc.n] = s;
                T += e - b;
                longest = std::max(longest, e - b);
                pc.tok0[++pc.n] = T;
                if (pc.n == PREFILL_PIECES_MAX || k + 1 == pass.size()) {
                    STACK_CHECK(launch_prefill_setup(setup, pc, stream));
                    pc.first = (int)k + 1;
                    pc.n = 0;
                }
            }
            if (T == 0) continue;
            RopeAppendParams r;
            memset(&r, 0, sizeof r);
            r.qkv = bf(qkv); r.q_out = bf(q);
            r.inv_freq = inv_freq_.data_ptr<float>(); r.block_table = block_table.data_ptr<int>(); r.positions = positions; r.seq_ids = tok_rows;
            r.block_stride = strides[0]; r.kv_stride = strides[2]; r.head_stride = strides[3]; r.tok_stride = strides[4];
            r.tokens = T; r.q_heads = q_heads_; r.kv_heads = kv_heads_; r.max_blocks = (int)block_table.size(1); r.block_tokens = 16; r.eps = eps_;
            auto attention = [&](size_t li) {
                const __nv_bfloat16* layer_base = bf(pool) + (int64_t)li * strides[1];
                PrefillAttnParams a;
                memset(&a, 0, sizeof a);
                a.q = bf(q); a.kv = layer_base; a.out = bf(ao); a.block_table = block_table.data_ptr<int>(); a.seq_start = seq_start;
                a.block_stride = strides[0]; a.kv_stride = strides[2]; a.head_stride = strides[3]; a.tok_stride = strides[4];
                a.n_seqs = (int)pass.size(); a.q_heads = q_heads_; a.kv_heads = kv_heads_; a.max_blocks = (int)block_table.size(1);
                a.max_len = longest; a.total_tokens = T; a.scale = 1.0f / std::sqrt(128.0f); a.pos0 = pos0; a.seq_rows = rows;
                a.status = reinterpret_cast<LaunchStatus*>(attn_status.data_ptr());
                STACK_CHECK(launch_prefill_attn_tc(a, (pool.numel() - (int64_t)li * strides[1]) / 128, stream));
            };
            // Passes of few tokens take the projections of a decode step: QK-norm, rotary embedding and cache append in the epilogue of QKV.
            // The norms stay kernels of their own here: with them in the epilogues too (16 launches of 3 us less at 8 layers) the
            // rounding of every projection's input differs from the longer passes', and K and V of one prompt should not
            // depend on how it was cut into passes.
            const bool few = T <= DECODE_GEMM_MAX_ROWS && hidden_ % 64 == 0 && ffn_ % 64 == 0;
            auto status = reinterpret_cast<LaunchStatus*>(gemm_status.data_ptr());
            TORCH_CHECK(choices[i].size() == 4, "a choice for each of the four projections");
            auto projection = [&](const __nv_bfloat16* x, const torch::Tensor& w, __nv_bfloat16* y, int N, int K, bool gated, int which) {
                if (!few) return gemm(x, T, K, w, y, N, gated, choices[i][which], workspace, counters, gemm_status, stream);
                DecodeGemmParams p = project_base(T, 0, status);
                p.mode = DG_STORE; p.y = y; p.ldy = N;
                project(p, x, w, N, K, 0, gated, sms, stream);
            };
            for (size_t li = 0; li < layers_.size(); ++li) {
                const Layer& l = layers_[li];
                STACK_CHECK(launch_rmsnorm(li ? bf(h) : bf(resid), li ? bf(resid) : nullptr, bf(l.ln1), bf(xn), T, hidden_, eps_, stream));
                r.q_norm = bf(l.q_norm); r.k_norm = bf(l.k_norm); r.kv = bf(pool) + (int64_t)li * strides[1];
                if (few) {
                    DecodeGemmParams p = project_base(T, 0, status);
                    p.mode = DG_QKV; p.rope = r; p.round_product = 1;
                    project(p, bf(xn), l.qkv, qkv_cols_, hidden_, 0, false, sms, stream);
                } else {
                    projection(bf(xn), l.qkv, bf(qkv), qkv_cols_, hidden_, false, 0);
                    STACK_CHECK(launch_rope_append(r, stream));
                }
                attention(li);
                projection(bf(ao), l.o, bf(h), hidden_, q_heads_ * 128, false, 1);
                STACK_CHECK(launch_rmsnorm(bf(h), bf(resid), bf(l.ln2), bf(xn), T, hidden_, eps_, stream));
                projection(bf(xn), l.gate_up, bf(act), ffn_, hidden_, true, 2);
                projection(bf(act), l.down, bf(h), hidden_, ffn_, false, 3);
            }
            RowMap rm;                                     // prompts that end in this pass: their last row, normed
            rm.n = 0;
            int at = 0;
            for (size_t k = 0; k < pass.size(); ++k) {
                auto [s, b, e] = pass[k];
                at += e - b;
                if (e == lens[s]) { rm.src[rm.n] = at - 1; rm.dst[rm.n++] = s; }
                if (rm.n == ROW_MAP_MAX || (k + 1 == pass.size() && rm.n > 0)) {
                    STACK_CHECK(launch_rmsnorm_rows(bf(h), bf(resid), bf(final_norm_), bf(out), rm, hidden_, eps_, stream));
                    rm.n = 0;
                }
            }
        }
        return out;
    }

    // One decode step of the first `rows` slots up to the logits: an embedding gather, per layer QKV, attention, O, gate/up and down with the
    // norms, the rotary embedding and the cache append in their epilogues (decode_gemm.cu), and the output projection.
    //   splits: K slices of the five projections (QKV, O, gate/up, down, output), 0 = by the rule of decode_gemm.cu.
    void decode(int rows, torch::Tensor ids, torch::Tensor positions, torch::Tensor ctx_lens, torch::Tensor block_table, torch::Tensor resid, torch::Tensor xg,
                torch::Tensor ss, torch::Tensor q, torch::Tensor ao, torch::Tensor act, torch::Tensor lm_head, torch::Tensor logits, torch::Tensor pool,
                std::vector<int64_t> strides, int max_ctx, int chunk_tokens, bool tensor_cores, torch::Tensor part_o, torch::Tensor part_m, torch::Tensor part_l,
                torch::Tensor counters, torch::Tensor attn_status, torch::Tensor gemm_status, std::vector<int> splits) {
        c10::cuda::CUDAGuard guard(embed_.device());
        auto stream = at::cuda::getCurrentCUDAStream().stream();
        const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
        TORCH_CHECK(rows >= 1 && rows <= DECODE_GEMM_MAX_ROWS && hidden_ % 128 == 0 && splits.size() == 5 && strides.size() == 4, "decode: up to 256 rows, hidden a multiple of 128");
        for (auto& t : {ids, positions, ctx_lens, block_table}) TORCH_CHECK(t.is_cuda() && t.scalar_type() == torch::kInt32 && t.is_contiguous(), "indexes: contiguous CUDA int32");
        for (auto& t : {resid, xg, q, ao, act, logits, lm_head}) TORCH_CHECK(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.is_contiguous(), "activations: contiguous CUDA bf16");
        TORCH_CHECK(resid.size(0) >= rows && xg.size(0) >= rows && q.size(0) >= rows && ao.size(0) >= rows && act.size(0) >= rows && logits.size(0) >= rows &&
                    ids.numel() >= rows && positions.numel() >= rows && ctx_lens.numel() >= rows && block_table.size(0) >= rows, "buffers smaller than the batch");
        TORCH_CHECK(lm_head.size(1) == hidden_ && logits.size(1) == lm_head.size(0) && resid.size(1) == hidden_ && act.size(1) == ffn_, "shapes");
        const int tiles = hidden_ / 128, pitch = (int)ss.size(1);
        TORCH_CHECK(ss.is_cuda() && ss.scalar_type() == torch::kFloat32 && ss.is_contiguous() && ss.size(0) >= 2 * tiles && pitch >= rows, "ss: two blocks of hidden / 128 rows");
        TORCH_CHECK((int64_t)max_ctx <= block_table.size(1) * 16, "max_ctx = ", max_ctx, " but a block-table row covers ", block_table.size(1) * 16, " tokens");
        const int max_splits = (int)part_m.size(2);
        TORCH_CHECK(part_o.numel() >= (int64_t)rows * q_heads_ * max_splits * 128 && counters.numel() >= (int64_t)rows * kv_heads_, "attention scratch too small");
        STACK_CHECK(launch_embed_norm(ids.data_ptr<int>(), bf(embed_), (int)embed_.size(0), hidden_, rows, bf(layers_[0].ln1), bf(resid), bf(xg), ss.data_ptr<float>(), stream));
        RopeAppendParams r;
        memset(&r, 0, sizeof r);
        r.q_out = bf(q);
        r.inv_freq = inv_freq_.data_ptr<float>(); r.block_table = block_table.data_ptr<int>(); r.positions = positions.data_ptr<int>();
        r.block_stride = strides[0]; r.kv_stride = strides[2]; r.head_stride = strides[3]; r.tok_stride = 128;
        r.tokens = rows; r.q_heads = q_heads_; r.kv_heads = kv_heads_; r.max_blocks = (int)block_table.size(1); r.block_tokens = 16; r.eps = eps_;
        auto status = reinterpret_cast<LaunchStatus*>(gemm_status.data_ptr());
        FusedRows f{rows, pitch, bf(resid), bf(xg), bf(q), bf(ao), bf(act), ss.data_ptr<float>()};
        const int n_ss = fused_layers(f, r, bf(pool), strides[1], status, splits, sms, stream, [&](size_t li) {
            PagedAttnParams a;
            memset(&a, 0, sizeof a);
            a.q = bf(q); a.kv = bf(pool) + (int64_t)li * strides[1]; a.out = bf(ao); a.block_table = r.block_table; a.ctx_lens = ctx_lens.data_ptr<int>();
            a.block_stride = strides[0]; a.kv_stride = strides[2]; a.head_stride = strides[3];
            a.batch = rows; a.q_heads = q_heads_; a.kv_heads = kv_heads_; a.head_dim = 128; a.block_tokens = 16; a.max_blocks = r.max_blocks;
            a.num_blocks = (int)pool.size(0); a.max_ctx = max_ctx; a.chunk_tokens = chunk_tokens; a.scale = 1.0f / std::sqrt(128.0f); a.max_splits = max_splits;
            a.part_o = part_o.data_ptr<float>(); a.part_m = part_m.data_ptr<float>(); a.part_l = part_l.data_ptr<float>();
            a.counters = reinterpret_cast<unsigned int*>(counters.data_ptr());
            a.status = reinterpret_cast<LaunchStatus*>(attn_status.data_ptr());
            STACK_CHECK(tensor_cores ? launch_paged_attn_decode_tc(a, (pool.numel() - (int64_t)li * strides[1]) / 128, stream) : launch_paged_attn_decode(a, stream));
        });
        DecodeGemmParams p = project_base(f.n, f.pitch, status);
        p.mode = DG_STORE; p.ss_in = f.ss; p.n_ss = n_ss; p.y = bf(logits); p.ldy = logits.size(1);
        project(p, f.xg, lm_head, (int)lm_head.size(0), hidden_, splits[4], false, sms, stream);
    }

private:
    // The rows of a pass of at most DECODE_GEMM_MAX_ROWS tokens and the scratch that its layers share. ss: partial sums of squares, [2][hidden / 128]
    // [pitch]: first those of the rows that QKV and the output projection read, then those that gate/up reads.
    struct FusedRows { int n, pitch; __nv_bfloat16 *resid, *xg, *q, *ao, *act; float* ss; };

    DecodeGemmParams project_base(int rows, int pitch, LaunchStatus* status) const {
        DecodeGemmParams p;
        memset(&p, 0, sizeof p);
        p.M = rows; p.ss_pitch = pitch; p.norm_dim = hidden_; p.eps = eps_; p.status = status;
        return p;
    }
    void project(DecodeGemmParams& p, const __nv_bfloat16* x, const torch::Tensor& w, int N, int K, int splits, bool gated, int sms, cudaStream_t stream) const {
        p.x = x; p.w = bf(w); p.N = N; p.K = K; p.gated = gated;
        p.splits = splits > 0 ? splits : decode_gemm_splits(p.M, N, K, gated, sms);
        STACK_CHECK(launch_decode_gemm(p, stream));
    }
    // All layers over rows whose embedding (resid, and xg = resid * first gain, and one sum of squares per row) is in place; attention(layer)
    // launches the attention of q into ao. Returns the number of partial sums per row that the output projection finds in f.ss.
    template <typename Attention>
    int fused_layers(const FusedRows& f, RopeAppendParams rope, __nv_bfloat16* pool, int64_t layer_stride, LaunchStatus* status, const std::vector<int>& splits,
                     int sms, cudaStream_t stream, Attention attention) const {
        const int tiles = hidden_ / 128;
        float *ss_attn = f.ss, *ss_mlp = f.ss + (int64_t)tiles * f.pitch;
        for (size_t li = 0; li < layers_.size(); ++li) {
            const Layer& l = layers_[li];
            DecodeGemmParams p = project_base(f.n, f.pitch, status);
            p.mode = DG_QKV; p.ss_in = ss_attn; p.n_ss = li ? tiles : 1;
            p.rope = rope;
            p.rope.q_norm = bf(l.q_norm); p.rope.k_norm = bf(l.k_norm); p.rope.kv = pool + (int64_t)li * layer_stride;
            project(p, f.xg, l.qkv, qkv_cols_, hidden_, splits[0], false, sms, stream);
            attention(li);
            p = project_base(f.n, f.pitch, status);
            p.mode = DG_RESID; p.resid = f.resid; p.xg = f.xg; p.gain = bf(l.ln2); p.ss_out = ss_mlp;
            project(p, f.ao, l.o, hidden_, q_heads_ * 128, splits[1], false, sms, stream);
            p = project_base(f.n, f.pitch, status);
            p.mode = DG_STORE; p.ss_in = ss_mlp; p.n_ss = tiles; p.y = f.act; p.ldy = ffn_;
            project(p, f.xg, l.gate_up, ffn_, hidden_, splits[2], true, sms, stream);
            p = project_base(f.n, f.pitch, status);
            p.mode = DG_RESID; p.resid = f.resid; p.xg = f.xg; p.gain = li + 1 < layers_.size() ? bf(layers_[li + 1].ln1) : bf(final_norm_); p.ss_out = ss_attn;
            project(p, f.act, l.down, hidden_, ffn_, splits[3], false, sms, stream);
        }
        return tiles;
    }

    void gemm(const __nv_bfloat16* x, int M, int K, const torch::Tensor& w, __nv_bfloat16* y, int N, bool gated, const Choice& c,
              const torch::Tensor& workspace, const torch::Tensor& counters, const torch::Tensor& status, cudaStream_t stream) {
        GemmParams p;
        memset(&p, 0, sizeof p);
        p.x = x; p.w = bf(w); p.y = y; p.M = M; p.N = N; p.K = K; p.ldx = K; p.ldw = K; p.ldy = N;
        p.ntok = std::get<0>(c); p.splits = std::get<1>(c); p.cluster_split = std::get<2>(c); p.persistent = std::get<3>(c); p.gated = gated;
        if (p.splits > 1 && !p.cluster_split) {
            TORCH_CHECK((size_t)workspace.numel() >= gemm_workspace_floats(M, N, p.splits, gated, p.ntok) &&
                        (size_t)counters.numel() >= gemm_counter_count(M, N, gated, p.ntok), "split-K scratch too small");
            p.workspace = workspace.data_ptr<float>();
            p.counters = reinterpret_cast<unsigned int*>(counters.data_ptr());
        }
        p.status = reinterpret_cast<LaunchStatus*>(status.data_ptr());
        STACK_CHECK(launch_gemm(p, stream));
    }

    std::vector<Layer> layers_;
    torch::Tensor embed_, final_norm_, inv_freq_;
    int hidden_, q_heads_, kv_heads_, ffn_, qkv_cols_;
    float eps_;
};

}  // namespace

void bind_decoder_stack(py::module_& m) {
    py::class_<DecoderStack>(m, "DecoderStack")
        .def(py::init<std::vector<std::vector<torch::Tensor>>, torch::Tensor, torch::Tensor, torch::Tensor, int, int, int, double>(), py::arg("layers"),
             py::arg("embed"), py::arg("final_norm"), py::arg("inv_freq"), py::arg("q_heads"), py::arg("kv_heads"), py::arg("ffn"), py::arg("eps"))
        .def("fits", &DecoderStack::fits)
        .def("prefill", &DecoderStack::prefill, py::call_guard<py::gil_scoped_release>(), py::arg("ids"), py::arg("starts"), py::arg("lens"), py::arg("passes"),
             py::arg("choices"), py::arg("block_table"), py::arg("pool"), py::arg("strides"), py::arg("workspace"), py::arg("counters"),
             py::arg("gemm_status"), py::arg("attn_status"))
        .def("decode", &DecoderStack::decode, py::call_guard<py::gil_scoped_release>(), py::arg("rows"), py::arg("ids"), py::arg("positions"),
             py::arg("ctx_lens"), py::arg("block_table"), py::arg("resid"), py::arg("xg"), py::arg("ss"), py::arg("q"), py::arg("ao"), py::arg("act"),
             py::arg("lm_head"), py::arg("logits"), py::arg("pool"), py::arg("strides"), py::arg("max_ctx"), py::arg("chunk_tokens"),
             py::arg("tensor_cores"), py::arg("part_o"), py::arg("part_m"), py::arg("part_l"), py::arg("counters"), py::arg("attn_status"),
             py::arg("gemm_status"), py::arg("splits"));
}
