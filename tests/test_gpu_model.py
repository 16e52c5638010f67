"""Qwen3 decoder on the package's kernels against a plain PyTorch forward of the same weights."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(layers=2, max_batch=4, max_ctx=256, attn_impl="simt", attn_chunk=64):
    from skygdr_b200 import ops
    from skygdr_b200.models import Qwen3Config, Qwen3Decoder, Qwen3Weights

    cfg = Qwen3Config.tiny(layers=layers)
    w = Qwen3Weights(cfg, "cuda", seed=1, std=0.05)
    pool = ops.PagedKVPool(cfg.geometry, 64, "hnd")
    eng = Qwen3Decoder(cfg, w, pool, max_batch=max_batch, max_ctx=max_ctx, attn_chunk=attn_chunk, attn_impl=attn_impl)
    return cfg, w, pool, eng


def _tables(seq_lens, max_blocks, nblocks=64, seed=0):
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(nblocks, generator=g).int()
    table = torch.zeros((len(seq_lens), max_blocks), dtype=torch.int32)
    o = 0
    for i, n in enumerate(seq_lens):
        nb = (n + 15) // 16 + 1          # one spare block for generated tokens
        table[i, :nb] = perm[o:o + nb]
        o += nb
    return table.cuda()


@pytest.mark.parametrize("attn_impl,attn_chunk", [("simt", 64), ("tc", 128)])
def test_prefill_and_decode_match_reference(attn_impl, attn_chunk):
    from skygdr_b200.models import reference_forward

    cfg, w, pool, eng = _setup(attn_impl=attn_impl, attn_chunk=attn_chunk)
    torch.manual_seed(0)
    seq_lens = [37, 16, 50]
    prompts = [torch.randint(0, cfg.vocab, (n,), device="cuda") for n in seq_lens]
    table = _tables(seq_lens, eng.max_blocks)
    logits = eng.prefill(torch.cat(prompts), seq_lens, table)
    refs = [reference_forward(cfg, w, p) for p in prompts]
    for i in range(3):
        ref_last = refs[i][-1]
        err = (logits[i].float() - ref_last).abs().max() / ref_last.abs().max()
        assert err < 0.05, float(err)
    # decode 3 steps, always feeding the reference's greedy token
    ids = torch.stack([r[-1].argmax() for r in refs]).int()
    seqs = [p.clone() for p in prompts]
    for step in range(3):
        pos = torch.tensor([s.numel() for s in seqs], dtype=torch.int32, device="cuda")
        eng.set_batch(ids, pos, table)
        eng.step(b=3, max_ctx=128, advance=False)
        seqs = [torch.cat([s, i.view(1).long()]) for s, i in zip(seqs, ids)]
        new_ids = []
        for i in range(3):
            ref = reference_forward(cfg, w, seqs[i])[-1]
            got = eng.logits[i].float()
            err = (got - ref).abs().max() / ref.abs().max()
            assert err < 0.05, (step, i, float(err))
            new_ids.append(ref.argmax())
        ids = torch.stack(new_ids).int()


@pytest.mark.parametrize("chunk,attn", [(8192, "tc"), (48, "tc"), (100, "tc"), (48, "sdpa")])
def test_prefill_with_the_native_attention_kernel_matches_reference(chunk, attn):
    """The whole prefill path without a library kernel: tcgen05 GEMMs, fused small ops, paged causal attention. With a small
    chunk the prompts go through the stack in several passes and the later pieces attend to K/V that earlier passes appended."""
    from skygdr_b200.models import reference_forward

    cfg, w, pool, eng = _setup()
    torch.manual_seed(5)
    seq_lens = [37, 128, 50, 1]
    prompts = [torch.randint(0, cfg.vocab, (n,), device="cuda") for n in seq_lens]
    table = _tables(seq_lens, eng.max_blocks)
    logits = eng.prefill(torch.cat(prompts), seq_lens, table, attn=attn, chunk=chunk)
    torch.cuda.synchronize()
    for i, pr in enumerate(prompts):
        ref_last = reference_forward(cfg, w, pr)[-1]
        err = (logits[i].float() - ref_last).abs().max() / ref_last.abs().max()
        assert err < 0.05, (i, float(err))


def test_graph_replay_equals_eager():
    cfg, w, pool, eng = _setup()
    torch.manual_seed(1)
    seq_lens = [20, 33, 5, 48]
    table = _tables(seq_lens, eng.max_blocks, seed=3)
    prompts = torch.cat([torch.randint(0, cfg.vocab, (n,), device="cuda") for n in seq_lens])
    logits = eng.prefill(prompts, seq_lens, table)
    ids = logits.float().argmax(-1).int()
    pos = torch.tensor(seq_lens, dtype=torch.int32, device="cuda")
    snapshot = pool.data.clone()
    eng.set_batch(ids, pos, table)
    eager = [eng.step(max_ctx=128).clone() for _ in range(4)]
    pool.data.copy_(snapshot)
    eng.set_batch(ids, pos, table)
    eng.capture(max_ctx=128)
    graph = [eng.replay().clone() for _ in range(4)]
    for a, b in zip(eager, graph):
        assert torch.equal(a, b)


@pytest.mark.parametrize("b,splits", [(1, 0), (15, 3), (16, 8), (17, 2), (33, 5), (64, 4), (100, 0), (128, 1), (129, 7), (256, 0)])
def test_fused_decode_step_equals_the_op_by_op_step(b, splits):
    """The projections with norms, rotary embedding and cache append in their epilogues (csrc/kernels/decode_gemm.cu) against the
    separate kernels: token counts around the MMA's multiples of 16, every cluster size, uneven slices of K, rows behind the batch."""
    from skygdr_b200 import ops
    from skygdr_b200.models import Qwen3Config, Qwen3Decoder, Qwen3Weights

    cfg = Qwen3Config.tiny(layers=2, vocab=1000)                        # 1000: the last tile of the output projection is ragged
    w = Qwen3Weights(cfg, "cuda", seed=3, std=0.05)
    cap, g = b + 3, torch.Generator(device="cuda").manual_seed(b)
    pools = [ops.PagedKVPool(cfg.geometry, 2 * cap + 1, "hnd") for _ in range(2)]
    pools[0].data.normal_(generator=g)
    pools[1].data.copy_(pools[0].data)
    ids = torch.randint(0, cfg.vocab, (b,), device="cuda", generator=g).int()
    pos = torch.randint(0, 32, (b,), device="cuda", generator=g).int()
    table = (torch.randperm(2 * cap, device="cuda", generator=g) + 1).int().view(cap, 2)[:b].contiguous()
    engs = [Qwen3Decoder(cfg, w, pool, max_batch=cap, max_ctx=32, attn_chunk=128) for pool in pools]
    engs[0]._decode_splits = [splits] * 5
    assert engs[0]._decode_stack(b) is not None
    engs[1]._decode_stack = lambda _: None
    for e in engs:
        e.logits.fill_(7.0)
        e.set_batch(ids, pos, table)
        e.step(b=b, advance=False)
        assert e.check_status() == "OK"
    got, want = engs[0].logits[:b].float(), engs[1].logits[:b].float()
    # Both sides round to bf16 (2^-9 relative at most, 2^-9 / sqrt(3) rms) at nine ops of each layer and four outside: 22 independent
    # roundings a side add up to 2^-9 sqrt(2 * 22 / 3) = 0.0075 of the norm; twice that for what a layer amplifies.
    assert ((got - want).norm() / want.norm()).item() < 0.015
    assert ((pools[0].data.float() - pools[1].data.float()).norm() / pools[1].data.float().norm()).item() < 0.015
    touched = (pools[0].data != pools[1].data).flatten(1).any(1).nonzero().flatten()
    assert set(touched.tolist()) <= set(table.flatten().tolist())
    assert bool((engs[0].logits[b:] == 7.0).all())


@pytest.mark.parametrize("lens", [[1], [17, 1, 30], [129], [200, 56], [250, 7], [256, 300]])
@pytest.mark.parametrize("layout", ["hnd", "nhd"])
def test_prefill_of_few_tokens_equals_the_op_by_op_prefill(lens, layout):
    """Passes of up to 256 tokens take the fused projections, longer ones the separate kernels (257 tokens here, and 256 + 300
    tokens in passes of 300 and 256), in both page layouts; the K and V of the prompts, and only they, are written."""
    from skygdr_b200 import ops
    from skygdr_b200.models import Qwen3Config, Qwen3Decoder, Qwen3Weights

    cfg = Qwen3Config.tiny(layers=2, vocab=1000)
    w = Qwen3Weights(cfg, "cuda", seed=4, std=0.05)
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    ids = torch.randint(0, cfg.vocab, (sum(lens),), device="cuda", generator=g)
    table = _tables(lens, 24, nblocks=80)
    out = []
    for native in (True, False):
        pool = ops.PagedKVPool(cfg.geometry, 80, layout)
        pool.data.fill_(300.0)
        eng = Qwen3Decoder(cfg, w, pool if layout == "hnd" else ops.PagedKVPool(cfg.geometry, 2, "hnd"), max_batch=1, max_ctx=64, attn_chunk=128)
        if not native:
            eng._layer_stack = lambda: None
        logits = eng.prefill(ids, lens, table, pool=pool, chunk=300)
        assert eng.check_status() == "OK"
        out.append((logits.float(), pool.data.float()))
    (got, kv), (want, kv_want) = out
    assert ((got - want).norm() / want.norm()).item() < 0.015            # as derived for the decode step above
    assert torch.equal(kv == 300.0, kv_want == 300.0)                     # the same places stay untouched (no K or V is that large)
    at = kv != 300.0
    assert ((kv - kv_want)[at].norm() / kv_want[at].norm()).item() < 0.015


def test_weights_that_the_layer_stack_does_not_take_go_op_by_op():
    """Storage exchanged under a weight tensor, of another layout: the native drivers step aside, the next layout brings them back."""
    from skygdr_b200 import ops
    from skygdr_b200.models import Qwen3Config, Qwen3Decoder, Qwen3Weights

    cfg = Qwen3Config.tiny(layers=2, vocab=1000)
    w = Qwen3Weights(cfg, "cuda", seed=4, std=0.05)
    eng = Qwen3Decoder(cfg, w, ops.PagedKVPool(cfg.geometry, 4, "hnd"), max_batch=1, max_ctx=64, attn_chunk=128)
    assert eng._layer_stack() is not None
    gain = w.layers[1].ln1
    plain = gain.data
    gain.data = plain.repeat_interleave(2)[::2]
    assert eng._layer_stack() is None
    gain.data = plain
    assert eng._layer_stack() is not None


def test_tensor_parallel_shards_tile_the_full_weights():
    from skygdr_b200.models import Qwen3Config, Qwen3Weights

    cfg = Qwen3Config.tiny(layers=1)
    full = Qwen3Weights(cfg, "cuda", seed=5)
    shards = [Qwen3Weights(cfg, "cuda", seed=5, tp_rank=r, tp_world=2) for r in range(2)]
    D, qh, kh = cfg.head_dim, cfg.q_heads // 2, cfg.kv_heads // 2
    f = full.layers[0]
    q = torch.cat([s.layers[0].qkv[:qh * D] for s in shards])
    assert torch.equal(q, f.qkv[:cfg.q_heads * D])
    assert torch.equal(torch.cat([s.layers[0].o for s in shards], 1), f.o)
    assert torch.equal(torch.cat([s.layers[0].down for s in shards], 1), f.down)
    gate = torch.cat([s.layers[0].gate_up[:cfg.ffn // 2] for s in shards])
    assert torch.equal(gate, f.gate_up[:cfg.ffn])
    assert torch.equal(torch.cat([s.lm_head for s in shards]), full.lm_head)


@pytest.mark.parametrize("use_graph", [False, True])
def test_continuous_batching_gives_each_request_the_tokens_it_gets_alone(use_graph):
    """Requests of different lengths arrive while the batch is running and share engine steps; since every row of a step is
    computed independently of the other rows, a request must get exactly the tokens it gets when it runs alone."""
    from skygdr_b200 import ops
    from skygdr_b200.models import ContinuousBatcher, Request

    cfg, w, pool, eng = _setup(attn_impl="tc", attn_chunk=128)
    torch.manual_seed(5)
    prompts = [torch.randint(0, cfg.vocab, (n,)) for n in (20, 3, 47, 16, 9, 33)]
    new = [6, 9, 4, 7, 5, 8]

    def run(reqs, arrivals):
        alloc = ops.BlockAllocator(64, max_seqs=eng.max_batch, max_ctx=eng.max_ctx)
        b = ContinuousBatcher(eng, alloc, use_graph=use_graph)
        out, pending = {}, list(reqs)
        step = 0
        while pending or not b.idle():
            for _ in range(arrivals[step % len(arrivals)]):
                if pending:
                    b.submit(pending.pop(0))
            for rid, tok in b.step():
                out.setdefault(rid, []).append(tok)
            step += 1
        assert alloc.free_blocks == alloc.capacity and eng.check_status() == "OK"
        return out

    together = run([Request(i, p, n) for i, (p, n) in enumerate(zip(prompts, new))], arrivals=[2, 0, 1, 3])
    for i, (p, n) in enumerate(zip(prompts, new)):
        alone = run([Request(i, p, n)], arrivals=[1])
        assert together[i] == alone[i] and len(alone[i]) == n, (i, together[i], alone[i])
