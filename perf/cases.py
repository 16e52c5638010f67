"""What is timed of this framework: the calls its users make, at the sizes its configurations, tests and benchmark use.

Four kinds of work, each through the entry points that a user's program calls:

* ``decode``: one step of a decode batch, host token ids in, host token ids out (``DecodeSession.step`` on an engine from
  ``build_decode_engine``), greedy or with temperature sampling;
* ``prefill``: prompts through the stack into the paged pool (``Qwen3Decoder.prefill``), head-major pool (decode follows on the same
  GPU) or token-major pool (hand-off to a decode GPU follows);
* ``transfer``: one request's KV from the prefill pool into one or several decode pools (``KvTransferFlow.transfer`` and
  ``result``), bf16 or block-scaled fp8, one destination or a scatter over tensor-parallel ranks. Every flow has a credit page, as a
  registered flow has. The destinations are pools of the same GPU;
* ``offload``: one request's KV into pinned host memory, layout kept.

The decoder has the widths of Qwen3-8B and 8 of its 36 layers (a pipeline stage with the embedding and the output projection), with
tied embeddings: random weights then still decide every sampled token clearly, and the rounding of two correct implementations
stays small against the logits. Transfers carry all 36 layers."""
import math
import random

import torch

from skygdr_b200 import ops
from skygdr_b200.models import DecodeSession, Qwen3Config, Qwen3Decoder, Qwen3Weights
from skygdr_b200.ops.kv_cache import KVGeometry, PagedKVPool
from skygdr_b200.parallel.tp import build_decode_engine

LAYERS = 8              # decoder layers of decode and prefill cases
KV_LAYERS = 36          # layers that a transfer carries
MAX_KV_TOKENS = 330000  # context tokens of a decode batch: 10.8 GB of KV at 8 layers


def _decode(batch, lo, hi, dist="uniform", temperature=0.0, lens=1):
    return {"kind": "decode", "batch": batch, "lo": lo, "hi": hi, "dist": dist, "temperature": temperature, "lens": lens}


def _prefill(prompts, lo, hi, layout, lens=1):
    return {"kind": "prefill", "prompts": prompts, "lo": lo, "hi": hi, "dist": "uniform", "layout": layout, "lens": lens}


def _transfer(tokens, fp8=False, n_dst=1):
    return {"kind": "transfer", "tokens": tokens, "fp8": fp8, "n_dst": n_dst}


def listed():
    named = {
        # one user's chat turn: the lowest latency a step can have, all of it weights and launches
        "decode_b1_short": _decode(1, 300, 300),
        # the benchmark's batch: 16 sequences, contexts uniform 2k-16k
        "decode_b16_2k_16k": _decode(16, 2048, 16384),
        # many long contexts (median 8k, 1k-32k): KV traffic dominates
        "decode_b32_long": _decode(32, 1024, 32768, dist="lognormal"),
        # a busy chat server: a ragged batch of short contexts, sampled with a temperature
        "decode_b100_sampled": _decode(100, 64, 2000, temperature=0.7),
        # the first token of a short question
        "prefill_77": _prefill(1, 77, 77, "hnd"),
        # several prompts admitted together, ragged, for hand-off to a decode GPU
        "prefill_9_ragged": _prefill(9, 20, 900, "nhd"),
        # a long document, cut into chunks of 8192 tokens
        "prefill_16k": _prefill(1, 16384, 16384, "hnd"),
        # the last blocks of a request, or a very short one
        "transfer_17": _transfer(17),
        # a median hand-off
        "transfer_4k": _transfer(4096),
        # the longest request
        "transfer_64k": _transfer(65536),
        # packed to fp8 and scattered over four tensor-parallel decode ranks
        "transfer_9k_fp8_tp4": _transfer(9001, fp8=True, n_dst=4),
        # prefix KV of a finished request to pinned host memory
        "offload_1500": {"kind": "offload", "tokens": 1500},
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "transfer", "transfer", "offload"])
    if kind == "decode":
        batch = _log_int(rng, 1, 128)
        mid = _log_int(rng, 64, min(16384, MAX_KV_TOKENS // (2 * batch)))
        c = _decode(batch, max(1, mid // 8), 2 * mid, rng.choice(["uniform", "lognormal"]), rng.choice([0.0, 0.0, 0.7, 1.0]), rng.randrange(1 << 20))
    elif kind == "prefill":
        total = _log_int(rng, 16, 16384)
        prompts = rng.choice([1, 1, rng.randint(2, 12)])
        hi = max(2, total // prompts)
        c = _prefill(prompts, max(1, hi // 6) if prompts > 1 else hi, hi, rng.choice(["hnd", "nhd"]), rng.randrange(1 << 20))
    elif kind == "transfer":
        c = _transfer(_log_int(rng, 16, 65536), rng.choice([False, False, True]), rng.choice([1, 1, 2, 4]))
    else:
        c = {"kind": "offload", "tokens": _log_int(rng, 16, 2048)}
    return c


def _lengths(case):
    """The context or prompt lengths of a case: they belong to its size, so they follow from the case and not from the seed."""
    rng = random.Random(case["lens"])
    n, lo, hi = case.get("batch") or case.get("prompts"), case["lo"], case["hi"]
    if case["dist"] == "lognormal":
        median = math.sqrt(lo * hi) * 1.4
        return [min(hi, max(lo, int(median * math.exp(0.6 * rng.gauss(0.0, 1.0))))) for _ in range(n)]
    return [rng.randint(lo, hi) for _ in range(n)]


def _config():
    return Qwen3Config(layers=LAYERS)


def _block_table(lens, device):
    """Each sequence's own blocks in random order; block 0 is nobody's."""
    need = [(n + 15) // 16 for n in lens]
    table = torch.zeros((len(lens), max(need) + 8), dtype=torch.int32, device=device)
    perm = (torch.randperm(sum(need), device=device) + 1).int()
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = perm[at:at + n]
        at += n
    return table, sum(need) + 1


def _prepare_decode(case, seed):
    dev, cfg = torch.device("cuda", 0), _config()
    ctx = torch.tensor(_lengths(case))
    batch = ctx.numel()
    eng, table = build_decode_engine(cfg, dev, 0, 1, ctx, extra_tokens=64, seed=seed % 100000)
    eng.w.lm_head = eng.w.embed                                         # tied embeddings
    eng.temperature, eng.sample_seed = case["temperature"], seed & 0xFFFF
    ids = torch.randint(0, cfg.vocab, (batch,), device=dev).int().cpu()
    eng.set_batch(ids.to(dev), ctx.int().to(dev), table.to(dev))
    sess = DecodeSession(eng, batch)
    sess.start(ids, ctx.int(), table)
    return {"kind": "decode", "sess": sess, "eng": eng, "ids": ids, "pos": ctx.int()}


def _prepare_prefill(case, seed):
    dev, cfg = torch.device("cuda", 0), _config()
    lens = _lengths(case)
    weights = Qwen3Weights(cfg, dev, seed=seed % 100000)
    weights.lm_head = weights.embed
    table, n_blocks = _block_table(lens, dev)
    decode_pool = PagedKVPool(cfg.geometry, n_blocks if case["layout"] == "hnd" else 2, "hnd", device=dev)
    pool = decode_pool if case["layout"] == "hnd" else PagedKVPool(cfg.geometry, n_blocks, "nhd", device=dev)
    eng = Qwen3Decoder(cfg, weights, decode_pool, max_batch=1, max_ctx=256, attn_chunk=128)
    ids = torch.randint(0, cfg.vocab, (sum(lens),), device=dev)
    return {"kind": "prefill", "eng": eng, "ids": ids, "lens": lens, "table": table, "pool": pool}


def _source(tokens):
    """A prefill pool that holds one request of this length, and its blocks in random order. Values N(0, 1), as the caches of the
    benchmark have; K and V of a normed projection look like it."""
    geom = KVGeometry(layers=KV_LAYERS)
    n = geom.blocks_for(tokens)
    src = PagedKVPool(geom, n + 1, "nhd", device="cuda:0")
    src.data.normal_()
    blocks = (torch.randperm(n, device="cuda:0") + 1).int()
    return geom, n, src, blocks


def _prepare_transfer(case, seed):
    geom, n, src, src_blocks = _source(case["tokens"])
    dst_blocks = (torch.randperm(n, device="cuda:0") + 1).int()
    heads = geom.kv_heads // case["n_dst"]
    pages, remotes = [], []
    for _ in range(case["n_dst"]):
        if case["fp8"]:
            q = torch.zeros((n + 1, geom.layers, 2, heads, 16, 128), dtype=torch.uint8, device="cuda:0")
            s = torch.zeros((n + 1, geom.layers, 2, heads, 16, 4), dtype=torch.uint8, device="cuda:0")
            pages += [q, s]
            remotes.append(ops.RemotePool(q.data_ptr(), q.stride()[:3], heads, s.data_ptr(), 0, n + 1))
        else:
            pool = PagedKVPool(KVGeometry(geom.layers, heads), n + 1, "hnd", device="cuda:0")
            pages.append(pool.data)
            remotes.append(ops.RemotePool.of(pool))
    flow = ops.KvTransferFlow("cuda:0", page=ops.CreditPage(flow_id=1, unlimited=True))
    return {"kind": "transfer", "flow": flow, "src": src, "remotes": remotes, "src_blocks": src_blocks, "dst_blocks": dst_blocks, "fp8": case["fp8"],
            "keep": False, "pages": pages}


def _prepare_offload(case, seed):
    geom, n, src, src_blocks = _source(case["tokens"])
    host = torch.zeros((n, geom.block_elems), dtype=torch.bfloat16).pin_memory()
    remote = ops.RemotePool(host.data_ptr(), src.strides, geom.kv_heads, num_blocks=n)
    flow = ops.KvTransferFlow("cuda:0", page=ops.CreditPage(flow_id=2, unlimited=True))
    return {"kind": "offload", "flow": flow, "src": src, "remotes": [remote], "src_blocks": src_blocks, "dst_blocks": torch.arange(n, device="cuda:0").int(),
            "fp8": False, "keep": True, "pages": [host]}


def prepare(case, seed):
    torch.manual_seed(seed)
    return {"decode": _prepare_decode, "prefill": _prepare_prefill, "transfer": _prepare_transfer, "offload": _prepare_offload}[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "decode":
        sess, eng = state["sess"], state["eng"]
        sess.h_ids.copy_(state["ids"])          # the token each sequence continues with, and its position
        sess.h_pos.copy_(state["pos"])
        ids = sess.step()
        return {"ids": ids, "logits": eng.logits[:sess.batch], "kv": eng.pool.data}
    if state["kind"] == "prefill":
        logits = state["eng"].prefill(state["ids"], state["lens"], state["table"], pool=state["pool"])
        return {"logits": logits, "kv": state["pool"].data}
    flow = state["flow"]
    flow.transfer(state["src"], state["remotes"], state["src_blocks"], state["dst_blocks"], fp8=state["fp8"], keep_layout=state["keep"])
    done = flow.result()
    return {"status": done["status"], "bytes": done["bytes_done"], "pages": state["pages"]}


def work(case):
    if case["kind"] in ("transfer", "offload"):
        geom = KVGeometry(layers=KV_LAYERS)
        payload = geom.blocks_for(case["tokens"]) * geom.block_elems * 2
        written = payload // 2 + payload // 64 if case.get("fp8") else payload
        return {"bytes": payload + written, "flops": 0}
    cfg = _config()
    lens = _lengths(case)
    layer = (cfg.q_heads + 2 * cfg.kv_heads) * cfg.head_dim * cfg.hidden + cfg.q_heads * cfg.head_dim * cfg.hidden + 3 * cfg.ffn * cfg.hidden
    head = cfg.vocab * cfg.hidden
    kv_token = cfg.layers * 2 * cfg.kv_heads * cfg.head_dim * 2          # bytes of one token's K and V
    rows = len(lens)                                                     # rows of logits
    fixed = 2 * (cfg.layers * layer + head) + 2 * rows * cfg.vocab
    pair = 4 * cfg.q_heads * cfg.head_dim * cfg.layers                   # operations per (query, key)
    if case["kind"] == "decode":
        return {"bytes": fixed + (sum(lens) + rows) * kv_token + rows * cfg.hidden * 2 + 12 * rows,
                "flops": 2 * rows * (cfg.layers * layer + head) + pair * (sum(lens) + rows)}
    tokens = sum(lens)
    return {"bytes": fixed + tokens * (kv_token + min(cfg.hidden * 2, head * 2 // max(1, tokens)) + 8),
            "flops": 2 * (tokens * cfg.layers * layer + rows * head) + pair * sum(n * (n + 1) // 2 for n in lens)}


def tolerance(case):
    # A transfer moves bytes, and fp8 packing is defined bit by bit. The decoder rounds to bf16 at every op (2^-9 each, 8 layers
    # of nine ops): the logits of two summation orders differ by one to two per cent of their norm, single values by a few times that.
    return "exact" if case["kind"] in ("transfer", "offload") else {"rel": 0.02, "max": 0.25}
