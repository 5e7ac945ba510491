"""Performance cases: the work a user of this package has it do on one GPU, through its public entry points.

Five kinds of work:

``model``  a stack of decoder layers with embedding, final norm and vocabulary projection, replayed from CUDA graphs
           by ``ModelGraphRunner`` as a serving worker does it every step (Llama-3-8B shapes, four of its layers; the
           step's keys and values go into a paged KV cache).  Batches run from a few decodes to a full
           chunked-prefill budget of 2048 tokens.
``layer``  one decoder layer called eagerly, as a model file that imports ``LlamaDecoderLayer`` does (``fused``), or
           module by module as the unmodified model file does after ``install()`` (``unfused``), in bf16, fp16 or fp32.
``rank``   what one tensor-parallel rank computes of a layer between the collectives (projections, norms, rotary,
           SiLU*mul at 1/tp of the width), captured in a CUDA graph by ``LayerGraph``.
``moe``    a Mixtral-shaped mixture-of-experts block (router gate, routing, expert MLPs, residual add) of one rank.
``route``  the routing ops alone, as the reference's own fused_moe calls them through the drop-in modules.

Attention is outside this package: it is stood in for by ``attn_out = q`` everywhere, as in the benchmark.
"""
import math

import torch

from sarathi_serve_b200 import fused_moe, kv_cache_ops, parallel_state
from sarathi_serve_b200.decoder_layer import LlamaDecoderLayer, LlamaForCausalLM, MixtralMoE
from sarathi_serve_b200.graph_runner import LayerGraph
from sarathi_serve_b200.model_runner import ModelGraphRunner
from sarathi_serve_b200.nn_layers import RMSNorm, get_rope
from sarathi_serve_b200.tp_layers import ColumnParallelLinear, RowParallelLinear

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
PAGE = 16         # tokens per KV-cache page, as in the benchmark configurations
MAX_CONTEXT = 256  # longest context of a decoding request here: it sets the size of the cache, not the work
LAYERS = 4        # layers of the ``model`` cases

# hidden, q heads, kv heads, head_dim, intermediate, vocabulary, rope theta, eps
SHAPES = {
    "llama3-8b": dict(hidden=4096, nq=32, nkv=8, hd=128, inter=14336, vocab=128256, theta=500000.0, max_pos=8192),
    "llama3-70b": dict(hidden=8192, nq=64, nkv=8, hd=128, inter=28672, vocab=128256, theta=500000.0, max_pos=8192),
    "small": dict(hidden=1024, nq=16, nkv=4, hd=64, inter=2816, vocab=0, theta=10000.0, max_pos=2048),
}
MOE = dict(hidden=4096, inter=14336, experts=8, top_k=2)  # Mixtral-8x7B


def listed():
    return [
        # a decode-only step of a lightly loaded server: every weight is read for eight tokens
        {"name": "model_decode_8", "kind": "model", "prefill": 0, "decodes": 8},
        # a decode-only step with an odd number of running requests
        {"name": "model_decode_61", "kind": "model", "prefill": 0, "decodes": 61},
        # the mixed chunk of the headline benchmark: 448 prompt tokens and 64 decodes
        {"name": "model_mixed_512", "kind": "model", "prefill": 448, "decodes": 64},
        # the largest scheduler budget, not quite full
        {"name": "model_mixed_1999", "kind": "model", "prefill": 1790, "decodes": 209},
        # the drop-in decoder layer in a host's own eager loop, ragged chunk
        {"name": "layer_fused_bf16_300", "kind": "layer", "path": "fused", "shape": "llama3-8b", "dtype": "bf16", "tokens": 300},
        # the unmodified model file on this package's modules and ops, fp16, ragged chunk
        {"name": "layer_unfused_fp16_777", "kind": "layer", "path": "unfused", "shape": "llama3-8b", "dtype": "fp16",
         "tokens": 777},
        # the fp32 parity configuration: 256 prompt tokens and 32 decodes of a small layer
        {"name": "layer_fused_fp32_288", "kind": "layer", "path": "fused", "shape": "small", "dtype": "fp32", "tokens": 288},
        # one of eight ranks of the headline layer: short K, narrow N, launch costs count
        {"name": "rank_8b_tp8_512", "kind": "rank", "shape": "llama3-8b", "tp": 8, "tokens": 512},
        # one of eight ranks of the 70B-shaped layer on a large ragged chunk
        {"name": "rank_70b_tp8_1601", "kind": "rank", "shape": "llama3-70b", "tp": 8, "tokens": 1601},
        # one of eight ranks of the Mixtral-shaped block on the benchmark's 1024-token chunk
        {"name": "moe_tp8_1024", "kind": "moe", "tp": 8, "tokens": 1024},
        # decode-only step of the whole block on one GPU: all experts are read for a few tokens each
        {"name": "moe_tp1_24", "kind": "moe", "tp": 1, "tokens": 24},
        # the smallest call: routing of a small batch with the reference's block size
        {"name": "route_64", "kind": "route", "tokens": 64, "experts": 8, "top_k": 2, "block": 64, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["model", "model", "layer", "layer", "rank", "rank", "moe", "route"])
    if kind == "model":
        tokens = _log_int(rng, 1, 2000)
        decodes = tokens if rng.random() < 0.4 else min(tokens, _log_int(rng, 1, 256))
        decodes = min(decodes, 256)
        return {"kind": "model", "prefill": tokens - decodes, "decodes": decodes}
    if kind == "layer":
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        small = dtype == "fp32"
        return {"kind": "layer", "path": rng.choice(["fused", "unfused"]), "shape": "small" if small else "llama3-8b",
                "dtype": dtype, "tokens": _log_int(rng, 1, 512 if small else 2048)}
    if kind == "rank":
        shape = rng.choice(["llama3-8b", "llama3-70b"])
        tp = rng.choice([2, 4, 8] if shape == "llama3-8b" else [4, 8])
        return {"kind": "rank", "shape": shape, "tp": tp, "tokens": _log_int(rng, 1, 2048)}
    if kind == "moe":
        return {"kind": "moe", "tp": rng.choice([1, 2, 4, 8]), "tokens": _log_int(rng, 1, 2048)}
    experts = rng.choice([8, 16, 64, 128])
    return {"kind": "route", "tokens": _log_int(rng, 1, 8192), "experts": experts, "top_k": rng.choice([1, 2, 4, 6]),
            "block": rng.choice([16, 64, 128]), "dtype": rng.choice(["fp32", "bf16"])}


# ------------------------------------------------------------------ inputs
class _Config:
    """The attributes of a model configuration that the modules read."""

    def __init__(self, s, layers):
        self.hidden_size, self.intermediate_size, self.vocab_size = s["hidden"], s["inter"], s["vocab"]
        self.num_attention_heads, self.num_key_value_heads = s["nq"], s["nkv"]
        self.num_hidden_layers, self.rms_norm_eps, self.hidden_act = layers, 1e-5, "silu"
        self.rope_theta, self.rope_scaling, self.max_position_embeddings = s["theta"], None, s["max_pos"]


class _default_dtype:
    def __init__(self, dtype):
        self.dtype = dtype

    def __enter__(self):
        self.old = torch.get_default_dtype()
        torch.set_default_dtype(self.dtype)

    def __exit__(self, *exc):
        torch.set_default_dtype(self.old)


def _init_weights(module, gen):
    """N(0, 0.02) projections and embeddings, norm weights near one."""
    with torch.no_grad():
        for p in module.parameters():
            if p.dim() == 1:
                p.normal_(1.0, 0.02, generator=gen)
            else:
                p.normal_(0.0, 0.02, generator=gen)
    return module


class _Batch:
    """Token positions of a mixed batch and its page table: one prompt chunk, then one token per decoding request."""

    def __init__(self, prefill, decodes, padded, gen, dev):
        n = prefill + decodes
        context = torch.randint(16, MAX_CONTEXT, (decodes,), generator=gen, device=dev)
        lengths = torch.cat([torch.tensor([prefill], device=dev), context]) if prefill else context
        first = 1 if prefill else 0
        pages = (lengths + PAGE - 1) // PAGE
        self.num_pages = decodes * (MAX_CONTEXT // PAGE) + (prefill + PAGE - 1) // PAGE  # the pool, not all of it in use
        self.kv_indptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=dev), pages.cumsum(0)]).int()
        self.kv_indices = torch.randperm(self.num_pages, generator=gen, device=dev).int()  # the first of them are used
        owner = torch.cat([torch.zeros(prefill, dtype=torch.int64, device=dev), torch.arange(decodes, device=dev) + first])
        self.positions = torch.cat([torch.arange(prefill, device=dev), context - 1])
        # rows that only pad the batch are stored nowhere
        self.batch_indices = torch.full((padded,), -1, dtype=torch.int32, device=dev)
        self.batch_indices[:n] = owner.int()
        self.positions32 = torch.zeros(padded, dtype=torch.int32, device=dev)
        self.positions32[:n] = self.positions.int()
        # the rows whose next token is sampled: the end of the prompt chunk and every decode
        self.sampled = torch.arange(prefill - 1 if prefill else 0, n, device=dev)


def _kv_cache(batch, s, dtype, gen, dev):
    """A paged cache full of the keys and values of earlier steps."""
    cache = torch.empty(batch.num_pages, 2, PAGE, s["nkv"], s["hd"], dtype=dtype, device=dev)
    return cache.normal_(0.0, 1.0, generator=gen)


class _GraphAttention:
    """Attention stand-in of a captured model: the qkv projection stores keys and values into the paged cache."""

    def __init__(self, caches, slots):
        self.caches, self.slots = caches, slots

    def fused_kv_append(self, layer_cache_idx):
        return self.caches[layer_cache_idx], self.slots

    def forward(self, q, k, v, layer_cache_idx, softmax_scale=1.0, layer_id=None):
        return q


class _EagerAttention:
    """Attention stand-in of an eager layer; ``unfused`` callers append keys and values themselves."""

    def __init__(self, batch=None, cache=None):
        self.batch, self.cache = batch, cache

    def forward(self, q, k, v, layer_cache_idx, softmax_scale=1.0, layer_id=None):
        if self.cache is not None:
            b = self.batch
            kv_cache_ops.append_paged_kv_cache(k, v, b.batch_indices, b.positions32, self.cache, b.kv_indices, b.kv_indptr)
        return q


class _RankShare(torch.nn.Module):
    """What one of ``tp`` ranks computes of a decoder layer; the collectives between the parts are left out."""

    def __init__(self, s, tp, dtype):
        super().__init__()
        self.hidden_size = s["hidden"]
        nq, nkv, hd = s["nq"] // tp, s["nkv"] // tp, s["hd"]
        self.sizes = [nq * hd, nkv * hd, nkv * hd]
        one = dict(bias=False, params_dtype=dtype)
        self.qkv_proj = ColumnParallelLinear(s["hidden"], sum(self.sizes), gather_output=False, **one)
        self.o_proj = RowParallelLinear(nq * hd, s["hidden"], input_is_parallel=True, **one)
        self.gate_up_proj = ColumnParallelLinear(s["hidden"], 2 * s["inter"] // tp, gather_output=False, **one)
        self.down_proj = RowParallelLinear(s["inter"] // tp, s["hidden"], input_is_parallel=True, **one)
        self.norm1, self.norm2 = RMSNorm(s["hidden"], eps=1e-5), RMSNorm(s["hidden"], eps=1e-5)
        self.rotary_emb = get_rope(hd, hd, s["max_pos"], s["theta"], True, None)

    def forward(self, positions, hidden_states, layer_cache_idx, attention_backend_wrapper):
        qkv = self.qkv_proj.forward_rotary(hidden_states, positions, self.rotary_emb, self.sizes[0] + self.sizes[1])
        q, k, v = qkv.split(self.sizes, dim=-1)
        attn = attention_backend_wrapper.forward(q, k, v, layer_cache_idx)
        out, _ = self.o_proj(attn)
        h, residual = self.norm1.forward_add(out, hidden_states)
        out, _ = self.down_proj(self.gate_up_proj.forward_silu_mul(h))
        h, _ = self.norm2.forward_add(out, residual)
        return h


def _bucket(n):
    for b in (8, 16, 32, 64, 128, 256, 512, 1024, 2048):  # ModelGraphRunner's own buckets
        if n <= b:
            return b
    raise ValueError(n)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    if not parallel_state.model_parallel_is_initialized():
        parallel_state.initialize_model_parallel(1)
    kind = case["kind"]
    if kind == "model":
        s = SHAPES["llama3-8b"]
        n = case["prefill"] + case["decodes"]
        padded = _bucket(n)
        with _default_dtype(torch.bfloat16):
            model = _init_weights(LlamaForCausalLM(_Config(s, LAYERS)), gen)
        batch = _Batch(case["prefill"], case["decodes"], padded, gen, dev)
        caches = [_kv_cache(batch, s, torch.bfloat16, gen, dev) for _ in range(LAYERS)]
        slots = torch.full((padded,), -1, dtype=torch.int64, device=dev)
        runner = ModelGraphRunner(model.model, _GraphAttention(caches, slots))
        tokens = torch.randint(0, s["vocab"], (n,), generator=gen, device=dev)
        runner.run(tokens, batch.positions)  # a worker captures its graphs when it starts
        return {"kind": kind, "model": model, "runner": runner, "batch": batch, "caches": caches, "slots": slots,
                "tokens": tokens}
    if kind == "layer":
        s, dtype, n = SHAPES[case["shape"]], DTYPES[case["dtype"]], case["tokens"]
        with _default_dtype(dtype):
            layer = _init_weights(LlamaDecoderLayer(_Config(s, 1)), gen)
        decodes = min(n, 64) if n <= 64 else n // 8
        batch = _Batch(n - decodes, decodes, n, gen, dev)
        cache = None
        if case["path"] == "unfused":
            cache = _kv_cache(batch, s, dtype, gen, dev)
        x = torch.randn(n, s["hidden"], generator=gen, device=dev, dtype=torch.float32).to(dtype)
        return {"kind": kind, "path": case["path"], "layer": layer, "attn": _EagerAttention(batch, cache), "x": x,
                "positions": batch.positions, "cache": cache}
    if kind == "rank":
        s, n = SHAPES[case["shape"]], case["tokens"]
        with _default_dtype(torch.bfloat16):
            share = _init_weights(_RankShare(s, case["tp"], torch.bfloat16), gen)
        decodes = min(n, 64) if n <= 64 else n // 8
        batch = _Batch(n - decodes, decodes, n, gen, dev)
        x = torch.randn(n, s["hidden"], generator=gen, device=dev, dtype=torch.float32).to(torch.bfloat16)
        return {"kind": kind, "graph": LayerGraph(share, n, _EagerAttention()), "x": x, "positions": batch.positions}
    if kind == "moe":
        n = case["tokens"]
        with _default_dtype(torch.bfloat16):
            block = _init_weights(MixtralMoE(MOE["experts"], MOE["top_k"], MOE["hidden"], MOE["inter"] // case["tp"]), gen)
        x = torch.randn(n, MOE["hidden"], generator=gen, device=dev, dtype=torch.float32).to(torch.bfloat16)
        residual = torch.randn(n, MOE["hidden"], generator=gen, device=dev, dtype=torch.float32).to(torch.bfloat16)
        return {"kind": kind, "block": block, "x": x, "residual": residual}
    n = case["tokens"]
    x = torch.empty(n, 16, dtype=torch.bfloat16, device=dev)
    logits = torch.randn(n, case["experts"], generator=gen, device=dev, dtype=torch.float32).to(DTYPES[case["dtype"]])
    return {"kind": kind, "x": x, "logits": logits, "top_k": case["top_k"], "block": case["block"],
            "experts": case["experts"]}


def run(state):
    with torch.inference_mode():
        kind = state["kind"]
        if kind == "model":
            b = state["batch"]
            kv_cache_ops.slots(b.batch_indices, b.positions32, b.kv_indices, b.kv_indptr, PAGE, out=state["slots"])
            hidden = state["runner"].run(state["tokens"], b.positions)
            logits = state["model"].compute_logits(hidden.index_select(0, b.sampled))
            return {"logits": logits, "hidden": hidden, "caches": state["caches"]}
        if kind == "layer":
            layer = state["layer"]
            call = layer.forward if state["path"] == "fused" else layer.forward_unfused
            return {"out": call(state["positions"], state["x"], 0, state["attn"]), "cache": state["cache"]}
        if kind == "rank":
            return state["graph"](state["positions"], state["x"])
        if kind == "moe":
            return state["block"].forward_fused(state["x"], state["residual"])
        weights, ids = fused_moe.fused_topk(state["x"], state["logits"], state["top_k"], True)
        sorted_ids, expert_ids, post_pad = fused_moe.moe_align_block_size(ids, state["block"], state["experts"])
        # expert_ids is defined for the blocks in use only: not returned whole
        return {"weights": weights, "ids": ids, "sorted": sorted_ids, "post_pad": post_pad}


# ------------------------------------------------------------------ what a pass cannot do without
def _layer_work(s, tp, tokens, es, kv):
    hidden, qkv, att, inter = s["hidden"], (s["nq"] + 2 * s["nkv"]) * s["hd"] // tp, s["nq"] * s["hd"] // tp, s["inter"] // tp
    params = hidden * (qkv + att + 3 * inter)
    moved = params + tokens * 2 * hidden + (tokens * 2 * s["nkv"] * s["hd"] // tp if kv else 0)
    return 2.0 * tokens * params, float(moved * es)


def work(case):
    kind = case["kind"]
    if kind == "model":
        s, n = SHAPES["llama3-8b"], case["prefill"] + case["decodes"]
        rows = case["decodes"] + (1 if case["prefill"] else 0)
        flops, moved = _layer_work(s, 1, n, 2, True)
        head = s["vocab"] * s["hidden"]
        return {"flops": LAYERS * flops + 2.0 * rows * head,
                "bytes": LAYERS * (moved - n * 2 * s["hidden"] * 2) + 2.0 * (head + rows * s["vocab"] + 2 * n * s["hidden"])}
    if kind == "layer":
        es = 4 if case["dtype"] == "fp32" else 2
        flops, moved = _layer_work(SHAPES[case["shape"]], 1, case["tokens"], es, case["path"] == "unfused")
        return {"flops": flops, "bytes": moved}
    if kind == "rank":
        flops, moved = _layer_work(SHAPES[case["shape"]], case["tp"], case["tokens"], 2, False)
        return {"flops": flops, "bytes": moved}
    if kind == "moe":
        n, inter, e, k, hidden = case["tokens"], MOE["inter"] // case["tp"], MOE["experts"], MOE["top_k"], MOE["hidden"]
        used = e * (1.0 - (1.0 - k / e) ** n)  # experts that a batch of n tokens is expected to use
        return {"flops": 2.0 * n * (k * 3 * hidden * inter + hidden * e),
                "bytes": 2.0 * (used * 3 * hidden * inter + hidden * e + 3 * n * hidden)}
    n, e, k = case["tokens"], case["experts"], case["top_k"]
    padded = n * k + e * (case["block"] - 1)
    return {"flops": 8.0 * n * e, "bytes": n * e * (4 if case["dtype"] == "fp32" else 2) + 8.0 * n * k + 4.0 * padded + 4}


def tolerance(case):
    """About four times what the path differs by from itself with its projections summed in fp32 (fp32 cases: fp64) and
    rounded where the path rounds: the roundings to 16 bits between the operations decide, and four layers of bf16
    compound them (1.1e-2 on the logits, at most 3e-2 is stated).  Routing: ids and orders are exact, weights are fp32."""
    kind = case["kind"]
    if kind == "model":
        return {"rel": 3e-2, "max": 0.3}
    if kind == "layer":
        return {"bf16": {"rel": 1.3e-2, "max": 0.15}, "fp16": {"rel": 2e-3, "max": 0.03},
                "fp32": {"rel": 2e-6, "max": 1.5e-5}}[case["dtype"]]
    if kind == "rank":
        return {"rel": 1.3e-2, "max": 0.13}
    if kind == "moe":
        return {"rel": 5e-3, "max": 0.07}
    return {"rel": 1e-6, "differ": 0.0}
