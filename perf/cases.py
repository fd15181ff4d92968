"""The calls whose speed this framework is judged by: the operators and the models a user runs through it.

Every case is a plain dict. `listed()` names the fixed ones, `draw()` picks others of the same ranges,
`prepare()` makes what a program holds before the call, `run()` is one pass through the public entry
points, `work()` the bytes and operations that pass cannot do without, `tolerance()` how far two
correct implementations of the same precision may lie apart.

Paths ("path" of a case) and what they stand for:
  norm       one LayerNorm / RMSNorm call, with the residual add of pre-norm decoders where asked
  linear     one fused linear (bias + activation) as the rewrites call it
  attention  one fused attention over a whole sequence (encoder, or prefill when causal)
  decode_attention  one query row per sequence against a KV cache (a generated token)
  encoder    a BERT-shaped encoder: traced graph -> the rewrite pipeline -> the CUDA-graph wrapper
  prefill    the Llama-shaped decoder over a prompt (fills the KV cache)
  decode     one token of the same decoder, captured in a CUDA graph as a serving loop does
"""
import math

import torch

from kernl_b200.implementations.attention import attention_forward
from kernl_b200.implementations.attention_skinny import skinny_attention_forward
from kernl_b200.implementations.layer_norm import layer_norm
from kernl_b200.implementations.linear_layer import linear_layer
from kernl_b200.llama_tp import LlamaConfig, LlamaTP
from kernl_b200.optimizer.cuda_graph import cuda_graphs_wrapper
from kernl_b200.optimizer.dynamo_backend import dynamo_backend_ofi

DEVICE = "cuda"


def listed():
    return [
        # a layer norm of BERT-base at batch 1 x 128 tokens, called eagerly: launch and host latency
        {"name": "norm_128x768", "path": "norm", "rows": 128, "cols": 768, "rms": False, "residual": False, "dtype": "float16"},
        # add + RMSNorm of a 7B decoder's prefill (16384 tokens): the largest streaming case
        {"name": "add_rms_16384x4096", "path": "norm", "rows": 16384, "cols": 4096, "rms": True, "residual": True, "dtype": "bfloat16"},
        # a projection in a decode step: few rows, the weights are what has to be read
        {"name": "linear_16x4096x11008", "path": "linear", "M": 16, "K": 4096, "N": 11008, "activation": "", "bias": True, "dtype": "float16"},
        # BERT-base's feed-forward over a ragged batch of 1000 tokens
        {"name": "linear_1000x768x3072_gelu", "path": "linear", "M": 1000, "K": 768, "N": 3072, "activation": "gelu", "bias": True,
         "dtype": "float16"},
        # BERT-base attention over a padded batch
        {"name": "attn_pad_8x12x512", "path": "attention", "batch": 8, "heads": 12, "kv_heads": 12, "seq": 512, "dim": 64, "mask": "padding",
         "causal": False, "split_heads": False, "dtype": "float16"},
        # T5-base encoder attention: dense position bias, a length that fits no tile
        {"name": "attn_bias_3x12x333", "path": "attention", "batch": 3, "heads": 12, "kv_heads": 12, "seq": 333, "dim": 64, "mask": "bias",
         "causal": False, "split_heads": True, "dtype": "float16"},
        # causal prefill with grouped-query heads of 128
        {"name": "attn_causal_gqa_4x32x2048", "path": "attention", "batch": 4, "heads": 32, "kv_heads": 8, "seq": 2048, "dim": 128,
         "mask": "none", "causal": True, "split_heads": True, "dtype": "bfloat16"},
        # one generated token against a partly filled grouped-query cache
        {"name": "decode_attn_16x32x3000", "path": "decode_attention", "batch": 16, "heads": 32, "kv_heads": 8, "keys": 3000, "capacity": 4096,
         "dim": 128, "mask": "none", "dtype": "bfloat16"},
        # BERT-base, one short query (the latency of online inference)
        {"name": "encoder_1x128", "path": "encoder", "batch": 1, "seq": 128, "layers": 12, "padded": False},
        # BERT-base, a padded batch (offline inference)
        {"name": "encoder_32x256", "path": "encoder", "batch": 32, "seq": 256, "layers": 12, "padded": True},
        # eight layers of the 7B shape: a token for eight sequences at 2048 keys
        {"name": "decode_8x2048", "path": "decode", "batch": 8, "seq": 2048, "layers": 8},
        # four layers of the 7B shape over four prompts
        {"name": "prefill_4x2048", "path": "prefill", "batch": 4, "seq": 2048, "layers": 4},
    ]


def _log(rng, lo, hi, step=1):
    """A whole number in [lo, hi], a multiple of `step`, spread over the logarithm of the range."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return max(lo, min(hi, int(n) // step * step))


def draw(rng):
    path = rng.choice(("norm", "linear", "attention", "attention", "decode_attention", "encoder", "decode", "prefill"))
    dtype = rng.choice(("float16", "bfloat16"))
    if path == "norm":
        rms = rng.random() < 0.5
        return {"path": path, "rows": _log(rng, 1, 16384), "cols": _log(rng, 256, 8192, 8), "rms": rms,
                "residual": rng.random() < 0.5, "dtype": dtype}
    if path == "linear":
        act = rng.choice(("", "gelu", "relu", "swiglu"))
        return {"path": path, "M": _log(rng, 1, 8192), "K": _log(rng, 256, 11008, 8), "N": _log(rng, 256, 11008, 16), "activation": act,
                "bias": act != "swiglu" and rng.random() < 0.7, "dtype": dtype}
    if path == "attention":
        dim = rng.choice((64, 64, 64, 128, 128, 80))
        seq = _log(rng, 16, 4096)
        batch = _log(rng, 1, max(1, 16384 // seq))
        causal = rng.random() < 0.35
        heads = rng.choice((12, 16, 32))
        return {"path": path, "batch": batch, "heads": heads, "kv_heads": heads // 4 if rng.random() < 0.25 else heads, "seq": seq, "dim": dim,
                "mask": "none" if causal else rng.choice(("none", "padding", "bias")), "causal": causal, "split_heads": rng.random() < 0.6,
                "dtype": dtype}
    if path == "decode_attention":
        keys = _log(rng, 51, 8192)
        heads = rng.choice((12, 16, 32))
        return {"path": path, "batch": _log(rng, 1, 64), "heads": heads, "kv_heads": rng.choice((heads, heads // 4)), "keys": keys,
                "capacity": keys + rng.choice((0, 1, 100)), "dim": rng.choice((64, 128)), "mask": rng.choice(("none", "none", "bias")),
                "dtype": dtype}
    if path == "encoder":
        seq = _log(rng, 16, 512)
        return {"path": path, "batch": _log(rng, 1, min(32, 8192 // seq)), "seq": seq, "layers": rng.randint(4, 12), "padded": rng.random() < 0.6}
    if path == "decode":
        return {"path": path, "batch": _log(rng, 1, 64), "seq": _log(rng, 64, 2200), "layers": rng.randint(2, 4)}
    seq = _log(rng, 64, 2048)
    return {"path": path, "batch": _log(rng, 1, min(16, 8192 // seq)), "seq": seq, "layers": rng.randint(1, 4)}


class _EncoderLayer(torch.nn.Module):
    """Post-LayerNorm transformer block, written as a model author writes it in plain PyTorch."""

    def __init__(self, hidden, heads, ffn):
        super().__init__()
        self.heads = heads
        self.query, self.key, self.value = (torch.nn.Linear(hidden, hidden) for _ in range(3))
        self.dense = torch.nn.Linear(hidden, hidden)
        self.norm1 = torch.nn.LayerNorm(hidden, eps=1e-12)
        self.up = torch.nn.Linear(hidden, ffn)
        self.act = torch.nn.GELU()
        self.down = torch.nn.Linear(ffn, hidden)
        self.norm2 = torch.nn.LayerNorm(hidden, eps=1e-12)

    def forward(self, x, keep, batch, seq):
        q, k, v = (f(x).view(batch, seq, self.heads, -1).transpose(1, 2) for f in (self.query, self.key, self.value))
        a = torch.nn.functional.scaled_dot_product_attention(q, k, v, attn_mask=keep)
        a = a.transpose(1, 2).reshape(batch, seq, -1)
        x = self.norm1(self.dense(a) + x)
        return self.norm2(self.down(self.act(self.up(x))) + x)


class _Encoder(torch.nn.Module):
    def __init__(self, batch, seq, layers, hidden=768, heads=12, ffn=3072, vocab=30522, positions=512):
        super().__init__()
        self.batch, self.seq = batch, seq
        self.words = torch.nn.Embedding(vocab, hidden)
        self.positions = torch.nn.Parameter(torch.empty(positions, hidden))
        self.norm = torch.nn.LayerNorm(hidden, eps=1e-12)
        self.layers = torch.nn.ModuleList(_EncoderLayer(hidden, heads, ffn) for _ in range(layers))

    def forward(self, ids, keep):
        x = self.norm(self.words(ids) + self.positions[: self.seq])
        mask = keep.view(self.batch, 1, 1, self.seq).expand(self.batch, 1, self.seq, self.seq)
        for layer in self.layers:
            x = layer(x, mask, self.batch, self.seq)
        return x


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _lengths(batch, seq, g):
    """Valid lengths of a padded batch, uniform in [min(64, seq), seq]."""
    return torch.randint(min(64, seq), seq + 1, (batch,), generator=g, device=DEVICE)


def _prepare_encoder(case, g):
    batch, seq = case["batch"], case["seq"]
    with torch.device("meta"):
        model = _Encoder(batch, seq, case["layers"])
    model = model.half().to_empty(device=DEVICE).eval()
    with torch.no_grad():
        for name, p in model.named_parameters():
            p.normal_(0.0, 0.02, generator=g)
            if "norm" in name and name.endswith("weight"):
                p.add_(1.0)
    gm = dynamo_backend_ofi(torch.fx.symbolic_trace(model))
    ids = torch.randint(0, 30522, (batch, seq), generator=g, device=DEVICE)
    if case["padded"]:
        keep = torch.arange(seq, device=DEVICE)[None, :] < _lengths(batch, seq, g)[:, None]
    else:
        keep = torch.ones((batch, seq), dtype=torch.bool, device=DEVICE)
    with torch.inference_mode():
        forward = cuda_graphs_wrapper(gm, [ids, keep])
    return {"path": "encoder", "forward": forward, "ids": ids, "keep": keep}


def _prepare_llama(case, g, seed):
    cfg = LlamaConfig(n_layers=case["layers"], max_seq=2304)
    model = LlamaTP(cfg, device=DEVICE, dtype=torch.bfloat16, seed=int(seed) % 1000003)
    batch, seq = case["batch"], case["seq"]
    ids = torch.randint(0, cfg.vocab, (batch, seq), generator=g, device=DEVICE)
    if case["path"] == "prefill":
        with torch.inference_mode():
            model.alloc_cache(batch)
        return {"path": "prefill", "model": model, "ids": ids}
    # a serving loop: prompt in, then one graph per token; the logits stay on the device for the sampler
    with torch.inference_mode():
        tokens = model.prefill(ids).float().argmax(-1)

        def step():
            # the same token again at every call: back to the end of the prompt
            model.pos.fill_(seq)
            model.kv_len.fill_(seq)
            return model.decode_step(tokens)

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            logits = step()
    return {"path": "decode", "model": model, "graph": graph, "tokens": tokens, "logits": logits}


def prepare(case, seed):
    g = _generator(seed)
    path = case["path"]
    if path == "encoder":
        return _prepare_encoder(case, g)
    if path in ("prefill", "decode"):
        return _prepare_llama(case, g, seed)
    dtype = getattr(torch, case["dtype"])

    def normal(shape, std=1.0):
        return (torch.randn(shape, generator=g, device=DEVICE) * std).to(dtype)

    if path == "norm":
        rows, cols = case["rows"], case["cols"]
        return {
            "path": path, "rms": case["rms"], "x": normal((rows, cols)),
            "weight": (torch.rand(cols, generator=g, device=DEVICE) + 0.5).to(dtype),
            "bias": None if case["rms"] else normal((cols,), 0.1),
            "residual": normal((rows, cols)) if case["residual"] else None,
        }
    if path == "linear":
        m, k, n = case["M"], case["K"], case["N"]
        return {"path": path, "activation": case["activation"], "x": normal((m, k)), "weight": normal((n, k), 0.02),
                "bias": normal((n,), 0.02) if case["bias"] else None}
    batch, heads, kv_heads, dim = case["batch"], case["heads"], case["kv_heads"], case["dim"]
    if path == "attention":
        seq = case["seq"]

        def operand(h):
            # `split_heads`: the [B, H, S, D] view of a projection's [B, S, H * D] output
            return normal((batch, seq, h, dim)).transpose(1, 2) if case["split_heads"] else normal((batch, h, seq, dim))

        s = {"path": path, "causal": case["causal"], "q": operand(heads), "k": operand(kv_heads), "v": operand(kv_heads), "mask": None}
        if case["mask"] == "padding":
            live = torch.arange(seq, device=DEVICE)[None, :] < _lengths(batch, seq, g)[:, None]
            s["mask"] = torch.where(live, 0.0, float("-inf")).reshape(batch, 1, 1, seq).to(dtype)
        elif case["mask"] == "bias":
            s["mask"] = normal((1, heads, seq, seq), 0.5)
        return s
    assert path == "decode_attention"
    # a KV cache of `capacity` slots; the number of filled ones is read on the device
    s = {"path": path, "q": normal((batch, heads, 1, dim)), "k": normal((batch, kv_heads, case["capacity"], dim)),
         "v": normal((batch, kv_heads, case["capacity"], dim)), "mask": None,
         "kv_len": torch.tensor([case["keys"]], dtype=torch.int64, device=DEVICE)}
    if case["mask"] == "bias":
        s["mask"] = normal((1, heads, 1, case["capacity"]), 0.5)
    return s


@torch.inference_mode()
def run(state):
    path = state["path"]
    if path == "norm":
        return layer_norm(state["x"], state["weight"], state["bias"], 1e-5, use_rms_norm=state["rms"], residual=state["residual"])
    if path == "linear":
        return linear_layer(state["x"], state["weight"], state["bias"], state["activation"])
    if path == "attention":
        q = state["q"]
        return attention_forward(q, state["k"], state["v"], torch.empty_like(q), q.shape[-1] ** -0.5, state["causal"], state["mask"])
    if path == "decode_attention":
        q = state["q"]
        return skinny_attention_forward(q, state["k"], state["v"], torch.empty_like(q), q.shape[-1] ** -0.5, False, state["mask"],
                                        kv_len=state["kv_len"])
    if path == "encoder":
        return state["forward"](state["ids"], state["keep"])
    model = state["model"]
    if path == "prefill":
        logits = model.prefill(state["ids"])
    else:
        state["graph"].replay()
        logits = state["logits"]
    return {"logits": logits, "k": model.kcache, "v": model.vcache}


def _mean_keys(seq, padded):
    """Keys that count, on average over the lengths of a padded batch."""
    return (min(64, seq) + seq) / 2 if padded else seq


def work(case):
    path = case["path"]
    if path == "norm":
        rows, cols = case["rows"], case["cols"]
        return {"bytes": 2.0 * rows * cols * (4 if case["residual"] else 2) + 2.0 * cols * (1 if case["rms"] else 2), "flops": 5.0 * rows * cols}
    if path == "linear":
        m, k, n = case["M"], case["K"], case["N"]
        out = n // 2 if case["activation"] == "swiglu" else n
        return {"bytes": 2.0 * (m * k + n * k + m * out) + (2.0 * n if case["bias"] else 0.0), "flops": 2.0 * m * n * k}
    if path == "attention":
        b, h, hk, s, d = (case[k] for k in ("batch", "heads", "kv_heads", "seq", "dim"))
        keys = _mean_keys(s, case["mask"] == "padding")
        mask = {"none": 0, "padding": b * s, "bias": h * s * s}[case["mask"]]
        pairs = s * (s + 1) / 2 if case["causal"] else s * keys
        return {"bytes": 2.0 * (2 * b * h * s * d + 2 * b * hk * keys * d + mask), "flops": 4.0 * b * h * d * pairs}
    if path == "decode_attention":
        b, h, hk, n, d = (case[k] for k in ("batch", "heads", "kv_heads", "keys", "dim"))
        return {"bytes": 2.0 * (2 * b * h * d + 2 * b * hk * n * d + (h * n if case["mask"] == "bias" else 0)), "flops": 4.0 * b * h * n * d}
    b, s, layers = case["batch"], case["seq"], case["layers"]
    tokens = b * s
    if path == "encoder":
        weights = layers * (4 * 768 * 768 + 2 * 768 * 3072)
        keys = _mean_keys(s, case["padded"])
        # weights once, the embedding rows of the tokens, the hidden states out
        return {"bytes": 2.0 * (weights + 2 * tokens * 768), "flops": 2.0 * tokens * weights + layers * 4.0 * tokens * keys * 768}
    per_layer = 4 * 4096 * 4096 + 3 * 4096 * 11008
    if path == "prefill":
        cache = 2.0 * layers * 2 * tokens * 4096
        return {"bytes": 2.0 * (layers * per_layer + 32000 * 4096 + tokens * 4096) + cache + 2.0 * b * 32000,
                "flops": 2.0 * tokens * layers * per_layer + layers * 4.0 * b * 4096 * s * (s + 1) / 2 + 2.0 * b * 32000 * 4096}
    cache = 2.0 * layers * 2 * b * (s + 1) * 4096
    return {"bytes": 2.0 * (layers * per_layer + 32000 * 4096 + b * 32000) + cache,
            "flops": 2.0 * b * (layers * per_layer + 32000 * 4096) + layers * 4.0 * b * (s + 1) * 4096}


def tolerance(case):
    """Accumulation is fp32 everywhere; what differs between correct implementations is the rounding of
    16-bit intermediates (11 bits of fp16, 8 bits of bf16): one operator rounds its result and, in
    attention, the probabilities; a model does so once per operator and layer."""
    path = case["path"]
    if path == "encoder":
        return {"rel": 6e-3}
    if path in ("prefill", "decode"):
        return {"rel": 2e-2}
    return {"rel": 1e-3} if case["dtype"] == "float16" else {"rel": 8e-3}
