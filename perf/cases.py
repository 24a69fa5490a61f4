"""Cases for timing the framework: one forward step of a decoder, prompts or decoding, as the engine issues them.

A case is one model (sizes of ``ckpt.synthetic.SHAPES``, random weights) and one batch:

* ``decode``: ``seqs`` sequences, one new token each, on a paged cache that holds ``context`` to ``context + spread`` tokens per sequence. The
  step is captured in a CUDA graph beforehand, as the engine does per batch size; a pass copies the new token ids in and replays it.
* ``prefill``: ``seqs`` prompts of ``tokens - spread`` to ``tokens`` new tokens behind ``prefix`` tokens that are already cached (and shared by
  all prompts, as after a hit in the prefix cache). A pass starts from the token ids on the host.

A pass returns the final-normed hidden rows of every token of the step and the logits of the last row of every sequence.

``layers`` is the model's own depth for the two models that fit three times beside their caches, and a few layers of the others, whose
weights repeat layer by layer.
"""
from __future__ import annotations

import math
import random
import zlib

import torch

from deliverance_b200.ckpt.safetensors_io import Q4Tensor
from deliverance_b200.ckpt.synthetic import SHAPES
from deliverance_b200.config import parse_config
from deliverance_b200.kv.paged import KvCacheSettings, PagedKVCache
from deliverance_b200.models.batch import make_batch
from deliverance_b200.models.transformer import DecoderModel

PAGE = 32
LAYERS = {"qwen3-4b": 36, "tinyllama": 22, "mixtral-8x7b": 4, "qwen3-30b-a3b": 6, "gemma2-9b": 8}
QUANTISED = ("qwen3-4b", "qwen3-30b-a3b")  # JQ4 weights; the others are bf16
MAX_SEQS = {"qwen3-4b": 64, "tinyllama": 32, "mixtral-8x7b": 64, "qwen3-30b-a3b": 64, "gemma2-9b": 128}


def _case(name, model, kind, seqs, context=0, tokens=0, prefix=0, spread=0):
    return {"name": name, "model": model, "kind": kind, "seqs": seqs, "context": context, "tokens": tokens, "prefix": prefix, "spread": spread}


def listed():
    return [
        # one user who waits for a small model's answer: the step with the least work, latency and launches are what counts
        _case("tinyllama decode 1", "tinyllama", "decode", 1, context=150),
        # a single request against the 4-bit model, and a few at once: the interactive use of a local server
        _case("qwen3-4b decode 1", "qwen3-4b", "decode", 1, context=777),
        _case("qwen3-4b decode 8", "qwen3-4b", "decode", 8, context=500, spread=1500),
        # a loaded server: the batch of the headline benchmark, contexts behind 2048-token prompts
        _case("qwen3-4b decode 64", "qwen3-4b", "decode", 64, context=2049, spread=255),
        # a chat turn arrives alone: time to first token of a short prompt of odd length
        _case("qwen3-4b prefill 333", "qwen3-4b", "prefill", 1, tokens=333),
        # a full step of the scheduler (8,192 tokens) of long prompts
        _case("qwen3-4b prefill 4x2048", "qwen3-4b", "prefill", 4, tokens=2048),
        # mixture of few large experts in bf16: 64 requests of 1024-token prompts, their prompt steps and their decoding
        _case("mixtral decode 64", "mixtral-8x7b", "decode", 64, context=1025, spread=255),
        _case("mixtral prefill 8x1024", "mixtral-8x7b", "prefill", 8, tokens=1024, spread=100),
        # mixture of many small 4-bit experts: 32 requests of 512-token prompts
        _case("qwen3-30b-a3b decode 32", "qwen3-30b-a3b", "decode", 32, context=513, spread=127),
        _case("qwen3-30b-a3b prefill 16x512", "qwen3-30b-a3b", "prefill", 16, tokens=512),
        # 128 streams behind a shared 1536-token prefix, 256 tokens of their own each: windows, soft-caps, heads of 256, large vocabulary
        _case("gemma2-9b decode 128", "gemma2-9b", "decode", 128, context=1792, spread=256),
        _case("gemma2-9b prefill 32x256", "gemma2-9b", "prefill", 32, tokens=256, prefix=1536),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    model = rng.choice(sorted(LAYERS))
    limit = SHAPES[model]["max_position_embeddings"]
    if rng.random() < 0.5:
        seqs = _log_int(rng, 1, MAX_SEQS[model])
        context = min(_log_int(rng, 17, 4096), limit - 16, 147456 // seqs)
        spread = rng.randrange(0, max(1, min(context, limit - 16 - context, 147456 // seqs - context) + 1))
        return {k: v for k, v in _case("", model, "decode", seqs, context=context, spread=spread).items() if k != "name"}
    total = _log_int(rng, 19, 8192)
    seqs = min(_log_int(rng, 1, 32), max(1, total // 17))
    tokens = min(total // seqs, limit - 16)
    prefix = PAGE * rng.randrange(0, min(1536, limit - 16 - tokens) // PAGE + 1) if rng.random() < 0.4 else 0
    spread = rng.randrange(0, tokens // 2 + 1)
    return {k: v for k, v in _case("", model, "prefill", seqs, tokens=tokens, prefix=prefix, spread=spread).items() if k != "name"}


# ---------------------------------------------------------------------------------------------------------------- weights
def _shape(case):
    return dict(SHAPES[case["model"]], num_hidden_layers=LAYERS[case["model"]])


def _quantise(w):
    """JQ4 of ``[..., K]``: blocks of 32, scale = signed maximum / -8, byte j of a block holds elements j and j + 16."""
    b = w.float().reshape(-1, 32)
    scale = b.gather(1, b.abs().argmax(1, keepdim=True)) / -8.0
    inv = torch.where(scale != 0, 1.0 / scale, torch.zeros_like(scale))
    q = torch.trunc(b * inv + 8.5).clamp_(0, 15).to(torch.uint8)
    packed = q[:, :16] | (q[:, 16:] << 4)
    return packed.reshape(*w.shape[:-1], w.shape[-1] // 2), scale.reshape(*w.shape[:-1], w.shape[-1] // 32)


def _dequantise64(packed, scales):
    p = packed.reshape(-1, 16)
    v = torch.cat([p & 15, p >> 4], 1).double().sub_(8.0).mul_(scales.reshape(-1, 1).double())
    return v.reshape(*packed.shape[:-1], packed.shape[-1] * 2)


class Weights:
    """A random checkpoint in the shape that a model's loader reads, made on the GPU tensor by tensor from the seed."""

    def __init__(self, case, seed, device="cuda"):
        self.s, self.seed, self.device = _shape(case), int(seed), device
        self.q4 = case["model"] in QUANTISED
        self.tied = self.s["tie_word_embeddings"]
        self._experts: dict = {}

    def _normal(self, name, shape, std):
        g = torch.Generator(device=self.device).manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
        return torch.empty(shape, dtype=torch.bfloat16, device=self.device).normal_(0.0, std, generator=g)

    def _dims(self, name):
        s = self.s
        h, hd = s["hidden_size"], s.get("head_dim") or s["hidden_size"] // s["num_attention_heads"]
        inner = s.get("moe_intermediate_size") or s["intermediate_size"]
        E = s.get("num_experts") or s.get("num_local_experts") or 0
        end = name.split(".")[-2]
        return {"embed_tokens": (s["vocab_size"], h), "lm_head": (s["vocab_size"], h), "q_proj": (s["num_attention_heads"] * hd, h),
                "k_proj": (s["num_key_value_heads"] * hd, h), "v_proj": (s["num_key_value_heads"] * hd, h), "o_proj": (h, s["num_attention_heads"] * hd),
                "gate_proj": (inner, h), "up_proj": (inner, h), "down_proj": (h, inner), "w1": (inner, h), "w3": (inner, h), "w2": (h, inner),
                "gate": (E, h), "q_norm": (hd,), "k_norm": (hd,)}.get(end, (h,))

    def dense(self, name):
        """The checkpoint's bf16 tensor."""
        shape = self._dims(name)
        if name.endswith("norm.weight"):
            gemma = self.s["model_type"] == "gemma2"  # stored as w - 1; the norms behind its sublayers scale what enters the stream
            return self._normal(name, shape, 0.02) + ((-0.7 if name.endswith(("post_attention_layernorm.weight", "post_feedforward_layernorm.weight")) else 0.0) if gemma else 1.0)
        if name.endswith(".gate.weight"):  # router: logits of about 8, so that rounding does not decide who is chosen
            return self._normal(name, shape, 8.0 / math.sqrt(shape[1]))
        return self._normal(name, shape, self._std(name))

    def _std(self, name):
        """Spread of a projection: 0.02, less for those that write to the residual stream (by the root of their number, so that depth does not
        magnify rounding), and embeddings that start the stream at about 1."""
        if "embed_tokens" in name:
            return 0.02 if self.s["model_type"] == "gemma2" else 1.0
        if name.endswith(("o_proj.weight", "down_proj.weight", "w2.weight")):
            return 0.7 / math.sqrt(self._dims(name)[1] * 2 * self.s["num_hidden_layers"])
        return 0.02

    def stacked(self, prefix, end):
        """``[experts, N, K]`` of one projection of a layer's experts, as stored."""
        name = f"{prefix}{end}.weight"
        if name not in self._experts:
            if len(self._experts) >= 3:
                self._experts.clear()
            E = self.s.get("num_experts") or self.s["num_local_experts"]
            w = self._normal(name, (E,) + self._dims(name), self._std(name))
            self._experts[name] = _quantise(w) if self.q4 else w
        return self._experts[name]

    def has(self, name):
        return not (name == "lm_head.weight" and self.tied) and not name.endswith(".bias") and (
            not name.endswith(("q_norm.weight", "k_norm.weight")) or self.s["model_type"] in ("qwen3", "qwen3_moe"))

    def is_q4(self, name):
        return self.q4 and "_proj." in name

    def load(self, name, shard=None):
        if ".experts." in name:
            prefix, rest = name.split("experts.")
            e, end = rest.split(".")[:2]
            w = self.stacked(prefix + "experts.", end)
            if not self.q4:
                return w[int(e)]
            return Q4Tensor(w[0][int(e)], w[1][int(e)], self._dims(name))
        w = self.dense(name)
        return Q4Tensor(*_quantise(w), tuple(w.shape)) if self.is_q4(name) else w

    def load_dense(self, name, dtype=torch.float32, shard=None):
        return self.dense(name).to(dtype)


# ---------------------------------------------------------------------------------------------------------------- inputs
def _plan(case, seed):
    """Host-side description of the batch: per sequence new tokens, first position and pages; and the number of pages."""
    rng, lengths = random.Random(int(seed)), random.Random(7)  # the lengths belong to the case, the tokens to the seed
    vocab = SHAPES[case["model"]]["vocab_size"]
    seqs, shared = [], case["prefix"] // PAGE
    for _ in range(case["seqs"]):
        if case["kind"] == "decode":
            start, n = case["context"] + lengths.randint(0, case["spread"]) - 1, 1
        else:
            start, n = case["prefix"], case["tokens"] - lengths.randint(0, case["spread"])
        seqs.append({"tokens": [rng.randrange(vocab) for _ in range(n)], "start": start})
    own = [(s["start"] + len(s["tokens"]) + PAGE - 1) // PAGE - shared for s in seqs]
    order = list(range(1 + shared, 1 + shared + sum(own)))
    rng.shuffle(order)  # a pool that has been in use hands out pages in any order; page 0 is nobody's
    for s, n in zip(seqs, own):
        s["pages"] = list(range(1, 1 + shared)) + order[:n]
        order = order[n:]
    return seqs, 1 + shared + sum(own)


def _fill(kv, seed):
    g = torch.Generator(device=kv.k[0].device).manual_seed(int(seed) & 0x7FFFFFFF)
    for k, v in zip(kv.k, kv.v):
        k.normal_(0.0, 1.0, generator=g)
        v.normal_(0.0, 1.0, generator=g)


def _splits(seqs, kv_heads):
    """Split-KV factor of decode attention, as the engine picks it: the smallest that fills two CTAs per SM evenly."""
    best, share = 1, 0.0
    for s in range(1, 33):
        n = max(1, seqs * kv_heads) * s
        if n / (-(-n // 296) * 296) > share + 0.03:
            best, share = s, n / (-(-n // 296) * 296)
    return best


def _forward(model, kv, batch):
    h = model.forward_hidden(batch, kv)
    rows = h if batch.is_decode else h.index_select(0, batch.logits_rows)
    return {"hidden": h, "logits": model.logits(rows)}


def prepare(case, seed):
    dev = torch.device("cuda")
    model = DecoderModel(parse_config(_shape(case)), dev, torch.bfloat16).load(Weights(case, seed), head_quant="Q4" if case["model"] in QUANTISED else None)
    seqs, pages = _plan(case, seed)
    kv = PagedKVCache(model.kv_layout(), pages, dev, torch.bfloat16, KvCacheSettings(enabled=False, block_size=PAGE))
    _fill(kv, seed)
    state = {"model": model, "kv": kv, "seqs": seqs}
    if case["kind"] == "decode":
        batch = make_batch(seqs, PAGE, dev)
        batch.decode_splits = _splits(case["seqs"], model.n_kv)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                _forward(model, kv, batch)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _forward(model, kv, batch)
        state.update(batch=batch, graph=graph, out=out, ids=batch.token_ids.cpu().pin_memory())
    return state


def run(state):
    if "graph" in state:
        state["batch"].token_ids.copy_(state["ids"], non_blocking=True)
        state["graph"].replay()
        return state["out"]
    batch = make_batch(state["seqs"], PAGE, state["model"].device)
    return _forward(state["model"], state["kv"], batch)


# ---------------------------------------------------------------------------------------------------------------- what a pass needs
def work(case):
    """Weights that take part once (4-bit blocks: 0.625 bytes per weight), cached keys and values that are visible once, new ones, hidden
    rows and logits. Shared prefixes are read once. For experts, the expected number of distinct ones that uniform routing touches."""
    s = _shape(case)
    L, h, H, KV = s["num_hidden_layers"], s["hidden_size"], s["num_attention_heads"], s["num_key_value_heads"]
    hd = s.get("head_dim") or h // H
    E, k = s.get("num_experts") or s.get("num_local_experts") or 0, s.get("num_experts_per_tok", 0)
    inner = s.get("moe_intermediate_size") if E and s.get("moe_intermediate_size") else s["intermediate_size"]
    per = 0.625 if case["model"] in QUANTISED else 2.0
    S, decode = case["seqs"], case["kind"] == "decode"
    n = 1 if decode else case["tokens"] - case["spread"] / 2
    start = case["context"] + case["spread"] / 2 - 1 if decode else case["prefix"]
    T = S * n
    attn = h * hd * (2 * H + 2 * KV)
    touched = E * (1 - (1 - k / E) ** T) if E else 1
    weights = L * (attn + 3 * h * inner * touched) * per + L * E * h * 2 + s["vocab_size"] * h * per
    window = s.get("sliding_window") or 0
    scores = kv_rows = 0.0
    for i in range(L):
        w = window if window and i % 2 == 0 else 1 << 30
        scores += S * n * min(w, start + (n + 1) / 2)
        seen = min(w + n, start + n)
        kv_rows += S * seen if decode or not case["prefix"] else S * n + start
    flops = 2.0 * T * L * (attn + 3 * h * inner * max(1, k) + E * h) + 2.0 * S * s["vocab_size"] * h + 4.0 * scores * H * hd
    moved = weights + kv_rows * KV * hd * 2 * 2 + T * h * 2 * 2 + S * s["vocab_size"] * 4
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """bf16 activations and residual stream: against 64 bits the rows are 0.006 (4 layers) to 0.015 (36 layers) off in the 2-norm and single values
    up to 0.08. Where two experts are nearly tied, rounding can choose the other one, and a row of that token is off as a whole."""
    return {"rel": 0.03, "max": 0.99 if case["model"] == "mixtral-8x7b" else 0.4}


# ---------------------------------------------------------------------------------------------------------------- 64 bits
def exact(case, seed):
    """The same step in 64-bit torch: dequantised weights, dense attention over the cached rows, every chosen expert."""
    s, W, dev = _shape(case), Weights(case, seed), torch.device("cuda")
    seqs, pages = _plan(case, seed)
    L, h, H, KV, eps = s["num_hidden_layers"], s["hidden_size"], s["num_attention_heads"], s["num_key_value_heads"], s["rms_norm_eps"]
    hd = s.get("head_dim") or h // H
    gemma, kind = s["model_type"] == "gemma2", s["model_type"]
    cap, window = s.get("attn_logit_softcapping") or 0.0, s.get("sliding_window") or 0
    scale = (s.get("query_pre_attn_scalar") or hd) ** -0.5
    g = torch.Generator(device=dev).manual_seed(int(seed) & 0x7FFFFFFF)
    cache = torch.empty(pages, KV, PAGE, hd, dtype=torch.bfloat16, device=dev)

    def lin(x, name):
        w = W.dense(name)
        w = _dequantise64(*_quantise(w)) if W.is_q4(name) else w.double()
        return x @ w.t()

    def norm(x, name):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * (W.dense(name).double() + (1.0 if gemma else 0.0))

    def act(x):
        return torch.nn.functional.gelu(x, approximate="tanh") if gemma else torch.nn.functional.silu(x)

    pos = torch.cat([torch.arange(q["start"], q["start"] + len(q["tokens"])) for q in seqs]).to(dev)
    angle = pos.double()[:, None] * (float(s["rope_theta"]) ** (-torch.arange(0, hd, 2, dtype=torch.float64, device=dev) / hd))[None]
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rotate(x):
        a, b = x[..., : hd // 2], x[..., hd // 2 :]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def attention(x, p, i):
        q, k, v = (lin(x, p + f"self_attn.{n}_proj.weight").reshape(x.shape[0], -1, hd) for n in "qkv")
        if W.has(p + "self_attn.q_norm.weight"):
            q, k = norm(q, p + "self_attn.q_norm.weight"), norm(k, p + "self_attn.k_norm.weight")
        q, k = rotate(q), rotate(k)
        old = [cache.normal_(0.0, 1.0, generator=g).clone() for _ in range(2)]
        out, row = torch.empty_like(q), 0
        for sq in seqs:
            n, start = len(sq["tokens"]), sq["start"]
            idx = torch.tensor(sq["pages"], device=dev)
            K, V = (torch.cat([o[idx].permute(1, 0, 2, 3).reshape(KV, -1, hd)[:, :start].double(), t[row : row + n].transpose(0, 1)], 1) for o, t in zip(old, (k, v)))
            Q = q[row : row + n].reshape(n, KV, H // KV, hd).permute(1, 2, 0, 3)
            sc = torch.einsum("kgqd,kjd->kgqj", Q, K) * scale
            if cap:
                sc = torch.tanh(sc / cap) * cap
            at, j = torch.arange(start, start + n, device=dev)[:, None], torch.arange(start + n, device=dev)[None]
            hide = j > at
            if window and gemma and i % 2 == 0:
                hide = hide | (j <= at - window)
            out[row : row + n] = torch.einsum("kgqj,kjd->qkgd", torch.softmax(sc.masked_fill_(hide, -math.inf), -1), V).reshape(n, H, hd)
            row += n
        return lin(out.reshape(x.shape[0], -1), p + "self_attn.o_proj.weight")

    def experts(x, p):
        mix = kind == "mixtral"
        logits = lin(x, p + ("block_sparse_moe.gate.weight" if mix else "mlp.gate.weight"))
        prob, idx = torch.softmax(logits, -1).topk(s["num_experts_per_tok"], -1)
        prob = prob / prob.sum(-1, keepdim=True)
        ep, ends = (p + "block_sparse_moe.experts.", ("w1", "w3", "w2")) if mix else (p + "mlp.experts.", ("gate_proj", "up_proj", "down_proj"))
        ws = [W.stacked(ep, e) for e in ends]
        y = torch.zeros_like(x)
        for e in range(logits.shape[1]):
            rows, slot = (idx == e).nonzero(as_tuple=True)
            if rows.numel():
                gate, up, down = (_dequantise64(w[0][e], w[1][e]) if W.q4 else w[e].double() for w in ws)
                y.index_add_(0, rows, (act(x[rows] @ gate.t()) * (x[rows] @ up.t())) @ down.t() * prob[rows, slot][:, None])
        return y

    embed = W.dense("model.embed_tokens.weight")
    x = embed[torch.tensor([t for q in seqs for t in q["tokens"]], device=dev)].double()
    if gemma:
        x = x * float(torch.tensor(math.sqrt(h)).to(torch.bfloat16))
    for i in range(L):
        p = f"model.layers.{i}."
        a = attention(norm(x, p + "input_layernorm.weight"), p, i)
        x = x + (norm(a, p + "post_attention_layernorm.weight") if gemma else a)
        f = norm(x, p + ("pre_feedforward_layernorm.weight" if gemma else "post_attention_layernorm.weight"))
        if "num_experts_per_tok" in s:
            f = experts(f, p)
        else:
            f = lin(act(lin(f, p + "mlp.gate_proj.weight")) * lin(f, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
        x = x + (norm(f, p + "post_feedforward_layernorm.weight") if gemma else f)
    x = norm(x, "model.norm.weight")
    ends, at = [], 0
    for q in seqs:
        at += len(q["tokens"])
        ends.append(at - 1)
    head = embed if W.tied else W.dense("lm_head.weight")
    head = _dequantise64(*_quantise(head)) if W.q4 else head.double()
    return {"hidden": x, "logits": x[torch.tensor(ends, device=dev)] @ head.t()}
