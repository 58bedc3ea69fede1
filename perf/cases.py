"""The engine's work as its users have it done: prompts, decode turns and whole batches of requests.

Three kinds of pass:

* "prompt": one request's prompt through the step function (`EngineCore.stepper.step`, what `bin/trace_run` drives), in
  portions of at most 2,048 tokens; the last token's logits.
* "decode": one turn of continuous batching with nothing but live requests in it (`LocalModel.backend.run`, what the
  scheduler calls every turn: a captured graph, sampling, the tokens read back), each at some length; logits. The
  requests are rolled back afterwards, so that every pass does the same.
* "serve": whole requests through `LocalModel.generate` (scheduler, prompt portions beside decoding requests, captured
  decode steps, sampling), several at a time. The reply is given, as in scoring: with random weights a token is decided
  by the last bit now and then, and everything after it would be another text. The sampled tokens are drawn and read
  back as always, then replaced. The result is every request's logits for its last token.

Models: the Llama-3.1-8B widths with sixteen layers and the Llama-3.2-1B shape with eight (the benchmark's shapes), a
Llama of the 1B widths in 32-bit, and the three recurrent designs at the benchmark's "1b" widths. Their feed-forwards are the
dense ones: a routed layer sends a token to another expert on a near tie, and no two implementations would agree.
"""
from __future__ import annotations

import gc
import math

import torch

from cuca_b200 import BatchingConfig, LocalModel, LocalModelConfig, RandomWeights
from cuca_b200.config.registry import build_spec
from cuca_b200.engine.core import EngineCore
from cuca_b200.engine.graphs import DecodeGraphs
from cuca_b200.engine.scheduler import Plan, Request, Sequence_
from cuca_b200.engine.step import StepEntry
from cuca_b200.models.model import Model
from cuca_b200.weights.loader import WeightSource

PORTION = 2048  # tokens of one step at most
PAGE = 16


# ------------------------------------------------------------------------------------------------------- models
def _llama(layers, width, heads, kv, dim, ff, vocab, factor, tied):
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": layers,
            "hidden_size": width, "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": dim,
            "intermediate_size": ff, "vocab_size": vocab, "max_position_embeddings": 131072, "rms_norm_eps": 1e-5,
            "rope_theta": 500000.0, "tie_word_embeddings": tied,
            "rope_scaling": {"rope_type": "llama3", "factor": factor, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                             "original_max_position_embeddings": 8192}}


def _config(model):
    """config.json of a case's model."""
    width, ff, H, vocab, window = 2048, 8192, 16, 32000, 1024
    if model == "llama-8b":
        return _llama(16, 4096, 32, 8, 128, 14336, 128256, 8.0, False)
    if model == "llama-1b":
        return _llama(8, 2048, 32, 8, 64, 8192, 128256, 32.0, True)
    if model == "llama-f32":
        return _llama(4, 2048, 32, 8, 64, 8192, 32000, 32.0, True)
    if model == "bananex":
        dense = {"kind": "dense", "ff": ff}
        d = width // H
        kinds = [{"type": "latent_attention", "mlp": dense,
                  "mixer": {"heads": H, "dim": d, "rot_dim": d // 2, "vdim": d, "kv_rank": 4 * d, "mask": {"size": window},
                            "rot": {"base": 10000.0, "dims": d // 2}, "scale": (d + d // 2) ** -0.5}},
                 {"type": "mingru", "mlp": dense, "mixer": {"width": width}},
                 {"type": "mamba2", "mlp": dense,
                  "mixer": {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}}]
        return {"architecture": "Bananex", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "logit_scale": 1.0,
                "layers": [kinds[i % 3] for i in range(6)], "loop": {"start": 0, "stop": 3, "times": 2}}
    if model == "dupenex":
        dense = {"kind": "dense", "ff": ff}
        delta = {"type": "channel_delta", "mlp": dense,
                 "mixer": {"heads": H, "kv_heads": H, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}}
        side = {"type": "parallel", "mlp": dense,
                "mixer": {"left": {"heads": H // 2, "kv_heads": H // 4, "dim": 128, "vdim": 256, "mask": {"size": window},
                                   "rot": {"base": 250000.0, "dims": 64}, "scale": 128 ** -0.5},
                          "right": {"heads": H // 4, "dim": 128, "vdim": 256, "gate_cap": 15.0}}}
        return {"architecture": "Dupenex", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "streams": 4,
                "layers": [side if i % 3 == 1 else delta for i in range(6)]}
    if model == "pudinex":
        dense = {"kind": "dense", "ff": ff, "limit": 7.0}
        attention = {"type": "attention", "mlp": dense,
                     "mixer": {"heads": H, "kv_heads": H // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
                               "rot": {"base": 10000.0, "dims": 64,
                                       "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
        forget = {"type": "hgrn2", "mlp": dense, "mixer": {"heads": H, "dim": 128, "vdim": 128}}
        return {"architecture": "Pudinex", "vocab": vocab, "width": width, "norm": {"eps": 1e-6, "groups": 2},
                "embedding": {"scale": 1.0}, "layers": [attention if i % 3 == 2 else forget for i in range(6)]}
    raise ValueError(model)


def _dtype(model):
    return torch.float32 if model == "llama-f32" else torch.bfloat16


class _Weights(WeightSource):
    """Weights in memory, one normal stream a model: matrices with unit gain, norm weights about 1, and what is no matrix
    (decays, step sizes, biases, mixes of the streams) spread so that every mechanism does something."""

    def __init__(self, model, seed):
        self.needs = Model(build_spec(_config(model)), runtime=None).tensor_needs()
        self.dtype = _dtype(model)
        self.seed = seed
        self.embed_gain = 0.05 if _config(model).get("tie_word_embeddings") else 1.0  # a tied table is the head too

    def shapes(self):
        return {n: tuple(t.shape) for n, t in self.needs.items()}

    def read(self, name):
        need = self.needs[name]
        shape, dev = tuple(need.shape), "cuda"
        g = torch.Generator(device=dev).manual_seed((self.seed * 1000003 + sum((i + 1) * ord(c) for i, c in enumerate(name))) % (1 << 62))
        big = len(shape) == 2 and min(shape) > 8
        if big:
            v = torch.randn(shape, device=dev, generator=g, dtype=self.dtype)
            return v.mul_(self.embed_gain if "embed" in name else shape[-1] ** -0.5)
        normal = lambda mean, std: mean + std * torch.randn(shape, device=dev, generator=g)  # noqa: E731
        even = lambda a, b: a + (b - a) * torch.rand(shape, device=dev, generator=g)  # noqa: E731
        if name.endswith(".hc1.mix") or name.endswith(".hc2.mix"):
            v = 0.8 * torch.eye(shape[0], device=dev) + normal(0.0, 0.1)
        elif name.endswith(".hc1.in") or name.endswith(".hc2.in"):
            v = even(0.3, 0.6)
        elif name.endswith(".hc1.out") or name.endswith(".hc2.out"):
            v = normal(0.6, 0.2)
        elif name.endswith(".shift"):
            v = even(0.0, 1.0)
        elif name.endswith("A_log"):
            v = even(-1.5, 1.0)
        elif name.endswith("dt_bias"):
            v = even(-2.0, 1.0)
        elif name.endswith(".lower"):
            v = even(0.0, 0.9)
        elif name.endswith(".f.b"):
            v = normal(2.0, 1.0)
        elif name.endswith(".conv"):
            v = normal(0.0, 0.5)
        elif name.endswith(".D") or need.init == "ones":
            v = normal(1.0, 0.1)
        elif name.endswith(".b") or name == "loop.step":
            v = normal(0.0, 0.3)
        else:
            v = normal(0.0, shape[-1] ** -0.5)
        return v.to(self.dtype)


# -------------------------------------------------------------------------------------------------------- cases
def listed():
    """Chosen by use: the benchmark's decode batches and prompt, prompts on both sides of it, a mixed batch under continuous
    batching, the 32-bit mode in both directions, and the recurrent designs in both."""
    return [
        # a chat with one user: every token waits for the whole model
        {"name": "llama-8b decode 1", "kind": "decode", "model": "llama-8b", "batch": 1, "context": 1035},
        # a small server's turn, the benchmark's default
        {"name": "llama-8b decode 8", "kind": "decode", "model": "llama-8b", "batch": 8, "context": 1035},
        # the largest batch the engine takes
        {"name": "llama-8b decode 64", "kind": "decode", "model": "llama-8b", "batch": 64, "context": 1035},
        # a question in a chat: ragged, below the default portion of 256
        {"name": "llama-8b prompt 203", "kind": "prompt", "model": "llama-8b", "tokens": 203},
        # the benchmark's prompt: one whole portion
        {"name": "llama-8b prompt 2048", "kind": "prompt", "model": "llama-8b", "tokens": 2048},
        # a document: three portions, the last one ragged, over keys of the earlier ones
        {"name": "llama-8b prompt 6001", "kind": "prompt", "model": "llama-8b", "tokens": 6001},
        # requests of mixed length under continuous batching, head size 64, sampled
        {"name": "llama-1b serve 24", "kind": "serve", "model": "llama-1b", "batch": 24, "tokens": 400, "reply": 24,
         "temperature": 0.8},
        # checking a checkpoint in the true 32-bit mode, both directions
        {"name": "f32 prompt 700", "kind": "prompt", "model": "llama-f32", "tokens": 700},
        {"name": "f32 decode 4", "kind": "decode", "model": "llama-f32", "batch": 4, "context": 515},
        # the recurrent designs: a long prompt each way, and a batch of short requests
        {"name": "bananex prompt 2048", "kind": "prompt", "model": "bananex", "tokens": 2048},
        {"name": "dupenex prompt 1501", "kind": "prompt", "model": "dupenex", "tokens": 1501},
        {"name": "pudinex serve 8", "kind": "serve", "model": "pudinex", "batch": 8, "tokens": 250, "reply": 24,
         "temperature": 0.0},
    ]


def draw(rng):
    def between(a, b):
        """Log-uniform whole number, a..b."""
        return min(b, max(a, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    model = rng.choice(["llama-8b", "llama-8b", "llama-8b", "llama-1b", "llama-f32", "bananex", "dupenex", "pudinex"])
    recurrent = model in ("bananex", "dupenex", "pudinex")
    kind = rng.choice(["prompt", "serve"] if recurrent else ["serve"] if model == "llama-1b" else ["prompt", "decode"])
    if kind == "prompt":
        top = {"llama-8b": 6000, "llama-f32": 700}.get(model, 2048)
        return {"kind": kind, "model": model, "tokens": between(16, top)}
    if kind == "decode":
        return {"kind": kind, "model": model, "batch": between(1, 64 if model == "llama-8b" else 8),
                "context": between(16, 1035 if model == "llama-8b" else 700)}
    return {"kind": kind, "model": model, "batch": between(1, 8 if recurrent else 24), "tokens": between(16, 400),
            "reply": rng.randint(16, 24), "temperature": rng.choice([0.0, 0.8])}


def _prompt_lengths(case):
    """Request i's prompt: between a half and three halves of `tokens`, spread by the golden ratio."""
    return [max(1, int(case["tokens"] * (0.5 + (i * 0.6180339887 + 0.31) % 1.0))) for i in range(case["batch"])]


def _tokens(case, seed, n):
    vocab = _vocab(case["model"])
    g = torch.Generator().manual_seed(seed * 7919 + 17)
    return torch.randint(0, vocab, (n,), generator=g).tolist()


def _vocab(model):
    c = _config(model)
    return c["vocab_size"] if "vocab_size" in c else c["vocab"]


class _GivenReply:
    """The engine's backend with a given reply in the place of the sampled tokens."""

    def __init__(self, backend):
        self.backend, self.first_id, self.replies, self.logits = backend, 0, [], []

    def start(self, seq):
        self.backend.start(seq)

    def run(self, plans):
        self.backend.run(plans)
        out = []
        for i, p in enumerate(plans):
            if not p.want_last:
                continue
            r, at = p.seq.id - self.first_id, len(p.seq.completion)
            out.append(self.replies[r][at])
            if at + 1 == len(self.replies[r]):
                self.logits[r] = self.backend.last_graph.logits[i].clone()
        return out


def prepare(case, seed):
    gc.collect()  # (a dropped engine's graphs and tensors hang in reference cycles)
    model, kind = case["model"], case["kind"]
    cfg = _config(model)
    if kind == "prompt":
        n, batch, context = case["tokens"], 1, case["tokens"] + PAGE
        kv = context + PAGE
    elif kind == "decode":
        n, batch, context = case["batch"] * (case["context"] + 1), case["batch"], case["context"] + 2 * PAGE
        kv = batch * (context + PAGE)
    else:
        lengths = _prompt_lengths(case)
        n, batch = sum(lengths) + case["batch"] * case["reply"], case["batch"]
        context = max(lengths) + case["reply"] + PAGE
        kv = max(sum(lengths) + batch * (case["reply"] + 2 * PAGE), context + PAGE)
    ids = _tokens(case, seed, n)
    config = LocalModelConfig(model_config=cfg, random_weights=RandomWeights(), context_length=context, kv_block_size=PAGE,
                              dtype="float32" if _dtype(model) == torch.float32 else "bfloat16",
                              batching=BatchingConfig(max_sequences=batch, kv_tokens=kv, max_step_tokens=PORTION,
                                                      prefill_chunk=PORTION))
    sizes = config.resolve(1 << 20)
    core = EngineCore(build_spec(cfg), _Weights(model, seed), dtype=_dtype(model), context_length=context,
                      kv_tokens=sizes["kv_tokens"], max_sequences=batch, block_size=PAGE, max_step_tokens=PORTION)
    if kind == "prompt":
        return {"case": case, "core": core, "tokens": ids}
    DecodeGraphs.keep_logits = True
    local = LocalModel(core, config, sizes, None)
    if kind == "serve":
        forced = _GivenReply(local.backend)
        local.scheduler.backend = forced
        prompts, replies, at = [], [], 0
        for length in lengths:
            prompts.append(ids[at:at + length])
            replies.append(ids[at + length:at + length + case["reply"]])
            at += length + case["reply"]
        return {"case": case, "local": local, "forced": forced, "prompts": prompts, "replies": replies}
    # decode: requests of `context` cached tokens, each with its next token
    seqs, tokens, length = [], [], case["context"]
    for i in range(batch):
        mine = ids[i * (length + 1):(i + 1) * (length + 1)]
        seq = Sequence_(Request(mine[:length], temperature=0.0), i, mine[:length], length, 1, 0)
        seq.blocks, seq.slot = core.pools.new_seq(), core.slots.alloc()
        local.backend.start(seq)
        for a in range(0, length, PORTION):
            part = mine[a:min(length, a + PORTION)]
            core.pools.reserve(seq.blocks, a + len(part))
            core.stepper.step([StepEntry(seq.blocks, seq.slot, part, [])])
        seqs.append(seq)
        tokens.append(mine[length])
    return {"case": case, "local": local, "seqs": seqs, "tokens": tokens}


def run(state):
    kind = state["case"]["kind"]
    if kind == "prompt":
        core, tokens = state["core"], state["tokens"]
        blocks, slot = core.pools.new_seq(), core.slots.alloc()
        core.cache.clear_slot(slot)
        for a in range(0, len(tokens), PORTION):
            part = tokens[a:a + PORTION]
            core.pools.reserve(blocks, a + len(part))
            last = a + len(part) == len(tokens)
            logits = core.stepper.step([StepEntry(blocks, slot, part, [len(part) - 1] if last else [])])
        core.pools.release(blocks)
        core.slots.release(slot)
        return {"logits": logits, "cache": _cache(core)}
    local = state["local"]
    if kind == "serve":
        forced, case = state["forced"], state["case"]
        forced.first_id, forced.replies = local.scheduler._next_id, state["replies"]
        forced.logits = [None] * case["batch"]
        local.generate(state["prompts"], max_tokens=case["reply"], temperature=case["temperature"], top_k=64, top_p=0.95, seed=7)
        return {"logits": torch.stack(forced.logits)}
    length, pools = state["case"]["context"], local.core.pools
    for seq in state["seqs"]:
        pools.reserve(seq.blocks, length + 1)
    local.backend.run([Plan(seq, [t], True, length) for seq, t in zip(state["seqs"], state["tokens"])])
    for seq in state["seqs"]:
        pools.truncate(seq.blocks, length)
    return {"logits": local.backend.last_graph.logits[:len(state["seqs"])], "cache": _cache(local.core)}


def _cache(core):
    """The keys, values and states that a pass leaves behind: the engine's own buffers."""
    return [t for t in core.cache.k + core.cache.v if t is not None] + list(core.cache._state_tensors())


# --------------------------------------------------------------------------------------------- what a pass costs
def _counts(model):
    """(parameters a token is multiplied with except the head, the head's, bytes of a parameter, cached values a token,
    flops a token and earlier token in the attentions, window of the attentions or None, state values a request)."""
    c, needs = _config(model), Model(build_spec(_config(model)), runtime=None).tensor_needs()
    size = 4 if _dtype(model) == torch.float32 else 2
    mats = {n: t.shape[0] * t.shape[1] for n, t in needs.items() if len(t.shape) == 2}
    if "hidden_size" in c:
        L, H, G, d = c["num_hidden_layers"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        head = c["vocab_size"] * c["hidden_size"]
        body = sum(v for n, v in mats.items() if "embed" not in n and "lm_head" not in n)
        return body, head, size, 2 * G * d * L, 4 * H * d * L, None, 0
    head, body, runs = mats["head"], 0, _runs(c)
    cached = attend = kept = 0
    for i in runs:
        body += sum(v for n, v in mats.items() if n.startswith("l%d." % i))
        kind, m = c["layers"][i]["type"], c["layers"][i]["mixer"]
        if kind == "latent_attention":
            cached += m["kv_rank"] + m["rot_dim"]
            attend += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif kind == "mingru":
            kept += m["width"]
        elif kind == "mamba2":
            kept += m["heads"] * m["vdim"] * m["state"]
        elif kind in ("channel_delta", "hgrn2"):
            kept += m["heads"] * m["dim"] * m["vdim"]
        elif kind == "attention":
            cached += m["kv_heads"] * (m["dim"] + m["vdim"])
            attend += 2 * m["heads"] * (m["dim"] + m["vdim"])
        elif kind == "parallel":
            a, r = m["left"], m["right"]
            cached += a["kv_heads"] * (a["dim"] + a["vdim"])
            attend += 2 * a["heads"] * (a["dim"] + a["vdim"])
            kept += r["heads"] * r["dim"] * r["vdim"]
    window = None if model == "pudinex" else 1024
    return body, head, size, cached, attend, window, kept


def work(case):
    body, head, size, cached, attend, window, kept = _counts(case["model"])

    def pairs(first, n):
        """(token, visible token) pairs of tokens first .. first + n - 1"""
        if window is None:
            return n * first + n * (n + 1) / 2
        return sum(min(window, p + 1) for p in range(first, first + n))

    def state(n_requests):  # read and written, 32-bit
        return 8 * kept * n_requests

    if case["kind"] == "prompt":
        n = case["tokens"]
        steps = -(-n // PORTION)
        return {"bytes": (body * steps + head) * size + n * cached * size + state(steps),
                "flops": 2.0 * body * n + 2.0 * head + attend * pairs(0, n) + 4.0 * kept * n}
    if case["kind"] == "decode":
        b, p = case["batch"], case["context"]
        return {"bytes": (body + head) * size + b * (p + 1) * cached * size + state(b) + 4 * b * _vocab(case["model"]),
                "flops": 2.0 * (body + head) * b + attend * b * pairs(p, 1) + 4.0 * kept * b}
    # serve: the prompts' portions, then every further token of the replies reads the model again
    b, r, lengths = case["batch"], case["reply"], _prompt_lengths(case)
    steps = -(-sum(lengths) // PORTION) + r - 1
    seen = sum(min(window or 1 << 30, l + j) for l in lengths for j in range(1, r))
    return {"bytes": (body + head) * size * steps + (seen + sum(lengths)) * cached * size + state(b * r),
            "flops": 2.0 * body * (sum(lengths) + b * (r - 1)) + 2.0 * head * b * r
                     + attend * sum(pairs(0, l + r - 1) for l in lengths) + 4.0 * kept * (sum(lengths) + b * (r - 1))}


def tolerance(case):
    """Four times what the engine is off from 64 bits: 4.6e-6 in 32-bit; in bfloat16 0.004 to 0.006, 0.01 with eight layers
    under a tied table or with the matrix memory's division."""
    if _dtype(case["model"]) == torch.float32:
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 0.03 if case["model"] in ("llama-1b", "dupenex") else 0.025, "max": 0.5}


# ------------------------------------------------------------------------------- the same in 64 bits, plain torch
def exact(case, seed):
    """Logits in 64 bits; None in the place of what the cache keeps."""
    model = case["model"]
    if case["kind"] == "decode" and case["batch"] * case["context"] > 40000:
        return None  # (tens of seconds)
    torch.cuda.empty_cache()
    c, source = _config(model), _Weights(model, seed)

    def w(name):
        return source.read(name).double()

    if case["kind"] == "serve":
        lengths, ids, rows, at = _prompt_lengths(case), None, [], 0
        ids = _tokens(case, seed, sum(lengths) + case["batch"] * case["reply"])
        groups = []
        for length in lengths:  # the last token of a reply is sampled, not fed
            n = length + case["reply"]
            groups.append(ids[at:at + n - 1])
            at += n
        logits = _forward(c, w, groups)
        return {"logits": logits}
    if case["kind"] == "prompt":
        return {"logits": _forward(c, w, [_tokens(case, seed, case["tokens"])]), "cache": None}
    n = case["context"] + 1
    ids = _tokens(case, seed, case["batch"] * n)
    return {"logits": _forward(c, w, [ids[i * n:(i + 1) * n] for i in range(case["batch"])]), "cache": None}


def _runs(c):
    lp, n = c.get("loop"), len(c["layers"])
    if not lp:
        return list(range(n))
    return list(range(lp["start"])) + list(range(lp["start"], lp["stop"])) * lp["times"] + list(range(lp["stop"], n))


def _rms(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def _turn(v, f, pairs, mag=1.0):
    """v [T, heads, d]: the first 2 len(f) entries turn, pair i by position times f[i]."""
    a = torch.arange(v.shape[0], device=v.device, dtype=torch.float64)[:, None] * f[None, :]
    cos, sin = (torch.cos(a) * mag)[:, None, :], (torch.sin(a) * mag)[:, None, :]
    half, out = f.shape[0], v.clone()
    one, two = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if pairs == "adjacent" else (slice(0, half), slice(half, 2 * half))
    out[..., one] = v[..., one] * cos - v[..., two] * sin
    out[..., two] = v[..., two] * cos + v[..., one] * sin
    return out


def _attend(q, k, v, scale, window=None, cap=None, sink=False):
    """Causal attention of one sequence. q [T, H, d], k [T, G, d], v [T, G, dv]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], device=q.device, dtype=q.dtype)
    at = torch.arange(T, device=q.device)
    for g in range(G):
        for a in range(0, T, 1024):
            rows = at[a:a + 1024]
            mask = at[None, :] > rows[:, None]
            if window is not None:
                mask |= at[None, :] <= rows[:, None] - window
            for h in range(g * (H // G), (g + 1) * (H // G)):
                s = (q[a:a + 1024, h] @ k[:, g].T) * scale
                if cap:
                    s = cap * torch.tanh(s / cap)
                s = s.masked_fill(mask, -math.inf)
                if sink:
                    s = torch.cat([s, torch.zeros(s.shape[0], 1, device=s.device, dtype=s.dtype)], 1)
                p = torch.softmax(s, -1)
                out[a:a + 1024, h] = (p[:, :T] if sink else p) @ v[:, g]
    return out


def _steps(x, ends):
    """The sequences of a concatenation of sequences."""
    a = 0
    for b in ends:
        yield slice(a, b)
        a = b


def _conv(x, taps, ends):
    """Causal convolution per channel along every sequence."""
    K, out = taps.shape[1], torch.zeros_like(x)
    for s in _steps(x, ends):
        part = torch.cat([torch.zeros(K - 1, x.shape[1], device=x.device, dtype=x.dtype), x[s]])
        out[s] = sum(part[j:j + s.stop - s.start] * taps[:, j] for j in range(K))
    return out


def _scan(step, state, n_rows, ends, shape, like):
    """`step(state, row) -> (state, out)` along every sequence."""
    out = torch.empty(n_rows, *shape, device=like.device, dtype=like.dtype)
    for s in _steps(like, ends):
        S = state()
        for t in range(s.start, s.stop):
            S, out[t] = step(S, t)
    return out


def _each(fn, ends, *parts):
    """`fn` on every sequence's rows of `parts`, put together again."""
    return torch.cat([fn(*(p[s] for p in parts)) for s in _steps(parts[0], ends)])


def _forward(c, w, sequences):
    """Logits [sequences, vocab] of every sequence's last token."""
    dev = torch.device("cuda")
    ends, n = [], 0
    for s in sequences:
        n += len(s)
        ends.append(n)
    ids = torch.tensor([t for s in sequences for t in s], device=dev)
    last = torch.tensor(ends, device=dev) - 1
    zeros = lambda *shape: torch.zeros(*shape, device=dev, dtype=torch.float64)  # noqa: E731
    silu = torch.nn.functional.silu
    if "hidden_size" in c:
        return _llama_forward(c, w, ids, last, ends, silu)
    eps = c["norm"]["eps"]
    x = w("embed")[ids]
    if c["architecture"] == "Bananex":
        return _bananex_forward(c, w, x, eps, last, ends, n, zeros, silu)
    if c["architecture"] == "Dupenex":
        return _dupenex_forward(c, w, x, eps, last, ends, n, zeros, silu)
    return _pudinex_forward(c, w, x, eps, last, ends, n, zeros, silu)


def _llama_forward(c, w, ids, last, ends, silu):
    eps, d, H, G = c["rms_norm_eps"], c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"]
    i = torch.arange(d // 2, device=ids.device, dtype=torch.float64)
    f = c["rope_theta"] ** (-2.0 * i / d)
    sc = c["rope_scaling"]
    wave = 2.0 * math.pi / f
    original, lo, hi = sc["original_max_position_embeddings"], sc["low_freq_factor"], sc["high_freq_factor"]
    smooth = (original / wave - lo) / (hi - lo)
    mixed = (1.0 - smooth) * f / sc["factor"] + smooth * f
    f = torch.where(wave > original / lo, f / sc["factor"], torch.where(wave < original / hi, f, mixed))
    x = w("model.embed_tokens.weight")[ids]
    for l in range(c["num_hidden_layers"]):
        p = "model.layers.%d." % l
        h = _rms(x, eps) * w(p + "input_layernorm.weight")
        q, k, v = ((h @ w(p + "self_attn.%s_proj.weight" % s).T).view(len(ids), -1, d) for s in "qkv")
        y = _each(lambda a, b, e: _attend(_turn(a, f, "half"), _turn(b, f, "half"), e, d ** -0.5), ends, q, k, v)
        x = x + y.reshape(len(ids), H * d) @ w(p + "self_attn.o_proj.weight").T
        del q, k, v, y
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
        h = silu(h @ w(p + "mlp.gate_proj.weight").T).mul_(h @ w(p + "mlp.up_proj.weight").T)
        x = x + h @ w(p + "mlp.down_proj.weight").T
    x = _rms(x[last], eps) * w("model.norm.weight")
    return x @ w("model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight").T


def _powers(base, dims, dev):
    return float(base) ** (-2.0 * torch.arange(dims // 2, device=dev, dtype=torch.float64) / dims)


def _bananex_forward(c, w, x, eps, last, ends, n, zeros, silu):
    dev, e, lp = x.device, x.clone(), c["loop"]
    entered = 0
    for i in _runs(c):
        if i == lp["start"] and entered < lp["times"]:
            x = torch.cat([x, e], 1) @ w("loop.in").T + w("loop.step")[entered]
            entered += 1
        p, m, kind = "l%d." % i, c["layers"][i]["mixer"], c["layers"][i]["type"]
        h = _rms(x, eps) * w(p + "norm1")
        before = _each(lambda a: torch.cat([torch.zeros_like(a[:1]), a[:-1]]), ends, h)
        h = h + (before - h) * w(p + "shift")
        q = p + "mix."
        if kind == "latent_attention":
            H, dn, dr, dv, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            f = _powers(m["rot"]["base"], m["rot"]["dims"], dev)
            qs, low = (h @ w(q + "q").T).view(n, H, dn + dr), h @ w(q + "dkv").T
            lat = _rms(low[:, :r], eps) * w(q + "dkv.norm")
            k, v = (lat @ w(q + "uk").T).view(n, H, dn), (lat @ w(q + "uv").T).view(n, H, dv)

            def attend(a, b, t, u):
                a = torch.cat([a[..., :dn], _turn(a[..., dn:], f, "adjacent")], -1)
                t = _turn(t[:, None, :], f, "adjacent").expand(-1, H, -1)
                return _attend(a, torch.cat([b, t], -1), u, m["scale"], m["mask"]["size"])
            y = _each(attend, ends, qs, k, low[:, r:], v).reshape(n, H * dv)
            y = (y * torch.sigmoid(h @ w(q + "g").T)) @ w(q + "o").T
        elif kind == "mingru":
            z = torch.sigmoid(h @ w(q + "z").T + w(q + "z.b"))
            u = h @ w(q + "x").T + w(q + "x.b")
            cand = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))

            def step(S, t):
                S = (1.0 - z[t]) * S + z[t] * cand[t]
                return S, S
            S = _scan(step, lambda: zeros(m["width"]), n, ends, (m["width"],), x)
            y = (S * silu(h @ w(q + "g").T)) @ w(q + "o").T
        else:
            H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            inner = H * P
            proj = h @ w(q + "in").T
            z, xbc, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * G * N], proj[:, 2 * inner + 2 * G * N:]
            xbc = silu(_conv(xbc, w(q + "conv"), ends) + w(q + "conv.b"))
            xs = xbc[:, :inner].reshape(n, H, P)
            B = xbc[:, inner:inner + G * N].reshape(n, G, N).repeat_interleave(H // G, 1)
            C = xbc[:, inner + G * N:].reshape(n, G, N).repeat_interleave(H // G, 1)
            dt = torch.nn.functional.softplus(dt + w(q + "dt_bias"), threshold=60)
            decay, D = torch.exp(-torch.exp(w(q + "A_log")) * dt), w(q + "D")

            def step(S, t):
                S = S * decay[t][:, None, None] + (dt[t][:, None] * B[t])[:, :, None] * xs[t][:, None, :]
                return S, (S * C[t][:, :, None]).sum(1)
            y = _scan(step, lambda: zeros(H, N, P), n, ends, (H, P), x) + D[:, None] * xs
            y = y.reshape(n, inner) * silu(z)
            parts = m["norm_groups"]
            y = (_rms(y.view(n, parts, -1), eps).reshape(n, inner) * w(q + "norm")) @ w(q + "o").T
        x = x + _rms(y, eps) * w(p + "norm1b")
        h = _rms(x, eps) * w(p + "norm2")
        y = torch.nn.functional.gelu(h @ w(p + "mlp.up").T + w(p + "mlp.up.b")) @ w(p + "mlp.down").T + w(p + "mlp.down.b")
        x = x + _rms(y, eps) * w(p + "norm2b")
    return (_rms(x[last], eps) * w("final.norm")) @ w("head").T * c["logit_scale"]


def _dupenex_forward(c, w, x, eps, last, ends, n, zeros, silu):
    dev = x.device

    def delta(h, q, m):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        qs, ks, vs = (silu(_conv(h @ w(q + s).T, w(q + s + ".conv"), ends)) for s in "qkv")
        qs, ks, vs = qs.view(n, G, d), ks.view(n, G, d), vs.view(n, H, dv)
        qs = qs / torch.sqrt((qs * qs).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
        ks = ks / torch.sqrt((ks * ks).sum(-1, keepdim=True) + 1e-6)
        qs, ks = qs.repeat_interleave(H // G, 1), ks.repeat_interleave(H // G, 1)
        beta = torch.sigmoid(h @ w(q + "b").T)
        rate = torch.nn.functional.softplus((h @ w(q + "a1").T) @ w(q + "a2").T + w(q + "dt_bias"), threshold=60).view(n, H, d)
        g = torch.exp(-torch.exp(w(q + "A_log"))[None, :, None] * rate)

        def step(S, t):
            S = S * g[t][:, :, None]
            u = beta[t][:, None] * (vs[t] - (S * ks[t][:, :, None]).sum(1))
            S = S + ks[t][:, :, None] * u[:, None, :]
            return S, (S * qs[t][:, :, None]).sum(1)
        y = _scan(step, lambda: zeros(H, d, dv), n, ends, (H, dv), h)
        y = _rms(y, eps) * w(q + "norm") * torch.sigmoid((h @ w(q + "g1").T) @ w(q + "g2").T).view(n, H, dv)
        return y.reshape(n, H * dv) @ w(q + "o").T

    def attention(h, q, m):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        f = _powers(m["rot"]["base"], m["rot"]["dims"], dev)
        qs, ks, vs = (h @ w(q + "q").T).view(n, H, d), (h @ w(q + "k").T).view(n, G, d), (h @ w(q + "v").T).view(n, G, dv)
        y = _each(lambda a, b, e: _attend(_turn(a, f, "adjacent"), _turn(b, f, "adjacent"), e, m["scale"], m["mask"]["size"]),
                  ends, qs, ks, vs)
        return (y.reshape(n, H * dv) * torch.sigmoid(h @ w(q + "g").T)) @ w(q + "o").T

    def memory(h, q, m):
        H, d, dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        qs, ks, vs = (h @ w(q + "q").T).view(n, H, d) * d ** -0.5, (h @ w(q + "k").T).view(n, H, d), (h @ w(q + "v").T).view(n, H, dv)
        gi = cap * torch.tanh((h @ w(q + "i").T + w(q + "i.b")) / cap)
        gf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w(q + "f").T + w(q + "f.b")) / cap))

        def step(state, t):
            S, z, r = state
            new = torch.maximum(gf[t] + r, gi[t])
            keep, take = torch.exp(gf[t] + r - new), torch.exp(gi[t] - new)
            S = keep[:, None, None] * S + take[:, None, None] * ks[t][:, :, None] * vs[t][:, None, :]
            z = keep[:, None] * z + take[:, None] * ks[t]
            low = torch.maximum((z * qs[t]).sum(-1).abs(), torch.exp(-new)) + 1e-6
            return (S, z, new), (S * qs[t][:, :, None]).sum(1) / low[:, None]
        y = _scan(step, lambda: (zeros(H, d, dv), zeros(H, d), zeros(H)), n, ends, (H, dv), h)
        y = _rms(y, eps).reshape(n, H * dv) * w(q + "norm") * torch.sigmoid(h @ w(q + "g").T)
        return y @ w(q + "o").T

    def mixer(h, i):
        q, layer = "l%d.mix." % i, c["layers"][i]
        if layer["type"] == "channel_delta":
            return delta(h, q, layer["mixer"])
        left = attention(h, q + "left.", layer["mixer"]["left"])
        right = memory(h, q + "right.", layer["mixer"]["right"])
        return 0.5 * (_rms(left, eps) * w(q + "left.out") + _rms(right, eps) * w(q + "right.out"))

    def unit(h, i):
        p = "l%d.mlp." % i
        return (silu(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T

    X = torch.stack([x] * c["streams"])
    for i in _runs(c):
        for k, part in ((1, mixer), (2, unit)):
            p = "l%d.hc%d." % (i, k)
            h = _rms(torch.einsum("a,ane->ne", w(p + "in").view(-1), X), eps) * w("l%d.norm%d" % (i, k))
            y = part(h, i)
            X = torch.einsum("ab,ane->bne", w(p + "mix"), X) + w(p + "out").view(-1)[:, None, None] * y[None]
    return (_rms(X.sum(0)[last], eps) * w("final.norm")) @ w("head").T


def _pudinex_forward(c, w, x, eps, last, ends, n, zeros, silu):
    dev, groups = x.device, c["norm"]["groups"]

    def norm(v, weight):
        return _rms(v.view(v.shape[0], groups, -1), eps).reshape(v.shape) * weight

    x = x * c["embedding"]["scale"]
    for i in _runs(c):
        p, layer = "l%d." % i, c["layers"][i]
        h, m, q = norm(x, w(p + "norm1")), layer["mixer"], p + "mix."
        if layer["type"] == "attention":
            H, G, d, dv, rot = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["rot"]
            f, sc, dims = _powers(rot["base"], rot["dims"], dev), rot["scaling"], rot["dims"]
            pair = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))  # noqa: E731
            lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), dims - 1)
            ramp = ((torch.arange(dims // 2, device=dev, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
            f = f / sc["factor"] * ramp + f * (1.0 - ramp)
            mag = 0.1 * math.log(sc["factor"]) + 1.0
            qs = _rms((h @ w(q + "q").T).view(n, H, d), eps) * w(q + "q.norm")
            ks = _rms((h @ w(q + "k").T).view(n, G, d), eps) * w(q + "k.norm")
            vs = _rms((h @ w(q + "v").T).view(n, G, dv), eps)
            y = _each(lambda a, b, e: _attend(_turn(a, f, "half", mag), _turn(b, f, "half", mag), e, m["scale"], None,
                                              m["softcap"], True), ends, qs, ks, vs)
            y = y.reshape(n, H * dv) @ w(q + "o").T
        else:
            H, d, dv = m["heads"], m["dim"], m["vdim"]
            qs, vs, low = silu(h @ w(q + "q").T).view(n, H, d), (h @ w(q + "v").T).view(n, H, dv), w(q + "lower").reshape(-1)
            f = (low + (1.0 - low) * torch.sigmoid(h @ w(q + "f").T + w(q + "f.b").reshape(-1))).view(n, H, d)

            def step(S, t):
                S = f[t][:, :, None] * S + (1.0 - f[t])[:, :, None] * vs[t][:, None, :]
                return S, (S * qs[t][:, :, None]).sum(1)
            y = _rms(_scan(step, lambda: zeros(H, d, dv), n, ends, (H, dv), x), eps) * w(q + "norm")
            y = y.reshape(n, H * dv) @ w(q + "o").T
        cap = layer["mlp"]["limit"]
        g = torch.clamp(h @ w(p + "mlp.gate").T, max=cap)
        u = torch.clamp(h @ w(p + "mlp.up").T, -cap, cap)
        x = x + y + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + "mlp.down").T
    return norm(x[last], w("final.norm")) @ w("head").T
