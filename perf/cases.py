"""What the library is timed on: generation and prompt steps through `Engine.generate` and `Engine.step`.

A case is a model, a number format and a set of requests.  With `new` > 0 the requests go through `Engine.generate` (their
prompts in one step, then a decode step per token, host token ids in and out); with `new` 0 their prompts go through one
`Engine.step`, which returns the logits of each prompt's last position, or of every position (`want` "all": documents that
are scored).  The lengths of a case's prompts are spread evenly, on a logarithmic scale, from `shortest` to `longest`.

Models are those the repository's benchmark runs: three sizes of the LFM3 hybrid (dense, larger dense, experts) and one of
the Zekivik and of the Lenesun design.  Weights are random: every matrix with a standard deviation of 1 / sqrt(columns),
the ones that write to the residual stream divided by sqrt(2 * layers) as is usual for training, embeddings of unit
variance, and output rows that are the embedding's.  Residual stream, norms and scores then have the magnitudes of a
trained model, and a generated token is as clear a choice as a trained model's, so that its value does not hang on rounding.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

# ---- the models ------------------------------------------------------------------------------------------------------
VOCAB = 65536


def _lfm3(layers: int, attention_at: list[int], **kw) -> dict:
    return dict({"architectures": ["Lfm3ForCausalLM"], "model_type": "lfm3", "vocab_size": VOCAB, "hidden_size": 2048,
                 "num_hidden_layers": layers, "layer_types": ["attention" if i in attention_at else "conv" for i in range(layers)],
                 "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 64, "rope_theta": 1000000.0,
                 "conv_L_cache": 3, "norm_eps": 1e-5, "tie_embedding": True, "max_position_embeddings": 128000}, **kw)


def _zekivik() -> dict:
    att = {"heads": 32, "kv_heads": 8, "dim": 64, "vdim": 64, "conv": 4, "scale": 0.125, "rot": {"dims": 64, "base": 1000000.0}}
    ret = {"heads": 16, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - (i % 8)) for i in range(16)],
           "rot": {"dims": 128, "base": 10000.0}}
    layers = [{"type": "attention" if i % 2 else "retention", "mixer": att if i % 2 else ret, "mlp": {"kind": "dense", "ff": 5632}}
              for i in range(6)]
    return {"architecture": "Zekivik", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-5}, "layers": layers,
            "loop": {"start": 0, "stop": 2, "times": 2}}


def _lenesun() -> dict:
    def mixer(i):
        m = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 768, "kv_rank": 512, "scale": 192 ** -0.5,
             "rot": {"dims": 64, "base": 10000.0}}
        return dict(m, kv_from=3) if i >= 4 else m
    mlp = {"kind": "moe", "router": {"experts": 32, "top": 4}, "expert": {"ff": 1024, "limit": 7.0}}
    return {"architecture": "Lenesun", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "residual_mult": 0.5, "layers": [{"type": "latent_attention", "mixer": mixer(i), "mlp": mlp} for i in range(6)]}


MODELS = {
    "1.2b": _lfm3(16, [2, 5, 8, 10, 12, 14], intermediate_size=5632),
    "2.6b": _lfm3(30, [2, 6, 10, 14, 18, 21, 24, 27], intermediate_size=7168),
    "8b-a1b": _lfm3(24, [2, 6, 10, 14, 18, 21], intermediate_size=7168, num_dense_layers=2, num_experts=32,
                    num_experts_per_tok=4, moe_intermediate_size=1792, norm_topk_prob=True, use_expert_bias=True,
                    routed_scaling_factor=1.0),
    "zekivik": _zekivik(),
    "lenesun": _lenesun(),
}


def _vocab(cfg: dict) -> int:
    return cfg["vocab_size"] if "vocab_size" in cfg else cfg["vocab"]


def _shapes(cfg: dict) -> dict[str, tuple]:
    """Every tensor of a model: name -> (shape, kind).  Kinds: "in" and "out" are matrices (out: they write to the residual
    stream), "expert in" and "expert out" those of one expert, "float" matrices are held in 32 bits."""
    t: dict[str, tuple] = {}
    if "vocab_size" in cfg:
        D, F, hd, L = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"], cfg["num_hidden_layers"]
        nh, nkv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
        t["embed_tokens.weight"] = ((cfg["vocab_size"], D), "embedding")
        t["embedding_norm.weight"] = ((D,), "norm")
        for i, kind in enumerate(cfg["layer_types"]):
            p = f"layers.{i}."
            t[p + "operator_norm.weight"] = t[p + "ffn_norm.weight"] = ((D,), "norm")
            if kind == "conv":
                t[p + "conv.in_proj.weight"] = ((3 * D, D), "in")
                t[p + "conv.conv.weight"] = ((D, 1, cfg["conv_L_cache"]), "taps")
                t[p + "conv.out_proj.weight"] = ((D, D), "out")
            else:
                for n, rows in (("q_proj", nh * hd), ("k_proj", nkv * hd), ("v_proj", nkv * hd)):
                    t[p + f"self_attn.{n}.weight"] = ((rows, D), "in")
                t[p + "self_attn.q_layernorm.weight"] = t[p + "self_attn.k_layernorm.weight"] = ((hd,), "norm")
                t[p + "self_attn.out_proj.weight"] = ((D, nh * hd), "out")
            E = cfg.get("num_experts", 0)
            if E and i >= cfg["num_dense_layers"]:
                Fe = cfg["moe_intermediate_size"]
                t[p + "feed_forward.gate.weight"] = ((E, D), "float")
                t[p + "feed_forward.expert_bias"] = ((E,), "bias")
                for e in range(E):
                    q = p + f"feed_forward.experts.{e}."
                    t[q + "w1.weight"] = t[q + "w3.weight"] = ((Fe, D), "expert in")
                    t[q + "w2.weight"] = ((D, Fe), "expert out")
            else:
                t[p + "feed_forward.w1.weight"] = t[p + "feed_forward.w3.weight"] = ((F, D), "in")
                t[p + "feed_forward.w2.weight"] = ((D, F), "out")
        return t
    W, V = cfg["width"], cfg["vocab"]
    t["embed.weight"] = ((V, W), "embedding")
    if cfg["architecture"] == "Zekivik":
        t["head.weight"], t["final.norm.weight"] = ((V, W), "embedding"), ((W,), "norm0")
        t["loop.step"] = ((cfg["loop"]["times"], W), "vector")
    else:
        t["final.norm.weight"] = ((W,), "norm")
    for i, lay in enumerate(cfg["layers"]):
        m, f, p = lay["mixer"], lay["mlp"], f"l{i}."
        H = m["heads"]
        if cfg["architecture"] == "Zekivik":
            G = m.get("kv_heads", H)
            t[p + "norm1.weight"] = t[p + "norm2.weight"] = ((W,), "norm0")
            t[p + "rg1"] = t[p + "rg2"] = ((W, W), "in")
            t[p + "rg1.b"] = t[p + "rg2.b"] = ((W,), "bias")
            for n, rows in (("q", H * m["dim"]), ("k", G * m["dim"]), ("v", G * m["vdim"])):
                t[p + "mix." + n] = ((rows, W), "in")
                if lay["type"] == "attention":
                    t[p + f"mix.{n}.conv"] = ((rows, m["conv"]), "taps")
            t[p + "mix.g"] = ((H if lay["type"] == "attention" else H * m["vdim"], W), "in")
            t[p + "mix.o"] = ((W, H * m["vdim"]), "out")
            t[p + "mlp.gate"] = t[p + "mlp.up"] = ((f["ff"], W), "in")
            t[p + "mlp.down"] = ((W, f["ff"]), "out")
        else:
            rq, rk, ff, E = m["q_rank"], m["kv_rank"], f["expert"]["ff"], f["router"]["experts"]
            t[p + "norm1.weight"] = ((W,), "norm")
            t[p + "mix.dq"], t[p + "mix.dq.norm"] = ((rq, W), "in"), ((rq,), "norm")
            t[p + "mix.uq"] = ((H * (m["dim"] + m["rot_dim"]), rq), "in")
            if "kv_from" not in m:
                t[p + "mix.dkv"], t[p + "mix.dkv.norm"] = ((rk + m["rot_dim"], W), "in"), ((rk,), "norm")
            t[p + "mix.uk"], t[p + "mix.uv"] = ((H * m["dim"], rk), "in"), ((H * m["vdim"], rk), "in")
            t[p + "mix.o"], t[p + "mix.sink"] = ((W, H * m["vdim"]), "out"), ((H,), "vector")
            t[p + "mlp.router"], t[p + "mlp.router.b"] = ((E, W), "float"), ((E,), "bias")
            for e in range(E):
                t[p + f"mlp.e{e}.gate"] = t[p + f"mlp.e{e}.up"] = ((ff, W), "expert in")
                t[p + f"mlp.e{e}.down"] = ((W, ff), "expert out")
    return t


class _Weights:
    """The model's tensors one by one; each has a generator of its own, so its values do not depend on which others are made.
    All are rounded to bfloat16, as a checkpoint's are, except biases."""

    def __init__(self, model: str):
        self.cfg, self.shapes = MODELS[model], _shapes(MODELS[model])
        self.depth = 2 * len(self.cfg.get("layer_types", self.cfg.get("layers")))
        self.model = model

    def __getitem__(self, name: str) -> torch.Tensor:
        shape, kind = self.shapes[name]
        seed = zlib.crc32(f"{self.model}:{'embed.weight' if name == 'head.weight' else name}".encode())
        v = torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
        if kind in ("norm", "norm0"):
            v = 0.1 * v + (1.0 if kind == "norm" else 0.0)
        elif kind in ("taps", "vector"):
            v = 0.5 * v
        elif kind == "bias":
            return 0.1 * v
        elif kind != "embedding":
            v = v * (shape[-1] * (self.depth if kind.endswith("out") else 1)) ** -0.5
            if kind == "expert out":
                v = 0.4 * v      # rounding decides near-ties between experts; one expert is then a small part of the stream
        return v.to(torch.bfloat16).float()

    def held(self, dtype: torch.dtype) -> dict[str, torch.Tensor]:
        return {n: self[n].to(dtype if k in ("in", "out", "expert in", "expert out", "embedding") else torch.float32)
                for n, (_, k) in self.shapes.items()}


_engines: dict = {}     # a program keeps its engine, weights and all, from one request to the next


def _engine(model: str, dtype: str):
    eng = _engines.get((model, dtype))
    if eng is None:
        from lastengine_b200 import Engine
        from lastengine_b200.registry import plan_from_config
        eng = _engines[model, dtype] = Engine(plan_from_config(MODELS[model]), dtype=dtype, max_tokens=65536, max_seqs=128)
        eng.model.load(_Weights(model).held(eng.dtype))
        eng.loaded = True
    return eng


# ---- the cases -------------------------------------------------------------------------------------------------------
def _case(name, model, requests, shortest, longest, new, want="last", sampled=False, dtype="bfloat16") -> dict:
    c = {"model": model, "dtype": dtype, "requests": requests, "shortest": shortest, "longest": longest, "new": new,
         "want": want, "sampled": sampled}
    return dict(c, name=name) if name else c


def listed() -> list[dict]:
    return [
        # the shortest useful call: a short question and the first two tokens of its answer
        _case("first_tokens", "1.2b", 1, 37, 37, 2),
        # one user's chat turn, with the sampling a request gets by default
        _case("chat", "1.2b", 1, 512, 512, 64, sampled=True),
        # a few users deep in long conversations
        _case("long_context", "1.2b", 8, 3968, 3968, 128),
        # a full batch of requests of unequal lengths on the larger dense model
        _case("many_requests", "2.6b", 64, 32, 512, 48),
        # one ordinary prompt
        _case("prompt", "1.2b", 1, 2048, 2048, 0),
        # prompts of very unequal lengths that start together
        _case("prompt_batch", "1.2b", 16, 64, 2048, 0),
        # a whole book chapter in one prompt, of odd length, longer than one pass over the layers takes
        _case("document", "1.2b", 1, 32767, 32767, 0),
        # documents that are scored: the logits of every position
        _case("scoring", "1.2b", 3, 301, 700, 0, want="all"),
        # a batch on the model with experts
        _case("moe", "8b-a1b", 8, 200, 500, 24),
        # true 32-bit arithmetic, as it is used to check a bfloat16 run
        _case("float32", "1.2b", 2, 190, 333, 8, dtype="float32"),
        # retention and convolved attention: one prompt and its answer
        _case("retention", "zekivik", 1, 2048, 2048, 32),
        # latent attention and experts: a batch of unequal prompts and their answers
        _case("latent", "lenesun", 8, 128, 700, 32),
    ]


def lengths(case: dict) -> list[int]:
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    if n == 1:
        return [hi]
    stride = next(s for s in range(n // 2 + 1, n + 2) if math.gcd(s, n) == 1)      # long and short ones mixed
    return [round(lo * (hi / lo) ** ((i * stride % n) / (n - 1))) for i in range(n)]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    most = max(_seconds(c) for c in listed())
    while True:
        model = rng.choice(["1.2b", "1.2b", "2.6b", "8b-a1b", "zekivik", "lenesun"])
        f32 = model == "1.2b" and rng.random() < 0.2
        longest = _log(rng, 24, 600 if f32 else 4000)
        if rng.random() < 0.6:
            c = _case(None, model, _log(rng, 1, 8 if f32 else 64), _log(rng, 8, longest), longest, _log(rng, 2, 16 if f32 else 128),
                      sampled=rng.random() < 0.3, dtype="float32" if f32 else "bfloat16")
        else:
            if not f32 and rng.random() < 0.2:
                longest = _log(rng, 4000, 32767)
            c = _case(None, model, _log(rng, 1, 16), _log(rng, 8, longest), longest, 0, want=rng.choice(["last", "last", "all"]),
                      dtype="float32" if f32 else "bfloat16")
        rows = sum(lengths(c))
        if _seconds(c) <= most and rows <= 40000 and (c["want"] == "last" or rows <= 2048):
            return c


def _seconds(case: dict) -> float:
    """Roughly what a pass takes, to keep drawn cases within the listed ones' cost."""
    w = work(case)
    return w["bytes"] / 4e12 + w["flops"] / (2e13 if case["dtype"] == "float32" else 8e14) + 5e-4 * case["new"]


def prepare(case: dict, seed: int) -> dict:
    eng = _engine(case["model"], case["dtype"])
    rng = np.random.default_rng(seed)
    prompts = [rng.integers(0, eng.vocab_size, size=n).tolist() for n in lengths(case)]
    return {"engine": eng, "case": case, "prompts": prompts, "sampling_seed": int(rng.integers(1 << 20)),
            "everywhere": [list(range(len(p))) for p in prompts]}


def run(state: dict):
    eng, case, prompts = state["engine"], state["case"], state["prompts"]
    if case["new"] == 0:
        seqs = [eng.new_sequence() for _ in prompts]
        logits = eng.step(seqs, prompts, state["everywhere"] if case["want"] == "all" else "last")
        eng.release(seqs)
        return {"logits": logits}
    from lastengine_b200 import SamplingParams
    sampling = SamplingParams(seed=state["sampling_seed"]) if case["sampled"] else SamplingParams(temperature=0.0)
    res = eng.generate(prompts, sampling, max_new_tokens=case["new"], stop_token_ids=[])
    return {"tokens": np.array(res.tokens), "logits": _last_logits(eng, res, len(prompts))}


def _last_logits(eng, res, n: int) -> torch.Tensor:
    """The logits the last tokens were chosen from: they lie in the scratch memory of the decode steps of this batch size."""
    from lastengine_b200.engine.graph import bucket_for
    b = bucket_for(n)
    return res.backend.graphs[("scratch", b)].get("model.logits", (b, eng.vocab_size), torch.float32)[:n]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _runs(cfg: dict) -> list[int]:
    """Layers in the order they run."""
    if "layer_types" in cfg:
        return list(range(cfg["num_hidden_layers"]))
    n, lp = len(cfg["layers"]), cfg.get("loop")
    return list(range(n)) if not lp else [*range(lp["start"])] + [*range(lp["start"], lp["stop"])] * lp["times"] + [*range(lp["stop"], n)]


def _cost(cfg: dict) -> dict:
    """Numbers of one model: weights a row meets outside experts, weights of all experts, the share of them a row meets,
    weights of the output rows; per position and run of an attention layer cached numbers, and flops per (query, key)."""
    shapes, runs = _shapes(cfg), _runs(cfg)
    times = {f"layers.{i}." if "layer_types" in cfg else f"l{i}.": runs.count(i) for i in runs}
    dense = experts = 0
    for n, (s, k) in shapes.items():
        if k in ("in", "out", "float", "expert in", "expert out"):
            size = math.prod(s) * next(t for p, t in times.items() if n.startswith(p))
            if k.startswith("expert"):
                experts += size
            else:
                dense += size
    cached, pair, state = 0, 0, 0
    for i in runs:
        if "layer_types" in cfg:
            if cfg["layer_types"][i] == "attention":
                cached += 2 * cfg["num_key_value_heads"] * cfg["head_dim"]
                pair += 4 * cfg["num_attention_heads"] * cfg["head_dim"]
            else:
                state += cfg["hidden_size"] * (cfg["conv_L_cache"] - 1)
        else:
            m = cfg["layers"][i]["mixer"]
            if "q_rank" in m:
                cached += 0 if "kv_from" in m else m["kv_rank"] + m["rot_dim"]
                pair += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            elif "kv_heads" in m:
                cached += m["kv_heads"] * (m["dim"] + m["vdim"])
                pair += 2 * m["heads"] * (m["dim"] + m["vdim"])
            else:
                state += m["heads"] * m["dim"] * m["vdim"]
    moe = cfg if "num_experts" in cfg else cfg.get("layers", [{}])[0].get("mlp", {}).get("router")
    share = 1.0 if not experts else moe["num_experts_per_tok"] / moe["num_experts"] if "num_experts" in moe else moe["top"] / moe["experts"]
    head = _vocab(cfg) * cfg.get("hidden_size", cfg.get("width"))
    return {"dense": dense, "experts": experts, "share": share, "head": head, "cached": cached, "pair": pair, "state": state}


def work(case: dict) -> dict:
    c, lens, n = _cost(MODELS[case["model"]]), lengths(case), case["requests"]
    size = 4 if case["dtype"] == "float32" else 2
    rows = sum(lens)
    per_row = 2 * (c["dense"] + c["share"] * c["experts"]) + 4 * c["state"]
    vocab = _vocab(MODELS[case["model"]])

    def weights(r):      # bytes of weights a step of r rows is expected to meet
        return size * (c["dense"] + c["head"] + c["experts"] * (1 - (1 - c["share"]) ** r))
    wanted = rows if case["want"] == "all" else n
    flops = rows * per_row + wanted * 2 * c["head"] + c["pair"] * sum(t * (t + 1) // 2 for t in lens)
    data = weights(rows) + rows * c["cached"] * size + n * c["state"] * 4 + 4 * wanted * vocab
    for k in range(max(0, case["new"] - 1)):
        live = sum(t + k + 1 for t in lens)
        flops += n * (per_row + 2 * c["head"]) + c["pair"] * live
        data += weights(n) + live * c["cached"] * size + n * c["state"] * 8 + 4 * n * vocab
    return {"bytes": data, "flops": flops}


def tolerance(case: dict) -> dict:
    # measured against 64 bits: 1.4e-6 in 32 bits, 0.003 in bfloat16, 0.007 with experts (near-ties of their scores)
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "differ": 0.0}
    return {"rel": 0.025 if case["model"] in ("8b-a1b", "lenesun") else 0.012, "differ": 0.0}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(v, base, dims, neighbours=False):
    """v [T, heads, d]: pairs of the first `dims` numbers turned by position * base^(-2i / dims)."""
    half = dims // 2
    i = torch.arange(half, dtype=v.dtype, device=v.device)
    a = torch.arange(v.shape[0], dtype=v.dtype, device=v.device)[:, None, None] * base ** (-2.0 * i / dims)
    c, s = torch.cos(a), torch.sin(a)
    x, y = (v[..., 0:dims:2], v[..., 1:dims:2]) if neighbours else (v[..., :half], v[..., half:dims])
    first, second = x * c - y * s, y * c + x * s
    turned = torch.stack([first, second], -1).flatten(-2) if neighbours else torch.cat([first, second], -1)
    return torch.cat([turned, v[..., dims:]], -1)


def _conv(u, w):
    """u [T, C], w [C, taps]: causal, zeros before the start."""
    taps = w.shape[1]
    pad = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    return sum(pad[j:j + len(u)] * w[:, j] for j in range(taps))


def _attend(q, k, v, scale, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, e]; a sink is a logit per head in the denominator alone."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = q.new_empty(T, H, v.shape[2])
    step = max(64, (1 << 26) // T)
    for h in range(H):
        kh, vh = k[:, h * G // H], v[:, h * G // H]
        for lo in range(0, T, step):
            hi = min(T, lo + step)
            s = (q[lo:hi, h] @ kh[:hi].T) * scale
            s.masked_fill_(torch.ones(hi - lo, hi, dtype=torch.bool, device=q.device).triu_(lo + 1), -math.inf)
            den = torch.logsumexp(s, -1, keepdim=True)
            if sink is not None:
                den = torch.logaddexp(den, sink[h])
            out[lo:hi, h] = torch.exp(s - den) @ vh[:hi]
    return out.flatten(1)


def _each(cuts, *xs):
    """The rows of every sequence of `xs`, sequence after sequence."""
    return zip(*(x.split(cuts) for x in xs))


def _experts(h, ids, wts, expert, E):
    out = torch.zeros_like(h)
    for e in range(E):
        row, j = (ids == e).nonzero(as_tuple=True)
        if len(row):
            out.index_add_(0, row, wts[row, j, None] * expert(e, h[row]))
    return out


def _lfm3_layer(cfg, w, i, x, cuts):
    p, eps, nh, nkv, hd = f"layers.{i}.", cfg["norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    h = _unit(x, eps) * w(p + "operator_norm.weight")
    if cfg["layer_types"][i] == "conv":
        b, c, u = (h @ w(p + "conv.in_proj.weight").T).chunk(3, -1)
        y = c * torch.cat([_conv(t, w(p + "conv.conv.weight")[:, 0]) for t in (b * u).split(cuts)])
        x = x + y @ w(p + "conv.out_proj.weight").T
    else:
        q, k, v = ((h @ w(p + f"self_attn.{n}_proj.weight").T).unflatten(1, (-1, hd)) for n in "qkv")
        q, k = _unit(q, eps) * w(p + "self_attn.q_layernorm.weight"), _unit(k, eps) * w(p + "self_attn.k_layernorm.weight")
        o = torch.cat([_attend(_turn(a, cfg["rope_theta"], hd), _turn(b, cfg["rope_theta"], hd), c, hd ** -0.5)
                       for a, b, c in _each(cuts, q, k, v)])
        x = x + o @ w(p + "self_attn.out_proj.weight").T
    h = _unit(x, eps) * w(p + "ffn_norm.weight")

    def gated(h, q):
        return (torch.nn.functional.silu(h @ w(q + "w1.weight").T) * (h @ w(q + "w3.weight").T)) @ w(q + "w2.weight").T
    p += "feed_forward."
    if not cfg.get("num_experts") or i < cfg["num_dense_layers"]:
        return x + gated(h, p)
    s = torch.sigmoid(h @ w(p + "gate.weight").T)
    ids = torch.topk(s + w(p + "expert_bias"), cfg["num_experts_per_tok"], -1).indices
    wts = s.gather(1, ids)
    return x + _experts(h, ids, wts / wts.sum(-1, keepdim=True), lambda e, r: gated(r, p + f"experts.{e}."), cfg["num_experts"])


def _zekivik_layer(cfg, w, i, x, cuts):
    lay, p, eps = cfg["layers"][i], f"l{i}.", cfg["norm"]["eps"]
    m, base, dims = lay["mixer"], lay["mixer"]["rot"]["base"], lay["mixer"]["rot"]["dims"]
    h = _unit(x, eps) * (1 + w(p + "norm1.weight"))
    q, k, v, g = (h @ w(p + "mix." + n).T for n in "qkvg")
    heads = lambda t, d: t.unflatten(1, (-1, d))  # noqa: E731
    out = []
    if lay["type"] == "attention":
        for a, b, c in _each(cuts, q, k, v):
            a, b, c = (heads(_conv(t, w(p + f"mix.{n}.conv")), d) for t, n, d in ((a, "q", m["dim"]), (b, "k", m["dim"]), (c, "v", m["vdim"])))
            out.append(_attend(_unit(_turn(a, base, dims), eps), _unit(_turn(b, base, dims), eps), _unit(c, eps), m["scale"]))
        y = heads(torch.cat(out), m["vdim"]) * torch.sigmoid(g)[:, :, None]
    else:
        for a, b, c in _each(cuts, heads(q, m["dim"]), heads(k, m["dim"]), heads(v, m["vdim"])):
            a, b = _turn(a, base, dims), _turn(b, base, dims) * m["dim"] ** -0.5
            t = torch.arange(len(a), dtype=x.dtype, device=x.device)
            ago = t[:, None] - t[None, :]
            o = [((a[:, j] @ b[:, j].T) * torch.where(ago >= 0, m["decay"][j] ** ago.clamp(min=0), 0.0)) @ c[:, j] for j in range(m["heads"])]
            out.append(_unit(torch.stack(o, 1), eps))
        y = torch.cat(out) * heads(torch.nn.functional.silu(g), m["vdim"])
    y = y.flatten(1) @ w(p + "mix.o").T
    x = x + torch.sigmoid(h @ w(p + "rg1").T + w(p + "rg1.b")) * y
    h = _unit(x, eps) * (1 + w(p + "norm2.weight"))
    y = (torch.nn.functional.gelu(h @ w(p + "mlp.gate").T, approximate="tanh") * (h @ w(p + "mlp.up").T)) @ w(p + "mlp.down").T
    return x + torch.sigmoid(h @ w(p + "rg2").T + w(p + "rg2.b")) * y


def _layer_norm(x, weight, eps):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], weight, None, eps)


def _lenesun_layer(cfg, w, i, x, cuts, rows):
    lay, p, eps = cfg["layers"][i], f"l{i}.", cfg["norm"]["eps"]
    m, f = lay["mixer"], lay["mlp"]
    base, dims, H = m["rot"]["base"], m["rot"]["dims"], m["heads"]
    h = _layer_norm(x, w(p + "norm1.weight"), eps)
    q = ((_unit(h @ w(p + "mix.dq").T, eps) * w(p + "mix.dq.norm")) @ w(p + "mix.uq").T).unflatten(1, (H, -1))
    if "kv_from" not in m:
        c, r = (h @ w(p + "mix.dkv").T).split([m["kv_rank"], m["rot_dim"]], -1)
        rows[i] = _unit(c, eps) * w(p + "mix.dkv.norm"), r
    c, r = rows[m.get("kv_from", i)]
    k, v = (c @ w(p + "mix.uk").T).unflatten(1, (H, -1)), (c @ w(p + "mix.uv").T).unflatten(1, (H, -1))
    out = []
    for a, b, t, u in _each(cuts, q, k, r, v):
        a = torch.cat([a[..., :m["dim"]], _turn(a[..., m["dim"]:], base, dims, True)], -1)
        t = _turn(t[:, None], base, dims, True).expand(-1, H, -1)
        out.append(_attend(a, torch.cat([b, t], -1), u, m["scale"], w(p + "mix.sink")))
    y = torch.cat(out) @ w(p + "mix.o").T
    z = h @ w(p + "mlp.router").T + w(p + "mlp.router.b")
    zc, ids = torch.topk(z, f["router"]["top"], -1)
    limit = f["expert"]["limit"]

    def expert(e, t):
        g = (t @ w(p + f"mlp.e{e}.gate").T).clamp(max=limit)
        u = (t @ w(p + f"mlp.e{e}.up").T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(p + f"mlp.e{e}.down").T
    return x + cfg["residual_mult"] * (y + _experts(h, ids, torch.softmax(zc, -1), expert, f["router"]["experts"]))


def _forward(model: str, seqs: list, places: list) -> torch.Tensor:
    """Logits, in 64 bits, of places[i] of sequence i, one after the other."""
    cfg, made = MODELS[model], _Weights(model)
    w = lambda name: made[name].double()  # noqa: E731
    cuts = [len(s) for s in seqs]
    table = w("embed_tokens.weight" if "layer_types" in cfg else "embed.weight")
    x = table[torch.as_tensor(np.concatenate(seqs), device="cuda")]
    first, rows, passes = x, {}, 0
    for i in _runs(cfg):
        if "layer_types" in cfg:
            x = _lfm3_layer(cfg, w, i, x, cuts)
        elif cfg["architecture"] == "Zekivik":
            if i == cfg["loop"]["start"]:
                x = x + w("loop.step")[passes] + (first if passes else 0.0)
                passes += 1
            x = _zekivik_layer(cfg, w, i, x, cuts)
        else:
            x = _lenesun_layer(cfg, w, i, x, cuts, rows)
    starts = np.cumsum([0] + cuts[:-1])
    x = x[torch.as_tensor(np.concatenate([s + np.asarray(p) for s, p in zip(starts, places)]), device="cuda")]
    if "layer_types" in cfg:
        return (_unit(x, cfg["norm_eps"]) * w("embedding_norm.weight")) @ table.T
    eps = cfg["norm"]["eps"]
    if cfg["architecture"] == "Zekivik":
        return (_unit(x, eps) * (1 + w("final.norm.weight"))) @ w("head.weight").T
    return _layer_norm(x, w("final.norm.weight"), eps) @ table.T


def exact(case: dict, seed: int):
    rng = np.random.default_rng(seed)
    prompts = [rng.integers(0, _vocab(MODELS[case["model"]]), size=n) for n in lengths(case)]
    new = case["new"]
    if new == 0:
        places = [range(len(p)) if case["want"] == "all" else [len(p) - 1] for p in prompts]
        return {"logits": _forward(case["model"], prompts, places)}
    # the tokens are guessed, and each forward pass puts the first wrong one of every request right
    tokens = np.repeat(np.array([p[-1] for p in prompts])[:, None], new, 1)
    for _ in range(4):
        places = [range(len(p) - 1, len(p) - 1 + new) for p in prompts]
        logits = _forward(case["model"], [np.concatenate([p, t[:-1]]) for p, t in zip(prompts, tokens)], places).unflatten(0, (-1, new))
        chosen = logits.argmax(-1).cpu().numpy()
        if (chosen == tokens).all():
            return {"tokens": tokens, "logits": logits[:, -1]}
        for t, c in zip(tokens, chosen):
            wrong = np.flatnonzero(t != c)
            if len(wrong):
                t[wrong[0]:] = c[wrong[0]]
    return None
