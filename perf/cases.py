"""What the library is timed on: passes that a program which serves these models makes, through the public entry points.

Two kinds of pass.

* ``turn``: a batch of conversations that the cache already holds goes on.  Every conversation brings the tokens of its next
  message (one prompt step on top of what is there), then the answer is decoded token by token.  Behind the pass the turn is
  taken back, as a program does that lets an answer be written again, so that a pass can be repeated.
* ``request``: prompts that nothing is held of.  Slots are taken, the prompts run in one step, the answers are decoded token by
  token, the slots are given back.  ``new`` = 1 is a prompt whose first answer token is all that is wanted.

Every step is ``Model.step_and_choose``: host token ids in, the chosen ids back on the host, the logits they were chosen from
beside them.  The tokens of the answers are given instead of being the chosen ones, so that one near-tie does not make the rest
of a pass another computation.  Weights are random with sizes that keep every part of a layer at work; what a conversation has
said before a turn is random keys and values of the size that the projections make.

``exact`` computes the same logits in 64 bits with plain torch, whole sequences at a time.
"""
import math

import numpy as np
import torch

import llmi_b200 as L
from llmi_b200.config.registry import parse_config
from llmi_b200.engine.model import Model
from llmi_b200.sampling import Sampler, UniformStream

DEVICE = "cuda:0"


# ----------------------------------------------------------------------------- the models

def _llama(layers, hidden, heads, kv_heads, head_dim, inner, vocab, theta, tied=True):
    return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": layers, "hidden_size": hidden, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "head_dim": head_dim, "intermediate_size": inner, "vocab_size": vocab,
            "rope_theta": theta, "rms_norm_eps": 1e-5, "tie_word_embeddings": tied, "max_position_embeddings": 8192,
            "hidden_act": "silu"}


def _garodra(width, heads, dim, rot_dim, kv_rank, q_rank, kv_heads, ff, experts, top, expert_ff, layers, vocab):
    att = {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": dim, "kv_rank": kv_rank, "q_rank": q_rank,
           "scale": (dim + rot_dim) ** -0.5, "rot": {"base": 10000.0, "dims": rot_dim}}
    delta = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "conv": 4}
    dense = {"kind": "dense", "ff": ff}
    moe = {"kind": "moe", "expert": {"ff": expert_ff}, "router": {"experts": experts, "top": top}}
    kinds = [("latent_attention", att, dense), ("latent_attention", att, moe), ("delta", delta, dense), ("delta", delta, moe)]
    return {"architecture": "Garodra", "vocab": vocab, "width": width, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
            "layers": [{"type": t, "mixer": m, "mlp": f} for t, m, f in (kinds[i % 4] for i in range(layers))]}


def _fusazen(width, heads, kv_heads, dim, delta_heads, ff, vocab, block):
    diff = {"heads": heads // 2, "kv_heads": kv_heads // 2, "dim": dim, "vdim": 2 * dim, "diff": 0.5, "mask": {"size": block},
            "rot": {"base": 10000.0, "dims": dim // 2}, "scale": dim ** -0.5}
    normed = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "mask": {"size": block}, "scale": 1.0 / dim}
    delta = {"heads": delta_heads, "dim": dim}
    mlp = {"kind": "dense", "ff": ff}
    kinds = [("attention", diff), ("general_delta", delta), ("attention_2", normed), ("general_delta", delta),
             ("attention", dict(diff, kv_from=0)), ("general_delta", delta), ("attention_2", normed), ("general_delta", delta)]
    return {"architecture": "Fusazen", "vocab": vocab, "width": width, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
            "canon": {"taps": 4}, "layers": [{"type": t, "mixer": m, "mlp": mlp} for t, m in kinds]}


def _sobezen(width, heads, kv_heads, dim, rot_dim, kv_rank, q_rank, ff, vocab):
    rot = {"base": 10000.0, "dims": rot_dim, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    lat = {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": dim, "kv_rank": kv_rank, "q_rank": q_rank,
           "scale": (dim + rot_dim) ** -0.5, "rot": rot}
    delta = {"heads": heads, "kv_heads": heads, "dim": dim, "vdim": dim, "conv": 4}
    att = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "rot": {"base": 10000.0, "dims": dim}}
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    layers = []
    for first in (0, 4):
        layers += [("latent_attention", lat, mlp), ("channel_delta", delta, None), ("attention", att, mlp),
                   ("latent_attention", dict(lat, kv_from=first), mlp)]
    return {"architecture": "Sobezen", "vocab": vocab, "width": width, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
            "logit_scale": 0.5, "layers": [{"type": t, "mixer": m, "mlp": f} for t, m, f in layers]}


CONFIGS = {
    "smollm2-135m": _llama(30, 576, 9, 3, 64, 1536, 49152, 100000.0),
    "smollm2-360m": _llama(32, 960, 15, 5, 64, 2560, 49152, 100000.0),
    "smollm2-1.7b": _llama(24, 2048, 32, 32, 64, 8192, 49152, 130000.0),
    "llama-4096": _llama(4, 4096, 32, 8, 128, 14336, 32000, 500000.0, tied=False),     # four layers of an 8B Llama's width
    "garodra-2048": _garodra(2048, 16, 128, 64, 512, 1024, 8, 8192, 8, 2, 2048, 8, 49152),
    "garodra-1024": _garodra(1024, 8, 64, 32, 256, 384, 4, 4096, 8, 2, 1024, 8, 49152),
    "fusazen-2048": _fusazen(2048, 32, 8, 64, 32, 8192, 49152, 8192),
    "fusazen-1024": _fusazen(1024, 16, 4, 64, 16, 4096, 49152, 8192),
    "sobezen-2048": _sobezen(2048, 16, 4, 128, 64, 512, 1536, 8192, 49152),
    "sobezen-1024": _sobezen(1024, 8, 2, 64, 32, 256, 768, 4096, 49152),
}
LLAMAS = ("smollm2-135m", "smollm2-360m", "smollm2-1.7b", "llama-4096")
DESIGNS = ("garodra-2048", "garodra-1024", "fusazen-2048", "fusazen-1024", "sobezen-2048", "sobezen-1024")
BYTES = {"bfloat16": 2, "float32": 4}


# ----------------------------------------------------------------------------- the cases

def _turn(model, batch, shortest, longest, message, new, dtype="bfloat16", temperature=0.0, top_k=0, top_p=1.0):
    return {"kind": "turn", "model": model, "dtype": dtype, "batch": batch, "shortest": shortest, "longest": longest,
            "message": message, "new": new, "temperature": temperature, "top_k": top_k, "top_p": top_p}


def _request(model, batch, shortest, longest, new, dtype="bfloat16", temperature=0.0, top_k=0, top_p=1.0):
    return {"kind": "request", "model": model, "dtype": dtype, "batch": batch, "shortest": shortest, "longest": longest,
            "message": 0, "new": new, "temperature": temperature, "top_k": top_k, "top_p": top_p}


def listed():
    return [
        # one user at the smallest model, a short conversation: launches and latency are all there is
        dict(_turn("smollm2-135m", 1, 333, 333, 13, 16), name="chat-135m"),
        # one user at the headline model, a long conversation, with the options that chats are sampled with
        dict(_turn("smollm2-1.7b", 1, 3989, 3989, 21, 16, temperature=0.8, top_k=50, top_p=0.95), name="chat-1.7b"),
        # the headline serving point: eight conversations at about 4,096 positions
        dict(_turn("smollm2-1.7b", 8, 3700, 4060, 16, 16), name="batch8-1.7b"),
        # a full server: 64 conversations of unequal lengths
        dict(_turn("smollm2-1.7b", 64, 1000, 2040, 8, 8), name="batch64-1.7b"),
        # grouped queries over heads of 128 at an 8B model's width, a batch that is no power of two
        dict(_turn("llama-4096", 24, 500, 3900, 9, 12), name="batch24-4096"),
        # a prompt to its first token: the headline length, and one near the context's end
        dict(_request("smollm2-1.7b", 1, 2048, 2048, 1), name="prompt-1.7b"),
        dict(_request("smollm2-1.7b", 1, 7931, 7931, 1), name="long-prompt-1.7b"),
        # eight unequal requests from first to last token
        dict(_request("smollm2-360m", 8, 16, 1024, 16), name="requests-360m"),
        # the same in the 32-bit path, which is what results are checked with
        dict(_request("smollm2-360m", 4, 30, 401, 8, dtype="float32"), name="requests-360m-float32"),
        # requests to designs with recurrent states, latent attention, experts, maps: prompts and answers
        dict(_request("garodra-2048", 2, 701, 1900, 8), name="requests-garodra"),
        dict(_request("fusazen-2048", 2, 701, 1900, 8), name="requests-fusazen"),
        dict(_request("sobezen-2048", 2, 701, 1900, 8), name="requests-sobezen"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    sampling = rng.choice([{}, {"temperature": round(rng.uniform(0.5, 1.2), 2), "top_k": rng.choice([20, 40, 50]),
                                "top_p": rng.choice([0.9, 0.95, 1.0])}])
    kind = rng.choice(["turn", "turn", "turn", "request", "request", "float32", "design", "design"])
    if kind == "turn":
        model = rng.choice(LLAMAS)
        batch = log_int(1, 64)
        longest = log_int(64, min(8000, 85000 // batch))
        return _turn(model, batch, rng.randint(max(16, longest // 4), longest), longest, rng.randint(2, 48), rng.randint(4, 16), **sampling)
    if kind == "float32":
        batch = rng.randint(1, 6)
        longest = log_int(8, 900 // batch)
        return _request(rng.choice(LLAMAS[:2]), batch, rng.randint(max(2, longest // 8), longest), longest, rng.randint(1, 8),
                        dtype="float32", **sampling)
    if kind == "request":
        batch = log_int(1, 16)
        longest = log_int(16, 7900 // batch)
        return _request(rng.choice(LLAMAS), batch, rng.randint(max(2, longest // 8), longest), longest, rng.randint(1, 16), **sampling)
    batch = rng.randint(1, 6)
    longest = log_int(40, 2600 // batch)
    return _request(rng.choice(DESIGNS), batch, rng.randint(max(2, longest // 4), longest), longest, rng.randint(1, 12), **sampling)


def _lengths(case):
    """Positions held (``turn``) or prompt tokens (``request``) of each sequence: spread unevenly, the longest among them."""
    lo, hi, n = case["shortest"], case["longest"], case["batch"]
    return [hi - int((hi - lo) * ((i * 0.6180339887498949) % 1.0)) for i in range(n)]


def _given(case):
    """Tokens of each sequence's first step."""
    return [case["message"]] * case["batch"] if case["kind"] == "turn" else _lengths(case)


def _held(case):
    return _lengths(case) if case["kind"] == "turn" else [0] * case["batch"]


# ----------------------------------------------------------------------------- inputs, made from the seed alone

def _generator(seed, *what):
    mixed = seed
    for k in what:
        mixed = (mixed * 1000003 + 7919 * k + 12345) % (1 << 62)
    return torch.Generator(device=DEVICE).manual_seed(mixed)


def _weights(case, seed):
    """name -> tensor as a model file would hold it.  The head is near the embedding table, as trained ones are: the choice of a
    token then hangs on no near-tie, which random heads of 49,152 rows give every few dozen tokens."""
    cfg, dtype = CONFIGS[case["model"]], getattr(torch, case["dtype"])
    gen = _generator(seed, 1)
    w = {}

    def vec(name, n, std, around=0.0):
        w[name] = (around + std * torch.randn(n, generator=gen, device=DEVICE)).to(dtype)

    def mat(name, out, inp, gain=1.0):
        w[name] = torch.randn((out, inp), generator=gen, device=DEVICE, dtype=dtype).mul_(gain / math.sqrt(inp))

    if cfg.get("architecture") is None:
        H, F, V, D = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["head_dim"]
        q, kv = cfg["num_attention_heads"] * D, cfg["num_key_value_heads"] * D
        w["model.embed_tokens.weight"] = torch.randn((V, H), generator=gen, device=DEVICE, dtype=dtype)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            vec(p + "input_layernorm.weight", H, 0.1, 1.0)
            mat(p + "self_attn.q_proj.weight", q, H)
            mat(p + "self_attn.k_proj.weight", kv, H)
            mat(p + "self_attn.v_proj.weight", kv, H)
            mat(p + "self_attn.o_proj.weight", H, q, 0.5)
            vec(p + "post_attention_layernorm.weight", H, 0.1, 1.0)
            mat(p + "mlp.gate_proj.weight", F, H)
            mat(p + "mlp.up_proj.weight", F, H)
            mat(p + "mlp.down_proj.weight", H, F, 0.5)
        tied = cfg["tie_word_embeddings"]
        vec("model.norm.weight", H, 6.0 / H if tied else 0.1, 60.0 / H if tied else 1.0)
        if not tied:
            mat("lm_head.weight", V, H, 0.75)
            w["lm_head.weight"].add_(w["model.embed_tokens.weight"], alpha=60.0 / H)
        return w

    W, V = cfg["width"], cfg["vocab"]
    garodra = cfg["architecture"] == "Garodra"

    def norm(name):
        vec(name, W, 0.2, 1.0)
        if garodra:                                     # a Dynamic Tanh
            vec(name + ".b", W, 0.2)
            w[name + ".alpha"] = (0.4 + 0.8 * torch.rand((), generator=gen, device=DEVICE)).to(dtype)

    w["embed"] = torch.randn((V, W), generator=gen, device=DEVICE, dtype=dtype)
    mat("head", V, W, 0.75)
    w["head"].add_(w["embed"], alpha=60.0 / W)
    norm("final.norm")
    for i, layer in enumerate(cfg["layers"]):
        p, m, kind = f"l{i}.", layer["mixer"], layer["type"]
        x = p + "mix."
        norm(p + "norm1")
        if garodra:
            norm(p + "norm1b")
        if cfg["architecture"] == "Sobezen":
            vec(p + "ls1", W, 0.5, 1.0)
        if cfg["architecture"] == "Fusazen":
            vec(p + "canon1", (W, cfg["canon"]["taps"]), 0.3)
        H, D = m["heads"], m["dim"]
        if kind == "latent_attention":
            R, C, Q = m["rot_dim"], m["kv_rank"], m["q_rank"]
            mat(x + "dq", Q, W)
            vec(x + "dq.norm", Q, 0.2, 1.0)
            mat(x + "uq", H * (D + R), Q, 1.5)
            if m.get("kv_from") is None:
                mat(x + "dkv", C + R, W, 1.5)
                vec(x + "dkv.norm", C, 0.2, 1.0)
            mat(x + "uk", H * D, C, 1.5)
            mat(x + "uv", H * m["vdim"], C)
            mat(x + "o", W, H * m["vdim"])
        elif kind in ("delta", "channel_delta"):
            for n, rows in (("q", m["kv_heads"] * D), ("k", m["kv_heads"] * D), ("v", H * m["vdim"])):
                mat(x + n, rows, W, 1.5)
                vec(x + n + ".conv", (rows, m["conv"]), 0.5)
            mat(x + "b", H, W, 2.0)
            if kind == "delta":
                mat(x + "a", H, W)
                vec(x + "dt_bias", H, 1.0)
                mat(x + "g", H * m["vdim"], W, 2.0)
            else:
                mat(x + "a1", W // 16, W)
                mat(x + "a2", H * D, W // 16, 2.0)
                vec(x + "dt_bias", H * D, 1.0)
                mat(x + "g1", W // 16, W)
                mat(x + "g2", H * m["vdim"], W // 16, 2.0)
            w[x + "A_log"] = torch.log(0.02 + 1.5 * torch.rand(H, generator=gen, device=DEVICE)).to(dtype)
            vec(x + "norm", m["vdim"], 0.2, 1.0)
            mat(x + "o", W, H * m["vdim"])
        elif kind == "general_delta":
            for n in ("r", "k", "v", "a", "g"):
                mat(x + n, H * D, W)
            mat(x + "w1", W // 16, W)
            mat(x + "w2", H * D, W // 16, 2.0)
            vec(x + "w0", H * D, 1.0, -1.0)
            vec(x + "a.b", H * D, 0.5)
            vec(x + "norm", H * D, 0.2, 1.0)
            mat(x + "o", W, H * D)
        else:
            maps = 2 if "diff" in m else 1
            mat(x + "q", H * maps * D, W)
            if m.get("kv_from") is None:
                mat(x + "k", m["kv_heads"] * maps * D, W)
            if cfg["architecture"] == "Sobezen":
                vec(x + "q.b", H * D, 0.5)
                vec(x + "k.b", m["kv_heads"] * D, 0.5)
            elif m.get("kv_from") is None:
                mat(x + "v", m["kv_heads"] * m["vdim"], W)
            if maps == 2:
                for n in ("lq1", "lk1", "lq2", "lk2"):
                    vec(x + n, D, 0.1)
            if kind == "attention_2":
                vec(x + "q.norm", H * D, 0.2, 1.0)
                vec(x + "k.norm", m["kv_heads"] * D, 0.2, 1.0)
                vec(x + "temp", H, 2.0, 8.0)
            mat(x + "o", W, H * m["vdim"])
        mlp = layer["mlp"]
        if mlp is None:
            continue
        norm(p + "norm2")
        if garodra:
            norm(p + "norm2b")
        if cfg["architecture"] == "Sobezen":
            vec(p + "ls2", W, 0.5, 1.0)
        y = p + "mlp."
        if mlp["kind"] == "moe":
            # a trained router is decisive: each token's row of the table leans toward the experts that are to be its own, so
            # that no choice hangs on the last bit (the recurrences would carry one expert's difference through all that follows)
            experts, top = mlp["router"]["experts"], mlp["router"]["top"]
            mat(y + "router", experts, W, 3.0)
            own = torch.rand((V, experts), generator=gen, device=DEVICE).argsort(dim=1) < top
            lean = torch.nn.functional.normalize(w[y + "router"].float(), dim=1)
            w["embed"].add_((own.float() @ lean).to(dtype), alpha=20.0)
            for e in range(mlp["router"]["experts"]):
                mat(y + f"e{e}.gate", mlp["expert"]["ff"], W, 1.5)
                mat(y + f"e{e}.up", mlp["expert"]["ff"], W)
                mat(y + f"e{e}.down", W, mlp["expert"]["ff"])
            continue
        names = ("up",) if cfg["architecture"] == "Fusazen" else ("gate", "up")
        for n in names:
            mat(y + n, mlp["ff"], W)
            if not garodra:
                vec(y + n + ".b", mlp["ff"], 0.3)
        mat(y + "down", W, mlp["ff"])
        if not garodra:
            vec(y + "down.b", W, 0.3)
    return w


def _tokens(case, seed):
    """Per sequence the tokens that it brings: those of its first step, then the answer's."""
    cfg = CONFIGS[case["model"]]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    rng = np.random.default_rng([seed, 2])
    return [rng.integers(0, vocab, n + case["new"] - 1).tolist() for n in _given(case)]


def _history(case, seed, layer):
    """Keys and values [positions of all conversations, heads, size] that a layer's cache holds before a turn."""
    cfg, dtype = CONFIGS[case["model"]], getattr(torch, case["dtype"])
    shape = (sum(_held(case)), cfg["num_key_value_heads"], cfg["head_dim"])
    gen = _generator(seed, 3, layer)
    return [torch.randn(shape, generator=gen, device=DEVICE, dtype=dtype) for _ in range(2)]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    dtype = getattr(torch, case["dtype"])
    arch, cfg = parse_config(CONFIGS[case["model"]])
    s.model = Model(arch.model_spec(cfg), _weights(case, seed), dtype, DEVICE, config=cfg)
    held, given, page = _held(case), _given(case), 64
    tokens = sum((h + n + case["new"] + page - 1) // page * page for h, n in zip(held, given))
    s.cache = s.model.new_cache(tokens, n_slots=case["batch"])
    s.params = L.SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=seed)
    s.sampler = Sampler(s.params, s.model.rt)
    s.tokens = _tokens(case, seed)
    if case["kind"] == "turn":
        s.slots = []
        pages, places = [], []
        for n in held:
            slot = s.cache.alloc_slot()
            s.cache.extend(slot, n)
            table = torch.tensor(s.cache.kv_groups[0].pool.table(slot))
            at = torch.arange(n)
            pages.append(table[at // page])
            places.append(at % page)
            s.slots.append(slot)
        pages, places = torch.cat(pages).to(DEVICE), torch.cat(places).to(DEVICE)
        for i, binding in enumerate(s.cache.bindings):
            k, v = _history(case, seed, i)
            binding.group.k[binding.index][pages, :, places] = k
            binding.group.v[binding.index][pages, :, places] = v
    return s


# ----------------------------------------------------------------------------- a pass

def _take_back(cache, slots, n):
    """The last ``n`` positions of every conversation are forgotten (their storage is written again by the next pass)."""
    cache.settle()
    for slot in slots:
        for group in cache.kv_groups:
            for _ in range(n):
                group.pool.shrink_by_one(slot)
        cache._length[slot] -= n


def run(state):
    case, model, cache, sampler = state.case, state.model, state.cache, state.sampler
    turn = case["kind"] == "turn"
    slots = state.slots if turn else [cache.alloc_slot() for _ in range(case["batch"])]
    streams = None if state.params.greedy else [UniformStream(state.params.seed, i) for i in range(case["batch"])]
    given = _given(case)
    logits, ids = [], []
    for step in range(case["new"]):
        seqs = []
        for slot, tokens, n in zip(slots, state.tokens, given):
            brings = tokens[:n] if step == 0 else [tokens[n + step - 1]]
            seqs.append(L.SequenceStep(slot, brings, [len(brings) - 1]))
        ids.append(model.step_and_choose(cache, seqs, sampler, streams))
        logits.append(model.last_logits.clone())
    if turn:
        _take_back(cache, slots, case["message"] + case["new"] - 1)
    else:
        for slot in slots:
            cache.free_slot(slot)
    return {"logits": torch.stack(logits), "ids": torch.stack(ids)}


# ----------------------------------------------------------------------------- bytes and operations

def _llama_layer_matrix(cfg):
    H, D = cfg["hidden_size"], cfg["head_dim"]
    q, kv = cfg["num_attention_heads"] * D, cfg["num_key_value_heads"] * D
    return H * (2 * q + 2 * kv) + 3 * H * cfg["intermediate_size"]


def work(case):
    """Every step reads the weights that it uses once (the steps of a pass follow one another, and a model is larger than
    the caches of the chip), the cache rows that its queries see, and writes its own rows and the logits."""
    cfg, size = CONFIGS[case["model"]], BYTES[case["dtype"]]
    given, held, new = _given(case), _held(case), case["new"]
    tokens = sum(given) + case["batch"] * (new - 1)
    # per sequence: (queries x visible keys) of the first step and of the answer, and the rows that are read
    pairs = sum(n * h + n * (n + 1) // 2 + sum(h + n + j + 1 for j in range(new - 1)) for n, h in zip(given, held))
    read = sum(h + sum(h + n + j for j in range(new - 1)) for n, h in zip(given, held))
    if cfg.get("architecture") is None:
        V, H = cfg["vocab_size"], cfg["hidden_size"]
        layers, matrix = cfg["num_hidden_layers"], _llama_layer_matrix(cfg)
        row = 2 * cfg["num_key_value_heads"] * cfg["head_dim"] * size
        by = new * (layers * matrix + V * H) * size + layers * row * (read + tokens)
        fl = 2 * tokens * layers * matrix + layers * 4 * cfg["num_attention_heads"] * cfg["head_dim"] * pairs
    else:
        V, H = cfg["vocab"], cfg["width"]
        by, fl = new * V * H * size, 0
        for layer in cfg["layers"]:
            m, mlp = layer["mixer"], layer["mlp"]
            h, d, dv = m["heads"], m["dim"], m.get("vdim", m["dim"])
            state = attends = 0
            if layer["type"] == "latent_attention":
                own = m.get("kv_from") is None
                r, c, q = m["rot_dim"], m["kv_rank"], m["q_rank"]
                matrix = H * q + q * h * (d + r) + (H * (c + r) if own else 0) + c * h * (d + dv) + h * dv * H
                row, attends = c + r, 2 * h * (d + r + dv)
            elif layer["type"] in ("delta", "channel_delta", "general_delta"):
                if layer["type"] == "general_delta":
                    matrix = 5 * H * h * d + 2 * H * (H // 16) + h * d * H
                else:
                    matrix = H * (2 * m["kv_heads"] * d + h * dv) + H * h * dv + (2 * H * h * dv if layer["type"] == "delta" else H * (H // 4))
                row, state = 0, h * d * dv
            else:
                maps, g = (2 if "diff" in m else 1), m["kv_heads"]
                matrix = H * h * maps * d + h * dv * H + (H * g * (maps * d + dv) if m.get("kv_from") is None else 0)
                row, attends = g * (maps * d + dv), 2 * h * maps * (d + dv)
            if mlp is None:
                used = read_m = 0
            elif mlp["kind"] == "moe":
                top, experts = mlp["router"]["top"], mlp["router"]["experts"]
                one = 3 * H * mlp["expert"]["ff"]
                used = top * one
                # a step of many tokens touches every expert, one of few at most as many as it has choices
                read_m = one * (experts + (new - 1) * min(experts, top * case["batch"])) / new
            else:
                used = read_m = (2 if cfg["architecture"] == "Fusazen" else 3) * H * mlp["ff"]
            by += new * (matrix + read_m) * size + row * size * (read + tokens) + 4 * state * case["batch"] * (2 * new - 1)
            fl += 2 * tokens * (matrix + used) + attends * pairs + 6 * state * tokens
    rows = case["batch"] * new
    return {"bytes": float(by + 4 * V * rows), "flops": float(fl + 2 * rows * V * H)}


def tolerance(case):
    """bf16 products with 32-bit sums through a stack of layers: the logits are 2e-3 to 7e-3 off the exact ones (their largest
    difference 4e-2 of a logit's size), those of the 32-bit path 2e-6 (1.2e-5).  Four times that and less; the chosen tokens are
    clear of near-ties (see _weights)."""
    if case["dtype"] == "float32":
        return {"rel": 8e-6, "max": 5e-5, "differ": 0.01}
    return {"rel": 0.02, "max": 0.15, "differ": 0.01}


# ----------------------------------------------------------------------------- the same in 64 bits, plain torch

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu_tanh(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _softmax_attention(q, k, v, scale, first=0):
    """q [T, H, D] at positions first.., k [S, G, D], v [S, G, Dv]; query head i reads key head i // (H / G)."""
    T, H, S = q.shape[0], q.shape[1], k.shape[0]
    rep = H // k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    hidden = torch.arange(S, device=q.device)[None, :] > torch.arange(first, first + T, device=q.device)[:, None]
    for i in range(H):
        s = (q[:, i] @ k[:, i // rep].T) * (scale if not torch.is_tensor(scale) else scale[i])
        out[:, i] = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1) @ v[:, i // rep]
    return out


def _exact_llama(case, seed):
    cfg, w = CONFIGS[case["model"]], _weights(case, seed)
    heads, kv, D, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], float(np.float32(cfg["rms_norm_eps"]))
    i = np.arange(D // 2)
    freq = (np.float32(1.0) / np.power(np.float32(cfg["rope_theta"]), (2 * i).astype(np.float32) / np.float32(D))).astype(np.float32)

    def rotated(v, first):
        at = np.arange(first, first + v.shape[0], dtype=np.float32)
        angle = torch.from_numpy((at[:, None] * freq[None, :]).astype(np.float32).astype(np.float64)).to(DEVICE)
        c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
        a, b = v[..., :D // 2], v[..., D // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], dim=-1)

    tokens, held = _tokens(case, seed), _held(case)
    table = w["model.embed_tokens.weight"]
    xs = [table[torch.tensor(t, device=DEVICE)].double() for t in tokens]
    starts = np.concatenate([[0], np.cumsum(held)])
    cut = [len(t) for t in tokens]
    for n in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{n}."
        get = lambda name: w[p + name + ".weight"].double()      # noqa: E731
        past = _history(case, seed, n) if case["kind"] == "turn" else None
        x = torch.cat(xs)
        h = _rms(x, eps) * get("input_layernorm")
        q, k, v = (torch.split((h @ get(f"self_attn.{c}_proj").T).view(-1, m, D), cut) for c, m in (("q", heads), ("k", kv), ("v", kv)))
        outs = []
        for b, base in enumerate(held):
            kb, vb = rotated(k[b], base), v[b]
            if past is not None:
                kb = torch.cat([past[0][starts[b]:starts[b + 1]].double(), kb])
                vb = torch.cat([past[1][starts[b]:starts[b + 1]].double(), vb])
            outs.append(_softmax_attention(rotated(q[b], base), kb, vb, D ** -0.5, base).reshape(cut[b], -1))
        x = x + torch.cat(outs) @ get("self_attn.o_proj").T
        h = _rms(x, eps) * get("post_attention_layernorm")
        x = x + (_silu(h @ get("mlp.gate_proj").T) * (h @ get("mlp.up_proj").T)) @ get("mlp.down_proj").T
        xs = list(torch.split(x, cut))
    head = (table if cfg["tie_word_embeddings"] else w["lm_head.weight"]).double()
    return [(_rms(x, eps) * w["model.norm.weight"].double())[-case["new"]:] @ head.T for x in xs]


def _turned(v, rot, halves=False):
    """v [T, ..., D]: the first ``dims`` entries turned by position, neighbours or halves in pairs; stretched where asked."""
    if not rot or not rot["dims"]:
        return v
    d, base, s = rot["dims"], float(rot["base"]), rot.get("scaling")
    i = torch.arange(d // 2, dtype=torch.float64, device=v.device)
    f, amp = base ** (-2.0 * i / d), 1.0
    if s is not None:
        index = lambda turns: d * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))      # noqa: E731
        lo, hi = max(math.floor(index(s["fast"])), 0), min(math.ceil(index(s["slow"])), d - 1)
        share = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, amp = f / s["factor"] * share + f * (1.0 - share), 0.1 * math.log(s["factor"]) + 1.0
    angle = torch.arange(v.shape[0], dtype=torch.float64, device=v.device)[:, None] * f
    angle = angle.view(v.shape[0], *(1,) * (v.dim() - 2), d // 2)
    c, s = amp * torch.cos(angle), amp * torch.sin(angle)
    out = v.clone()
    lo, hi = (slice(0, d // 2), slice(d // 2, d)) if halves else (slice(0, d, 2), slice(1, d, 2))
    out[..., lo] = v[..., lo] * c - v[..., hi] * s
    out[..., hi] = v[..., hi] * c + v[..., lo] * s
    return out


def _over_time(x, taps):
    T, K = x.shape[0], taps.shape[1]
    padded = torch.cat([torch.zeros((K - 1, x.shape[1]), dtype=x.dtype, device=x.device), x])
    return sum(padded[j:j + T] * taps[:, j] for j in range(K))


def _mixer(h, get, layer, eps, rows, index):
    m, kind, T = layer["mixer"], layer["type"], h.shape[0]
    H, D = m["heads"], m["dim"]
    if kind == "latent_attention":
        C, source = m["kv_rank"], m.get("kv_from")
        if source is None:
            down = h @ get("dkv").T
            rows[index] = (_rms(down[:, :C], eps) * get("dkv.norm"), _turned(down[:, C:], m["rot"]))
        c, k_rot = rows[index if source is None else source]
        q = ((_rms(h @ get("dq").T, eps) * get("dq.norm")) @ get("uq").T).view(T, H, -1)
        q = torch.cat([q[..., :D], _turned(q[..., D:], m["rot"])], dim=-1)
        k = torch.cat([(c @ get("uk").T).view(T, H, D), k_rot[:, None].expand(T, H, k_rot.shape[1])], dim=-1)
        return _softmax_attention(q, k, (c @ get("uv").T).view(T, H, -1), m["scale"]).reshape(T, -1) @ get("o").T
    if kind in ("delta", "channel_delta"):
        Hk, Dv = m["kv_heads"], m["vdim"]
        q, k, v = (_silu(_over_time(h @ get(n).T, get(n + ".conv"))).view(T, heads, -1) for n, heads in (("q", Hk), ("k", Hk), ("v", H)))
        unit = lambda a: a / torch.sqrt((a * a).sum(dim=-1, keepdim=True) + 1e-6)      # noqa: E731
        q, k = (unit(a).repeat_interleave(H // Hk, dim=1) for a in (q, k))
        q, beta = q * D ** -0.5, torch.sigmoid(h @ get("b").T)
        soft = torch.nn.functional.softplus
        if kind == "delta":
            decay = torch.exp(-torch.exp(get("A_log")) * soft(h @ get("a").T + get("dt_bias"), threshold=700.0))[..., None, None]
            gate = _silu(h @ get("g").T).view(T, H, Dv)
        else:
            z = ((h @ get("a1").T) @ get("a2").T + get("dt_bias")).view(T, H, D)
            decay = torch.exp(-torch.exp(get("A_log"))[None, :, None] * soft(z, threshold=700.0))[..., None]
            gate = torch.sigmoid((h @ get("g1").T) @ get("g2").T).view(T, H, Dv)
        S, out = torch.zeros((H, D, Dv), dtype=h.dtype, device=h.device), torch.empty((T, H, Dv), dtype=h.dtype, device=h.device)
        for t in range(T):
            S = decay[t] * S
            u = beta[t, :, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            out[t] = (q[t][:, None] @ S)[:, 0]
        return (_rms(out, eps) * get("norm") * gate).reshape(T, -1) @ get("o").T
    if kind == "general_delta":
        r, k, v = ((h @ get(n).T).view(T, H, D) for n in "rkv")
        d = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ get("w1").T) @ get("w2").T + get("w0"))).view(T, H, D, 1)
        u = k / torch.sqrt((k * k).sum(dim=-1, keepdim=True) + 1e-6)
        au = torch.sigmoid(h @ get("a").T + get("a.b")).view(T, H, D) * u
        S, out = torch.zeros((H, D, D), dtype=h.dtype, device=h.device), torch.empty_like(v)
        for t in range(T):
            S = d[t] * S - au[t][:, :, None] * (u[t][:, None] @ S) + k[t][:, :, None] * v[t][:, None]
            out[t] = (r[t][:, None] @ S)[:, 0]
        return (_rms(out, eps).reshape(T, -1) * get("norm") * torch.sigmoid(h @ get("g").T)) @ get("o").T
    G = m["kv_heads"]
    if kind == "attention_2":
        q = (_rms(h @ get("q").T, eps) * get("q.norm")).view(T, H, D)
        k = (_rms(h @ get("k").T, eps) * get("k.norm")).view(T, G, D)
        return _softmax_attention(q, k, (h @ get("v").T).view(T, G, -1), m["scale"] * get("temp")).reshape(T, -1) @ get("o").T
    if "diff" in m:
        if m.get("kv_from") is None:
            k = _turned((h @ get("k").T).view(T, G, 2, D), m["rot"], halves=True)
            rows[index] = (k, (h @ get("v").T).view(T, G, -1))
        k, v = rows[index if m.get("kv_from") is None else m["kv_from"]]
        q = _turned((h @ get("q").T).view(T, H, 2, D), m["rot"], halves=True)
        lam = torch.exp((get("lq1") * get("lk1")).sum()) - torch.exp((get("lq2") * get("lk2")).sum()) + m["diff"]
        a = _softmax_attention(q[:, :, 0], k[:, :, 0], v, m["scale"]) - lam * _softmax_attention(q[:, :, 1], k[:, :, 1], v, m["scale"])
        return (_rms(a, eps) * (1.0 - m["diff"])).reshape(T, -1) @ get("o").T
    q = _turned((h @ get("q").T + get("q.b")).view(T, H, D), m["rot"])
    v = (h @ get("k").T + get("k.b")).view(T, G, D)
    return _softmax_attention(q, _turned(v, m["rot"]), v, m["scale"]).reshape(T, -1) @ get("o").T


def _feed_forward(h, get, mlp, design):
    if design == "Fusazen":
        return torch.relu(h @ get("up").T + get("up.b")) ** 2 @ get("down").T + get("down.b")
    if design == "Sobezen":
        z = (h @ get("gate").T + get("gate.b")).clamp(max=mlp["limit"])
        u = (h @ get("up").T + get("up.b")).clamp(-mlp["limit"], mlp["limit"])
        return (z * torch.sigmoid(1.702 * z) * (u + 1.0)) @ get("down").T + get("down.b")
    if mlp["kind"] == "dense":
        return (_gelu_tanh(h @ get("gate").T) * (h @ get("up").T)) @ get("down").T
    best, which = torch.topk(h @ get("router").T, mlp["router"]["top"], dim=-1)
    share, out = torch.softmax(best, dim=-1), torch.zeros_like(h)
    for e in range(mlp["router"]["experts"]):
        rows, place = (which == e).nonzero(as_tuple=True)
        one = h[rows]
        y = (_silu(one @ get(f"e{e}.gate").T) * (one @ get(f"e{e}.up").T)) @ get(f"e{e}.down").T
        out.index_add_(0, rows, share[rows, place][:, None] * y)
    return out


def _exact_design(case, seed):
    cfg, w = CONFIGS[case["model"]], _weights(case, seed)
    design, eps = cfg["architecture"], cfg["norm"]["eps"]

    def norm(x, name):
        if design == "Garodra":
            return torch.tanh(w[name + ".alpha"].double() * x) * w[name].double() + w[name + ".b"].double()
        return _rms(x, eps) * w[name].double()

    results = []
    for tokens in _tokens(case, seed):
        x, rows = w["embed"][torch.tensor(tokens, device=DEVICE)].double(), {}
        for i, layer in enumerate(cfg["layers"]):
            p = f"l{i}."
            h = norm(x, p + "norm1")
            if design == "Fusazen":
                h = h + _over_time(h, w[p + "canon1"].double())
            y = _mixer(h, lambda n: w[p + "mix." + n].double(), layer, eps, rows, i)
            x = x + (norm(y, p + "norm1b") if design == "Garodra" else y * w[p + "ls1"].double() if design == "Sobezen" else y)
            if layer["mlp"] is not None:
                y = _feed_forward(norm(x, p + "norm2"), lambda n: w[p + "mlp." + n].double(), layer["mlp"], design)
                x = x + (norm(y, p + "norm2b") if design == "Garodra" else y * w[p + "ls2"].double() if design == "Sobezen" else y)
        results.append(norm(x[-case["new"]:], "final.norm") @ w["head"].double().T * cfg.get("logit_scale", 1.0))
    return results


def exact(case, seed):
    each = (_exact_llama if CONFIGS[case["model"]].get("architecture") is None else _exact_design)(case, seed)
    logits = torch.stack(each, dim=1)
    return {"logits": logits, "ids": logits.argmax(dim=-1).to(torch.int32) if case["temperature"] <= 0.0 else None}
