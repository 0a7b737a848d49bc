"""The engine's work as a serving program gives it, one pass at a time, for measuring it.

A case is one pass of `Engine.step` calls over live requests: `decode` requests that each take one more token, beside
`prompts` new prompts that are cut into portions so that a step brings at most `budget` tokens (each decoding request's
token first, then prompt portions, oldest first: what the scheduler does).  A pass without prompts is one step; a pass
with prompts admits them, runs steps until their last token's logits are there, and releases them.  The models are the
three benchmark sizes of this repository (with fewer layers where all of them would only repeat the same work), in
bfloat16 with float32 or bfloat16 recurrent states, and in float32.

`prepare` gives what a server has in hand: an engine whose graphs are captured (one engine serves all states of the
same case that are alive, as it serves all requests of a server) and requests whose contexts are in the cache.  Weights
are a property of the model and the same for every seed, as a checkpoint is; token ids come from the seed.
"""
from __future__ import annotations

import json
import math
import os
import shutil
import tempfile
import weakref

import numpy as np
import torch

_MULTIPLIERS = {
    "embedding_multiplier": 5.0, "lm_head_multiplier": 0.25, "attention_in_multiplier": 1.5,
    "attention_out_multiplier": 0.8, "key_multiplier": 0.5, "ssm_in_multiplier": 1.2, "ssm_out_multiplier": 0.7,
    "ssm_multipliers": [0.6, 1.1, 0.9, 1.3, 0.8], "mlp_multipliers": [0.9, 1.1],
}
_COMMON = {
    "architectures": ["FalconH1ForCausalLM"], "model_type": "falcon_h1", "rms_norm_eps": 1e-5, "rope_theta": 1e11,
    "mamba_n_groups": 1, "mamba_d_conv": 4, "mamba_chunk_size": 128, "mamba_conv_bias": True, "mamba_proj_bias": False,
    "projectors_bias": False, "mamba_rms_norm": False, "mamba_norm_before_gate": False,
    "hidden_act": "silu", "attention_bias": False, "mlp_bias": False, **_MULTIPLIERS,
}
MODELS = {
    "0p5b": {**_COMMON, "hidden_size": 1024, "num_attention_heads": 8, "num_key_value_heads": 2, "head_dim": 64,
             "intermediate_size": 2048, "vocab_size": 32784, "max_position_embeddings": 8192, "tie_word_embeddings": True,
             "mamba_d_ssm": 1536, "mamba_n_heads": 24, "mamba_d_head": 64, "mamba_d_state": 128},
    "1p5b-deep": {**_COMMON, "hidden_size": 1280, "num_attention_heads": 6, "num_key_value_heads": 2, "head_dim": 128,
                  "intermediate_size": 3072, "vocab_size": 65536, "max_position_embeddings": 8192,
                  "tie_word_embeddings": True, "mamba_d_ssm": 1536, "mamba_n_heads": 24, "mamba_d_head": 64,
                  "mamba_d_state": 256},
    "7b": {**_COMMON, "hidden_size": 3072, "num_attention_heads": 12, "num_key_value_heads": 2, "head_dim": 128,
           "intermediate_size": 12288, "vocab_size": 130048, "max_position_embeddings": 40960,
           "tie_word_embeddings": False, "mamba_d_ssm": 3072, "mamba_n_heads": 24, "mamba_d_head": 128,
           "mamba_d_state": 256},
}
PAGE = 64
_DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def _case(name, model, layers, dtype="bfloat16", state="float32", decode=0, low=0, high=0, prompts=0, short=0, long=0,
          budget=8192):
    """`decode` requests with contexts from `low` to `high` tokens; `prompts` prompts of `short` to `long` tokens."""
    case = {"model": model, "layers": layers, "dtype": dtype, "state": state, "decode": decode, "low": low, "high": high,
            "prompts": prompts, "short": short, "long": long, "budget": budget}
    return {"name": name, **case} if name else case


def listed():
    return [
        # one user's chat: a token at a time, the smallest call
        _case("decode-1", "0p5b", 36, decode=1, low=2048, high=2048),
        # a small server in the steady state of decoding
        _case("decode-8", "0p5b", 36, decode=8, low=2048, high=2048),
        # a full server: 64 requests decode
        _case("decode-64", "0p5b", 36, decode=64, low=2048, high=2048),
        # an odd number of requests that came at different times
        _case("decode-13-ragged", "1p5b-deep", 16, decode=13, low=37, high=4001),
        # the time to the first token of one document
        _case("prompt-2048", "0p5b", 36, prompts=1, short=2048, long=2048),
        # several users' chat turns arrive together, none of a round length
        _case("prompts-short", "0p5b", 36, prompts=5, short=19, long=203),
        # continuous serving: a prompt in portions beside the requests that decode
        _case("mixed-24", "1p5b-deep", 16, decode=24, low=128, high=4096, prompts=1, short=976, long=976, budget=512),
        # a full server of the largest model: the most bytes a decode step reads
        _case("decode-64-large", "7b", 4, decode=64, low=4096, high=4096),
        # recurrent states kept in the activations' type, contexts of all lengths
        _case("decode-24-state16", "7b", 4, state="activation", decode=24, low=203, high=3001),
        # a book as one prompt: the most operations
        _case("prompt-32768", "7b", 4, prompts=1, short=32768, long=32768),
        # the 32-bit path, decoding: someone checks a model's numbers
        _case("float32-decode", "0p5b", 12, dtype="float32", decode=4, low=301, high=702),
        # ... and its prompts
        _case("float32-prompts", "0p5b", 12, dtype="float32", prompts=2, short=91, long=350),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    model = rng.choice(["0p5b", "0p5b", "1p5b-deep", "7b"])
    layers = {"0p5b": 36, "1p5b-deep": 16, "7b": 4}[model]
    kind = rng.choice(["decode", "decode", "prompts", "prompts", "mixed", "float32"])
    state = "activation" if rng.random() < 0.15 else "float32"
    if kind == "float32":
        half = rng.random() < 0.5
        a, b = sorted((log_int(16, 700), log_int(16, 700)))
        if half:
            return _case(None, "0p5b", 12, dtype="float32", decode=log_int(1, 16), low=a, high=b)
        return _case(None, "0p5b", 12, dtype="float32", prompts=rng.randint(1, 3), short=min(a, 350), long=min(b, 350))
    a, b = sorted((log_int(32, 4096), log_int(32, 4096)))
    if kind == "decode":
        return _case(None, model, layers, state=state, decode=log_int(1, 64), low=a, high=b)
    if kind == "prompts":
        if rng.random() < 0.3:
            n = log_int(512, 16384 if model == "7b" else 7000)
            return _case(None, model, layers, state=state, prompts=1, short=n, long=n, budget=rng.choice([2048, 8192]))
        return _case(None, model, layers, state=state, prompts=rng.randint(1, 8), short=max(2, a // 8), long=max(16, b // 4))
    n = log_int(64, 1500)
    return _case(None, model, layers, state=state, decode=log_int(1, 32), low=a, high=b, prompts=1, short=n, long=n, budget=512)


# --------------------------------------------------------------------------- sizes of a case
def _spread(count, low, high):
    """`count` lengths from `low` to `high`, in no order (a low-discrepancy walk), the largest among them."""
    if count <= 1:
        return [high] * count
    return [low + int(round((high - low) * ((1 + i * 0.6180339887498949) % 1.0))) if i else high for i in range(count)]


def _contexts(case):
    return _spread(case["decode"], case["low"], case["high"])


def _prompts(case):
    return _spread(case["prompts"], case["short"], case["long"])


def _new_tokens(case):
    """Tokens a request may decode before it ends and another one of the same context takes its place."""
    if not case["decode"]:
        return 0
    return min(16384 // case["decode"] + 1024, 8192 - case["high"] - 8)


def _steps(case):
    """The steps of a pass: lists of (prompt, first token, end) beside one token of every decoding request."""
    left = [[i, 0, n] for i, n in enumerate(_prompts(case))]
    if not left:
        return [[]]
    steps = []
    while left:
        room, portions = case["budget"] - case["decode"], []
        while left and room > 0:
            i, lo, n = left[0]
            hi = min(n, lo + room)
            portions.append((i, lo, hi))
            room -= hi - lo
            left[0][1] = hi
            if hi == n:
                left.pop(0)
        steps.append(portions)
    return steps


def _config(case):
    return {**MODELS[case["model"]], "num_hidden_layers": case["layers"], "torch_dtype": case["dtype"]}


def work(case):
    c, size = _config(case), 4 if case["dtype"] == "float32" else 2
    H, inter, V, L = c["hidden_size"], c["intermediate_size"], c["vocab_size"], c["num_hidden_layers"]
    Hq, Hkv, hd = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    nh, P, N = c["mamba_n_heads"], c["mamba_d_head"], c["mamba_d_state"]
    inner, conv = nh * P, nh * P + 2 * N
    matrices = L * (H * (Hq + 2 * Hkv) * hd + Hq * hd * H + H * (inner + conv + nh) + inner * H + 3 * H * inter)
    per_key = L * 2 * Hkv * hd * size
    state = L * (nh * P * N * (2 if case["state"] == "activation" else size if size == 4 else 4) + conv * 3 * size)
    steps, contexts, prompts = _steps(case), _contexts(case), _prompts(case)
    decoded = len(steps) * len(contexts)
    wanted = decoded + len(prompts)
    tokens = decoded + sum(prompts)
    pairs = sum(s + i + 1 for s in contexts for i in range(len(steps))) + sum(n * (n + 1) // 2 for n in prompts)
    byts = (matrices + V * H) * size + wanted * V * 4 + tokens * H * size + tokens * per_key
    byts += sum(contexts) * per_key + len(contexts) * 2 * state + len(prompts) * state
    ssd = L * 4 * nh * P * N
    flops = tokens * (2 * matrices + ssd) + L * 4 * Hq * hd * pairs + 2 * V * H * wanted
    return {"bytes": float(byts), "flops": float(flops)}


def tolerance(case):
    return {"rel": 2e-5} if case["dtype"] == "float32" else {"rel": 0.03}


# --------------------------------------------------------------------------- the model
def _weights(case, layer=None):
    """The model's tensors on the GPU, by their checkpoint names: those of one layer, or (None) those outside of all
    layers.  Drawn as this repository's random models are, with its norms, biases and skips off their plain values."""
    c, dtype = _config(case), _DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(7001 + (0 if layer is None else 1 + layer))

    def normal(*shape, std=0.02, mean=0.0):
        return torch.randn(shape, generator=gen, device="cuda").mul_(std).add_(mean).to(dtype)

    H, inter = c["hidden_size"], c["intermediate_size"]
    if layer is None:
        out = {"model.embed_tokens.weight": normal(c["vocab_size"], H), "model.final_layernorm.weight": normal(H, std=0.1, mean=1.0)}
        if not c["tie_word_embeddings"]:
            out["lm_head.weight"] = normal(c["vocab_size"], H)
        return out
    q, kv = c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
    nh, inner = c["mamba_n_heads"], c["mamba_d_ssm"]
    conv = inner + 2 * c["mamba_n_groups"] * c["mamba_d_state"]
    step = torch.exp(torch.empty(nh, device="cuda").uniform_(math.log(1e-3), math.log(1e-1), generator=gen))
    tensors = {
        "input_layernorm.weight": normal(H, std=0.1, mean=1.0),
        "self_attn.q_proj.weight": normal(q, H), "self_attn.k_proj.weight": normal(kv, H),
        "self_attn.v_proj.weight": normal(kv, H), "self_attn.o_proj.weight": normal(H, q),
        "mamba.in_proj.weight": normal(inner + conv + nh, H),
        "mamba.conv1d.weight": normal(conv, 1, c["mamba_d_conv"], std=0.2), "mamba.conv1d.bias": normal(conv),
        "mamba.A_log": torch.log(torch.empty(nh, device="cuda").uniform_(1.0, 16.0, generator=gen)),
        "mamba.dt_bias": (step + torch.log(-torch.expm1(-step))).to(dtype), "mamba.D": normal(nh, std=0.1, mean=1.0),
        "mamba.out_proj.weight": normal(H, inner),
        "pre_ff_layernorm.weight": normal(H, std=0.1, mean=1.0),
        "feed_forward.gate_proj.weight": normal(inter, H), "feed_forward.up_proj.weight": normal(inter, H),
        "feed_forward.down_proj.weight": normal(H, inter),
    }
    return {f"model.layers.{layer}.{k}": v for k, v in tensors.items()}


def _write_model(case, folder):
    """config.json and model.safetensors (a header of 8 bytes of length and JSON, then the tensors' bytes)."""
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(_config(case), f)
    groups = [None, *range(case["layers"])]
    header, at = {}, 0
    for g in groups:
        for name, t in _weights(case, g).items():
            n = t.numel() * t.element_size()
            kind = {torch.bfloat16: "BF16", torch.float32: "F32"}[t.dtype]
            header[name] = {"dtype": kind, "shape": list(t.shape), "data_offsets": [at, at + n]}
            at += n
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(len(text).to_bytes(8, "little"))
        f.write(text)
        for g in groups:
            for t in _weights(case, g).values():
                t.reshape(-1).view(torch.uint8).cpu().numpy().tofile(f)


_engines = weakref.WeakValueDictionary()        # the engines that states in use hold, by their case
_STATES = 3                                     # states of a case that may be in use at once


def _engine(case):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    engine = _engines.get(key)
    if engine is None:
        from logssms_b200.engine import Engine
        rows = _STATES * (case["decode"] + case["prompts"])
        longest = max([n + _new_tokens(case) for n in _contexts(case)] + _prompts(case)) + 8
        pages = sum(-(-(n + _new_tokens(case)) // PAGE) + 1 for n in _contexts(case)) + sum(-(-n // PAGE) for n in _prompts(case))
        limit = max(8192, -(-longest // PAGE) * PAGE)
        folder = tempfile.mkdtemp(prefix="logssms_b200_cases_")
        try:
            _write_model(case, folder)
            engine = Engine(folder, case["dtype"], max_requests=max(rows, 4), max_seq_len=limit, page_size=PAGE,
                            num_pages=_STATES * pages + 16, ssm_state_dtype=case["state"])
        finally:
            shutil.rmtree(folder, ignore_errors=True)
        torch.cuda.empty_cache()
        _engines[key] = engine
        _warm(engine, case)
    return engine


def _warm(engine, case):
    """What a server has behind it when a request comes: kernels loaded, graphs captured."""
    if not case["prompts"]:
        engine.capture_decode_graphs([case["decode"]])
        return
    fits = all(case["decode"] + sum(hi - lo for _, lo, hi in s) <= engine.max_graph_tokens for s in _steps(case))
    state = _state(engine, case, 0)
    for _ in range(engine.exact_after + 4 if fits else 2):
        run(state)
    torch.cuda.synchronize()


# --------------------------------------------------------------------------- a state and a pass
class _Live:
    """The decoding requests of a state; they are released with it."""

    def __init__(self, engine, contexts):
        from logssms_b200.engine import StepEntry
        self.engine, self.requests = engine, []
        for ids in contexts:
            request = engine.new_request()
            self.requests.append(request)
        # contexts go into the cache in steps of at most 8,192 tokens
        pending = [[r, ids, 0] for r, ids in zip(self.requests, contexts)]
        while pending:
            room, entries = 8192, []
            while pending and room > 0:
                r, ids, lo = pending[0]
                hi = min(len(ids), lo + room)
                entries.append(StepEntry(r, ids[lo:hi]))
                room -= hi - lo
                pending[0][2] = hi
                if hi == len(ids):
                    pending.pop(0)
            engine.step(entries)

    def __del__(self):
        for r in reversed(self.requests):
            self.engine.release(r)


def _ids(case, seed):
    """Token ids: per decoding request its context and the tokens that follow, per prompt its tokens."""
    V = MODELS[case["model"]]["vocab_size"]
    rng = np.random.default_rng([seed, 17])
    contexts = [rng.integers(0, V, n).tolist() for n in _contexts(case)]
    prompts = [rng.integers(0, V, n).tolist() for n in _prompts(case)]
    new = [rng.integers(0, V, _new_tokens(case)).tolist() for _ in contexts]
    return contexts, prompts, new


def _state(engine, case, seed):
    contexts, prompts, new = _ids(case, seed)
    return {"engine": engine, "live": _Live(engine, contexts), "contexts": contexts, "prompts": prompts, "new": new,
            "steps": _steps(case), "room": _new_tokens(case), "at": 0}


def prepare(case, seed):
    return _state(_engine(case), case, seed)


def _rows(states, requests):
    rows = [r.row for r in requests]
    if rows == list(range(rows[0], rows[0] + len(rows))):
        return states[rows[0]:rows[0] + len(rows)]
    return states[rows]


def run(state):
    """One pass.  Returns the logits of every step and the last layer's recurrent states after it (whose inputs have
    gone through all the other layers)."""
    from logssms_b200.engine import StepEntry
    engine, prompts, steps = state["engine"], state["prompts"], state["steps"]
    if state["contexts"] and state["at"] + len(steps) > state["room"]:
        state["live"] = None                       # these requests are done: others take their places
        state["live"], state["at"] = _Live(engine, state["contexts"]), 0
    live = state["live"].requests
    coming = [engine.new_request() for _ in prompts]
    logits = []
    for portions in steps:
        at = state["at"]
        entries = [StepEntry(r, [ids[at]], [0]) for r, ids in zip(live, state["new"])]
        for i, lo, hi in portions:
            entries.append(StepEntry(coming[i], prompts[i][lo:hi], [hi - lo - 1] if hi == len(prompts[i]) else []))
        out = engine.step(entries)
        # a step's logits are the engine's own buffer until its next step
        logits.append(out.clone() if len(steps) > 1 else out)
        state["at"] += 1
    last = engine.cache.states[-1]["ssm"]
    result = {"logits": [x for x in logits if x.shape[0]], "states": [_rows(last, r) for r in (live, coming) if r]}
    for r in reversed(coming):
        engine.release(r)
    return result


# --------------------------------------------------------------------------- the same in 64 bits
def _norm(x, weight, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight


def _attention(x, w, c):
    T, hd = x.shape[0], c["head_dim"]
    Hq, Hkv = c["num_attention_heads"], c["num_key_value_heads"]
    q = (x @ w["self_attn.q_proj.weight"].T).view(T, Hq, hd)
    k = (x @ w["self_attn.k_proj.weight"].T).view(T, Hkv, hd) * c["key_multiplier"]
    v = (x @ w["self_attn.v_proj.weight"].T).view(T, Hkv, hd)
    inv = 1.0 / (c["rope_theta"] ** (torch.arange(0, hd, 2, dtype=torch.float32) / hd))
    angle = (torch.arange(T, dtype=torch.float32)[:, None] * inv).cuda().double()[:, None, :]
    cos, sin = angle.cos(), angle.sin()

    def rotate(t):
        a, b = t[..., :hd // 2], t[..., hd // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    q = rotate(q).view(T, Hkv, Hq // Hkv, hd).permute(1, 2, 0, 3)              # [Hkv, group, T, hd]
    k, v = rotate(k).transpose(0, 1)[:, None], v.transpose(0, 1)[:, None]      # [Hkv, 1, T, hd]
    out, rows = torch.empty_like(q), max(64, min(T, (1 << 27) // (Hq * T)))
    for lo in range(0, T, rows):
        hi = min(T, lo + rows)
        scores = q[:, :, lo:hi] @ k[:, :, :hi].transpose(-1, -2) * hd ** -0.5
        mask = torch.arange(hi, device="cuda")[None, :] > torch.arange(lo, hi, device="cuda")[:, None]
        out[:, :, lo:hi] = torch.softmax(scores.masked_fill_(mask, float("-inf")), -1) @ v[:, :, :hi]
    return out.permute(2, 0, 1, 3).reshape(T, Hq * hd) @ w["self_attn.o_proj.weight"].T


def _mamba(x, w, c, Q=64):
    """The mixer's rows and its recurrent state after the last one, by chunks of Q tokens."""
    T, nh, P, N = x.shape[0], c["mamba_n_heads"], c["mamba_d_head"], c["mamba_d_state"]
    inner, K, m = nh * P, c["mamba_d_conv"], c["ssm_multipliers"]
    z, xbc, dt = (x @ w["mamba.in_proj.weight"].T).split([inner, inner + 2 * N, nh], -1)
    scale = torch.cat([torch.full((n,), s, dtype=torch.float64, device="cuda") for n, s in ((inner, m[1]), (N, m[2]), (N, m[3]))])
    padded = torch.cat([xbc.new_zeros(K - 1, inner + 2 * N), xbc * scale])
    conv = sum(padded[j:j + T] * w["mamba.conv1d.weight"][:, 0, j] for j in range(K)) + w["mamba.conv1d.bias"]
    conv = torch.nn.functional.pad(torch.nn.functional.silu(conv), (0, 0, 0, -T % Q))
    n = conv.shape[0] // Q
    u, B, C = conv[:, :inner].view(n, Q, nh, P), conv[:, inner:inner + N].view(n, Q, N), conv[:, inner + N:].view(n, Q, N)
    dt = torch.nn.functional.softplus(dt * m[4] + w["mamba.dt_bias"], threshold=1e9)
    dt = torch.nn.functional.pad(dt, (0, 0, 0, -T % Q)).view(n, Q, nh)          # a filled-up token: no step, nothing decays
    cum = (-torch.exp(w["mamba.A_log"]) * dt).cumsum(1)                        # [n, Q, nh]
    own = u * dt[..., None]
    later = torch.ones(Q, Q, dtype=torch.bool, device="cuda").triu(1)
    state, y = x.new_zeros(nh, P, N), torch.empty_like(u)
    added = (own * torch.exp(cum[:, -1:] - cum)[..., None]).permute(0, 2, 3, 1) @ B[:, None]        # [n, nh, P, N]
    for i in range(n):
        decay = torch.exp((cum[i][:, None] - cum[i][None, :]).masked_fill(later[..., None], float("-inf")))   # [Q, Q, nh]
        mix = (C[i] @ B[i].T)[..., None] * decay
        y[i] = torch.einsum("qsh,shp->qhp", mix, own[i]) + torch.einsum("qn,hpn,qh->qhp", C[i], state, torch.exp(cum[i]))
        state = state * torch.exp(cum[i, -1])[:, None, None] + added[i]
    y = (y + w["mamba.D"][:, None] * u).view(n * Q, inner)[:T]
    return (y * torch.nn.functional.silu(z * m[0])) @ w["mamba.out_proj.weight"].T, state


def _sequences(case, sequences, wanted):
    """For whole sequences: the logits of the last `wanted` tokens of each, and the last layer's state at its end."""
    c = _config(case)
    outer = {k: v.double() for k, v in _weights(case).items()}
    embed, eps = outer["model.embed_tokens.weight"], c["rms_norm_eps"]
    rows = [embed[torch.tensor(ids, device="cuda")] * c["embedding_multiplier"] for ids in sequences]
    states = [None] * len(rows)
    for layer in range(case["layers"]):
        w = {k.split(".", 3)[3]: v.double() for k, v in _weights(case, layer).items()}
        for i, x in enumerate(rows):
            h = _norm(x, w["input_layernorm.weight"], eps)
            mixed, states[i] = _mamba(h * c["ssm_in_multiplier"], w, c)
            x = x + c["attention_out_multiplier"] * _attention(h * c["attention_in_multiplier"], w, c) + c["ssm_out_multiplier"] * mixed
            h = _norm(x, w["pre_ff_layernorm.weight"], eps)
            gate = torch.nn.functional.silu(h @ w["feed_forward.gate_proj.weight"].T * c["mlp_multipliers"][0])
            rows[i] = x + gate * (h @ w["feed_forward.up_proj.weight"].T) @ w["feed_forward.down_proj.weight"].T * c["mlp_multipliers"][1]
    head = outer.get("lm_head.weight", embed)
    out = [_norm(x[-n:], outer["model.final_layernorm.weight"], eps) @ head.T * c["lm_head_multiplier"] for x, n in zip(rows, wanted)]
    return out, states


def exact(case, seed):
    contexts, prompts, new = _ids(case, seed)
    steps = _steps(case)
    sequences = [ids + more[:len(steps)] for ids, more in zip(contexts, new)] + prompts
    if sum(map(len, sequences)) * (work({**case, "decode": 0, "prompts": 1, "short": 1, "long": 1})["flops"]) > 6e14:
        return None
    out, states = _sequences(case, sequences, [len(steps)] * len(contexts) + [1] * len(prompts))
    logits, B = [], len(contexts)
    for k, portions in enumerate(steps):
        rows = [out[b][k] for b in range(B)] + [out[B + i][0] for i, _, hi in portions if hi == len(prompts[i])]
        if rows:
            logits.append(torch.stack(rows))
    return {"logits": logits, "states": [torch.stack(s) for s in (states[:B], states[B:]) if s]}
