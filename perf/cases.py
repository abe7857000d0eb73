"""The work that the engine is timed on, as calls of its public entry points with inputs made from a seed.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same ranges, ``prepare(case, seed)`` builds what a
program has in hand before the call (an engine with random weights, requests whose prompts are in the cache, the steps'
shapes seen before, as a server does before it takes requests), ``run(state)`` is one pass, ``exact(case, seed)`` the
same outputs as plain torch forms them in 64 bits.

Two kinds of pass:

``step``      one step of the batch through ``Engine.step_raw``: ``decode`` requests bring one token each, after contexts of
              ``context`` tokens (``ragged``: of context / 16 to context tokens), and ``prompts`` new requests bring their
              whole prompts of ``tokens`` tokens (``ragged``: tokens / 4 to tokens); logits after every decoded token and
              at the last ``want`` places of every prompt.  The decoding requests keep their tokens from pass to pass,
              as in serving; the prompts' requests end with the pass.
``generate``  ``Engine.generate``: ``prompts`` greedy requests of ``tokens`` tokens, ``new`` generated tokens each.
"""

import math

import torch

from ferrisinfer_b200 import Engine, SamplingParams, SchedulerConfig
from ferrisinfer_b200.engine.runner import StepEntry
from ferrisinfer_b200.weights.random_init import random_tensors

DEVICE = "cuda"
PAGE = 16
ROOM = 4096  # tokens that a decoding request can grow by before its conversation begins anew
PREPARE_TOKENS = 8192  # of the steps that bring the contexts in
WARM = 2  # passes of other tokens before the first one

QWEN_05B = {
    "architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": 151936, "hidden_size": 896,
    "intermediate_size": 4864, "num_hidden_layers": 24, "num_attention_heads": 14, "num_key_value_heads": 2,
    "max_position_embeddings": 32768, "rms_norm_eps": 1e-6, "rope_theta": 1000000.0, "hidden_act": "silu",
    "tie_word_embeddings": True, "use_sliding_window": False, "sliding_window": None, "max_window_layers": 24,
}
QWEN_15B = dict(QWEN_05B, hidden_size=1536, intermediate_size=8960, num_hidden_layers=28, num_attention_heads=12,
                max_window_layers=28)
QWEN_7B = dict(QWEN_05B, vocab_size=152064, hidden_size=3584, intermediate_size=18944, num_hidden_layers=28,
               num_attention_heads=28, num_key_value_heads=4, tie_word_embeddings=False, max_window_layers=28)

# the sizes at which the benchmark puts the designs side by side: width 2048, 16 heads of 128 over 4, 12 layer runs
_WIDTH, _HEADS, _KV, _DIM, _FF, _WINDOW, _VOCAB = 2048, 16, 4, 128, 8192, 1024, 32000
_DECAY = [round(1.0 - 2.0 ** (-2 - 6 * h / _HEADS), 6) for h in range(_HEADS)]
_K_ATT = {"type": "attention", "mlp": {"kind": "dense", "ff": _FF},
          "mixer": {"heads": _HEADS, "kv_heads": _KV, "dim": _DIM, "vdim": _DIM, "scale": _DIM ** -0.5,
                    "mask": {"size": _WINDOW}, "q_temp": {"coef": 0.3, "every": 128}}}
_K_LIN = {"type": "lightning", "mlp": {"kind": "dense", "ff": _FF},
          "mixer": {"heads": _HEADS, "dim": _DIM, "vdim": _DIM, "decay": _DECAY}}
KUGILIX = {"architecture": "Kugilix", "vocab": _VOCAB, "width": _WIDTH, "embedding": {"scale": _WIDTH ** 0.5},
           "norm": {"eps": 1e-6, "groups": 4}, "canon": {"taps": 4}, "loop": {"start": 2, "stop": 6, "times": 2},
           "layers": [_K_ATT, _K_LIN, _K_LIN, _K_ATT, _K_LIN, _K_LIN, _K_ATT, _K_LIN]}
_N_MLP = {"kind": "moe", "expert": {"ff": 2688}, "router": {"experts": 8, "top": 2}}
_N_ATT = {"type": "attention", "mlp": _N_MLP,
          "mixer": {"heads": _HEADS, "kv_heads": _KV, "dim": _DIM, "vdim": _DIM, "scale": _DIM ** -0.5,
                    "mask": {"size": _WINDOW},
                    "rot": {"base": 10000.0, "dims": _DIM,
                            "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}}}
_N_RET = {"type": "retention", "mlp": _N_MLP,
          "mixer": {"heads": _HEADS, "dim": _DIM, "vdim": _DIM, "rot": {"base": 1000000.0, "dims": _DIM}, "decay": _DECAY}}
NETINEX = {"architecture": "Netinex", "vocab": _VOCAB, "width": _WIDTH, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
           "layers": [_N_ATT, _N_RET, _N_RET] * 4}

MODELS = {"qwen-0.5b": QWEN_05B, "qwen-1.5b": QWEN_15B, "qwen-7b": QWEN_7B, "kugilix": KUGILIX, "netinex": NETINEX}


def _step(model, dtype="bfloat16", decode=0, context=0, prompts=0, tokens=0, want=1, ragged=False):
    return {"kind": "step", "model": model, "dtype": dtype, "decode": decode, "context": context, "prompts": prompts,
            "tokens": tokens, "want": want, "ragged": ragged}


def _generate(model, dtype, prompts, tokens, new):
    return {"kind": "generate", "model": model, "dtype": dtype, "prompts": prompts, "tokens": tokens, "new": new}


def listed():
    return [
        # one user's next token in a long conversation: the smallest step, all latency
        dict(_step("qwen-0.5b", decode=1, context=4096), name="decode-1"),
        # the benchmark's headline: eight users
        dict(_step("qwen-0.5b", decode=8, context=4096), name="decode-8"),
        # a busy server's decode step
        dict(_step("qwen-0.5b", decode=64, context=4096), name="decode-64"),
        # one long prompt
        dict(_step("qwen-0.5b", prompts=1, tokens=2048), name="prompt-2048"),
        # the step of continuous batching: requests at all lengths decode beside a portion of a new prompt
        dict(_step("qwen-1.5b", decode=31, context=2000, prompts=1, tokens=481, ragged=True), name="mixed-1.5b"),
        # short prompts of different lengths that arrive together
        dict(_step("qwen-1.5b", prompts=6, tokens=700, ragged=True), name="prompts-1.5b"),
        # the largest published sizes: decode of a small batch, one prompt
        dict(_step("qwen-7b", decode=8, context=1024), name="decode-8-7b"),
        dict(_step("qwen-7b", prompts=1, tokens=2048), name="prompt-2048-7b"),
        # the 32-bit path: a trace replayed with logits at several places, as checks of a model do
        dict(_step("qwen-0.5b", dtype="float32", prompts=1, tokens=777, want=16), name="replay-fp32"),
        # the 32-bit path from prompts to tokens
        dict(_generate("qwen-0.5b", "float32", prompts=4, tokens=96, new=24), name="generate-fp32"),
        # another design's long prompt: linear attention, windowed attention with slopes, short convolutions
        dict(_step("kugilix", prompts=1, tokens=2048, want=16), name="prompt-2048-kugilix"),
        # another design's busy decode step: mixtures of experts, retention, attention over chunks
        dict(_step("netinex", decode=64, context=1000), name="decode-64-netinex"),
    ]


def draw(rng):
    def between(lo, hi):  # a whole number, spread over its logarithm
        return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))

    what = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "fp32", "generate", "design"])
    model = rng.choice(["qwen-0.5b", "qwen-0.5b", "qwen-1.5b", "qwen-7b"])
    cached = {"qwen-0.5b": 65536, "qwen-1.5b": 32768, "qwen-7b": 8192}.get(model)
    ragged = rng.random() < 0.5
    if what == "decode":
        batch = between(1, 64)
        return _step(model, decode=batch, context=between(40, min(4096, cached // batch)), ragged=ragged)
    if what == "prompt":
        prompts = between(1, 8)
        return _step(model, prompts=prompts, tokens=between(16, 2048 // prompts), ragged=ragged)
    if what == "mixed":
        batch = between(1, 63)
        return _step(model, decode=batch, context=between(40, min(2000, cached // batch)), prompts=1,
                     tokens=between(16, 1024), ragged=True)
    if what == "fp32":
        if rng.random() < 0.5:
            batch = between(1, 32)
            return _step("qwen-0.5b", dtype="float32", decode=batch, context=between(40, min(2000, 16384 // batch)), ragged=ragged)
        return _step("qwen-0.5b", dtype="float32", prompts=between(1, 2), tokens=between(16, 1024), want=8, ragged=ragged)
    if what == "generate":
        return _generate("qwen-0.5b", "float32", between(1, 8), between(16, 192), between(4, 24))
    model = rng.choice(["kugilix", "netinex"])
    if rng.random() < 0.5:
        batch = between(8, 64)
        return _step(model, decode=batch, context=between(40, 65536 // batch if batch > 40 else 1500), ragged=ragged)
    return _step(model, prompts=between(1, 2), tokens=between(64, 1024), want=16, ragged=ragged)


# ------------------------------------------------------------------------------------------------------- inputs
def _vocab(case):
    cfg = MODELS[case["model"]]
    return cfg.get("vocab_size") or cfg["vocab"]


def _ids(case, seed, name, count):
    # integer seeds of their own for every list: lists do not depend on which others are made
    g = torch.Generator().manual_seed((int(seed) * 1000003 + name) & 0x7FFFFFFF)
    return torch.randint(0, _vocab(case), (count,), generator=g).tolist()


def _spread(count, low, high):
    """``count`` lengths from low to high, the longest first, in steps of one ratio, made odd."""
    if count == 1:
        return [high]
    return [max(1, round(high * (low / high) ** (i / (count - 1)))) | (1 if i else 0) for i in range(count)]


def _contexts(case):
    n, c = case["decode"], case["context"]
    return _spread(n, max(8, c // 16), c) if case["ragged"] else [c] * n


def _lengths(case):
    n, t = case["prompts"], case["tokens"]
    return _spread(n, max(2, t // 4), t) if case.get("ragged") else [t] * n


def _weights_seed(seed):
    return int(seed) & 0xFFFF


def _bring_contexts(state):
    """The decoding requests' contexts go into the cache, several requests a step."""
    engine, entries, tokens = state["engine"], [], 0
    for rid, ids in enumerate(state["contexts"]):
        if engine.runner.has_request(rid):
            engine.runner.free_request(rid)
        for at in range(0, len(ids), PREPARE_TOKENS):
            part = ids[at:at + PREPARE_TOKENS]
            if tokens + len(part) > PREPARE_TOKENS:
                engine.step_raw(entries)
                entries, tokens = [], 0
            entries.append(StepEntry(rid, part))
            tokens += len(part)
    if entries:
        engine.step_raw(entries)
    state["grown"] = 0


def prepare(case, seed):
    cfg = MODELS[case["model"]]
    decode = case.get("decode", 0)
    lengths = _lengths(case)
    longest = max([case["context"] + WARM + ROOM + 8 if decode else 0, case["tokens"] + case.get("new", 0) + 8])
    rows = decode * longest + sum(lengths) + len(lengths) * (case.get("new", 0) + 8)
    requests = decode + len(lengths)
    scheduler = SchedulerConfig(max_batch_size=requests, max_sequence_length=longest, max_prefill_chunk_tokens=2048,
                                max_prefill_batch_tokens=max(2048, requests), max_generated_tokens=max(1, case.get("new", 1)))
    engine = Engine(config=cfg, seed=_weights_seed(seed), dtype=case["dtype"], init_device=DEVICE, page_size=PAGE,
                    num_pages=-(-rows // PAGE) + 2 * requests + 4, scheduler=scheduler, prefix_sharing=False)
    if case["kind"] == "generate":
        state = {"engine": engine, "params": SamplingParams.greedy(max_new_tokens=case["new"]),
                 "prompts": [_ids(case, seed, 100000 + i, n) for i, n in enumerate(lengths)]}
        engine.generate([_ids(case, seed, 200000 + i, n) for i, n in enumerate(lengths)], state["params"])
        return state
    state = {"engine": engine, "decode": decode, "want": case["want"], "passes": 0, "grown": 0,
             "contexts": [_ids(case, seed, i, n) for i, n in enumerate(_contexts(case))],
             "next": [_ids(case, seed, 300000 + i, decode) for i in range(WARM + 64)]}
    _bring_contexts(state)
    for i in range(WARM):
        state["prompts"] = [_ids(case, seed, 200000 + 1000 * i + k, n) for k, n in enumerate(lengths)]
        run(state)
    state["prompts"] = [_ids(case, seed, 100000 + k, n) for k, n in enumerate(lengths)]
    return state


# --------------------------------------------------------------------------------------------------------- pass
def run(state):
    engine = state["engine"]
    if "params" in state:
        outs = engine.generate(state["prompts"], state["params"])
        return {"tokens": torch.tensor([[t.token_id for t in o.generated_tokens] for o in outs]),
                "probabilities": torch.tensor([[t.probability for t in o.generated_tokens] for o in outs])}
    if state["grown"] >= ROOM:
        _bring_contexts(state)
    tokens = state["next"][state["passes"] % len(state["next"])]
    entries = [StepEntry(rid, [tokens[rid]], [0]) for rid in range(state["decode"])]
    for k, prompt in enumerate(state["prompts"]):
        n = len(prompt)
        entries.append(StepEntry(("prompt", k), prompt, list(range(max(0, n - state["want"]), n))))
    logits = engine.step_raw(entries)
    for k in range(len(state["prompts"])):
        engine.runner.free_request(("prompt", k))
    state["passes"] += 1
    state["grown"] += 1
    return logits


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def _sizes(cfg):
    """(weights of the layers that one token meets, weights of the layers that a step reads, output head, layers with a
    cache of keys, elements of a token's keys and values there, heads x head size, window)."""
    if "hidden_size" in cfg:
        H, I, L = cfg["hidden_size"], cfg["intermediate_size"], cfg["num_hidden_layers"]
        nh, kv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
        d = H // nh
        layers = L * (2 * H * nh * d + 2 * H * kv * d + 3 * H * I)
        return layers, layers, cfg["vocab_size"] * H, L, 2 * kv * d, nh * d, None
    W, hd, runs = cfg["width"], _HEADS * _DIM, 12
    att, lin = W * (2 * hd + 2 * _KV * _DIM), W * 5 * hd
    attended = [layer["type"] == "attention" for layer in cfg["layers"]]
    if "loop" in cfg:  # a span of layers runs twice over the same weights
        attended = attended[:2] + attended[2:6] * 2 + attended[6:]
        met = sum(att if a else lin for a in attended) + runs * 2 * W * _FF
        read = sum(att if layer["type"] == "attention" else lin for layer in cfg["layers"]) + 8 * 2 * W * _FF
        return met, read, cfg["vocab"] * W, sum(attended), 2 * _KV * _DIM, hd, _WINDOW
    att -= W * _KV * _DIM  # the values are the keys
    met = sum(att if a else lin for a in attended) + runs * 2 * 3 * W * 2688
    read = sum(att if a else lin for a in attended) + runs * 8 * 3 * W * 2688
    return met, read, cfg["vocab"] * W, sum(attended), 2 * _KV * _DIM, hd, _WINDOW


def work(case):
    cfg = MODELS[case["model"]]
    met, read, head, attended, row, hd, window = _sizes(cfg)
    size = 4 if case["dtype"] == "float32" else 2
    contexts, lengths, steps = [], _lengths(case), case.get("new", 1)
    if case["kind"] == "step":
        contexts = [c + WARM for c in _contexts(case)]
        logits = len(contexts) + sum(min(case["want"], n) for n in lengths)
        tokens = len(contexts) + sum(lengths)
    else:
        logits, tokens = len(lengths) * steps, sum(lengths) + len(lengths) * (steps - 1)
    seen = sum(min(c + 1, window or c + 1) for c in contexts)  # keys that the single tokens read
    cached = seen
    pairs = float(seen)
    for n in lengths:
        pairs += n * (n + 1) / 2.0 if not window or n <= window else n * window - window * (window - 1) / 2.0
        cached += n
        for k in range(1, steps):
            pairs += n + k
            cached += n + k
    if "hidden_size" not in cfg and "loop" not in cfg and tokens < 8:
        read -= 12 * (8 - min(8, 2 * tokens)) * 3 * cfg["width"] * 2688  # experts that no token takes
    state = 0 if "hidden_size" in cfg else (12 - attended) * _HEADS * _DIM * _DIM  # of the recurrent layers, a request
    held = len(contexts) + len(lengths)
    flops = 2.0 * met * tokens + 2.0 * head * logits + 4.0 * hd * pairs * attended + 6.0 * state * tokens
    bytes_ = steps * (read + head) * size + cached * row * attended * size + logits * (cfg.get("vocab_size") or cfg["vocab"]) * 4.0
    return {"bytes": float(bytes_ + 8.0 * state * held), "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        # 32-bit sums in another order through all layers; a greedy token may fall to a tie
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.01 if case["kind"] == "generate" else 0.0}
    # bf16 operands and activations through all layers: two correct orders of the sums differ by what each is off
    return {"rel": 0.03, "max": 0.3}


# -------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(z):
    return z * torch.sigmoid(z)


def _angles(positions, freqs):
    return positions.double()[:, None] * torch.tensor(freqs, dtype=torch.float64, device=DEVICE)


def _rotate(x, angles, factor=1.0, neighbours=False):
    """x [T, heads, dim]; pairs are (i, i + dim / 2), or (2i, 2i + 1)."""
    c, s = (factor * torch.cos(angles))[:, None], (factor * torch.sin(angles))[:, None]
    if neighbours:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(q, k, v, scale, bias):
    """q [T, H, d], k and v [T, G, d], bias [H or 1, T, T] added to the scores (minus infinity where unseen)."""
    G = k.shape[1]
    out = torch.empty_like(q)
    per = q.shape[1] // G
    for g in range(G):
        qg = q[:, g * per:(g + 1) * per].transpose(0, 1)
        s = (qg @ k[:, g].T) * scale
        s += bias if bias.shape[0] == 1 else bias[g * per:(g + 1) * per]
        out[:, g * per:(g + 1) * per] = (torch.softmax(s, -1) @ v[:, g]).transpose(0, 1)
    return out.flatten(1)


def _far(T):
    """How far key j lies before query t, and minus infinity where j is after t."""
    t = torch.arange(T, device=DEVICE, dtype=torch.float64)
    dist = t[:, None] - t[None]
    return dist, torch.zeros_like(dist).masked_fill_(dist < 0, -math.inf)


def _qwen(cfg, w, seqs, wanted):
    """Logits at the wanted places of each sequence, all rows through a layer together, attention sequence by sequence."""
    H, nh, kv, eps = cfg["hidden_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"]
    d = H // nh
    freqs = [cfg["rope_theta"] ** (-2.0 * i / d) for i in range(d // 2)]
    x = w["model.embed_tokens.weight"][torch.tensor([t for s in seqs for t in s], device=DEVICE)].double()
    spans, at = [], 0
    for s in seqs:
        spans.append((at, at + len(s)))
        at += len(s)
    angles = _angles(torch.cat([torch.arange(len(s), device=DEVICE) for s in seqs]), freqs)
    masks = {T: _far(T)[1][None] for T in {len(s) for s in seqs}}
    for i in range(cfg["num_hidden_layers"]):
        def W(name):
            return w[f"model.layers.{i}.{name}"].double()
        y = _rms(x, W("input_layernorm.weight"), eps)
        q, k, v = (y @ W(f"self_attn.{n}_proj.weight").T + W(f"self_attn.{n}_proj.bias") for n in "qkv")
        q, k, v = _rotate(q.view(-1, nh, d), angles), _rotate(k.view(-1, kv, d), angles), v.view(-1, kv, d)
        o = torch.cat([_attend(q[a:b], k[a:b], v[a:b], d ** -0.5, masks[b - a]) for a, b in spans])
        x = x + o @ W("self_attn.o_proj.weight").T
        y = _rms(x, W("post_attention_layernorm.weight"), eps)
        x = x + (_silu(y @ W("mlp.gate_proj.weight").T) * (y @ W("mlp.up_proj.weight").T)) @ W("mlp.down_proj.weight").T
    rows = torch.tensor([a + p for (a, _), places in zip(spans, wanted) for p in places], device=DEVICE)
    head = w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"].double()
    return _rms(x[rows], w["model.norm.weight"].double(), eps) @ head.T


def _kugilix(cfg, w, ids, places):
    eps, T = cfg["norm"]["eps"], len(ids)

    def norm(x, name):
        return _rms(x.view(T, cfg["norm"]["groups"], -1), 1.0, eps).flatten(1) * w[name].double()

    t = torch.arange(T, device=DEVICE)
    wave = _angles(t, [10000.0 ** (-2.0 * i / _WIDTH) for i in range(_WIDTH // 2)])
    first = w["embed"][torch.tensor(ids, device=DEVICE)].double() * cfg["embedding"]["scale"]
    first = first + torch.stack([torch.sin(wave), torch.cos(wave)], -1).flatten(1)
    dist, unseen = _far(T)
    slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / _HEADS) for h in range(_HEADS)], dtype=torch.float64, device=DEVICE)
    bias = unseen.masked_fill(dist >= _WINDOW, -math.inf)[None] - slopes[:, None, None] * dist
    log_decay = torch.log(torch.tensor(_DECAY, dtype=torch.float64, device=DEVICE))
    x = first
    for n, i in enumerate([0, 1, 2, 3, 4, 5, 2, 3, 4, 5, 6, 7]):
        layer, p = cfg["layers"][i], f"l{i}"

        def W(name):
            return w[p + name].double()
        if n == 6:
            x = x + first
        y = norm(x, p + ".norm1")
        taps, u = W(".canon1"), y
        for j in range(taps.shape[1]):
            back = taps.shape[1] - 1 - j
            u = u + taps[:, j] * torch.cat([torch.zeros_like(y[:back]), y[:T - back]])
        q, k, v = (u @ W(f".mix.{m}").T for m in "qkv")
        if layer["type"] == "attention":
            temp = 1.0 + layer["mixer"]["q_temp"]["coef"] * torch.log((t + 1) // layer["mixer"]["q_temp"]["every"] + 1.0).double()
            q = _rms(q.view(T, _HEADS, -1), 1.0, eps) * temp[:, None, None]
            o = _attend(q, _rms(k.view(T, _KV, -1), 1.0, eps), v.view(T, _KV, -1), layer["mixer"]["scale"], bias)
        else:
            q, k, v = (_silu(z).view(T, _HEADS, -1) for z in (q, k, v))
            o = torch.empty_like(v)
            for h in range(_HEADS):
                o[:, h] = ((q[:, h] @ k[:, h].T) * torch.exp(log_decay[h] * dist.clamp_min(0) + unseen)) @ v[:, h]
            o = _rms(o.flatten(1), W(".mix.norm"), eps) * torch.sigmoid(u @ W(".mix.g").T)
        a, b = (torch.nn.functional.softplus(W(".mlp.act"))[m] for m in (0, 1))
        z = norm(x, p + ".norm2") @ W(".mlp.up").T
        act = torch.where(z > 0, a * z * z, (0.5 + b) * (torch.expm1(z.clamp(max=0.0)) - z)) + z / 2
        x = x + o @ W(".mix.o").T + act @ W(".mlp.down").T
    return norm(x, "final.norm")[torch.tensor(places, device=DEVICE)] @ w["head"].double().T


def _netinex(cfg, w, ids, places):
    eps, T = cfg["norm"]["eps"], len(ids)
    t = torch.arange(T, device=DEVICE)
    _, unseen = _far(T)
    bias = unseen.masked_fill(t[:, None] // _WINDOW != t[None] // _WINDOW, -math.inf)[None]
    dist = _far(T)[0].clamp_min(0)
    log_decay = torch.log(torch.tensor(_DECAY, dtype=torch.float64, device=DEVICE))

    def norm(x, name):
        return torch.tanh(x * w[name + ".alpha"].double()) * w[name].double() + w[name + ".b"].double()

    def turn(rot):  # (angles, factor)
        R, base, sc = rot["dims"], rot["base"], rot.get("scaling")
        f = [base ** (-2.0 * i / R) for i in range(R // 2)]
        if not sc:
            return _angles(t, f), 1.0
        lo, hi = (R * math.log(sc["original"] / (2.0 * math.pi * sc[n])) / (2.0 * math.log(base)) for n in ("fast", "slow"))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), R - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(R // 2)]
        f = [fi / sc["factor"] * r + fi * (1.0 - r) for fi, r in zip(f, ramp)]
        return _angles(t, f), 0.1 * math.log(sc["factor"]) + 1.0

    x = w["embed"][torch.tensor(ids, device=DEVICE)].double()
    for i, layer in enumerate(cfg["layers"]):
        def W(name):
            return w[f"l{i}{name}"].double()
        y = norm(x, f"l{i}.norm1")
        angles, factor = turn(layer["mixer"]["rot"])
        q, k = y @ W(".mix.q").T, y @ W(".mix.k").T
        if layer["type"] == "attention":
            v = k.view(T, _KV, -1)
            q = _rotate(_rms(q, W(".mix.q.norm"), eps).view(T, _HEADS, -1), angles, factor, True)
            k = _rotate(_rms(k, W(".mix.k.norm"), eps).view(T, _KV, -1), angles, factor, True)
            o = _attend(q, k, v, layer["mixer"]["scale"], bias)
        else:
            q, k = (_rotate(z.view(T, _HEADS, -1), angles, factor) for z in (q, k))
            v = (y @ W(".mix.v").T).view(T, _HEADS, -1)
            o = torch.empty_like(v)
            for h in range(_HEADS):
                o[:, h] = ((q[:, h] @ k[:, h].T) * torch.exp(log_decay[h] * dist + unseen)) @ v[:, h] * _DIM ** -0.5
            o = _rms(o, 1.0, eps).flatten(1) * _silu(y @ W(".mix.g").T)
        x = x + o @ W(".mix.o").T
        y = norm(x, f"l{i}.norm2")
        z = y @ W(".mlp.router").T + W(".mlp.router.b")
        best, chosen = torch.topk(z, layer["mlp"]["router"]["top"], -1)
        weight = torch.zeros_like(z).scatter_(1, chosen, torch.softmax(best, -1))
        for e in range(z.shape[1]):
            rows = weight[:, e].nonzero()[:, 0]
            a = _silu(y[rows] @ W(f".mlp.e{e}.gate").T) * (y[rows] @ W(f".mlp.e{e}.up").T)
            x = x.index_add(0, rows, weight[rows, e][:, None] * (a @ W(f".mlp.e{e}.down").T))
    logits = norm(x, "final.norm")[torch.tensor(places, device=DEVICE)] @ w["embed"].double().T
    return cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])


def _logits(cfg, w, seqs, wanted):
    if "hidden_size" not in cfg:
        of = _kugilix if cfg["architecture"] == "Kugilix" else _netinex
        return torch.cat([of(cfg, w, s, p) for s, p in zip(seqs, wanted)])
    out, lo = [], 0
    while lo < len(seqs):  # as many sequences at a time as their 64-bit activations leave room for
        hi, rows = lo, 0
        while hi < len(seqs) and (hi == lo or rows + len(seqs[hi]) <= 32768):
            rows += len(seqs[hi])
            hi += 1
        out.append(_qwen(cfg, w, seqs[lo:hi], wanted[lo:hi]))
        lo = hi
    return torch.cat(out)


def exact(case, seed):
    cfg, lengths = MODELS[case["model"]], _lengths(case)
    w = random_tensors(cfg, _weights_seed(seed), "bfloat16", device=DEVICE)
    prompts = [_ids(case, seed, 100000 + k, n) for k, n in enumerate(lengths)]
    if case["kind"] == "generate":
        tokens, probabilities = [[] for _ in prompts], [[] for _ in prompts]
        for _ in range(case["new"]):
            seqs = [p + t for p, t in zip(prompts, tokens)]
            best, at = torch.softmax(_logits(cfg, w, seqs, [[len(s) - 1] for s in seqs]), -1).max(-1)
            for k, (p, t) in enumerate(zip(best.tolist(), at.tolist())):
                tokens[k].append(t)
                probabilities[k].append(p)
        return {"tokens": torch.tensor(tokens), "probabilities": torch.tensor(probabilities, dtype=torch.float64)}
    seqs, wanted = [], []
    for rid, n in enumerate(_contexts(case)):
        fed = [_ids(case, seed, 300000 + i, case["decode"])[rid] for i in range(WARM + 1)]
        seqs.append(_ids(case, seed, rid, n) + fed)
        wanted.append([n + WARM])
    for p in prompts:
        seqs.append(p)
        wanted.append(list(range(max(0, len(p) - case["want"]), len(p))))
    return _logits(cfg, w, seqs, wanted)
