"""What a program that uses this library has it do, as cases that can be timed and checked.

A case is a step of the engine as its two callers issue it: ``decode`` is a stretch of single-token steps of a batch of
sequences (the generation loop), ``prompt`` is one step that brings unequal prompts, or a further portion behind tokens
that are already evaluated (a chat session's next turn), and ``sample`` is the choice of a batch's next tokens from its
logits.  The models are the named configurations of ``gophonic_b200/config/presets`` with random weights: the dense decoder
in two sizes, a design whose layers are matrix-state recurrences and windowed attention with a sink, and a design of
latent and differential attention with mixtures of experts.  Larger configurations keep fewer layers, of full size each.

``exact`` runs the same models in 64 bits, in plain torch: whole sequences, no cache.
"""
import math
import random

import torch

from gophonic_b200 import registry
from gophonic_b200.config.presets import preset
from gophonic_b200.engine.model import Model, dtype_mode, make_runtime
from gophonic_b200.engine.step import Engine
from gophonic_b200.sampling import DeviceSampler, Options
from gophonic_b200.weights import declare_model

DEVICE = "cuda:0"
VOCAB = 151936
LAYERS = {"1.7b": 28, "8b": 12, "pugalix-2k": 8, "kimilix-2k": 8}
LAYERS_F32 = 8          # of the configurations that also run in 32 bits
ROUTED = 64             # channels of the routed design's residual that tell its routers what a token is


def listed():
    return [
        # the next tokens of a full batch, each sequence with options of its own: the end of every generated step
        {"name": "sample-16", "work": "sample", "seqs": 16},
        # one user waiting for one token: latency and launches
        {"name": "token-1", "work": "decode", "model": "1.7b", "dtype": "bfloat16", "seqs": 1, "longest": 700, "steps": 1},
        # the benchmark's batch: eight sequences at contexts up to 4096, bound by weights and cache
        {"name": "tokens-8", "work": "decode", "model": "8b", "dtype": "bfloat16", "seqs": 8, "longest": 4096, "steps": 2},
        # a busy server of a small model: an odd number of sequences of very different lengths
        {"name": "tokens-50", "work": "decode", "model": "1.7b", "dtype": "bfloat16", "seqs": 50, "longest": 1900, "steps": 4},
        # the 32-bit path, as a reference run or a check of the other one takes it
        {"name": "tokens-3-f32", "work": "decode", "model": "1.7b", "dtype": "float32", "seqs": 3, "longest": 333, "steps": 2},
        # a chat's next turn: a short message behind an evaluated context, scored at every place
        {"name": "turn-90", "work": "prompt", "model": "8b", "dtype": "bfloat16", "seqs": 1, "context": 1000, "longest": 90, "every": True},
        # prompts that start together: unequal, packed into one step; the most work a step of this list does
        {"name": "prompts-8", "work": "prompt", "model": "8b", "dtype": "bfloat16", "seqs": 8, "context": 0, "longest": 2048, "every": False},
        {"name": "prompts-2-f32", "work": "prompt", "model": "1.7b", "dtype": "float32", "seqs": 2, "context": 0, "longest": 201, "every": False},
        # matrix-state layers and windowed attention: a long prompt of one user, and a batch that decodes
        {"name": "states-prompt", "work": "prompt", "model": "pugalix-2k", "dtype": "bfloat16", "seqs": 1, "context": 0, "longest": 1611, "every": False},
        {"name": "states-tokens-16", "work": "decode", "model": "pugalix-2k", "dtype": "bfloat16", "seqs": 16, "longest": 1500, "steps": 8},
        # latent attention and mixtures of experts: two prompts, and a batch that decodes
        {"name": "latents-prompts-2", "work": "prompt", "model": "kimilix-2k", "dtype": "bfloat16", "seqs": 2, "context": 0, "longest": 2048, "every": False},
        {"name": "latents-tokens-24", "work": "decode", "model": "kimilix-2k", "dtype": "bfloat16", "seqs": 24, "longest": 1500, "steps": 4},
    ]


def _log_int(rng, low, high):
    return min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        work = rng.choice(["sample"] + 4 * ["decode"] + 5 * ["prompt"])
        if work == "sample":
            case = {"work": work, "seqs": _log_int(rng, 1, 64)}
        else:
            model = rng.choice(sorted(LAYERS))
            dtype = "float32" if model == "1.7b" and rng.random() < 0.4 else "bfloat16"
            case = {"work": work, "model": model, "dtype": dtype}
            if work == "decode":
                case.update(seqs=_log_int(rng, 1, 8 if dtype == "float32" else 64), longest=_log_int(rng, 64, 512 if dtype == "float32" else 4096),
                            steps=rng.randint(1, 8))
                if case["seqs"] * case["longest"] > 65536:
                    continue
            else:
                case.update(seqs=_log_int(rng, 1, 8), context=rng.choice([0, 0, _log_int(rng, 64, 2048)]),
                            longest=_log_int(rng, 8, 256 if dtype == "float32" else 2048))
                case["every"] = case["longest"] * case["seqs"] <= 256 and rng.random() < 0.3
        if _cost(case) <= largest:
            return case


# ---- the inputs ---------------------------------------------------------------------------------------------
def _lengths(case):
    """The sequences' lengths (tokens evaluated before a decode step, or brought by a prompt): the longest as stated, the
    others spread over a factor of 16 below it."""
    r = random.Random(case["seqs"] * 1000003 + case["longest"])
    low = max(1, case["longest"] // 16)
    return [case["longest"]] + [_log_int(r, low, case["longest"]) for _ in range(case["seqs"] - 1)]


def _config(case):
    raw = preset(case["model"])
    config = registry.config_class(registry.architecture_of(raw)).from_dict(raw)
    return config.with_layers(LAYERS_F32 if case["dtype"] == "float32" else LAYERS[case["model"]])


def _declared(case):
    """The tensors of the case's checkpoint: name -> shape; a head that is tied to the embedding has none of its own."""
    config = _config(case)
    tied = case["model"] == "1.7b" or case["model"].startswith("kimilix")
    spec = config.model_spec()
    return {d.name: tuple(d.shape) for d in declare_model(spec) if not (tied and d.name == spec.head.name)}


def _law(model, name, shape):
    """(mean, deviation) of a tensor's values: matrices keep their input's size, norms and scales stand near one (a norm
    that multiplies by 1 + w: near zero), decays and forget gates near one so that a state lives for a while."""
    last = name.rsplit(".", 1)[-1]
    if "norm" in name:
        less_one = model.startswith("kimilix") and last in ("norm1", "norm2") or name == "final.norm" and model.startswith("kimilix")
        return (0.0 if less_one else 1.0), 0.2
    if last in ("ls1", "ls2"):
        return 1.0, 0.2
    if last in ("lq1", "lk1", "lq2", "lk2"):
        return 0.0, 0.2
    if name.endswith(("a2.b", "f.b")):
        return 2.0, 1.0
    if last == "b":
        return 0.0, 0.2
    if last == "router":
        return 0.0, 0.1 / math.sqrt(shape[-1])
    if name == "embed" and model.startswith("kimilix"):
        return 0.0, 1.0
    return 0.0, 1.0 / math.sqrt(shape[-1])


def _weights(case, seed):
    """The checkpoint's tensors on the GPU, as bfloat16 stores them (a 32-bit run widens them)."""
    gen = torch.Generator(DEVICE).manual_seed(seed)
    out = {}
    for name, shape in _declared(case).items():
        mean, dev = _law(case["model"], name, shape)
        t = torch.randn(shape, generator=gen, device=DEVICE).mul_(dev).add_(mean).to(torch.bfloat16)
        out[name] = t.float() if "norm" in name or case["dtype"] == "float32" else t
    if case["model"].startswith("kimilix"):
        _decide_routes(out, gen)
    return out


def _decide_routes(w, gen):
    """A trained router has a clear opinion of a token; a random one all but ties its experts, and then rounding chooses.
    Here the first channels of the embedding say which two experts a token prefers, every router reads them, and the
    final norm keeps them out of the logits."""
    experts = next(t.shape[0] for n, t in w.items() if n.endswith(".router"))
    codes = torch.ones((1, 1), device=DEVICE)
    while codes.shape[0] < ROUTED:
        codes = torch.cat([torch.cat([codes, codes], 1), torch.cat([codes, -codes], 1)])
    codes = codes[1:experts + 1]
    tokens = w["embed"].shape[0]
    first = torch.randint(experts, (tokens,), generator=gen, device=DEVICE)
    second = (first + 1 + torch.randint(experts - 1, (tokens,), generator=gen, device=DEVICE)) % experts
    w["embed"][:, :ROUTED] = (4.0 * codes[first] + 2.4 * codes[second]).to(w["embed"].dtype)
    for n, t in w.items():
        if n.endswith(".router"):
            t[:, :ROUTED] = (0.02 * codes).to(t.dtype)
    w["final.norm"][:ROUTED] = -1.0


def _tokens(case, seed):
    """Every sequence's token ids: what a prompt's context or a decode step's prompt holds, then what the pass brings."""
    r = random.Random(seed)
    if case["work"] == "decode":
        parts = [(n, case["steps"]) for n in _lengths(case)]
    else:
        parts = [(case["context"], n) for n in _lengths(case)]
    return [([r.randrange(VOCAB) for _ in range(a)], [r.randrange(VOCAB) for _ in range(b)]) for a, b in parts]


def prepare(case, seed):
    if case["work"] == "sample":
        return _prepare_sample(case, seed)
    tokens = _tokens(case, seed)
    config = _config(case)
    model = Model(config.model_spec(), _weights(case, seed), make_runtime(dtype_mode(case["dtype"]), DEVICE), config)
    room = sum((len(a) + len(b) + 63) // 64 * 64 for a, b in tokens)
    engine = Engine(model, max_tokens=room, max_slots=len(tokens))
    state = {"work": case["work"], "engine": engine, "marks": None}
    if tokens[0][0]:
        # sequences that are already evaluated, and the mark that every pass begins from
        slots = [engine.new_sequence() for _ in tokens]
        for slot, (known, _) in zip(slots, tokens):
            engine.step([(slot, known)])
        state["slots"] = slots
        state["marks"] = [engine.checkpoint(s) for s in slots]
    if case["work"] == "decode":
        n = len(tokens)
        state["source"] = torch.tensor([b[t] for t in range(case["steps"]) for _, b in tokens], dtype=torch.int32, device=DEVICE)
        state["places"] = [range(t * n, (t + 1) * n) for t in range(case["steps"])]
        run(state)      # a server has its steps captured
    else:
        state["prompts"] = [b for _, b in tokens]
        state["want"] = [list(range(len(b))) for _, b in tokens] if case["every"] else None
    return state


def _prepare_sample(case, seed):
    gen = torch.Generator(DEVICE).manual_seed(seed)
    sampler = DeviceSampler(VOCAB, case["seqs"], DEVICE)
    kinds = [Options(Temperature=0.7, TopK=40, TopP=0.9), Options(Temperature=1.0, TopP=0.95), Options(Temperature=0.6, TopK=20), Options()]
    for row in range(case["seqs"]):
        sampler.start(row, kinds[row % len(kinds)], seed + row)
    logits = torch.randn((case["seqs"], VOCAB), generator=gen, device=DEVICE).mul_(3.0)
    return {"work": "sample", "sampler": sampler, "logits": logits, "rows": list(range(case["seqs"]))}


# ---- one pass -----------------------------------------------------------------------------------------------
def run(state):
    if state["work"] == "sample":
        return state["sampler"].select_device(state["logits"], state["rows"])
    engine = state["engine"]
    if state["work"] == "decode":
        # the generation loop's step: tokens come from where the last step's were left on the device
        out = [engine.step_from(state["slots"], state["source"], places) for places in state["places"]]
    elif state["marks"] is None:
        slots = [engine.new_sequence() for _ in state["prompts"]]
        out = engine.step(list(zip(slots, state["prompts"])), state["want"])
        for slot in slots:
            engine.end_sequence(slot)
        return out
    else:
        out = engine.step(list(zip(state["slots"], state["prompts"])), state["want"])
    for slot, mark in zip(state["slots"], state["marks"]):
        engine.restore(slot, mark)
    return out


# ---- what a pass cannot do without --------------------------------------------------------------------------
def _pairs(new, known, limit=0, block=0, kept=0):
    """(row, key) pairs that ``new`` rows behind ``known`` tokens see."""
    total = 0
    for i in range(known, known + new):
        seen = i + 1
        if block:
            seen = i % block + 1
        elif limit:
            seen = min(seen, limit + min(kept, max(0, seen - limit)))
        total += seen
    return total


def work(case):
    if case["work"] == "sample":
        return {"bytes": 4 * case["seqs"] * (VOCAB + 1), "flops": 0}
    decode = case["work"] == "decode"
    elem = 4 if case["dtype"] == "float32" else 2
    passes = case["steps"] if decode else 1
    if decode:
        parts = [(1, n) for n in _lengths(case)]
    else:
        parts = [(n, case["context"]) for n in _lengths(case)]
    rows = sum(n for n, _ in parts)
    wanted = rows if decode or case.get("every") else len(parts)
    config = _config(case).to_dict()
    nbytes = 4.0 * wanted * VOCAB
    flops = 0.0
    experts = top = 0
    for layer in config.get("layers", []):
        if layer.get("mlp") and layer["mlp"]["kind"] == "moe":
            experts, top = layer["mlp"]["router"]["experts"], layer["mlp"]["router"]["top"]
    for name, shape in _declared(case).items():
        n = math.prod(shape)
        if name in ("embed", "model.embed_tokens.weight"):
            nbytes += elem * rows * shape[1]
            if case["model"] != "1.7b" and not case["model"].startswith("kimilix"):
                continue
            name = "head"       # the tied head reads the table
        if len(shape) < 2:
            nbytes += elem * n
            continue
        head = name in ("head", "lm_head.weight")
        expert = ".mlp.e" in name
        nbytes += elem * n * (min(1.0, rows * top / experts) if expert else 1.0)
        flops += 2.0 * n * (wanted if head else rows * top / experts if expert else rows)
    known = sum(k for _, k in parts)
    if "layers" not in config:
        H, G, d, L = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"], config["num_hidden_layers"]
        nbytes += L * elem * 2 * G * d * (known + rows)
        flops += L * 4.0 * H * d * sum(_pairs(n, k) for n, k in parts)
    for layer in config.get("layers", []):
        m, kind = layer["mixer"], layer["type"]
        H, d, dv = m["heads"], m["dim"], m.get("vdim", m["dim"])
        size, kept = m.get("mask", {}).get("size", 0), m.get("mask", {}).get("keep_first", 0)
        if kind in ("gla", "mlstm"):
            nbytes += 4 * 2 * len(parts) * H * d * dv
            flops += 4.0 * rows * H * d * dv
            continue
        if kind == "latent_attention":
            seen = sum(min(k, size) + n for n, k in parts)
            nbytes += elem * (m["kv_rank"] + m["rot_dim"]) * seen
            flops += 2.0 * H * (d + m["rot_dim"] + dv) * sum(_pairs(n, k, limit=size) for n, k in parts)
        elif "diff" in m:
            seen = sum(min(k, size) + n for n, k in parts)
            nbytes += elem * m["kv_heads"] * (2 * d + dv) * seen
            flops += 2.0 * H * 2 * (d + dv) * sum(_pairs(n, k, block=size) for n, k in parts)
        else:
            seen = sum(min(k, size + kept) + n for n, k in parts)
            nbytes += elem * m["kv_heads"] * (d + dv) * seen
            flops += 2.0 * H * (d + dv) * sum(_pairs(n, k, limit=size, kept=kept) for n, k in parts)
    return {"bytes": passes * nbytes, "flops": passes * flops}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def tolerance(case):
    if case["work"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5}     # against 64 bits: 4.5e-6
    return {"rel": 0.03}         # against 64 bits: 0.005 to 0.011, each side with roundings of its own


# ---- the same models in 64 bits -----------------------------------------------------------------------------
def exact(case, seed):
    if case["work"] == "sample":
        return None
    tokens = _tokens(case, seed)
    if case["work"] == "decode":
        want = [range(len(a), len(a) + len(b)) for a, b in tokens]
    else:
        want = [range(len(a) if case["every"] else len(a) + len(b) - 1, len(a) + len(b)) for a, b in tokens]
    lengths = [len(a) + len(b) for a, b in tokens]
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    at = {"parts": list(zip(starts, lengths)), "pos": torch.cat([torch.arange(n, device=DEVICE) for n in lengths])}
    ids = torch.tensor([t for a, b in tokens for t in a + b], device=DEVICE)
    rows = torch.tensor([s + i for s, r in zip(starts, want) for i in r], device=DEVICE)
    config = _config(case).to_dict()
    plain = _qwen3 if "layers" not in config else _pugalix if case["model"].startswith("pugalix") else _kimilix
    logits = plain(config, _weights(case, seed), ids, at, rows)
    if case["work"] == "prompt":
        return logits
    logits = logits.view(case["seqs"], case["steps"], VOCAB)
    return [logits[:, t].contiguous() for t in range(case["steps"])]


def _mul(x, w):
    return x @ w.double().T


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, pos, freqs, pairs):
    """x [rows, heads, d]: the first 2 len(freqs) channels turn, channel i with i + len(freqs) or neighbours together."""
    n = len(freqs)
    ang = pos.double()[:, None] * torch.tensor(freqs, dtype=torch.float64, device=DEVICE)[None]
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    out = x.clone()
    u, v = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if pairs else (x[..., :n], x[..., n:2 * n])
    a, b = u * c - v * s, v * c + u * s
    if pairs:
        out[..., 0:2 * n:2], out[..., 1:2 * n:2] = a, b
    else:
        out[..., :n], out[..., n:2 * n] = a, b
    return out


def _frequencies(dims, base, scaling=None):
    out = []
    for i in range(dims // 2):
        f = base ** (-2.0 * i / dims)
        if scaling:
            wave = 2.0 * math.pi / f
            low, high, orig = scaling["low"], scaling["high"], scaling["original"]
            if wave > orig / low:
                f /= scaling["factor"]
            elif wave >= orig / high:
                s = (orig / wave - low) / (high - low)
                f = (1.0 - s) * f / scaling["factor"] + s * f
        out.append(f)
    return out


def _attend(q, k, v, scale, at, window=0, block=0, kept=0, sink=False):
    """Softmax attention inside every sequence: q [rows, H, d], k [rows, G, d], v [rows, Gv, dv] -> [rows, H, dv]."""
    H, G, Gv = q.shape[1], k.shape[1], v.shape[1]
    out = torch.empty((q.shape[0], H, v.shape[2]), dtype=torch.float64, device=DEVICE)
    for a, n in at["parts"]:
        i = torch.arange(n, device=DEVICE)
        see = i[None] <= i[:, None]
        if window:
            see &= (i[:, None] - i[None] < window) | (i[None] < kept)
        if block:
            see &= i[:, None] // block == i[None] // block
        few = max(1, (1 << 26) // (n * n))
        for h in range(0, H, few):
            hs = torch.arange(h, min(H, h + few), device=DEVICE)
            s = torch.einsum("ihd,jhd->hij", q[a:a + n, hs], k[a:a + n, hs // (H // G)]) * scale
            s.masked_fill_(~see, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink:
                top.clamp_(min=0.0)
            s.sub_(top).exp_()
            total = s.sum(-1, keepdim=True)
            if sink:
                total += torch.exp(-top)
            s.div_(total)
            out[a:a + n, hs] = torch.einsum("hij,jhd->ihd", s, v[a:a + n, hs // (H // Gv)])
    return out


def _gated(x, w, gate, up, down):
    g = _mul(x, w[gate])
    return _mul(g * torch.sigmoid(g) * _mul(x, w[up]), w[down])


def _qwen3(c, w, ids, at, rows):
    eps, H, G, d = c["rms_norm_eps"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    freqs = _frequencies(d, c["rope_theta"])
    x = w["model.embed_tokens.weight"][ids].double()
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        h = _unit(x, eps) * w[p + "input_layernorm.weight"]
        q = _unit(_mul(h, w[a + "q_proj.weight"]).view(-1, H, d), eps) * w[a + "q_norm.weight"]
        k = _unit(_mul(h, w[a + "k_proj.weight"]).view(-1, G, d), eps) * w[a + "k_norm.weight"]
        v = _mul(h, w[a + "v_proj.weight"]).view(-1, G, d)
        q, k = _rotate(q, at["pos"], freqs, False), _rotate(k, at["pos"], freqs, False)
        x = x + _mul(_attend(q, k, v, d ** -0.5, at).reshape(-1, H * d), w[a + "o_proj.weight"])
        h = _unit(x, eps) * w[p + "post_attention_layernorm.weight"]
        x = x + _gated(h, w, *(f"{p}mlp.{n}_proj.weight" for n in ("gate", "up", "down")))
    x = _unit(x[rows], eps) * w["model.norm.weight"]
    return _mul(x, w["lm_head.weight"] if "lm_head.weight" in w else w["model.embed_tokens.weight"])


def _padded(x, at):
    """Packed rows as [sequences, longest, ...]; a recurrence looks back, so what is behind a sequence's end changes nothing."""
    longest = max(n for _, n in at["parts"])
    out = torch.zeros((len(at["parts"]), longest) + x.shape[1:], dtype=x.dtype, device=DEVICE)
    for i, (a, n) in enumerate(at["parts"]):
        out[i, :n] = x[a:a + n]
    return out


def _packed(x, at):
    return torch.cat([x[i, :n] for i, (_, n) in enumerate(at["parts"])])


def _gla(h, w, p, m, eps, at):
    H, d, dv = m["heads"], m["dim"], m["vdim"]
    q = _mul(h, w[p + "q"]).view(-1, H, d) / math.sqrt(d)
    k, v = _mul(h, w[p + "k"]).view(-1, H, d), _mul(h, w[p + "v"]).view(-1, H, dv)
    z = _mul(_mul(h, w[p + "a1"]), w[p + "a2"]) + w[p + "a2.b"].double()
    decay = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).view(-1, H, d)
    q, k, v, decay = (_padded(t, at) for t in (q, k, v, decay))
    S = torch.zeros((q.shape[0], H, d, dv), dtype=torch.float64, device=DEVICE)
    o = torch.empty_like(v)
    for t in range(q.shape[1]):
        S.mul_(decay[:, t, :, :, None]).addcmul_(k[:, t, :, :, None], v[:, t, :, None, :])
        o[:, t] = torch.matmul(q[:, t, :, None], S)[:, :, 0]
    o = (_unit(_packed(o, at), eps) * w[p + "norm"].double()).reshape(-1, H * dv)
    g = _mul(h, w[p + "g"])
    return _mul(o * g * torch.sigmoid(g), w[p + "o"])


def _mlstm(h, w, p, m, eps, at):
    H, d, dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q = _mul(h, w[p + "q"]).view(-1, H, d) / math.sqrt(d)
    k, v = _mul(h, w[p + "k"]).view(-1, H, d), _mul(h, w[p + "v"]).view(-1, H, dv)
    gi = cap * torch.tanh((_mul(h, w[p + "i"]) + w[p + "i.b"].double()) / cap)
    gf = torch.nn.functional.logsigmoid(cap * torch.tanh((_mul(h, w[p + "f"]) + w[p + "f.b"].double()) / cap))
    v = torch.cat([v, torch.ones_like(v[..., :1])], -1)      # the normaliser is one more column of the state
    q, k, v, gi, gf = (_padded(t, at) for t in (q, k, v, gi, gf))
    S = torch.zeros((q.shape[0], H, d, dv + 1), dtype=torch.float64, device=DEVICE)
    top = torch.zeros((q.shape[0], H), dtype=torch.float64, device=DEVICE)
    o = torch.empty_like(v)
    tops = torch.empty_like(gi)
    for t in range(q.shape[1]):
        new = torch.maximum(gf[:, t] + top, gi[:, t])
        keep, take = torch.exp(gf[:, t] + top - new), torch.exp(gi[:, t] - new)
        S.mul_(keep[..., None, None]).addcmul_((take[..., None] * k[:, t])[..., None], v[:, t, :, None, :])
        o[:, t] = torch.matmul(q[:, t, :, None], S)[:, :, 0]
        tops[:, t] = top = new
    o, tops = _packed(o, at), _packed(tops, at)
    o = o[..., :dv] / (torch.maximum(o[..., dv].abs(), torch.exp(-tops)) + 1e-6)[..., None]
    o = _unit(o, eps).reshape(-1, H * dv) * w[p + "norm"].double()
    return _mul(o * torch.sigmoid(_mul(h, w[p + "g"])), w[p + "o"])


def _pugalix(c, w, ids, at, rows):
    eps = c["norm"]["eps"]
    x = w["embed"][ids].double() * c["embedding"]["scale"]
    held = {}
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        h = _unit(x, eps) * w[f"l{i}.norm1"].double()
        if layer["type"] == "attention":
            H, d, dv = m["heads"], m["dim"], m["vdim"]
            freqs = _frequencies(m["rot"]["dims"], m["rot"]["base"])
            if m.get("kv_from") is None:
                k = (_mul(h, w[p + "k"]) + w[p + "k.b"].double()).view(-1, m["kv_heads"], d)
                v = (_mul(h, w[p + "v"]) + w[p + "v.b"].double()).view(-1, m["kv_heads"], dv)
                held[i] = _rotate(k, at["pos"], freqs, True), v
            k, v = held[m["kv_from"] if m.get("kv_from") is not None else i]
            q = _rotate((_mul(h, w[p + "q"]) + w[p + "q.b"].double()).view(-1, H, d), at["pos"], freqs, True)
            y = _attend(q, k, v, m["scale"], at, window=m["mask"]["size"], kept=m["mask"]["keep_first"], sink=True)
            x = x + _mul(y.reshape(-1, H * dv) * torch.sigmoid(_mul(h, w[p + "g"])), w[p + "o"])
        else:
            x = x + (_gla if layer["type"] == "gla" else _mlstm)(h, w, p, m, eps, at)
        if layer.get("mlp") is not None:
            x = x + _gated(_unit(x, eps) * w[f"l{i}.norm2"].double(), w, *(f"l{i}.mlp.{n}" for n in ("gate", "up", "down")))
    return _mul(_unit(x[rows], eps) * w["final.norm"].double(), w["head"])


def _differential(h, w, p, m, eps, at):
    H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    freqs = _frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
    q = _unit(_mul(h, w[p + "q"]).view(-1, 2 * H, d), eps) * w[p + "q.norm"].double()
    k = _unit(_mul(h, w[p + "k"]).view(-1, 2 * G, d), eps) * w[p + "k.norm"].double()
    v = _mul(h, w[p + "v"]).view(-1, G, dv)
    q, k = _rotate(q, at["pos"], freqs, False), _rotate(k, at["pos"], freqs, False)
    dot = lambda a, b: float((w[p + a].double() * w[p + b].double()).sum())  # noqa: E731
    lam = math.exp(dot("lq1", "lk1")) - math.exp(dot("lq2", "lk2")) + m["diff"]
    a1, a2 = (_attend(q[:, i::2], k[:, i::2], v, m["scale"], at, block=m["mask"]["size"]) for i in (0, 1))
    return _mul((_unit(a1 - lam * a2, eps) * (1.0 - m["diff"])).reshape(-1, H * dv), w[p + "o"])


def _latent(h, w, p, m, eps, at):
    H, d, dr, R, dv = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], m["vdim"]
    freqs = _frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
    q = _mul(_unit(_mul(h, w[p + "dq"]), eps) * w[p + "dq.norm"].double(), w[p + "uq"]).view(-1, H, d + dr)
    made = _mul(h, w[p + "dkv"])
    c = _unit(made[:, :R], eps) * w[p + "dkv.norm"].double()
    q = torch.cat([q[..., :d], _rotate(q[..., d:], at["pos"], freqs, True)], -1)
    turned = _rotate(made[:, None, R:], at["pos"], freqs, True)
    k = torch.cat([_mul(c, w[p + "uk"]).view(-1, H, d), turned.expand(-1, H, -1)], -1)
    y = _attend(q, k, _mul(c, w[p + "uv"]).view(-1, H, dv), m["scale"], at, window=m["mask"]["size"])
    return _mul(y.reshape(-1, H * dv), w[p + "o"])


def _clamped(x, w, p, limit):
    g = _mul(x, w[p + "gate"]).clamp(max=limit)
    return _mul(g * torch.sigmoid(1.702 * g) * (_mul(x, w[p + "up"]).clamp(-limit, limit) + 1.0), w[p + "down"])


def _mixture(x, w, p, mlp):
    z = _mul(x, w[p + "router"]) + w[p + "router.b"].double()
    z, index = z.topk(mlp["router"]["top"])
    weight = z.softmax(-1)
    out = torch.sigmoid(_mul(x, w[p + "shared.sg"])) * _clamped(x, w, p + "shared.", mlp["shared"]["limit"])
    for e in range(mlp["router"]["experts"]):
        r, j = (index == e).nonzero(as_tuple=True)
        out.index_add_(0, r, weight[r, j][:, None] * _clamped(x[r], w, f"{p}e{e}.", mlp["expert"]["limit"]))
    return out


def _kimilix(c, w, ids, at, rows):
    eps, mult = c["norm"]["eps"], c["residual_mult"]
    x = w["embed"][ids].double() * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        p = f"l{i}."
        mix = _differential if layer["type"] == "attention" else _latent
        y = mix(x, w, p + "mix.", layer["mixer"], eps, at)
        x = x + mult * w[p + "ls1"].double() * _unit(y, eps) * (1.0 + w[p + "norm1"].double())
        if layer["mlp"]["kind"] == "dense":
            y = _mul(_mul(x, w[p + "mlp.up"]).clamp(min=0.0) ** 2, w[p + "mlp.down"])
        else:
            y = _mixture(x, w, p + "mlp.", layer["mlp"])
        x = x + mult * w[p + "ls2"].double() * _unit(y, eps) * (1.0 + w[p + "norm2"].double())
    return _mul(_unit(x[rows], eps) * (1.0 + w["final.norm"].double()), w["embed"])
