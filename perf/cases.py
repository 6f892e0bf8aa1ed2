"""The work this library is measured on: steps and generations of models with random weights.

Three kinds of case, all through the engine's public calls:

prompt    every pass gives fresh slots whole prompts in one step, reads the logits of their last tokens and gives the
          slots back: time to the first token, or the throughput of a batch of prompts.
decode    the sequences are in the cache; every pass takes one more token for each of them and gives the logits, as a
          generation or a replayed trace does.  The sequences grow from pass to pass; once the cache's room is used up
          the next pass starts them over.
generate  one call of ``Engine.generate``: prompts, then token after token sampled on the device.

A case is a dictionary of plain values: the shape (a name of ``ziglm_b200.config.shapes``), the layers kept of it (0: all),
the storage type, the number of sequences and the range ``lo``..``hi`` of their lengths, spread evenly over it.  Weights
are normal with the library's own standard deviation (0.02), embeddings with 1 (the residual stream of a trained model is
as large), norms near one; token ids are uniform.  The three designs whose layers choose experts are left out: the choice
is not continuous, so that two correct bfloat16 implementations differ by whole experts and their logits cannot be held
to a tolerance.
"""
from __future__ import annotations

import gc
import math

import torch

from ziglm_b200 import Engine, EngineOptions, GenerationOptions, SamplerParams, config_from_dict
from ziglm_b200.config.shapes import shape
from ziglm_b200.engine.model import Model

DEVICE = "cuda:0"
PAGE = 64
STEP_TOKENS = 16384          # most prompt tokens brought into the cache by one step of a preparation


# ------------------------------------------------------------------------------------------------ the cases
def _case(kind, model, layers, dtype, seqs, lo, hi, new=0, sampler="none"):
    return {"kind": kind, "model": model, "layers": layers, "dtype": dtype, "seqs": seqs, "lo": lo, "hi": hi, "new": new,
            "sampler": sampler}


def listed():
    return [
        # one short chat at the small model: the fewest bytes a step can read, so launches and gaps count most
        dict(_case("decode", "llama-1b", 0, "bfloat16", 1, 130, 130), name="step-1b-one-sequence"),
        # a serving batch of short sequences of unequal length
        dict(_case("decode", "llama-1b", 0, "bfloat16", 64, 18, 1008), name="step-1b-64-ragged"),
        # the batch the library's own benchmark quotes, on a quarter of the layers
        dict(_case("decode", "llama-8b", 8, "bfloat16", 8, 4096, 4096), name="step-8b-8x4096"),
        # as many key/value heads as query heads: the cache is four times as heavy for a context
        dict(_case("decode", "llama-13b", 8, "bfloat16", 16, 700, 2048), name="step-13b-16-ragged"),
        # the first token of a short question
        dict(_case("prompt", "llama-1b", 0, "bfloat16", 1, 77, 77), name="prompt-1b-77"),
        # the prompt the library's own benchmark quotes
        dict(_case("prompt", "llama-8b", 8, "bfloat16", 1, 2048, 2048), name="prompt-8b-2048"),
        # a long document, not a whole number of pages or tiles
        dict(_case("prompt", "llama-8b", 4, "bfloat16", 1, 16001, 16001), name="prompt-8b-16001"),
        # a batch of requests from text ids in to text ids out: prompts, then sampled tokens, host loop included
        dict(_case("generate", "llama-1b", 0, "bfloat16", 64, 18, 1008, 32, "sample"), name="generate-1b-64-ragged"),
        # the true 32-bit path, which checks and replays of traces run on
        dict(_case("prompt", "llama-8b", 4, "float32", 3, 100, 300), name="prompt-8b-float32"),
        dict(_case("decode", "llama-8b", 4, "float32", 8, 1024, 1024), name="step-8b-float32-8x1024"),
        # two of the further designs: windows, sinks, a decayed linear state and a latent cache in one step ...
        dict(_case("decode", "vilazen-1b", 4, "bfloat16", 8, 2048, 2048), name="step-vilazen-8x2048"),
        # ... and residual streams and delta rules over a prompt
        dict(_case("prompt", "mopilorn-1b", 4, "bfloat16", 1, 2048, 2048), name="prompt-mopilorn-2048"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _floor_seconds(case):
    """A rough time of a pass, to keep drawn cases within the listed ones: at 6.5 TB/s and 1.6 PFLOP/s (75 TFLOP/s
    for 32-bit products)."""
    w = work(case)
    return w["bytes"] / 6.5e12 + w["flops"] / (1.6e15 if case["dtype"] == "bfloat16" else 7.5e13)


def draw(rng):
    most = max(_floor_seconds(c) for c in listed())
    while True:
        kind = rng.choice(["prompt", "decode", "decode", "prompt", "generate"])
        model, layers = rng.choice([("llama-1b", 16), ("llama-8b", 8), ("llama-13b", 8), ("llama-8b", 4), ("vilazen-1b", 4),
                                    ("mopilorn-1b", 4)])
        dtype = "float32" if kind != "generate" and model.startswith("llama") and rng.random() < 0.2 else "bfloat16"
        if dtype == "float32":
            layers = 4
        hi = _log_int(rng, 16, {"prompt": 16384, "decode": 8192, "generate": 1024}[kind])
        if model == "llama-13b":
            hi = min(hi, 3000)
        if dtype == "float32":
            hi = min(hi, 2048)
        if kind == "generate" and not model.startswith("llama"):
            model, layers = "llama-1b", 16
        if kind == "decode" and not model.startswith("llama"):
            hi = min(hi, 4096)
        lo = max(2, int(hi * rng.uniform(0.05, 1.0)))
        seqs = _log_int(rng, 1, 64) if kind != "prompt" else _log_int(rng, 1, 16)
        case = _case(kind, model, layers, dtype, seqs, lo, hi)
        if kind == "generate":
            case.update(new=rng.randint(8, 48), sampler=rng.choice(["greedy", "sample", "presence"]))
        if sum(lengths(case)) <= 65536 and _floor_seconds(case) <= most:
            return case


def lengths(case):
    """Tokens of every sequence, spread evenly over lo..hi in an order without a trend."""
    span = case["hi"] - case["lo"]
    return [case["lo"] + int(round(span * ((0.5 + i * 0.6180339887) % 1.0))) for i in range(case["seqs"])]


def _config(case):
    d = shape(case["model"])
    if case["layers"]:
        if "layers" in d:
            d["layers"] = d["layers"][:case["layers"]]
        else:
            d["num_hidden_layers"] = case["layers"]
    return d


# ------------------------------------------------------------------------------------------------ weights and ids
def _llama_sizes(d):
    H, G = d["num_attention_heads"], d["num_key_value_heads"]
    return d["hidden_size"], d["intermediate_size"], H, G, d["head_dim"], d["vocab_size"], d["num_hidden_layers"]


def _tensor_table(d):
    """(name, shape, mean, std) of every tensor of the model, from the configuration alone."""
    N = 0.02
    out = []
    if d.get("architectures"):
        w, ff, H, G, hd, vocab, layers = _llama_sizes(d)
        out.append(("model.embed_tokens.weight", (vocab, w), 0.0, 1.0))
        for i in range(layers):
            p = f"model.layers.{i}."
            out += [(p + "input_layernorm.weight", (w,), 1.0, 0.1), (p + "post_attention_layernorm.weight", (w,), 1.0, 0.1),
                    (p + "self_attn.q_proj.weight", (H * hd, w), 0.0, N), (p + "self_attn.k_proj.weight", (G * hd, w), 0.0, N),
                    (p + "self_attn.v_proj.weight", (G * hd, w), 0.0, N), (p + "self_attn.o_proj.weight", (w, H * hd), 0.0, N),
                    (p + "mlp.gate_proj.weight", (ff, w), 0.0, N), (p + "mlp.up_proj.weight", (ff, w), 0.0, N),
                    (p + "mlp.down_proj.weight", (w, ff), 0.0, N)]
        out.append(("model.norm.weight", (w,), 1.0, 0.1))
        if not d["tie_word_embeddings"]:
            out.append(("lm_head.weight", (vocab, w), 0.0, N))
        return out
    w, vocab = d["width"], d["vocab"]
    out += [("embed", (vocab, w), 0.0, 1.0), ("head", (vocab, w), 0.0, N)]
    if d["architecture"] == "Vilazen":
        out += [("embed.norm", (w,), 0.0, 0.1), ("final.norm", (w,), 0.0, 0.1)]
        for i, layer in enumerate(d["layers"]):
            p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
            out += [(p + "norm1", (w,), 0.0, 0.1), (p + "mlp.up", (ff, w), 0.0, N), (p + "mlp.down", (w, ff), 0.0, N)]
            if layer["type"] == "latent_attention":
                H, D, R, V, C = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
                out += [(p + "mix.dkv", (C + R, w), 0.0, N), (p + "mix.dkv.norm", (C,), 1.0, 0.1),
                        (p + "mix.uk", (H * D, C), 0.0, 0.1), (p + "mix.uv", (H * V, C), 0.0, 0.1),
                        (p + "mix.o", (w, H * V), 0.0, N), (p + "mix.q", (H * (D + R), w), 0.0, N)]
                continue
            a, q = (m["left"], p + "mix.left.") if layer["type"] == "parallel" else (m, p + "mix.")
            H, G, D, V = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
            out += [(q + "q", (H * D, w), 0.0, N), (q + "k", (G * D, w), 0.0, N), (q + "v", (G * V, w), 0.0, N),
                    (q + "o", (w, H * V), 0.0, N), (q + "g", (H, w), 0.0, N)]
            if layer["type"] == "attention":
                out += [(q + "q.norm", (H * D,), 1.0, 0.1), (q + "k.norm", (G * D,), 1.0, 0.1), (q + "vmix", (), 0.5, 0.1)]
                continue
            out += [(q + "q.b", (H * D,), 0.0, 0.1), (q + "k.b", (G * D,), 0.0, 0.1), (q + "v.b", (G * V,), 0.0, 0.1),
                    (q + "sink", (H,), 0.0, 1.0)]
            r, q = m["right"], p + "mix.right."
            H, D, V = r["heads"], r["dim"], r["vdim"]
            out += [(q + "q", (H * D, w), 0.0, N), (q + "k", (H * D, w), 0.0, N), (q + "v", (H * V, w), 0.0, N),
                    (q + "o", (w, H * V), 0.0, N), (q + "norm", (H * V,), 1.0, 0.1), (q + "g", (H * V, w), 0.0, N)]
        return out
    S = d["streams"]
    out.append(("final.norm", (w,), 1.0, 0.1))
    for i, layer in enumerate(d["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        for k in (1, 2):
            # streams that start alike and stay near their own selves, each giving its share to the sublayer
            out += [(f"{p}norm{k}", (w,), 1.0, 0.1), (f"{p}hc{k}.in", (S,), 1.0 / S, 0.05), (f"{p}hc{k}.out", (S,), 1.0, 0.1),
                    (f"{p}hc{k}.mix", (S, S), "eye", 0.05)]
        out += [(p + "mlp.gate", (ff, w), 0.0, N), (p + "mlp.up", (ff, w), 0.0, N), (p + "mlp.down", (w, ff), 0.0, N)]
        sides = [(p + "mix.", m, True)]
        if layer["type"] == "parallel":
            a, q = m["left"], p + "mix.left."
            H, G, D, V, K = a["heads"], a["kv_heads"], a["dim"], a["vdim"], a["conv"]
            out += [(q + "q", (H * D, w), 0.0, N), (q + "k", (G * D, w), 0.0, N), (q + "v", (G * V, w), 0.0, N),
                    (q + "o", (w, H * V), 0.0, N), (q + "q.conv", (H * D, K), 0.25, 0.3), (q + "k.conv", (G * D, K), 0.25, 0.3),
                    (q + "v.conv", (G * V, K), 0.25, 0.3), (q + "out", (w,), 1.0, 0.1), (p + "mix.right.out", (w,), 1.0, 0.1)]
            sides = [(p + "mix.right.", m["right"], False)]
        for q, r, channel in sides:
            H, G, D, V, K = r["heads"], r["kv_heads"], r["dim"], r["vdim"], r["conv"]
            out += [(q + "q", (G * D, w), 0.0, N), (q + "k", (G * D, w), 0.0, N), (q + "v", (H * V, w), 0.0, N),
                    (q + "q.conv", (G * D, K), 0.25, 0.3), (q + "k.conv", (G * D, K), 0.25, 0.3),
                    (q + "v.conv", (H * V, K), 0.25, 0.3), (q + "b", (H, w), 0.0, N), (q + "A_log", (H,), 0.0, 0.5),
                    (q + "norm", (V,), 1.0, 0.1), (q + "o", (w, H * V), 0.0, N)]
            if channel:
                rd, rg = r["decay_rank"], r["gate_rank"]
                out += [(q + "a1", (rd, w), 0.0, N), (q + "a2", (H * D, rd), 0.0, 0.05), (q + "dt_bias", (H * D,), -2.0, 0.5),
                        (q + "g1", (rg, w), 0.0, N), (q + "g2", (H * V, rg), 0.0, 0.05)]
            else:
                out += [(q + "a", (H, w), 0.0, N), (q + "dt_bias", (H,), -2.0, 0.5), (q + "g", (H * V, w), 0.0, N)]
    return out


def _tensors(case, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed * 2 + 1)
    dtype = getattr(torch, case["dtype"])
    made = {}
    for name, size, mean, std in _tensor_table(_config(case)):
        t = torch.empty(size, dtype=dtype, device=DEVICE).normal_(0.0, std, generator=g)
        if mean == "eye":
            t += torch.eye(size[0], dtype=dtype, device=DEVICE)
        elif mean != 0.0:
            t += mean
        made[name] = t
    if case["kind"] == "generate" and "lm_head.weight" in made:
        # the next token is decided by a wide margin, as it mostly is for a trained model: every row of the head stands
        # out for the embedding of one token (a tied head does so for the token itself)
        made["lm_head.weight"].copy_(made["model.embed_tokens.weight"].roll(17, dims=0))
    return made


def _ids(case, seed, more=0):
    """Token ids of every sequence: its length's worth and ``more`` to go on with."""
    d = _config(case)
    vocab = d.get("vocab_size") or d["vocab"]
    g = torch.Generator().manual_seed(seed * 2)
    return [torch.randint(0, vocab, (n + more,), generator=g).tolist() for n in lengths(case)]


# ------------------------------------------------------------------------------------------------ a pass
def _cache_bytes_a_token(case):
    """Bytes of cache a position takes in all layers together (windows left aside)."""
    d, size = _config(case), 2 if case["dtype"] == "bfloat16" else 4
    if d.get("architectures"):
        w, ff, H, G, hd, vocab, layers = _llama_sizes(d)
        return layers * 2 * G * hd * size
    total = 0
    for layer in d["layers"]:
        m = layer["mixer"]
        if layer["type"] == "latent_attention":
            total += (m["kv_rank"] + m["rot_dim"]) * size
        elif layer["type"] in ("attention", "parallel"):
            a = m.get("left", m)
            total += a["kv_heads"] * (a["dim"] + a["vdim"]) * size
    return total


def _room(case):
    """Tokens a sequence may grow by before it is started over: enough for some thousand passes of a small case, at
    most 4 GB of cache for a large one."""
    if case["kind"] != "decode":
        return case["new"]
    most = 4096 - 16 - case["hi"] if case["model"] == "llama-13b" else 4096
    return max(64, min(most, int(4e9 / (case["seqs"] * max(1, _cache_bytes_a_token(case))))))


def _start(state):
    """The sequences' prompts into the cache, some at a time."""
    engine, ids, lens = state["engine"], state["ids"], state["lens"]
    for slot in state["slots"]:
        engine.free_slot(slot)
    state["slots"] = [engine.alloc_slot() for _ in lens]
    state["at"] = 0
    at = 0
    while at < len(lens):
        end, tokens = at, 0
        while end < len(lens) and (end == at or tokens + lens[end] <= STEP_TOKENS):
            tokens += lens[end]
            end += 1
        engine.step([(state["slots"][i], ids[i][:lens[i]]) for i in range(at, end)])
        at = end


def prepare(case, seed):
    gc.collect()                                  # an engine dropped before gives its memory back first
    lens, room = lengths(case), _room(case)
    pages = sum(-(-(n + room + 1) // PAGE) for n in lens)
    config = config_from_dict(_config(case))
    dtype = getattr(torch, case["dtype"])
    model = Model(config.model_spec(), dtype, torch.device(DEVICE))
    model.bind(_tensors(case, seed))
    options = EngineOptions(dtype=case["dtype"], max_seq_len=max(lens) + room + 1, max_tokens=pages * PAGE,
                            max_batch=len(lens), device=DEVICE)
    state = {"kind": case["kind"], "engine": Engine(config, model, options), "lens": lens, "room": room, "slots": []}
    if case["kind"] == "decode":
        state["ids"] = _ids(case, seed, room)
        _start(state)
        return state
    state["ids"] = _ids(case, seed)
    if case["kind"] == "generate":
        state["options"] = GenerationOptions(max_tokens=case["new"], ignore_eos=True, sampler={
            "greedy": SamplerParams(greedy=True),
            "sample": SamplerParams(repetition_penalty=1.0, seed=seed),
            "presence": SamplerParams(repetition_penalty=1.0, presence_penalty=0.5, seed=seed)}[case["sampler"]])
    return state


def run(state):
    engine, ids, lens = state["engine"], state["ids"], state["lens"]
    if state["kind"] == "generate":
        results, _ = engine.generate(ids, state["options"])
        return torch.tensor([r.tokens for r in results])
    if state["kind"] == "prompt":
        slots = [engine.alloc_slot() for _ in ids]
        logits = engine.step(list(zip(slots, ids)))
        for slot in slots:
            engine.free_slot(slot)
        return logits
    if state["at"] >= state["room"]:
        _start(state)
    k = state["at"]
    state["at"] = k + 1
    return engine.step([(slot, [t[n + k]]) for slot, t, n in zip(state["slots"], ids, lens)])


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Weights read once a step, the cache read once a decode step and written for new tokens, logits written; two
    operations a weight and token, four a key, channel and head."""
    d, size = _config(case), 2 if case["dtype"] == "bfloat16" else 4
    table = _tensor_table(d)
    vocab, width = d.get("vocab_size") or d["vocab"], d.get("hidden_size") or d["width"]
    embed = vocab * width
    inner = sum(math.prod(s) for n, s, _, _ in table if s != (vocab, width))
    lens, cache = lengths(case), _cache_bytes_a_token(case)

    def attention_flops(keys):
        """Scores and weighted sums of one query of every layer over ``keys`` keys (or a window's worth)."""
        if d.get("architectures"):
            w, ff, H, G, hd, v, layers = _llama_sizes(d)
            return 4.0 * layers * H * hd * keys
        total = 0.0
        for layer in d["layers"]:
            m = layer["mixer"]
            for a in (m.get("left", m), m.get("right")):
                if a is None:
                    continue
                if "scale" in a:
                    seen = min(keys, ((a.get("mask") or {}).get("size") or keys) + (a.get("mask") or {}).get("keep_first", 0))
                    total += 2.0 * a["heads"] * (a["dim"] + a.get("rot_dim", 0) + a["vdim"]) * seen
                else:
                    total += 6.0 * a["heads"] * a["dim"] * a["vdim"]         # a state of matrices, once a token
        return total

    def step(new, past, cached):
        tokens, n = sum(new), len(new)
        flops = 2.0 * inner * tokens + 2.0 * embed * n
        for t, p in zip(new, past):
            flops += attention_flops(p + 1) if t == 1 else t * attention_flops((t + 1) / 2.0)
        return (inner + embed) * size + tokens * width * size + cached * cache + tokens * cache + 4.0 * n * vocab, flops

    if case["kind"] == "decode":
        b, f = step([1] * len(lens), lens, sum(lens))
    else:
        b, f = step(lens, [0] * len(lens), 0)
        for k in range(case["new"] - 1):
            c = step([1] * len(lens), [n + k for n in lens], sum(lens) + k * len(lens))
            b, f = b + c[0], f + c[1]
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    """Sampled ids are decided by a wide margin.  bfloat16 logits were seen 0.003 to 0.02 off the 64-bit ones, and 0.008
    from one run to the next where a prompt's sums are added in the order they arrive; 32-bit ones 6e-6 off."""
    if case["kind"] == "generate":
        return "exact"
    return {"rel": 2.5e-5} if case["dtype"] == "float32" else {"rel": 0.03}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _times(x, w):
    """x W^T in 64 bits, some rows at a time."""
    w = w.double().t()
    return torch.cat([part @ w for part in x.split(8192)])


def _angles(positions, rot, base, scaling=None):
    """Angles in 32 bits, as the design defines them: position * frequency.  ``scaling``: factor, low, high, original."""
    out = []
    for i in range(rot // 2):
        f = base ** (-2.0 * i / rot)
        if scaling:
            factor, lo, hi, n0 = scaling
            wave = 2.0 * math.pi / f
            if wave > n0 / lo:
                f = f / factor
            elif wave >= n0 / hi:
                share = (n0 / wave - lo) / (hi - lo)
                f = (1.0 - share) * f / factor + share * f
        out.append(f)
    a = positions.float()[:, None] * torch.tensor(out, dtype=torch.float64, device=DEVICE).float()[None, :]
    return a.double()


def _turn(x, a, adjacent):
    """x [T, heads, D]: the first 2 R dimensions turned by the angles a [T, R]; pairs (2i, 2i+1) or (i, i+R)."""
    R = a.shape[1]
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    y = x.clone()
    i, j = (slice(0, 2 * R, 2), slice(1, 2 * R, 2)) if adjacent else (slice(0, R), slice(R, 2 * R))
    y[..., i] = x[..., i] * c - x[..., j] * s
    y[..., j] = x[..., j] * c + x[..., i] * s
    return y


def _attend(q, k, v, scale, bounds, window=None, keep_first=0, sink=None):
    """Softmax attention of every sequence (rows bounds[b]..bounds[b+1]) over its own keys up to the query's place."""
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=torch.float64, device=DEVICE)
    group = q.shape[1] // k.shape[1]
    for at, end in zip(bounds[:-1], bounds[1:]):
        n = end - at
        heads = max(1, int(2e8 / (n * n)))
        i = torch.arange(n, device=DEVICE)
        hidden = i[None, :] > i[:, None]
        if window is not None:
            hidden |= (i[:, None] - i[None, :] >= window) & (i[None, :] >= keep_first)
        for h in range(0, q.shape[1], heads):
            hs = range(h, min(q.shape[1], h + heads))
            of = [x // group for x in hs]
            s = torch.einsum("qhd,khd->hqk", q[at:end, h:hs[-1] + 1], k[at:end][:, of]).mul_(scale).masked_fill_(hidden, -math.inf)
            m = s.amax(dim=-1, keepdim=True)
            if sink is not None:
                extra = sink[h:hs[-1] + 1].double()[:, None, None]
                m = torch.maximum(m, extra)
            s.sub_(m).exp_()
            den = s.sum(dim=-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(extra - m)
            out[at:end, h:hs[-1] + 1] = torch.einsum("hqk,khd->qhd", s.div_(den), v[at:end][:, of])
    return out


def _padded(x, bounds):
    """Rows of the sequences as [longest, sequences, ...], zeros behind the ends."""
    return torch.nn.utils.rnn.pad_sequence([x[a:b] for a, b in zip(bounds[:-1], bounds[1:])])


def _unpadded(x, bounds):
    return torch.cat([x[:b - a, i] for i, (a, b) in enumerate(zip(bounds[:-1], bounds[1:]))])


def _conv(x, w, bounds):
    """Causal convolution a channel: y_t = sum_j w[:, j] x_(t - (K-1) + j), zeros before the sequence."""
    w, K = w.double(), w.shape[1]
    y = torch.zeros_like(x)
    for a, b in zip(bounds[:-1], bounds[1:]):
        for j in range(K):
            back = K - 1 - j
            if b - a > back:
                y[a + back:b] += x[a:b - back] * w[:, j]
    return y


def _silu(z):
    return z * torch.sigmoid(z)


def _llama_layer(d, w, p, x, pos, bounds):
    width, ff, H, G, hd, _, _ = _llama_sizes(d)
    sc = d["rope_scaling"]
    sc = sc and (sc["factor"], sc["low_freq_factor"], sc["high_freq_factor"], sc["original_max_position_embeddings"])
    h = _rms(x, d["rms_norm_eps"]) * w[p + "input_layernorm.weight"].double()
    q, k, v = (_times(h, w[f"{p}self_attn.{n}_proj.weight"]).view(-1, heads, hd) for n, heads in (("q", H), ("k", G), ("v", G)))
    a = _angles(pos, hd, d["rope_theta"], sc)
    o = _attend(_turn(q, a, False), _turn(k, a, False), v, hd ** -0.5, bounds)
    x = x + _times(o.reshape(-1, H * hd), w[p + "self_attn.o_proj.weight"])
    h = _rms(x, d["rms_norm_eps"]) * w[p + "post_attention_layernorm.weight"].double()
    return x + torch.cat([_times(_silu(_times(r, w[p + "mlp.gate_proj.weight"])) * _times(r, w[p + "mlp.up_proj.weight"]),
                                 w[p + "mlp.down_proj.weight"]) for r in h.split(8192)])


def _vilazen_layer(d, w, i, x, pos, bounds, kept):
    eps, layer, p = d["norm"]["eps"], d["layers"][i], f"l{i}."
    m = layer["mixer"]
    h = _rms(x, eps) * (1.0 + w[p + "norm1"].double())
    up = torch.cat([_times(0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0))), w[p + "mlp.down"])
                    for z in (_times(r, w[p + "mlp.up"]) for r in h.split(8192))])
    if layer["type"] == "latent_attention":
        H, D, R, V, C = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        a = _angles(pos, R, m["rot"]["base"])
        q = _times(h, w[p + "mix.q"]).view(-1, H, D + R)
        down = _times(h, w[p + "mix.dkv"])
        c = _rms(down[:, :C], eps) * w[p + "mix.dkv.norm"].double()
        turned = _turn(down[:, None, C:], a, True).expand(-1, H, -1)
        k = torch.cat([_times(c, w[p + "mix.uk"]).view(-1, H, D), turned], dim=-1)
        q = torch.cat([q[..., :D], _turn(q[..., D:], a, True)], dim=-1)
        o = _attend(q, k, _times(c, w[p + "mix.uv"]).view(-1, H, V), m["scale"], bounds, (m.get("mask") or {}).get("size"))
        return x + up + _times(o.reshape(-1, H * V), w[p + "mix.o"])
    side = layer["type"] == "parallel"
    a, t = (m["left"], p + "mix.left.") if side else (m, p + "mix.")
    H, G, D, V = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
    q, k, v = (_times(h, w[t + n]) for n in "qkv")
    if side:
        q, k, v = (y + w[t + n + ".b"].double() for y, n in ((q, "q"), (k, "k"), (v, "v")))
    else:
        q, k = _rms(q, eps) * w[t + "q.norm"].double(), _rms(k, eps) * w[t + "k.norm"].double()
        if "v" in kept:
            lam = w[t + "vmix"].double()
            v = (1.0 - lam) * v + lam * kept["v"]
        else:
            kept["v"] = v
    ang = _angles(pos, a["rot"]["dims"], a["rot"]["base"])
    mask = a.get("mask") or {}
    o = _attend(_turn(q.view(-1, H, D), ang, True), _turn(k.view(-1, G, D), ang, True), v.view(-1, G, V), a["scale"], bounds,
                mask.get("size"), mask.get("keep_first", 0), w[t + "sink"] if side else None)
    o = o * torch.sigmoid(_times(h, w[t + "g"]))[:, :, None]
    y = up + (m["left_scale"] if side else 1.0) * _times(o.reshape(-1, H * V), w[t + "o"])
    if side:
        r, t = m["right"], p + "mix.right."
        H, D, V = r["heads"], r["dim"], r["vdim"]
        q, k, v = (_padded(_silu(_times(h, w[t + n])).view(-1, H, z), bounds) for n, z in (("q", D), ("k", D), ("v", V)))
        decay = torch.tensor(r["decay"], dtype=torch.float64, device=DEVICE)[None, :, None, None]
        S = torch.zeros(q.shape[1], H, D, V, dtype=torch.float64, device=DEVICE)
        o = torch.empty_like(v)
        for at in range(q.shape[0]):
            S.mul_(decay).add_(k[at][..., :, None] * v[at][..., None, :])
            o[at] = (q[at][..., None, :] @ S)[..., 0, :]
        o = _unpadded(o, bounds).reshape(-1, H * V)
        o = _rms(o, eps) * w[t + "norm"].double() * torch.sigmoid(_times(h, w[t + "g"]))
        y = y + m["right_scale"] * _times(o, w[t + "o"])
    return x + y


def _delta(h, w, t, r, eps, bounds):
    H, G, D, V = r["heads"], r["kv_heads"], r["dim"], r["vdim"]
    q, k, v = (_silu(_conv(_times(h, w[t + n]), w[t + n + ".conv"], bounds)) for n in "qkv")
    q, k = q.view(-1, G, D), k.view(-1, G, D)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = (y.repeat_interleave(H // G, dim=1) for y in (q, k))
    v, beta = v.view(-1, H, V), torch.sigmoid(_times(h, w[t + "b"]))
    rate = torch.exp(w[t + "A_log"].double())[None, :, None]
    if t + "a" in w:
        z = (_times(h, w[t + "a"]) + w[t + "dt_bias"].double()).view(-1, H, 1)
        gate = _silu(_times(h, w[t + "g"]))
    else:
        z = (_times(_times(h, w[t + "a1"]), w[t + "a2"]) + w[t + "dt_bias"].double()).view(-1, H, D)
        gate = torch.sigmoid(_times(_times(h, w[t + "g1"]), w[t + "g2"]))
    g = torch.exp(-rate * torch.nn.functional.softplus(z, threshold=40.0)).expand(-1, H, D)
    q, k, v, beta, g = (_padded(y, bounds) for y in (q, k, v, beta, g))
    S = torch.zeros(q.shape[1], H, D, V, dtype=torch.float64, device=DEVICE)
    o = torch.empty_like(v)
    for at in range(q.shape[0]):
        S.mul_(g[at][..., None])
        u = beta[at][..., None] * (v[at] - (k[at][..., None, :] @ S)[..., 0, :])
        S.add_(k[at][..., :, None] * u[..., None, :])
        o[at] = (q[at][..., None, :] @ S)[..., 0, :]
    o = _unpadded(o, bounds)
    return _times((_rms(o, eps) * w[t + "norm"].double()).reshape(-1, H * V) * gate, w[t + "o"])


def _mopilorn_layer(d, w, i, xs, pos, bounds):
    """xs: the residual streams [S, T, width]."""
    eps, layer, p = d["norm"]["eps"], d["layers"][i], f"l{i}."
    m = layer["mixer"]

    def into(k):
        return _rms(torch.einsum("a,atd->td", w[f"{p}hc{k}.in"].double(), xs), eps) * w[f"{p}norm{k}"].double()

    def spread(y, k):
        return (torch.einsum("ab,atd->btd", w[f"{p}hc{k}.mix"].double(), xs)
                + w[f"{p}hc{k}.out"].double()[:, None, None] * y[None])

    h = into(1)
    if layer["type"] == "parallel":
        a, t = m["left"], p + "mix.left."
        H, G, D, V = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
        q, k, v = (_conv(_times(h, w[t + n]), w[t + n + ".conv"], bounds) for n in "qkv")
        sc = a["rot"].get("scaling")
        ang = _angles(pos, a["rot"]["dims"], a["rot"]["base"], sc and (sc["factor"], sc["low"], sc["high"], sc["original"]))
        o = _attend(_turn(q.view(-1, H, D), ang, True), _turn(k.view(-1, G, D), ang, True), v.view(-1, G, V), a["scale"],
                    bounds, (a.get("mask") or {}).get("size"))
        left = _times(o.reshape(-1, H * V), w[t + "o"])
        right = _delta(h, w, p + "mix.right.", m["right"], eps, bounds)
        y = 0.5 * (_rms(left, eps) * w[t + "out"].double() + _rms(right, eps) * w[p + "mix.right.out"].double())
    else:
        y = _delta(h, w, p + "mix.", m, eps, bounds)
    xs = spread(y, 1)
    h = into(2)
    y = torch.cat([_times(_silu(_times(r, w[p + "mlp.gate"])) * _times(r, w[p + "mlp.up"]), w[p + "mlp.down"])
                   for r in h.split(8192)])
    return spread(y, 2)


def exact(case, seed):
    """The logits of the last token of every sequence (of the first token behind it for a decode step)."""
    if case["kind"] == "generate":
        return None                                   # ids only: nothing to be near to
    d, w = _config(case), _tensors(case, seed)
    # a decode step's first pass brings the token behind the prompt; what follows it is drawn as prepare() draws it
    ids = _ids(case, seed, _room(case))
    ids = [t[:n + 1] for t, n in zip(ids, lengths(case))] if case["kind"] == "decode" else _ids(case, seed)
    bounds = [0]
    for t in ids:
        bounds.append(bounds[-1] + len(t))
    pos = torch.cat([torch.arange(len(t), device=DEVICE) for t in ids])
    flat = torch.tensor([i for t in ids for i in t], device=DEVICE)
    last = torch.tensor(bounds[1:], device=DEVICE) - 1
    if d.get("architectures"):
        x = w["model.embed_tokens.weight"][flat].double()
        for i in range(d["num_hidden_layers"]):
            x = _llama_layer(d, w, f"model.layers.{i}.", x, pos, bounds)
        h = _rms(x[last], d["rms_norm_eps"]) * w["model.norm.weight"].double()
        return _times(h, w.get("lm_head.weight", w["model.embed_tokens.weight"]))
    eps = d["norm"]["eps"]
    if d["architecture"] == "Vilazen":
        x = _rms(w["embed"][flat].double(), eps) * (1.0 + w["embed.norm"].double())
        kept = {}
        for i in range(len(d["layers"])):
            x = _vilazen_layer(d, w, i, x, pos, bounds, kept)
        return _times(_rms(x[last], eps) * (1.0 + w["final.norm"].double()), w["head"])
    xs = w["embed"][flat].double()[None].repeat(d["streams"], 1, 1)
    for i in range(len(d["layers"])):
        xs = _mopilorn_layer(d, w, i, xs, pos, bounds)
    z = _times(_rms(xs.sum(dim=0)[last], eps) * w["final.norm"].double(), w["head"])
    return d["logit_softcap"] * torch.tanh(z / d["logit_softcap"])
