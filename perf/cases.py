"""The work this library is measured on: requests a program hands to ``Engine.generate`` and steps it hands to
``Runner.step``, at the layer sizes of ``bench.py``, with random weights.

A case names the model's layer sizes, the storage type, the call, and the batch: ``batch`` prompts of ``shortest`` to
``longest`` tokens.

* ``call`` "generate": ``Engine.generate`` of ``new`` greedy tokens a sequence (the prompts, then one step a token). A
  pass returns the tokens and the logits that the last of them were chosen from.
* ``call`` "step": a new sequence each, one ``Runner.step`` with their prompts, and, where ``follow`` is not 0, a second
  one of ``follow`` tokens each on top of what the first left in the cache. A pass returns the last step's logits at the
  last ``want`` places of each sequence. ``graph`` says whether the step may be replayed as a CUDA graph, which is how
  generation calls it; a check of given tokens does not ask for it.

Weights: matrices N(0, 0.02), norm weights 1 + N(0, 0.1), as ``random_model`` draws them, but for the embedding and the
head: the head's row of token t + vocab / 3 is the embedding's row of t, scaled to N(0, 0.02), and the embedding is N(0, 4),
of the order of what the layers add up to. So a token's logit stands out by some units as a trained model's does, and greedy
tokens do not hang on the rounding of near ties. Tokens: uniform in [1000, 100000) where the vocabulary has them, as the
command line draws them.
"""
import math

import numpy as np
import torch

import dryft_challenge_htn_2026_b200 as dk

# ------------------------------------------------------------------------------------------------ models
_QWEN3 = dict(architectures=["Qwen3ForCausalLM"], vocab_size=151936, num_key_value_heads=8, head_dim=128, rms_norm_eps=1e-6,
              rope_theta=1000000.0, max_position_embeddings=40960)
SIZES = {   # the layer sizes of bench.py
    "qwen3-4b": dict(_QWEN3, hidden_size=2560, intermediate_size=9728, num_hidden_layers=36, num_attention_heads=32,
                     tie_word_embeddings=True),
    "qwen3-8b": dict(_QWEN3, hidden_size=4096, intermediate_size=12288, num_hidden_layers=36, num_attention_heads=32,
                     tie_word_embeddings=False),
    "qwen3-14b": dict(_QWEN3, hidden_size=5120, intermediate_size=17408, num_hidden_layers=40, num_attention_heads=40,
                      tie_word_embeddings=False),
}
# the second design at the 4B widths, as bench.py --design lays it out: chunked attention beside decayed linear attention
NILIVIK = dict(vocab=32768, width=2560, layers=4, heads=32, kv_heads=8, dim=128, chunk=2048, right_heads=16, ff=7424, eps=1e-6,
               cap=30.0, mix=0.7)


def _decays():
    n = NILIVIK["right_heads"]
    return [1.0 - 2.0 ** -(3 + 5 * i / (n - 1)) for i in range(n)]


def _config(model):
    if model != "nilivik":
        return dict(SIZES[model])
    n = NILIVIK
    layer = {"type": "parallel",
             "mixer": {"left": {"heads": n["heads"], "kv_heads": n["kv_heads"], "dim": n["dim"], "vdim": n["dim"],
                                "mask": {"size": n["chunk"]}, "scale": n["dim"] ** -0.5},
                       "right": {"heads": n["right_heads"], "dim": n["dim"], "vdim": n["dim"], "decay": _decays()},
                       "left_scale": n["mix"], "right_scale": n["mix"]},
             "mlp": {"kind": "dense", "ff": n["ff"]}}
    return dict(architecture="Nilivik", vocab=n["vocab"], width=n["width"], embedding={"scale": 1.0}, norm={"eps": n["eps"]},
                logit_softcap=n["cap"], layers=[layer] * n["layers"])


def _vocab(model):
    return NILIVIK["vocab"] if model == "nilivik" else SIZES[model]["vocab_size"]


def _parameters(model):
    """[(name, shape, kind)]: kind "matrix" is kept in the model's storage type, the others in float32."""
    out = []
    if model == "nilivik":
        n = NILIVIK
        w, d = n["width"], n["dim"]
        for i in range(n["layers"]):
            p = "l%d." % i
            out += [(p + "norm1", (), "norm"), (p + "norm2", (), "norm"), (p + "mlp.act", (2,), "unit"),
                    (p + "mlp.up", (n["ff"], w), "matrix"), (p + "mlp.down", (w, n["ff"]), "matrix")]
            left, right = p + "mix.left.", p + "mix.right."
            rows = {"q": n["heads"] * d, "k": n["kv_heads"] * d, "v": n["kv_heads"] * d, "g": n["heads"] * d}
            out += [(left + k, (r, w), "matrix") for k, r in rows.items()]
            out += [(left + "o", (w, n["heads"] * d), "matrix"), (left + "sink", (n["heads"],), "unit"),
                    (left + "r1", (n["heads"],), "rate"), (left + "r2", (n["heads"],), "rate")]
            out += [(right + k, (n["right_heads"] * d, w), "matrix") for k in ("q", "k", "v", "g")]
            out += [(right + "o", (w, n["right_heads"] * d), "matrix"), (right + "norm", (n["right_heads"] * d,), "norm")]
        return out + [("final.norm", (), "norm")]
    c = SIZES[model]
    w, f, hd = c["hidden_size"], c["intermediate_size"], c["head_dim"]
    q, kv = c["num_attention_heads"] * hd, c["num_key_value_heads"] * hd
    for i in range(c["num_hidden_layers"]):
        p = "model.layers.%d." % i
        out += [(p + "input_layernorm.weight", (w,), "norm"), (p + "post_attention_layernorm.weight", (w,), "norm"),
                (p + "self_attn.q_norm.weight", (hd,), "norm"), (p + "self_attn.k_norm.weight", (hd,), "norm"),
                (p + "self_attn.q_proj.weight", (q, w), "matrix"), (p + "self_attn.k_proj.weight", (kv, w), "matrix"),
                (p + "self_attn.v_proj.weight", (kv, w), "matrix"), (p + "self_attn.o_proj.weight", (w, q), "matrix"),
                (p + "mlp.gate_proj.weight", (f, w), "matrix"), (p + "mlp.up_proj.weight", (f, w), "matrix"),
                (p + "mlp.down_proj.weight", (w, f), "matrix")]
    return out + [("model.norm.weight", (w,), "norm")]


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _weights(case, seed):
    model, gen = case["model"], torch.Generator(device="cuda").manual_seed(int(seed))
    draw = lambda shape: torch.randn(shape, generator=gen, dtype=torch.float32, device="cuda")  # noqa: E731
    out = {}
    for name, shape, kind in _parameters(model):
        x = draw(shape)
        if kind == "matrix":
            out[name] = (0.02 * x).to(_dtype(case))
        else:
            out[name] = 1.0 + 0.1 * x if kind == "norm" else 0.05 + 0.3 * x.abs() if kind == "rate" else x
    nilivik = model == "nilivik"
    e = draw((_vocab(model), NILIVIK["width"] if nilivik else SIZES[model]["hidden_size"]))
    out["head" if nilivik else "lm_head.weight"] = (0.02 * e.roll(_vocab(model) // 3, 0)).to(_dtype(case))
    out["embed" if nilivik else "model.embed_tokens.weight"] = (4.0 * e).to(_dtype(case))
    return out


# ------------------------------------------------------------------------------------------------ cases
def _case(name, model, call, batch, shortest, longest, dtype="bfloat16", **more):
    c = {"name": name, "model": model, "dtype": dtype, "call": call, "batch": batch, "shortest": shortest, "longest": longest}
    c.update({"new": 32} if call == "generate" else {"want": 1, "follow": 0, "graph": dtype != "float32"})
    c.update(more)
    return c


def listed():
    return [
        # the first token of a short question: latency, launches and one reading of the weights
        _case("first_token_1x9", "qwen3-4b", "step", 1, 9, 9),
        # one document, then the first token (the bench's prompt)
        _case("prompt_1x2048", "qwen3-4b", "step", 1, 2048, 2048),
        # the next turn of four conversations on top of what is cached
        _case("turn_4x700_41", "qwen3-4b", "step", 4, 300, 701, follow=41),
        # one user: the command line's first default shape
        _case("generate_1x512_32", "qwen3-4b", "generate", 1, 512, 512),
        # a small batch of unequal prompts: the bench's batch of 8
        _case("generate_8x2048_64", "qwen3-4b", "generate", 8, 1024, 2048, new=64),
        # the command line's third default shape
        _case("generate_16x512_128", "qwen3-4b", "generate", 16, 512, 512, new=128),
        # a large batch of short unequal prompts
        _case("generate_64x333_32", "qwen3-4b", "generate", 64, 64, 333),
        # a long document and a short answer
        _case("generate_1x16384_16", "qwen3-4b", "generate", 1, 16384, 16384, new=16),
        # the bench's next layer sizes, three users
        _case("generate_3x777_24_8b", "qwen3-8b", "generate", 3, 401, 777, new=24),
        # the command line's check of a sample: prompt and emitted tokens through the 32-bit path, logits of the emitted ones
        _case("check_1x544_f32", "qwen3-4b", "step", 1, 544, 544, dtype="float32", want=32),
        # generation in 32 bits: what a bfloat16 result is compared with
        _case("generate_2x100_12_f32", "qwen3-4b", "generate", 2, 61, 100, dtype="float32", new=12),
        # the second design: masked attention and a recurrence side by side
        _case("generate_8x3000_32_nilivik", "nilivik", "generate", 8, 1000, 3000),
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    most = max(_seconds(c) for c in listed())
    while True:
        model = rng.choice(["qwen3-4b"] * 5 + ["qwen3-8b", "qwen3-14b", "nilivik", "nilivik"])
        dtype = "float32" if model in ("qwen3-4b", "nilivik") and rng.random() < 0.25 else "bfloat16"
        batch = _spread(rng, 1, 64 if dtype == "bfloat16" else 8)
        longest = _spread(rng, 8, 16384 if dtype == "bfloat16" else 1024)
        shortest = rng.randint(max(1, longest // 5), longest)
        c = {"model": model, "dtype": dtype, "batch": batch, "shortest": shortest, "longest": longest}
        if rng.random() < 0.5:
            c.update(call="generate", new=_spread(rng, 4, 128 if dtype == "bfloat16" else 16))
        else:
            follow = rng.choice([0, 0, _spread(rng, 2, 64)])
            c.update(call="step", follow=follow, want=rng.choice([1, rng.randint(1, min(32, follow or shortest))]),
                     graph=dtype != "float32")
        if sum(_lengths(c)) <= (20000 if dtype == "bfloat16" else 1200) and _seconds(c) <= most:
            return c


def _lengths(case):
    """The prompts' lengths: spread evenly over shortest..longest, in no order."""
    b, lo, hi = case["batch"], case["shortest"], case["longest"]
    if b == 1:
        return [hi]
    order = np.random.RandomState(b).permutation(b)
    return [lo + (hi - lo) * int(i) // (b - 1) for i in order]


def _prompts(case, seed):
    gen = torch.Generator().manual_seed(int(seed))
    hi = min(100000, _vocab(case["model"]))
    return [torch.randint(1000, hi, (n + case.get("follow", 0),), generator=gen).tolist() for n in _lengths(case)]


# ------------------------------------------------------------------------------------------------ a pass
def prepare(case, seed):
    model = dk.CausalLM(dk.config_from_dict(_config(case["model"])).to_spec(), _dtype(case), "cuda")
    model.bind(_weights(case, seed), False)
    prompts = _prompts(case, seed)
    state = {"case": case, "prompts": prompts}
    if case["call"] == "generate":
        state["engine"] = dk.Engine(model=model)
    else:
        state["runner"] = dk.Runner(model, sum((len(p) + 63) // 64 * 64 for p in prompts), max_slots=len(prompts))
    return state


def run(state):
    case, prompts = state["case"], state["prompts"]
    if case["call"] == "generate":
        engine = state["engine"]
        tokens = list(engine.generate(prompts, case["new"]))
        return {"tokens": np.array(tokens, dtype=np.int64), "logits": engine.backend.state.logits[:len(prompts)]}
    runner, follow = state["runner"], case["follow"]
    slots = [runner.begin() for _ in prompts]
    if follow:
        runner.step([(s, p[:-follow], []) for s, p in zip(slots, prompts)], graph=case["graph"])
    last = [p[-follow:] for p in prompts] if follow else prompts
    logits = runner.step([(s, t, list(range(len(t) - case["want"], len(t)))) for s, t in zip(slots, last)], graph=case["graph"])
    for s in slots:
        runner.end(s)
    return {"logits": logits}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _layer_sizes(model):
    """(layers, matrix elements of a layer, elements of the head, K/V elements of a token and layer, attention multiply-adds of
    a query and key, the attention's reach, state elements of a sequence and layer)"""
    if model == "nilivik":
        n = NILIVIK
        at, r = n["heads"] * n["dim"], n["right_heads"] * n["dim"]
        m = n["width"] * (3 * at + 2 * n["kv_heads"] * n["dim"] + 5 * r + 2 * n["ff"])
        return n["layers"], m, n["vocab"] * n["width"], 2 * n["kv_heads"] * n["dim"], 2 * at, n["chunk"], r * n["dim"]
    c = SIZES[model]
    w, hd = c["hidden_size"], c["head_dim"]
    q, kv = c["num_attention_heads"] * hd, c["num_key_value_heads"] * hd
    m = w * (2 * q + 2 * kv + 3 * c["intermediate_size"])
    return c["num_hidden_layers"], m, c["vocab_size"] * w, 2 * kv, 2 * q, 1 << 30, 0


def _pairs(first, last, reach):
    """Keys that the queries at positions first..last-1 see, in sum; ``reach`` is the size of a chunk."""
    upto = lambda n: (n // reach) * (reach * (reach + 1) // 2) + (n % reach) * (n % reach + 1) // 2  # noqa: E731
    return upto(last) - upto(first)


def _steps(case):
    """The steps of a pass: [([(first, last) position of each sequence], logit rows)]"""
    lengths, follow = _lengths(case), case.get("follow", 0)
    if case["call"] == "generate":
        return [([(0, n) for n in lengths], len(lengths))] + \
            [([(n + k, n + k + 1) for n in lengths], len(lengths)) for k in range(case["new"] - 1)]
    if follow:
        return [([(0, n) for n in lengths], 0), ([(n, n + follow) for n in lengths], len(lengths) * case["want"])]
    return [([(0, n) for n in lengths], len(lengths) * case["want"])]


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    layers, matrix, head, kv, pair, reach, state = _layer_sizes(case["model"])
    total = flops = 0
    for seqs, rows in _steps(case):
        tokens = sum(b - a for a, b in seqs)
        read = sum(a % reach for a, b in seqs)     # what is cached and in sight; the step's own keys and values are written
        total += size * (layers * (matrix + kv * (read + tokens)) + (head if rows else 0)) + 8 * layers * state * len(seqs)
        total += 4 * rows * _vocab(case["model"])
        flops += 2 * (layers * (matrix * tokens + pair * sum(_pairs(a, b, reach) for a, b in seqs) + 2 * state * tokens) + head * rows)
    return {"bytes": float(total), "flops": float(flops)}


def _seconds(case):
    """Roughly what a pass takes at a B200's rates: 6.5 TB/s, 1,600 TFLOP/s (70 in 32 bits)."""
    w = work(case)
    return w["bytes"] / 6.5e12 + w["flops"] / (70e12 if case["dtype"] == "float32" else 1600e12)


def tolerance(case):
    """Relative differences of the logits; the tokens are the same. Measured against ``exact``: 0.003 to 0.01 in bfloat16, 2e-6 to
    5e-6 in float32; another implementation is as far off on another side."""
    if case["dtype"] == "float32":
        return {"rel": 2.5e-5, "max": 5e-4, "differ": 0.0}
    return {"rel": 0.02, "max": 0.25, "differ": 0.0}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
F64 = torch.float64


def _mm(x, w):
    return x @ w.to(F64).T


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.to(F64)


def _weighted_sums(q, k, v, weights):
    """q [S, H, D], k, v [S, G, D] of one sequence; ``weights(scores [H, n, m], i [n, 1], j [1, m])`` turns the products of the
    queries i with the keys j into the values' weights. -> [S, H * D]"""
    S, H, D = q.shape
    G = k.shape[1]
    q = q.transpose(0, 1).reshape(G, H // G, S, D)
    k, v = k.transpose(0, 1), v.transpose(0, 1)
    out = torch.empty(G, H // G, S, D, dtype=F64, device=q.device)
    for a in range(0, S, 512):
        b = min(S, a + 512)
        s = torch.matmul(q[:, :, a:b].reshape(G, -1, D), k[:, :b].transpose(1, 2)).view(H, b - a, b)
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(b, device=q.device)[None, :]
        p = weights(s, i, j).view(G, -1, b)
        out[:, :, a:b] = torch.matmul(p, v[:, :b]).view(G, H // G, b - a, D)
    return out.reshape(H, S, D).transpose(0, 1).reshape(S, H * D)


def _softmax(s, i, j):
    return torch.softmax(s.masked_fill(j > i, -math.inf), -1)


def _rotate(x, theta):
    S, _, D = x.shape
    inv = theta ** (-torch.arange(0, D, 2, device=x.device, dtype=F64) / D)
    a = torch.arange(S, device=x.device, dtype=F64)[:, None] * inv
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _by_sequence(fn, lengths, *xs):
    return torch.cat([fn(*parts) for parts in zip(*(x.split(lengths) for x in xs))])


def _qwen3_layers(c, t, h, lengths):
    eps, hd = c["rms_norm_eps"], c["head_dim"]

    def attend(q, k, v):
        q, k = _rotate(q, c["rope_theta"]), _rotate(k, c["rope_theta"])
        return _weighted_sums(q * hd ** -0.5, k, v, _softmax)

    for i in range(c["num_hidden_layers"]):
        p = "model.layers.%d." % i
        a = _rms(h, t[p + "input_layernorm.weight"], eps)
        q, k, v = (_mm(a, t[p + "self_attn.%s_proj.weight" % x]).view(len(h), -1, hd) for x in "qkv")
        q, k = _rms(q, t[p + "self_attn.q_norm.weight"], eps), _rms(k, t[p + "self_attn.k_norm.weight"], eps)
        h = h + _mm(_by_sequence(attend, lengths, q, k, v), t[p + "self_attn.o_proj.weight"])
        a = _rms(h, t[p + "post_attention_layernorm.weight"], eps)
        g = _mm(a, t[p + "mlp.gate_proj.weight"])
        h = h + _mm(g * torch.sigmoid(g) * _mm(a, t[p + "mlp.up_proj.weight"]), t[p + "mlp.down_proj.weight"])
    return _rms(h, t["model.norm.weight"], eps)


def _nilivik_layers(t, h, lengths):
    n = NILIVIK
    eps, hd = n["eps"], n["dim"]
    decay = torch.tensor(_decays(), dtype=F64, device=h.device).view(-1, 1, 1)

    def sinusoid(x):
        a = torch.arange(len(x), device=x.device, dtype=F64)[:, None] * \
            10000.0 ** (-torch.arange(0, x.shape[1], 2, device=x.device, dtype=F64) / x.shape[1])
        return x + torch.stack([a.sin(), a.cos()], -1).view(len(x), -1)

    h = _by_sequence(sinusoid, lengths, h)
    for l in range(n["layers"]):
        left, right, mlp = ("l%d.%s." % (l, x) for x in ("mix.left", "mix.right", "mlp"))
        r1, r2, sink = (t[left + x].to(F64).view(-1, 1, 1) for x in ("r1", "r2", "sink"))

        def chunked(s, i, j):
            s = s - r1 * torch.log1p(r2 * (i - j).clamp(min=0).to(F64))
            s = s.masked_fill((j > i) | (j // n["chunk"] != i // n["chunk"]), -math.inf)
            return torch.softmax(torch.cat([s, sink.expand(-1, s.shape[1], 1)], -1), -1)[..., :-1].contiguous()

        def decayed(s, i, j):
            return s * (decay ** (i - j).clamp(min=0).to(F64)).masked_fill(j > i, 0.0)

        a = _rms(h, t["l%d.norm1" % l], eps)
        q, k, v = (_mm(a, t[left + x]).view(len(h), -1, hd) for x in "qkv")
        o = _by_sequence(lambda q, k, v: _weighted_sums(q * hd ** -0.5, k, v, chunked), lengths, q, k, v)
        o = n["mix"] * _mm(o * torch.sigmoid(_mm(a, t[left + "g"])), t[left + "o"])
        silu = torch.nn.functional.silu
        q, k, v = (silu(_mm(a, t[right + x])).view(len(h), -1, hd) for x in "qkv")
        r = _by_sequence(lambda q, k, v: _weighted_sums(q, k, v, decayed), lengths, q, k, v)
        r = _rms(r, t[right + "norm"], eps) * torch.sigmoid(_mm(a, t[right + "g"]))
        h = h + o + n["mix"] * _mm(r, t[right + "o"])
        z = _mm(_rms(h, t["l%d.norm2" % l], eps), t[mlp + "up"])
        p, q = torch.nn.functional.softplus(t[mlp + "act"].to(F64))
        h = h + _mm(torch.where(z > 0, p * z * z, (0.5 + q) * (torch.expm1(z) - z)) + 0.5 * z, t[mlp + "down"])
    return _rms(h, t["final.norm"], eps)


def exact(case, seed):
    if work(case)["flops"] > 2.0e14:
        return None                # over about 20 seconds in 64 bits
    model, new = case["model"], case.get("new", 1)
    t, prompts, V = _weights(case, seed), _prompts(case, seed), _vocab(case["model"])
    # greedy tokens follow one another by the step the head is built with; the logits below say so again
    seqs = [p + [(p[-1] + k * (V // 3)) % V for k in range(1, new)] for p in prompts]
    lengths = [len(s) for s in seqs]
    tokens = torch.tensor([x for s in seqs for x in s], device="cuda")
    with torch.inference_mode():
        if model == "nilivik":
            h, head = _nilivik_layers(t, t["embed"][tokens].to(F64), lengths), t["head"]
        else:
            h = _qwen3_layers(SIZES[model], t, t["model.embed_tokens.weight"][tokens].to(F64), lengths)
            head = t["lm_head.weight"]
        head = head.to(F64)
        cap = lambda z: NILIVIK["cap"] * torch.tanh(z / NILIVIK["cap"]) if model == "nilivik" else z  # noqa: E731
        ends = np.cumsum(lengths)
        if case["call"] == "step":
            rows = [e - case["want"] + k for e in ends for k in range(case["want"])]
            return {"logits": cap(h[torch.tensor(rows, device="cuda")] @ head.T)}
        chosen = []
        for k in range(new):       # the k-th token of every sequence
            z = h[torch.tensor(ends - new + k, device="cuda")] @ head.T
            chosen.append(z.argmax(-1))
        return {"tokens": torch.stack(chosen), "logits": cap(z)}
