"""What the speed of this framework is measured on: passes through its step function and its sampler, as a program that
serves a model calls them, over the sizes such programs have.

Three kinds of pass:

* ``step``: one engine step over requests that hold cached tokens already: ``decodes`` requests bring one token each
  and, beside them or alone, one request brings a portion of ``portion`` prompt tokens behind ``behind`` cached ones.
  The wanted logits come back (the last token of each run, or every token of the portion where a text is scored).
  Behind the step each request is set back to what it held, as when several continuations of one text are tried.
* ``requests``: whole requests: they are admitted, their prompts run in steps of at most 2,048 tokens, then ``tokens``
  steps bring one given token per request, then they are released.  All logits come back.  Models whose layers keep a
  state, which cannot be set back, are measured this way, and so is the 32-bit path.
* ``sample``: token ids for rows of logits, with the options a request may choose.

Weights are random (matrices N(0, 0.02), norm weights 1 + N(0, 0.05)), token ids uniform.  Sizes are the ones of the
benchmark (bench.py): the Qwen3-1.7B shape whole, eight layers of the Qwen3-8B widths, and eight layers of the Fadosun
design at the 1.7B width; and the 0.6B widths of the tests for the 32-bit path.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from ember_b200 import SamplingParams, StepEntry
from ember_b200.api import LLM
from ember_b200.config import FadosunConfig, Qwen3Config
from ember_b200.engine.runner import ModelRunner
from ember_b200.sampling import device as device_sampler
from ember_b200.weights.loader import WeightStore

STEP_TOKENS = 2048              # the engine's default limit of a step and of a prompt portion
VOCAB = 151936

QWEN3 = {
    "1.7b": dict(hidden=2048, inter=6144, layers=28, heads=16, kv_heads=8, tied=True),
    "8b": dict(hidden=4096, inter=12288, layers=8, heads=32, kv_heads=8, tied=False),
    "0.6b": dict(hidden=1024, inter=3072, layers=28, heads=16, kv_heads=8, tied=True),
}
HEAD, THETA, EPS = 128, 1000000.0, 1e-6

DELTA = {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}
SIGMOID = {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 0.0884, "rot": {"dims": 64, "base": 1e6}}
SPACE = {"heads": 32, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}
MEMORY = {"heads": 8, "dim": 128, "vdim": 256, "gate_cap": 15.0}
FADOSUN_LAYERS = [
    {"type": "channel_delta", "mixer": DELTA},
    {"type": "parallel", "mixer": {"left": SIGMOID, "right": SPACE, "left_scale": 1.0, "right_scale": 1.0}},
    {"type": "mlstm", "mixer": MEMORY},
    {"type": "channel_delta", "mixer": DELTA},
] * 2
FADOSUN_WIDTH, FADOSUN_FF = 2048, 6144


# ------------------------------------------------------------------------------------------------------------- cases
def step(name, model="1.7b", decodes=0, context=0, portion=0, behind=0, every=False, page=64):
    return dict(name=name, kind="step", model=model, dtype="bfloat16", decodes=decodes, context=context, portion=portion,
                behind=behind, every=every, page=page)


def requests(name, model, dtype, count, prompt, tokens, page=64):
    return dict(name=name, kind="requests", model=model, dtype=dtype, count=count, prompt=prompt, tokens=tokens, page=page)


def sample(name, rows, temperature, top_k, top_p, min_p):
    return dict(name=name, kind="sample", rows=rows, temperature=temperature, top_k=top_k, top_p=top_p, min_p=min_p)


def listed():
    return [
        # one user's chat: the next token of one request, a short context
        step("decode-1", decodes=1, context=700),
        # the benchmark's default point: eight requests in the middle of their 4,096 positions
        step("decode-8", decodes=8, context=3072),
        # a server under load: 64 requests of different lengths
        step("decode-64", decodes=64, context=1024),
        # a question of a few lines, the first token's delay
        step("prompt-61", portion=61),
        # the benchmark's prompt: a step's limit of tokens in one portion
        step("prompt-2048", portion=2048),
        # a long document's later portion: attention over what is cached is as much work as the products
        step("prompt-2048-behind-8192", portion=2048, behind=8192),
        # a scheduler's mixed step: a 512-token prompt portion beside the requests that decode, at the 8B widths
        step("mixed-8b", model="8b", decodes=48, context=1200, portion=512, behind=512),
        # a text is scored: logits at each of its tokens; an odd size
        step("score-601", portion=601, every=True),
        # the 32-bit path
        requests("fp32-0.6b", "0.6b", "float32", count=4, prompt=75, tokens=4),
        # a model of recurrent layers: a long prompt and the tokens behind it, and many short requests at once
        requests("fadosun-long", "fadosun", "bfloat16", count=1, prompt=1500, tokens=8),
        requests("fadosun-many", "fadosun", "bfloat16", count=24, prompt=60, tokens=8),
        # the sampler with the model card's options, a batch of 32
        sample("sample-32", rows=32, temperature=0.6, top_k=20, top_p=0.95, min_p=0.0),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    what = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "later", "mixed", "score", "fp32", "fadosun", "fadosun", "sample"])
    page = rng.choice([16, 64, 64, 64])
    if what == "decode":
        batch = _log(rng, 1, 64)
        model = rng.choice(["1.7b", "1.7b", "8b"])
        return _unnamed(step("", model=model, decodes=batch, context=_log(rng, 64, min(8192, 65536 // batch)), page=page))
    if what == "prompt":
        return _unnamed(step("", model=rng.choice(["1.7b", "1.7b", "8b"]), portion=_log(rng, 5, 2048), page=page))
    if what == "later":
        return _unnamed(step("", portion=_log(rng, 200, 2048), behind=rng.randrange(1, 8193), page=page))
    if what == "mixed":
        return _unnamed(step("", model=rng.choice(["1.7b", "8b"]), decodes=_log(rng, 2, 60), context=_log(rng, 64, 1024),
                             portion=_log(rng, 30, 1024), behind=rng.choice([0, rng.randrange(1, 2048)]), page=page))
    if what == "score":
        return _unnamed(step("", portion=_log(rng, 20, 800), every=True, page=page))
    if what == "fp32":
        return _unnamed(requests("", "0.6b", "float32", count=_log(rng, 1, 8), prompt=_log(rng, 5, 80), tokens=rng.randrange(1, 6), page=page))
    if what == "fadosun":
        count = _log(rng, 1, 32)
        return _unnamed(requests("", "fadosun", "bfloat16", count=count, prompt=_log(rng, 5, min(1500, 2048 // count)), tokens=rng.randrange(1, 9), page=page))
    return _unnamed(sample("", rows=_log(rng, 1, 64), temperature=round(rng.uniform(0.2, 1.2), 2), top_k=rng.choice([0, 20, 40, rng.randrange(1, 200)]),
                           top_p=rng.choice([1.0, 0.8, 0.95]), min_p=rng.choice([0.0, 0.0, 0.05])))


def _unnamed(case):
    del case["name"]
    return case


def contexts(case):
    """Cached tokens of each decoding request: spread between half of ``context`` and all of it (one or eight requests,
    as the benchmark has them, hold all of it)."""
    n, c = case["decodes"], case["context"]
    return [c if n in (1, 8) else c - (i * (c // 2)) // n for i in range(n)]


def steps_of(lengths):
    """Prompts packed into steps of at most STEP_TOKENS tokens: [[(request, first, stop), ...], ...]."""
    out, room = [[]], STEP_TOKENS
    for r, n in enumerate(lengths):
        at = 0
        while at < n:
            if not room:
                out.append([])
                room = STEP_TOKENS
            m = min(room, n - at)
            out[-1].append((r, at, at + m))
            at, room = at + m, room - m
    return [s for s in out if s]


# ------------------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 1)


def _qwen3_names(m):
    h, q, kv = m["hidden"], m["heads"] * HEAD, m["kv_heads"] * HEAD
    yield "model.embed_tokens.weight", (VOCAB, h)
    for i in range(m["layers"]):
        p = "model.layers.%d." % i
        yield p + "input_layernorm.weight", (h,)
        yield p + "self_attn.q_proj.weight", (q, h)
        yield p + "self_attn.k_proj.weight", (kv, h)
        yield p + "self_attn.v_proj.weight", (kv, h)
        yield p + "self_attn.q_norm.weight", (HEAD,)
        yield p + "self_attn.k_norm.weight", (HEAD,)
        yield p + "self_attn.o_proj.weight", (h, q)
        yield p + "post_attention_layernorm.weight", (h,)
        yield p + "mlp.gate_proj.weight", (m["inter"], h)
        yield p + "mlp.up_proj.weight", (m["inter"], h)
        yield p + "mlp.down_proj.weight", (h, m["inter"])
    yield "model.norm.weight", (h,)
    if not m["tied"]:
        yield "lm_head.weight", (VOCAB, h)


def _fadosun_names():
    """(name, shape, range): range None for a matrix, "norm" for norm weights, "bias", or (low, high)."""
    w, f = FADOSUN_WIDTH, FADOSUN_FF
    yield "embed", (VOCAB, w), None
    yield "head", (VOCAB, w), None
    yield "final.norm", (w,), "norm"
    yield "final.norm.b", (w,), "bias"
    for i, layer in enumerate(FADOSUN_LAYERS):
        p, x, m = "l%d." % i, "l%d.mix." % i, layer["mixer"]
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            yield p + n, (w,), "norm"
            yield p + n + ".b", (w,), "bias"
        for n in ("rg1", "rg2"):
            yield p + n, (w, w), None
            yield p + n + ".b", (w,), "bias"
        for n in ("gate", "up"):
            yield p + "mlp." + n, (f, w), None
        yield p + "mlp.down", (w, f), None
        if layer["type"] == "channel_delta":
            inner = m["heads"] * m["dim"]
            for n in ("q", "k", "v"):
                yield x + n, (inner, w), None
                yield x + n + ".conv", (inner, m["conv"]), (-0.5, 0.5)
            yield x + "b", (m["heads"], w), None
            yield x + "A_log", (m["heads"],), (-1.0, 1.0)
            yield x + "norm", (m["vdim"],), "norm"
            yield x + "dt_bias", (inner,), (-3.0, 0.0)
            yield x + "o", (w, inner), None
            for n, rank in (("a", m["decay_rank"]), ("g", m["gate_rank"])):
                yield x + n + "1", (rank, w), None
                yield x + n + "2", (inner, rank), None
        elif layer["type"] == "mlstm":
            d, v = m["heads"] * m["dim"], m["heads"] * m["vdim"]
            for n, rows in (("q", d), ("k", d), ("v", v), ("g", v)):
                yield x + n, (rows, w), None
            yield x + "o", (w, v), None
            yield x + "norm", (v,), "norm"
            yield x + "i", (m["heads"], w), None
            yield x + "i.b", (m["heads"],), (-1.0, 1.0)
            yield x + "f", (m["heads"], w), None
            yield x + "f.b", (m["heads"],), (1.0, 4.0)
        else:
            a, b = m["left"], m["right"]
            for n, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                yield x + "left." + n, (rows, w), None
            yield x + "left.pb", (a["heads"],), (-4.0, -2.0)
            yield x + "left.o", (w, a["heads"] * a["vdim"]), None
            inner, mixed = b["heads"] * b["vdim"], b["heads"] * b["vdim"] + 2 * b["groups"] * b["state"]
            yield x + "right.in", (inner + mixed + b["heads"], w), None
            yield x + "right.conv", (mixed, b["conv"]), (-0.5, 0.5)
            yield x + "right.conv.b", (mixed,), "bias"
            yield x + "right.dt_bias", (b["heads"],), (-3.0, -1.0)
            yield x + "right.A_log", (b["heads"],), (0.0, 2.0)
            yield x + "right.D", (b["heads"],), "norm"
            yield x + "right.norm", (inner,), "norm"
            yield x + "right.o", (w, inner), None


def weights(model, seed):
    g, out = _generator(seed), {}
    named = _fadosun_names() if model == "fadosun" else (
        (n, s, "norm" if len(s) == 1 else None) for n, s in _qwen3_names(QWEN3[model]))
    for name, shape, kind in named:
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        if isinstance(kind, tuple):
            t.uniform_(kind[0], kind[1], generator=g)
        elif kind == "norm":
            t.copy_(torch.empty(shape, device="cuda").normal_(1.0, 0.05, generator=g))
        else:
            t.normal_(0.0, 0.02, generator=g)
        out[name] = t
    return out


def texts(seed, lengths):
    """Token ids, host lists as a tokenizer gives them."""
    g = torch.Generator().manual_seed(int(seed) + 2)
    return [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in lengths]


def lengths_of(case):
    """Tokens of every request of a case, those of the pass included."""
    if case["kind"] == "requests":
        return [case["prompt"] + case["tokens"]] * case["count"]
    return [c + 1 for c in contexts(case)] + ([case["behind"] + case["portion"]] if case["portion"] else [])


def model_config(model):
    if model == "fadosun":
        return FadosunConfig.from_json({"architecture": "Fadosun", "vocab": VOCAB, "width": FADOSUN_WIDTH, "norm": {"eps": EPS},
                                        "layers": [dict(l, mlp={"kind": "dense", "ff": FADOSUN_FF}) for l in FADOSUN_LAYERS]})
    m = QWEN3[model]
    return Qwen3Config.from_json(dict(
        architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=VOCAB, hidden_size=m["hidden"], intermediate_size=m["inter"],
        num_hidden_layers=m["layers"], num_attention_heads=m["heads"], num_key_value_heads=m["kv_heads"], head_dim=HEAD, rope_theta=THETA,
        rms_norm_eps=EPS, tie_word_embeddings=m["tied"], max_position_embeddings=40960))


def sampler_logits(case, seed):
    """Rows of logits as a model gives them: normal, a few words far above the rest."""
    g = _generator(seed)
    x = torch.empty(case["rows"], VOCAB, device="cuda").normal_(0.0, 2.0, generator=g)
    at = torch.randint(0, VOCAB, (case["rows"], 30), generator=g, device="cuda")
    return x.scatter_(1, at, torch.empty(case["rows"], 30, device="cuda").uniform_(6.0, 16.0, generator=g))


def prepare(case, seed):
    if case["kind"] == "sample":
        logits = sampler_logits(case, seed)
        params = [SamplingParams(temperature=case["temperature"], top_p=case["top_p"], top_k=case["top_k"], min_p=case["min_p"],
                                 seed=1 + seed + i) for i in range(case["rows"])]
        return {"case": case, "logits": logits, "params": params, "counters": [100 + 3 * i for i in range(case["rows"])],
                "out": torch.empty(case["rows"], dtype=torch.int32, device="cuda")}
    lengths, page = lengths_of(case), case["page"]
    room = sum((n + page - 1) // page * page for n in lengths)
    runner = ModelRunner(model_config(case["model"]).to_model_spec(), WeightStore.from_tensors(weights(case["model"], seed)), dtype=case["dtype"],
                         capacity_tokens=room, max_batch_tokens=STEP_TOKENS, max_requests=max(8, len(lengths)), page_tokens=page)
    llm = LLM(runner)
    ids = texts(seed, lengths)
    state = {"case": case, "llm": llm, "ids": ids}
    if case["kind"] == "step":
        held = contexts(case) + ([case["behind"]] if case["portion"] else [])
        for r in range(len(held)):
            assert runner.admit(r)
        for part in steps_of(held):
            for r, first, stop in part:
                assert runner.reserve(r, stop - first)
            llm.step([StepEntry(r, ids[r][first:stop]) for r, first, stop in part])
        runner.check_device()
        state["held"] = held
        wanted = [(0,)] * case["decodes"]
        if case["portion"]:
            wanted.append(tuple(range(case["portion"])) if case["every"] else (case["portion"] - 1,))
        state["entries"] = [StepEntry(r, ids[r][n:], wanted[r]) for r, n in enumerate(held)]
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return device_sampler.sample(state["logits"], state["params"], state["counters"], out=state["out"])
    llm, ids = state["llm"], state["ids"]
    runner = llm.runner
    if case["kind"] == "step":
        for e in state["entries"]:
            assert runner.reserve(e.request, len(e.tokens))
        logits = llm.step(state["entries"])
        for r, n in enumerate(state["held"]):
            runner.cache.advance(r, n)
        return logits
    count, prompt, outs = case["count"], case["prompt"], []
    for r in range(count):
        assert runner.admit(r)
    for part in steps_of([prompt] * count):
        for r, first, stop in part:
            assert runner.reserve(r, stop - first)
        logits = llm.step([StepEntry(r, ids[r][first:stop], (stop - first - 1,) if stop == prompt else ()) for r, first, stop in part])
        if logits is not None:
            outs.append(logits.clone())
    outs = [torch.cat(outs) if len(outs) > 1 else outs[0]]
    for t in range(case["tokens"]):
        for r in range(count):
            assert runner.reserve(r, 1)
        outs.append(llm.step([StepEntry(r, ids[r][prompt + t:prompt + t + 1], (0,)) for r in range(count)]).clone())
    for r in range(count):
        runner.release(r)
    return outs


# -------------------------------------------------------------------------------------------------------------- work
def work(case):
    if case["kind"] == "sample":
        return {"bytes": case["rows"] * (4.0 * VOCAB + 4), "flops": 0.0}
    size = 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "step":
        runs = [[(c, 1, 1) for c in contexts(case)]]                    # one step: (cached, new, wanted) of each run
        if case["portion"]:
            runs[0].append((case["behind"], case["portion"], case["portion"] if case["every"] else 1))
    else:
        runs = [[(a, b - a, int(b == case["prompt"])) for _, a, b in part] for part in steps_of([case["prompt"]] * case["count"])]
        runs += [[(case["prompt"] + t, 1, 1)] * case["count"] for t in range(case["tokens"])]
    if case["model"] == "fadosun":
        h, matrices, vectors, state = FADOSUN_WIDTH, 0, 0, 0
        for name, shape, kind in _fadosun_names():
            if name not in ("embed", "head"):
                matrices += shape[0] * shape[1] if kind is None else 0
                vectors += math.prod(shape) if kind is not None else 0
        kv = heads = 0
        for layer in FADOSUN_LAYERS:
            m = layer["mixer"]
            if layer["type"] == "channel_delta":
                state += m["heads"] * m["dim"] * m["vdim"]
            elif layer["type"] == "mlstm":
                state += m["heads"] * m["dim"] * (m["vdim"] + 1)
            else:
                state += m["right"]["heads"] * m["right"]["vdim"] * m["right"]["state"]
                kv += 2 * m["left"]["kv_heads"] * m["left"]["dim"]
                heads += m["left"]["heads"]
    else:
        m = QWEN3[case["model"]]
        h, q, g = m["hidden"], m["heads"] * HEAD, m["kv_heads"] * HEAD
        matrices = m["layers"] * (h * (q + 2 * g) + q * h + 3 * h * m["inter"])
        vectors, state = m["layers"] * (2 * h + 2 * HEAD) + h, 0
        kv, heads = 2 * m["layers"] * g, m["layers"] * m["heads"]
    total_bytes = total_flops = 0.0
    for one in runs:
        new, wanted = sum(n for _, n, _ in one), sum(w for _, _, w in one)
        pairs = sum(n * c + n * (n + 1) // 2 for c, n, _ in one)
        total_bytes += size * (matrices + (VOCAB * h if wanted else 0) + new * h) + 2 * vectors
        total_bytes += size * kv * sum(c + 2 * n for c, n, _ in one) + 8.0 * state * len(one) + 4.0 * wanted * VOCAB
        # each recurrence at least decays its state, adds to it and reads it
        total_flops += 2.0 * new * matrices + 2.0 * wanted * VOCAB * h + 4.0 * HEAD * heads * pairs + 6.0 * state * new
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-4}              # (2.3e-6 from the 64-bit values)
    return {"rel": 3e-2, "max": 0.25}                  # (1e-2 between two orders of the same sums, 2e-2 from the 64-bit values)


# ------------------------------------------------------------------------------------------------- 64-bit statements
def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _layer_norm(x, w, b):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt((d * d).mean(-1, keepdim=True) + EPS) * w + b


def _rotate(x, positions, dims, base):
    """Pairs (i, i + dims / 2) of the first ``dims`` entries turn by position * base^(-2i / dims), the angle a 32-bit product."""
    half = dims // 2
    inv = (1.0 / torch.tensor(base, dtype=torch.float32) ** (torch.arange(half, dtype=torch.float32) * 2 / dims)).to(x.device)
    a = (positions.to(torch.float32)[:, None] * inv).to(x.dtype)[:, None, :]
    u, w = x[..., :half], x[..., half:dims]
    return torch.cat([u * torch.cos(a) - w * torch.sin(a), w * torch.cos(a) + u * torch.sin(a), x[..., dims:]], -1)


def _attend(q, k, v, first, weigh):
    """Rows ``first``.. of a causal sequence: q [T, H, D] against k, v [first + T, G, D]."""
    group = q.shape[1] // k.shape[1]
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    for a in range(0, q.shape[0], 1024):
        b = min(a + 1024, q.shape[0])
        seen = torch.arange(first + b, device=q.device)[None, :] <= torch.arange(first + a, first + b, device=q.device)[:, None]
        for h in range(q.shape[1]):
            out[a:b, h] = weigh(q[a:b, h] @ k[:first + b, h // group].T, seen, h) @ v[:first + b, h // group]
    return out


def _qwen3_logits(model, w, tokens, want):
    """Logits of one sequence at the places ``want``, one layer's weights in 64 bits at a time."""
    m, dev = QWEN3[model], "cuda"
    wide = lambda n: w[n].double()                                                      # noqa: E731
    T, pos = len(tokens), torch.arange(len(tokens), device=dev)
    x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=dev)].double()
    scale = HEAD ** -0.5
    softmax = lambda s, seen, h: torch.softmax((s * scale).masked_fill(~seen, float("-inf")), -1)    # noqa: E731
    for i in range(m["layers"]):
        p = "model.layers.%d." % i
        n = _rms(x, wide(p + "input_layernorm.weight"))
        q, k, v = ((n @ wide(p + "self_attn.%s_proj.weight" % s).T).view(T, -1, HEAD) for s in "qkv")
        q = _rotate(_rms(q, wide(p + "self_attn.q_norm.weight")), pos, HEAD, THETA)
        k = _rotate(_rms(k, wide(p + "self_attn.k_norm.weight")), pos, HEAD, THETA)
        if i == m["layers"] - 1:                     # nothing reads the last layer's other rows
            rows = torch.tensor(want, device=dev)
            low = min(want)
            o = _attend(q[low:], k, v, low, softmax)[rows - low].reshape(len(want), -1)
            x = x[rows] + o @ wide(p + "self_attn.o_proj.weight").T
        else:
            x = x + _attend(q, k, v, 0, softmax).reshape(T, -1) @ wide(p + "self_attn.o_proj.weight").T
        n = _rms(x, wide(p + "post_attention_layernorm.weight"))
        x = x + (F.silu(n @ wide(p + "mlp.gate_proj.weight").T) * (n @ wide(p + "mlp.up_proj.weight").T)) @ wide(p + "mlp.down_proj.weight").T
    return _rms(x, wide("model.norm.weight")) @ wide("model.embed_tokens.weight" if m["tied"] else "lm_head.weight").T


def _conv(x, taps):
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(n))


def _channel_delta(h, w, p, m):
    T, H, D, V = h.shape[0], m["heads"], m["dim"], m["vdim"]
    q, k, v = (F.silu(_conv(h @ w(p + n).T, w(p + n + ".conv"))).view(T, H, -1) for n in "qkv")
    q = q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5
    k = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(h @ w(p + "b").T)
    decay = torch.exp(-torch.exp(w(p + "A_log"))[:, None] * F.softplus((h @ w(p + "a1").T) @ w(p + "a2").T + w(p + "dt_bias")).view(T, H, D))
    S, out = h.new_zeros(H, D, V), []
    for t in range(T):
        S = S * decay[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    gate = torch.sigmoid((h @ w(p + "g1").T) @ w(p + "g2").T).view(T, H, V)
    return (_rms(torch.stack(out), w(p + "norm")) * gate).reshape(T, H * V) @ w(p + "o").T


def _mlstm(h, w, p, m):
    T, H, D, V, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = (h @ w(p + "q").T * D ** -0.5).view(T, H, D), (h @ w(p + "k").T).view(T, H, D), (h @ w(p + "v").T).view(T, H, V)
    i = cap * torch.tanh((h @ w(p + "i").T + w(p + "i.b")) / cap)
    f = F.logsigmoid(cap * torch.tanh((h @ w(p + "f").T + w(p + "f.b")) / cap))
    S, n, top, out = h.new_zeros(H, D, V), h.new_zeros(H, D), h.new_zeros(H), []
    for t in range(T):
        new = torch.maximum(f[t] + top, i[t])
        keep, put = torch.exp(f[t] + top - new), torch.exp(i[t] - new)
        S = keep[:, None, None] * S + put[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
        n = keep[:, None] * n + put[:, None] * k[t]
        top = new
        below = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out.append(torch.einsum("hdv,hd->hv", S, q[t]) / below[:, None])
    return (_rms(torch.stack(out), 1.0).reshape(T, H * V) * w(p + "norm") * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T


def _sigmoid_attention(h, w, p, m):
    T, pos = h.shape[0], torch.arange(h.shape[0], device=h.device)
    q, k, v = (h @ w(p + "q").T).view(T, -1, m["dim"]), (h @ w(p + "k").T).view(T, -1, m["dim"]), (h @ w(p + "v").T).view(T, -1, m["vdim"])
    q, k = (_rotate(x, pos, m["rot"]["dims"], m["rot"]["base"]) for x in (q, k))
    bias = w(p + "pb")
    o = _attend(q, k, v, 0, lambda s, seen, i: torch.sigmoid(s * m["scale"] + bias[i]) * seen)
    return o.reshape(T, -1) @ w(p + "o").T


def _state_space(h, w, p, m):
    T, H, V, N = h.shape[0], m["heads"], m["vdim"], m["state"]
    z, mixed, dt = (h @ w(p + "in").T).split([H * V, H * V + 2 * N, H], dim=-1)
    x, B, C = F.silu(_conv(mixed, w(p + "conv")) + w(p + "conv.b")).split([H * V, N, N], dim=-1)
    x, dt = x.reshape(T, H, V), F.softplus(dt + w(p + "dt_bias"))
    decay = torch.exp(-torch.exp(w(p + "A_log")) * dt)
    S, out = h.new_zeros(H, N, V), []
    for t in range(T):
        S = decay[t][:, None, None] * S + B[t][None, :, None] * (dt[t][:, None] * x[t])[:, None, :]
        out.append(torch.einsum("hnv,n->hv", S, C[t]))
    y = (torch.stack(out) + w(p + "D")[:, None] * x).reshape(T, H * V) * F.silu(z)
    return _rms(y, w(p + "norm")) @ w(p + "o").T


def _fadosun_logits(weights_, tokens, want):
    w = lambda n: weights_[n].double()                                                  # noqa: E731
    norm = lambda n, t: _layer_norm(t, w(n), w(n + ".b"))                               # noqa: E731
    x = weights_["embed"][torch.tensor(tokens, device="cuda")].double()
    for i, layer in enumerate(FADOSUN_LAYERS):
        p, m = "l%d." % i, layer["mixer"]
        h = norm(p + "norm1", x)
        if layer["type"] == "channel_delta":
            y = _channel_delta(h, w, p + "mix.", m)
        elif layer["type"] == "mlstm":
            y = _mlstm(h, w, p + "mix.", m)
        else:
            y = m["left_scale"] * _sigmoid_attention(h, w, p + "mix.left.", m["left"]) + m["right_scale"] * _state_space(h, w, p + "mix.right.", m["right"])
        x = x + norm(p + "norm1b", y * torch.sigmoid(h @ w(p + "rg1").T + w(p + "rg1.b")))
        h = norm(p + "norm2", x)
        y = (torch.relu(h @ w(p + "mlp.gate").T) * (h @ w(p + "mlp.up").T)) @ w(p + "mlp.down").T
        x = x + norm(p + "norm2b", y * torch.sigmoid(h @ w(p + "rg2").T + w(p + "rg2.b")))
    return norm("final.norm", x[torch.tensor(want, device="cuda")]) @ w("head").T


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    w, ids = weights(case["model"], seed), texts(seed, lengths_of(case))
    logits = _fadosun_logits if case["model"] == "fadosun" else lambda *a: _qwen3_logits(case["model"], *a)
    if case["kind"] == "step":
        rows = []
        for r, text in enumerate(ids):
            every = case["every"] and r == case["decodes"]
            rows.append(logits(w, text, list(range(case["behind"], len(text))) if every else [len(text) - 1]))
        return torch.cat(rows)
    want = list(range(case["prompt"] - 1, case["prompt"] + case["tokens"]))
    rows = torch.stack([logits(w, text, want) for text in ids], 1)
    return list(rows)
