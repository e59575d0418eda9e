"""What a user of this framework has it do, as cases that can be timed and compared.

A case is one call of the step function (``ModelRunner.step``) on a model of one of the named
presets, or one draw of the device sampler, with what such a call meets in a serving program:

``decode``  one token for each of ``batch`` live requests whose lengths spread around ``context``.
            Requests that keep only keys and values are rewound behind the step
            (``cache.truncate``), so every pass decodes at the same place; a request with recurrent
            state cannot be rewound and moves on by a token a pass.
``prompt``  one prompt of ``tokens`` tokens into an empty request, logits at ``wants`` places
            spread to its end, then the request is closed.
``mixed``   a serving step: ``batch`` decoded tokens beside ``portions`` portions of prompts,
            ``tokens`` rows in all, some of the portions starting where an earlier one ended.
``sample``  the sampling chain on the logits of ``batch`` requests (temperature, top-k, top-p,
            min-p), tokens back on the host.

``preset`` names the sizes, ``layers`` how many of its layers run.  Weights are the framework's own
seeded random ones.  Two things are arranged as training leaves them, so that rounding does not grow
from layer to layer: a layer of the pre-norm models adds little to its residual stream, and the
experts of a token are clear (a coin toss between two would compare coins, not kernels).
"""
import math
import random

import torch

from llmario_b200 import Model, ModelRunner, SamplingParams, StepEntry
from llmario_b200.cli import PRESETS, preset_config
from llmario_b200.sampling.sampler import DeviceSampler, RequestSampler
from llmario_b200.weights import random_tensors
from llmario_b200.weights.loader import expected_tensors

DEV = "cuda:0"
F64 = torch.float64
RECURRENT = ("vunasun", "pavatar")      # their requests carry a state that cannot be rewound
CLUSTERS = 28                           # kinds of tokens of a routed model: pairs of eight experts


def listed():
    return [
        # a single user chatting with a small model: the least work a step can have
        dict(name="decode-1", kind="decode", preset="qwen3-0.6b", layers=28, dtype="bfloat16",
             batch=1, context=500, page=64),
        # the framework's headline: eight requests on the whole 8B model, pages of 16
        dict(name="decode-8", kind="decode", preset="qwen3-8b", layers=36, dtype="bfloat16",
             batch=8, context=1024, page=16),
        # a busy server: 64 requests of ragged lengths, where the cache weighs beside the weights
        dict(name="decode-64", kind="decode", preset="qwen3-8b", layers=8, dtype="bfloat16",
             batch=64, context=1400, page=64),
        # what follows every decode step of that server
        dict(name="sample-64", kind="sample", preset="qwen3-8b", batch=64),
        # the named prompt of the whole 8B model
        dict(name="prompt-2048", kind="prompt", preset="qwen3-8b", layers=36, dtype="bfloat16",
             tokens=2048, wants=16, page=16),
        # a long document, where attention weighs beside the products
        dict(name="prompt-8192", kind="prompt", preset="qwen3-8b", layers=12, dtype="bfloat16",
             tokens=8192, wants=16, page=64),
        # continuous batching on a small model: ragged portions beside decoded tokens
        dict(name="mixed-777", kind="mixed", preset="qwen3-0.6b", layers=28, dtype="bfloat16",
             batch=24, portions=4, tokens=777, context=900, page=64),
        # the true 32-bit path, used to check a model
        dict(name="prompt-211-float32", kind="prompt", preset="qwen3-0.6b", layers=28,
             dtype="float32", tokens=211, wants=16, page=64),
        # recurrent layers (gated linear attention, state-space mixer) beside chunked attention
        dict(name="recurrent-prompt-2048", kind="prompt", preset="vunasun-0.6b", layers=8,
             dtype="bfloat16", tokens=2048, wants=16, page=64),
        dict(name="recurrent-decode-32", kind="decode", preset="vunasun-8b", layers=8,
             dtype="bfloat16", batch=32, context=700, page=64),
        # the delta rule, attention and routed experts, an odd length
        dict(name="delta-prompt-1501", kind="prompt", preset="pavatar-8b", layers=8,
             dtype="bfloat16", tokens=1501, wants=16, page=64),
        # attention through latents and routed experts, one token for each of 16 requests
        dict(name="latent-decode-16", kind="decode", preset="momuvik-8b", layers=8,
             dtype="bfloat16", batch=16, context=1800, page=64),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prompt", "prompt", "prompt", "mixed",
                       "sample"))
    if kind == "sample":
        return dict(kind=kind, preset="qwen3-8b", batch=_spread(rng, 1, 96))
    small = rng.random() < 0.5
    size = "0.6b" if small else "8b"
    layers = rng.randint(4, 16 if small else 10)
    page = rng.choice((16, 64))
    if kind == "mixed":
        tokens = _spread(rng, 100, 2048)
        return dict(kind=kind, preset="qwen3-" + size, layers=layers, dtype="bfloat16",
                    batch=_spread(rng, 1, 48), portions=rng.randint(1, 6), tokens=tokens,
                    context=_spread(rng, 64, 1500), page=page)
    family = rng.choice(("qwen3", "qwen3", "qwen3", "vunasun", "momuvik")
                        + (("pavatar",) if kind == "prompt" else ()))
    if kind == "decode":
        batch = _spread(rng, 1, 64)
        return dict(kind=kind, preset=f"{family}-{size}", layers=layers, dtype="bfloat16",
                    batch=batch, context=_spread(rng, 64, min(4096, 90000 // batch)), page=page)
    dtype = "float32" if family == "qwen3" and small and rng.random() < 0.25 else "bfloat16"
    tokens = _spread(rng, 16, 512 if dtype == "float32" else 8192 if family == "qwen3" else 3072)
    return dict(kind=kind, preset=f"{family}-{size}", layers=layers, dtype=dtype, tokens=tokens,
                wants=min(16, tokens), page=page)


# ----------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------
def _family(case):
    return case["preset"].split("-")[0]


def _weights(case, spec, seed):
    """Every tensor of the model.  Pre-norm models get a wide embedding and small output
    projections (a GPT-2's initialisation: 1 / sqrt(2 layers)).  For routed models the embedding
    has a direction per kind of token and each router answers to it, two experts to a kind."""
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    w = random_tensors(spec, seed, dtype, DEV)
    if _family(case) == "qwen3":
        w["model.embed_tokens.weight"].mul_(25.0)
        for n in w:
            if n.endswith(("o_proj.weight", "down_proj.weight")):
                w[n].mul_((2 * case["layers"]) ** -0.5)
    routers = [n for n in w if n.endswith(".router")]
    if routers:
        g = torch.Generator(DEV).manual_seed(seed * 2 + 1)
        vocab, width = w["embed"].shape
        kinds = torch.randn(CLUSTERS, width, device=DEV, generator=g)
        own = torch.randn(vocab, width, device=DEV, generator=g)
        w["embed"] = (kinds[torch.arange(vocab, device=DEV) % CLUSTERS] + 0.5 * own).to(dtype)
        pairs = [(a, b) for a in range(8) for b in range(a)]
        for n in routers:
            r = 0.002 * torch.randn(w[n].shape, device=DEV, generator=g)
            for kind, pair in enumerate(pairs):
                for e in pair:
                    r[e] += 0.15 * kinds[kind] / width ** 0.5
            w[n] = r.to(w[n].dtype)
    return w


def _sequences(case, seed):
    """Per request: its tokens so far, the tokens of the step, and the places whose logits are
    wanted (within the step's tokens)."""
    rng = random.Random(seed)
    vocab = PRESETS["qwen3-8b"]["vocab_size"]
    toks = lambda n: [rng.randrange(vocab) for _ in range(n)]  # noqa: E731
    kind = case["kind"]
    if kind == "prompt":
        n, k = case["tokens"], case["wants"]
        return [([], toks(n), [n * (i + 1) // k - 1 for i in range(k)])]
    shape = random.Random(case["batch"])      # lengths belong to the case, not to the seed
    context = case["context"]
    lengths = [max(1, int(context * shape.uniform(0.5, 1.5))) for _ in range(case["batch"])]
    if case["batch"] == 1:
        lengths = [context]
    out = [(toks(n), toks(1), [0]) for n in lengths]
    if kind == "mixed":
        left = max(case["portions"], case["tokens"] - case["batch"])
        cuts = sorted(shape.sample(range(1, left), case["portions"] - 1)) if left > 1 else []
        for i, (a, b) in enumerate(zip([0] + cuts, cuts + [left])):
            n = b - a
            before = 0 if i % 2 == 0 else shape.randint(1, context)
            out.append((toks(before), toks(n), [n - 1]))
    return out


def prepare(case, seed):
    if case["kind"] == "sample":
        vocab = PRESETS[case["preset"]]["vocab_size"]
        g = torch.Generator(DEV).manual_seed(seed)
        logits = 2.5 * torch.randn(case["batch"], vocab, device=DEV, generator=g)
        params = [SamplingParams(temperature=0.7, top_k=40, top_p=0.9, seed=seed),
                  SamplingParams(temperature=1.0, top_p=0.95, seed=seed),
                  SamplingParams(temperature=0.8, min_p=0.05, seed=seed),
                  SamplingParams(temperature=0.0)]
        samplers = [RequestSampler(params[i % 4], vocab) for i in range(case["batch"])]
        return {"kind": "sample", "sampler": DeviceSampler(DEV), "samplers": samplers,
                "logits": logits}
    spec = preset_config(case["preset"], case["layers"]).to_spec()
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    weights = _weights(case, spec, seed)
    model = Model(spec, weights, dtype, DEV)
    weights.clear()
    seqs = _sequences(case, seed)
    grows = _family(case) in RECURRENT and case["kind"] == "decode"
    room = 32768 if grows else 0      # for the passes to come
    page = case["page"]
    rows = sum(len(s[1]) for s in seqs)
    longest = max(len(a) + len(b) for a, b, _ in seqs) + room + page
    # (a recurrent model's attention looks back over a chunk of 1,024 positions at most)
    held = [len(a) + (2048 + 2 * page if grows else len(b)) for a, b, _ in seqs]
    runner = ModelRunner(model, page_size=page, max_requests=len(seqs) + 1, max_context=longest,
                         n_pages=sum(-(-n // page) + 1 for n in held) + 1,
                         token_budget=max(rows, 2048))
    entries = []
    for i, (before, step, want) in enumerate(seqs):
        for at in range(0, len(before), 2048):
            runner.step([StepEntry(i, before[at:at + 2048], [])])
        entries.append(StepEntry(i, step, want))
    return {"kind": case["kind"], "runner": runner, "entries": entries, "grows": grows,
            "before": [len(s[0]) for s in seqs]}


def run(state):
    if state["kind"] == "sample":
        return torch.tensor(state["sampler"].sample(state["logits"], state["samplers"]))
    runner = state["runner"]
    logits = runner.step(state["entries"])
    if not state["grows"]:
        for e, n in zip(state["entries"], state["before"]):
            if n:
                runner.cache.truncate(e.request, n)
            else:
                runner.close(e.request)
    return logits


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4 * case["batch"] * PRESETS[case["preset"]]["vocab_size"], "flops": 0}
    raw = preset_config(case["preset"], case["layers"]).to_dict()
    spec = preset_config(case["preset"], case["layers"]).to_spec()
    shapes = {n: tuple(16 if d is None else d for d in s)
              for n, s in expected_tensors(spec).items()}
    seqs = _sequences(case, 0)
    rows = sum(len(s[1]) for s in seqs)
    wants = sum(len(s[2]) for s in seqs)
    size = 4 if case["dtype"] == "float32" else 2
    head = "lm_head.weight" if "lm_head.weight" in shapes else "head" if "head" in shapes else \
        "model.embed_tokens.weight" if "model.embed_tokens.weight" in shapes else "embed"
    nbytes = flops = 0.0
    for n, s in shapes.items():
        numel = math.prod(s)
        if n == head:
            nbytes, flops = nbytes + size * numel, flops + 2.0 * numel * wants
        elif n in ("embed", "model.embed_tokens.weight"):
            nbytes += size * rows * s[-1]
        elif len(s) == 2:
            # a token uses two of eight experts
            share = 0.25 if ".mlp.e" in n else 1.0
            met = 1.0 - (1.0 - share) ** rows
            nbytes, flops = nbytes + size * numel * met, flops + 2.0 * numel * share * rows
        else:
            nbytes += size * numel
    # attention and recurrences, layer by layer: (channels of a pair's two products, values kept
    # per token, state elements, positions a query sees)
    layers = raw.get("layers")
    family = _family(case)
    if layers is None:
        d, H, G = raw["head_dim"], raw["num_attention_heads"], raw["num_key_value_heads"]
        per = [(2 * H * d, 2 * G * d, 0, 1 << 30)] * raw["num_hidden_layers"]
    else:
        per = []
        for layer in layers:
            m, kind = layer["mixer"], layer["type"]
            if kind == "gla":
                per.append((0, 0, m["heads"] * m["dim"] * m["vdim"], 0))
            elif kind == "mamba2":
                per.append((0, 0, m["heads"] * m["state"] * m["vdim"], 0))
            elif kind == "delta":
                per.append((0, 0, m["heads"] * m["dim"] * m["vdim"], 0))
            elif kind == "parallel":
                a, r = m["left"], m["right"]
                per.append((2 * a["heads"] * a["dim"], 2 * a["kv_heads"] * a["dim"],
                            r["heads"] * r["dim"] * r["vdim"], 1 << 30))
            elif family == "momuvik":
                wide = m["kv_rank"] + m["rot_dim"]
                per.append((m["heads"] * (wide + m["kv_rank"]), wide, 0, 1 << 30))
            else:
                reach = m["mask"]["size"] if m.get("mask") else 1 << 30
                per.append((2 * m["heads"] * m["dim"], 2 * m["kv_heads"] * m["dim"], 0, reach))
    for pair, kept, state, reach in per:
        for before, step, _ in seqs:
            n, p = len(step), len(before)
            seen = sum(min(p + i + 1, reach) for i in range(n)) if reach else 0
            flops += 2.0 * pair * seen + 4.0 * state * n
            nbytes += size * kept * (min(p, reach) + n) + 8.0 * state
    return {"bytes": nbytes + 4.0 * wants * raw.get("vocab_size", raw.get("vocab", 0)),
            "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    # bfloat16: operands are rounded in every layer.  Two orders of the same sums came 0.2 to 0.9 %
    # apart, and 0.2 to 1.7 % from 64 bits (the most with 36 layers, and where a sublayer's output
    # is normed).  float32: 32-bit sums, up to 2e-6 from 64 bits.
    return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 0.03}


# ----------------------------------------------------------------------------------------------
# the same in 64 bits
# ----------------------------------------------------------------------------------------------
def _unit(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _lin(h, w):
    """h W^T in 64 bits, rows in slabs."""
    w = w.to(F64)
    return torch.cat([s @ w.T for s in h.split(16384)])


def _rotate(x, pos, dims, base):
    half = dims // 2
    ang = pos.to(F64)[:, None] * base ** (-2.0 * torch.arange(half, device=DEV, dtype=F64) / dims)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:dims]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


def _attend(q, k, v, scale, spans, chunk=0, sink=None, rows=None):
    """Causal softmax attention of each span of rows on itself, q [T, H, d], k / v [T, G, .]."""
    out = torch.zeros(q.shape[0], q.shape[1], v.shape[2], dtype=F64, device=DEV)
    share = q.shape[1] // k.shape[1]
    for a, b in spans:
        for i in range(a, b, 2048):
            j = min(b, i + 2048)
            first = a if not chunk else a + (i - a) // chunk * chunk
            qi = torch.arange(i, j, device=DEV)[:, None] - a
            ki = torch.arange(first, j, device=DEV)[None] - a
            hide = ki > qi
            if chunk:
                hide = hide | (ki // chunk != qi // chunk)
            for g in range(k.shape[1]):
                heads = slice(g * share, (g + 1) * share)
                s = torch.einsum("ihd,jd->hij", q[i:j, heads], k[first:j, g]) * scale
                s = s.masked_fill(hide, -math.inf)
                if sink is not None:
                    s = torch.cat([s, sink.to(F64)[heads, None, None].expand(-1, j - i, 1)], -1)
                p = torch.softmax(s, -1)[..., :j - first]
                out[i:j, heads] = torch.einsum("hij,jd->ihd", p, v[first:j, g])
    return out.flatten(1)


def _silu_mlp(h, w, p, gate="gate", up="up", down="down"):
    F = torch.nn.functional
    return torch.cat([_lin(F.silu(_lin(s, w[p + gate])) * _lin(s, w[p + up]), w[p + down])
                      for s in h.split(16384)])


def _exact_qwen3(raw, w, tokens, pos, spans):
    eps, d = raw["rms_norm_eps"], raw["head_dim"]
    x = w["model.embed_tokens.weight"][tokens].to(F64)
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        h = _unit(x, eps) * w[p + "input_layernorm.weight"].to(F64)
        q, k, v = (_lin(h, w[a + n + "_proj.weight"]).unflatten(1, (-1, d)) for n in "qkv")
        q = _unit(q, eps) * w[a + "q_norm.weight"].to(F64)
        k = _unit(k, eps) * w[a + "k_norm.weight"].to(F64)
        q, k = (_rotate(t, pos, d, raw["rope_theta"]) for t in (q, k))
        x = x + _lin(_attend(q, k, v, d ** -0.5, spans), w[a + "o_proj.weight"])
        h = _unit(x, eps) * w[p + "post_attention_layernorm.weight"].to(F64)
        x = x + _silu_mlp(h, w, p + "mlp.", "gate_proj.weight", "up_proj.weight",
                          "down_proj.weight")
    return _unit(x, eps) * w["model.norm.weight"].to(F64), \
        w["model.embed_tokens.weight" if raw["tie_word_embeddings"] else "lm_head.weight"]


def _walk(spans, step):
    """Every span's tokens in order, all spans side by side (``step(rows, live)``)."""
    for t in range(max(b - a for a, b in spans)):
        live = [i for i, (a, b) in enumerate(spans) if a + t < b]
        step(torch.tensor([spans[i][0] + t for i in live], device=DEV),
             torch.tensor(live, device=DEV))


def _conv(u, w, spans):
    """Causal convolution per channel; the last column meets the current token."""
    taps = w.shape[1]
    out = torch.empty_like(u)
    for a, b in spans:
        pad = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u[a:b]])
        out[a:b] = sum(pad[j:j + b - a] * w[:, j].to(F64) for j in range(taps))
    return out


def _exact_vunasun(raw, w, tokens, pos, spans):
    F = torch.nn.functional
    eps = raw["norm"]["eps"]
    x = w["embed"][tokens].to(F64)
    n, live = x.shape[0], len(spans)
    for i, layer in enumerate(raw["layers"]):
        L, m, kind = f"l{i}.", layer["mixer"], layer["type"]
        t = lambda name: w[L + "mix." + name].to(F64)  # noqa: E731
        lin = lambda name: _lin(x, w[L + "mix." + name])  # noqa: E731
        if kind == "attention":
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            q = (lin("q") + t("q.b")).view(n, H, d)
            v = (lin("k") + t("k.b")).view(n, G, d)
            q, k = _unit(q, eps) * t("q.norm"), _unit(v, eps) * t("k.norm")
            q, k = (_rotate(z, pos, m["rot"]["dims"], m["rot"]["base"]) for z in (q, k))
            y = _attend(q, k, v, m["scale"], spans, chunk=m["mask"]["size"]).view(n, H, d)
            y = (y * torch.sigmoid(lin("g"))[..., None]).flatten(1)
        elif kind == "gla":
            H, dk, dv = m["heads"], m["dim"], m["vdim"]
            q, k = (lin("q") * dk ** -0.5).view(n, H, dk), lin("k").view(n, H, dk)
            v = lin("v").view(n, H, dv)
            z = _lin(lin("a1"), w[L + "mix.a2"]) + t("a2.b")
            decay = torch.sigmoid(z).pow(1.0 / m["tau"]).view(n, H, dk)
            S = torch.zeros(live, H, dk, dv, dtype=F64, device=DEV)
            y = torch.empty(n, H, dv, dtype=F64, device=DEV)

            def step(r, s):
                S[s] = decay[r][..., None] * S[s] + k[r][..., None] * v[r][:, :, None]
                y[r] = torch.einsum("bhkv,bhk->bhv", S[s], q[r])

            _walk(spans, step)
            y = (_unit(y, eps) * t("norm")).flatten(1) * F.silu(lin("g"))
        else:
            H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            inner = H * P
            z, xbc, dt = lin("in").split([inner, inner + 2 * G * N, H], 1)
            xbc = F.silu(_conv(xbc, w[L + "mix.conv"], spans) + t("conv.b"))
            v = xbc[:, :inner].reshape(n, H, P)
            B, C = (c.reshape(n, G, N).repeat_interleave(H // G, 1)
                    for c in xbc[:, inner:].split(G * N, 1))
            dt = F.softplus(dt + t("dt_bias"))
            decay = torch.exp(-torch.exp(t("A_log")) * dt)
            S = torch.zeros(live, H, N, P, dtype=F64, device=DEV)
            y = torch.empty(n, H, P, dtype=F64, device=DEV)

            def step(r, s):
                S[s] = decay[r][..., None, None] * S[s] + \
                    (dt[r][..., None] * B[r])[..., None] * v[r][:, :, None]
                y[r] = torch.einsum("bhkv,bhk->bhv", S[s], C[r])

            _walk(spans, step)
            y = (y + t("D")[:, None] * v).flatten(1) * F.silu(z)
            y = _unit(y.view(n, m["norm_groups"], -1), eps).flatten(1) * t("norm")
        y = _lin(y, w[L + "mix.o"])
        x = x + _unit(y, eps) * w[L + "norm1"].to(F64) * w[L + "ls1"].to(F64)
        y = _silu_mlp(x, w, L + "mlp.")
        x = x + _unit(y, eps) * w[L + "norm2"].to(F64) * w[L + "ls2"].to(F64)
    return _unit(x, eps) * w["final.norm"].to(F64), w["head"]


def _exact_delta(h, t, m, eps, spans, low_rank):
    F = torch.nn.functional
    n, H, G, d, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (F.silu(_conv(_lin(h, t(c)), t(c + ".conv"), spans)) for c in "qkv")
    q, k = (z.view(n, G, d) for z in (q, k))
    q, k = (z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
    q, k = ((z * f).repeat_interleave(H // G, 1) for z, f in ((q, d ** -0.5), (k, 1.0)))
    v, beta, rate = v.view(n, H, dv), torch.sigmoid(_lin(h, t("b"))), t("A_log").to(F64).exp()
    if low_rank:
        z = (_lin(_lin(h, t("a1")), t("a2")) + t("dt_bias").to(F64)).view(n, H, d)
        gate = torch.sigmoid(_lin(_lin(h, t("g1")), t("g2")))
    else:
        z = (_lin(h, t("a")) + t("dt_bias").to(F64))[..., None]
        gate = F.silu(_lin(h, t("g")))
    decay = torch.exp(-rate[:, None] * F.softplus(z))
    S = torch.zeros(len(spans), H, d, dv, dtype=F64, device=DEV)
    y = torch.empty(n, H, dv, dtype=F64, device=DEV)

    def step(r, s):
        now = decay[r][..., None] * S[s]
        u = beta[r][..., None] * (v[r] - torch.einsum("bhkv,bhk->bhv", now, k[r]))
        S[s] = now + k[r][..., None] * u[:, :, None]
        y[r] = torch.einsum("bhkv,bhk->bhv", S[s], q[r])

    _walk(spans, step)
    return _lin((_unit(y, eps) * t("norm").to(F64)).flatten(1) * gate, t("o"))


def _exact_pavatar(raw, w, tokens, pos, spans):
    eps = raw["norm"]["eps"]
    x = w["embed"][tokens].to(F64) * raw["embedding"]["scale"]
    n, first = x.shape[0], None
    for i, layer in enumerate(raw["layers"]):
        L, m, kind = f"l{i}.", layer["mixer"], layer["type"]
        t = lambda name: w[L + "mix." + name]  # noqa: E731
        h = _unit(x, eps) * w[L + "norm1"].to(F64)
        if kind == "delta":
            y = _exact_delta(h, t, m, eps, spans, False)
        elif kind == "parallel":
            a = m["left"]
            q, k, v = (_lin(h, t("left." + c)).view(n, -1, a["dim"]) for c in "qkv")
            q = _unit(q, eps) * t("left.q.norm").to(F64)
            k = _unit(k, eps) * t("left.k.norm").to(F64)
            q, k = (_rotate(z, pos, a["rot"]["dims"], a["rot"]["base"]) for z in (q, k))
            left = _attend(q, k, v, a["scale"], spans) * torch.sigmoid(_lin(h, t("left.g")))
            left = _lin(left, t("left.o"))
            right = _exact_delta(h, lambda c: t("right." + c), m["right"], eps, spans, True)
            y = 0.5 * (_unit(left, eps) * t("left.out").to(F64)
                       + _unit(right, eps) * t("right.out").to(F64))
        else:
            q, k, v = ((_lin(h, t(c)) + t(c + ".b").to(F64)).view(n, -1, m["dim"])
                       for c in "qkv")
            warm = torch.floor((pos.to(F64) + 1) / m["q_temp"]["every"])
            q = q * (1 + m["q_temp"]["coef"] * torch.log1p(warm))[:, None, None]
            if first is None:
                first = v
            else:
                mix = t("vmix").to(F64).reshape(())
                v = (1 - mix) * v + mix * first
            y = _attend(q, k, v, m["scale"], spans).view(n, m["heads"], -1)
            y = _lin((y * torch.sigmoid(_lin(h, t("g")))[..., None]).flatten(1), t("o"))
        f = lambda name: w[L + "mlp." + name]  # noqa: E731
        s = torch.softmax(_lin(h, f("router")), -1)
        ids = (s + f("correction").to(F64)).topk(layer["mlp"]["router"]["top"], -1).indices
        wt = s.gather(1, ids)
        wt = wt / wt.sum(-1, keepdim=True) * layer["mlp"]["router"]["scale"]
        for e in range(s.shape[1]):
            own = (wt * (ids == e)).sum(-1)
            r = own.nonzero()[:, 0]
            up = _lin(h[r], f(f"e{e}.up")).relu().square()
            y[r] += own[r, None] * _lin(up, f(f"e{e}.down"))
        x = x + y
    return _unit(x, eps) * w["final.norm"].to(F64), w["embed"]


def _exact_momuvik(raw, w, tokens, pos, spans):
    eps = raw["norm"]["eps"]
    x = w["embed"][tokens].to(F64) * raw["embedding"]["scale"]
    n = x.shape[0]
    for i, layer in enumerate(raw["layers"]):
        L, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        t = lambda name: w[L + "mix." + name]  # noqa: E731
        H, d, r, base = m["heads"], m["dim"], m["rot_dim"], m["rot"]["base"]
        h = _unit(x, eps) * (1 + w[L + "norm1"].to(F64))
        both = _lin(h, t("dkv"))
        c = _unit(both[:, :m["kv_rank"]], eps) * t("dkv.norm").to(F64)
        turned = _rotate(both[:, None, m["kv_rank"]:], pos, r, base)
        q = _lin(_unit(_lin(h, t("dq")), eps) * t("dq.norm").to(F64), t("uq")).view(n, H, d + r)
        q = torch.cat([q[..., :d], _rotate(q[..., d:], pos, r, base)], -1)
        k = torch.cat([_lin(c, t("uk")).view(n, H, d), turned.expand(-1, H, -1)], -1)
        v = _lin(c, t("uv")).view(n, H, -1)
        y = _lin(_attend(q, k, v, m["scale"], spans, sink=t("sink")), t("o"))
        x = x + raw["residual_mult"] * y
        h = _unit(x, eps) * (1 + w[L + "norm2"].to(F64))
        if mlp["kind"] == "dense":
            y = _silu_mlp(h, w, L + "mlp.")
        else:
            def expert(z, p, limit):
                g = _lin(z, w[p + "gate"]).clamp(max=limit)
                u = _lin(z, w[p + "up"]).clamp(-limit, limit)
                return _lin(g * torch.sigmoid(1.702 * g) * (u + 1), w[p + "down"])

            y = expert(h, L + "mlp.shared.", mlp["shared"]["limit"])
            top, ids = _lin(h, w[L + "mlp.router"]).topk(mlp["router"]["top"], -1)
            for e in range(mlp["router"]["experts"]):
                own = (torch.sigmoid(top) * (ids == e)).sum(-1)
                at = own.nonzero()[:, 0]
                y[at] += expert(own[at, None] * h[at], f"{L}mlp.e{e}.", mlp["expert"]["limit"])
        x = x + raw["residual_mult"] * y
    return _unit(x, eps) * (1 + w["final.norm"].to(F64)), w["embed"]


def exact(case, seed):
    if case["kind"] == "sample":
        return None                       # whole numbers
    config = preset_config(case["preset"], case["layers"])
    raw = config.to_dict()
    seqs = _sequences(case, seed)
    total = sum(len(a) + len(b) for a, b, _ in seqs)
    shapes = expected_tensors(config.to_spec())
    dense = sum(math.prod(s) for n, s in shapes.items()
                if len(s) == 2 and None not in s and s[0] < PRESETS["qwen3-8b"]["vocab_size"])
    if total * dense * 2.0 > 4.5e14:
        return None                       # over some 15 seconds of 64-bit products
    w = _weights(case, config.to_spec(), seed)
    tokens, pos, spans, want = [], [], [], []
    for before, step, wants in seqs:
        a = len(tokens)
        tokens += before + step
        pos += range(len(before) + len(step))
        spans.append((a, len(tokens)))
        want += [a + len(before) + i for i in wants]
    of = {"qwen3": _exact_qwen3, "vunasun": _exact_vunasun, "pavatar": _exact_pavatar,
          "momuvik": _exact_momuvik}[_family(case)]
    x, head = of(raw, w, torch.tensor(tokens, device=DEV), torch.tensor(pos, device=DEV), spans)
    logits = x[torch.tensor(want, device=DEV)] @ head.to(F64).T
    cap = raw.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits
