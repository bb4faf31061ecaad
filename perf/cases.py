"""What the speed of this library is measured on: passes through the engine's public entry points.

A pass of kind "trace" plays one batch of requests through ``Engine.step`` the way trace replay and a serving
loop do: sequences are opened, their prompts go in (all in one step, or in chunks beside the tokens of the
sequences that are already decoding), then every sequence brings one token a step, and the sequences are
closed.  The tokens are given, so the logits of every step can be compared; they are what a pass returns.  A
pass of kind "sample" is the device sampler's choice of a token for every row of a step's logits.

A program loads a model once and serves many batches with it, so the engine (random weights of the named layer
sizes) is kept from one ``prepare`` to the next of the same model; the requests come from the seed.  Routed
feed-forwards are left out: with random weights the scores of the last expert chosen and the first one left
out are often nearer than the rounding of 16-bit activations, and two correct runs then differ by a whole expert."""
import hashlib
import math

import numpy as np
import torch

from grout_b200.engine import Engine
from grout_b200.sampling import DeviceSampler, SamplingParams

MAX_SEQ, MAX_BATCH, MAX_TOKENS = 4096, 64, 40960     # what an engine's cache is built for
# (width, query heads, kv heads, head size, feed-forward rows, layers, vocabulary): the layer sizes of bench.py
SIZES = {"1b": (2048, 16, 8, 128, 6144, 16, 65536), "4b": (2560, 32, 8, 128, 9728, 36, 151936)}


def listed():
    def trace(name, model, dtype, seqs, low, high, steps, chunk=0):
        return dict(name=name, kind="trace", model=model, dtype=dtype, seqs=seqs, low=low, high=high, steps=steps,
                    chunk=chunk)

    return [
        # the smallest call: a few tokens in and out of a small model
        trace("small", "qwen3-1b", "bfloat16", 1, 5, 5, 3),
        # a question and its answer, one user: prompt of 18 tokens and 36 tokens generated (the reference's own cell)
        trace("chat", "qwen3-4b", "bfloat16", 1, 18, 18, 35),
        # reading one document: a prompt of 2,048 tokens, the logits behind its last
        trace("prompt", "qwen3-4b", "bfloat16", 1, 2048, 2048, 0),
        # the batch of the default benchmark: eight prompts of 2,048 tokens, then decode steps
        trace("batch", "qwen3-4b", "bfloat16", 8, 2048, 2048, 32),
        # a full server: 64 requests of very unequal lengths
        trace("serve", "qwen3-4b", "bfloat16", 64, 17, 700, 16),
        # continuous batching: prompts come in chunks of 384 tokens beside the tokens of those already decoding
        trace("chunks", "qwen3-1b", "bfloat16", 6, 300, 1500, 8, 384),
        # the true 32-bit path: one request, and a small batch of unequal prompts
        trace("float32-chat", "qwen3-1b", "float32", 1, 45, 45, 12),
        trace("float32-batch", "qwen3-1b", "float32", 4, 100, 600, 6),
        # a sampled token for one user and for a full batch whose requests ask for different limits
        dict(name="sample-one", kind="sample", rows=1, vocab=151936),
        dict(name="sample-batch", kind="sample", rows=64, vocab=151936),
        # models with a recurrent state beside attention: a document through the gated delta rule, and a ragged
        # batch through the delta rule with a decay per channel, latent and windowed attention
        trace("sonalorn", "sonalorn-1b", "bfloat16", 1, 2048, 2048, 12),
        trace("keralix", "keralix-1b", "bfloat16", 4, 250, 1200, 12),
    ]


def draw(rng):
    def log(a, b):
        return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    kind = rng.choice(["qwen3-4b", "qwen3-4b", "qwen3-1b", "qwen3-1b", "float32", "sample", "sonalorn-1b", "keralix-1b"])
    if kind == "sample":
        return dict(kind="sample", rows=log(1, 64), vocab=rng.randint(32000, 151936))
    if kind == "float32":
        seqs, most, dtype, kind = log(1, 8), 600, "float32", "qwen3-1b"
    else:
        seqs, most, dtype = log(1, 64), 2048, "bfloat16"
    high = log(5, min(most, {"float32": 2400, "bfloat16": 16000}[dtype] // seqs))
    low = max(1, int(high * rng.uniform(0.1, 1.0)))
    chunk = rng.choice([0, 0, rng.randint(64, 1024)])
    return dict(kind="trace", model=kind, dtype=dtype, seqs=seqs, low=low, high=high, steps=rng.randint(0, 24),
                chunk=chunk if chunk < high and seqs <= 12 and chunk * 24 >= seqs * high else 0)


# -- the requests -----------------------------------------------------------
def lengths(case):
    """Prompt lengths of a case: spread from low to high over their logarithm, in an order without a trend."""
    n, lo, hi = case["seqs"], case["low"], case["high"]
    out = [int(round(lo * (hi / lo) ** (i / (n - 1)))) if n > 1 else hi for i in range(n)]
    order = sorted(range(n), key=lambda i: hashlib.sha256(b"%d" % i).digest())
    return [out[i] for i in order]


def plan(case):
    """The steps of a pass: lists of (sequence, first place, tokens, whether the last one's logits are wanted)."""
    lens, steps = lengths(case), []
    held, left = [0] * len(lens), [case["steps"]] * len(lens)
    if not case["chunk"]:
        steps.append([(i, 0, n, True) for i, n in enumerate(lens)])
        held = list(lens)
    else:
        for i, n in enumerate(lens):
            while held[i] < n:
                k = min(case["chunk"], n - held[i])
                step = [(i, held[i], k, held[i] + k == n)]
                for j in range(i):
                    if left[j]:
                        step.append((j, held[j], 1, True))
                        left[j] -= 1
                for j, _at, m, _w in step:
                    held[j] += m
                steps.append(step)
    while any(left):
        step = [(j, held[j], 1, True) for j in range(len(lens)) if left[j]]
        for j, _at, _n, _w in step:
            held[j] += 1
            left[j] -= 1
        steps.append(step)
    return steps


def tokens_of(case, seed):
    vocab = SIZES[case["model"].split("-")[1]][6]
    rs = np.random.RandomState(seed % (1 << 31))
    return [rs.randint(0, vocab, n + case["steps"]).tolist() for n in lengths(case)]


# -- the models -------------------------------------------------------------
def config(model):
    family, size = model.split("-")
    W, nq, nkv, D, ff, n, V = SIZES[size]
    dense = {"kind": "dense", "ff": ff}
    if family == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=V, hidden_size=W,
                    intermediate_size=ff, num_hidden_layers=n, num_attention_heads=nq, num_key_value_heads=nkv,
                    head_dim=D, rope_theta=1000000.0, rms_norm_eps=1e-6, max_position_embeddings=40960,
                    tie_word_embeddings=True, use_sliding_window=False, eos_token_id=V - 1)
    if family == "sonalorn":     # three layers of the delta rule to one of attention
        delta = dict(heads=nq, kv_heads=nkv, dim=D, vdim=D, conv=4)
        attn = dict(heads=nq, kv_heads=nkv, dim=D, vdim=D, scale=D ** -0.5, q_temp={"coef": 0.1, "every": 256})
        layers = [dict(type="attention" if i % 4 == 3 else "delta", mixer=attn if i % 4 == 3 else delta, mlp=dense)
                  for i in range(n)]
        return dict(architecture="Sonalorn", vocab=V, width=W, max_positions=MAX_SEQ, norm={"eps": 1e-6}, layers=layers)
    lat = dict(heads=nq, dim=D, vdim=D, kv_rank=128, q_rank=3 * W // 8 // 64 * 64, scale=D ** -0.5)
    delta = dict(heads=nq, kv_heads=nq, dim=D, vdim=D, conv=4)
    attn = dict(heads=nq, kv_heads=nkv, dim=D, vdim=D, conv=4, scale=D ** -0.5, softcap=50.0, mask={"size": 1024},
                rot={"base": 1000000.0, "dims": D})
    kinds = (("latent_attention", lat), ("channel_delta", delta), ("attention", attn))
    return dict(architecture="Keralix", vocab=V, width=W, streams=4, norm={"eps": 1e-6}, embedding={"scale": W ** 0.5},
                layers=[dict(type=kinds[i % 3][0], mixer=kinds[i % 3][1], mlp=dense) for i in range(n)])


def shapes(model):
    """name -> (shape, kind) of every tensor of a model."""
    cfg = config(model)
    family, size = model.split("-")
    W, nq, nkv, D, ff, n, V = SIZES[size]
    q, kv, out = nq * D, nkv * D, {}

    def add(prefix, **tensors):
        for name, (kind, *shape) in tensors.items():
            out[prefix + name.replace("__", ".")] = (tuple(shape), kind)

    for i in range(n):
        if family == "qwen3":
            add(f"model.layers.{i}.", input_layernorm__weight=("vector", W), post_attention_layernorm__weight=("vector", W),
                self_attn__q_proj__weight=("matrix", q, W), self_attn__k_proj__weight=("matrix", kv, W),
                self_attn__v_proj__weight=("matrix", kv, W), self_attn__o_proj__weight=("matrix", W, q),
                self_attn__q_norm__weight=("vector", D), self_attn__k_norm__weight=("vector", D),
                mlp__gate_proj__weight=("matrix", ff, W), mlp__up_proj__weight=("matrix", ff, W),
                mlp__down_proj__weight=("matrix", W, ff))
            continue
        p, layer = f"l{i}.", cfg["layers"][i]
        add(p, norm1=("vector", W), norm2=("vector", W), mlp__gate=("matrix", ff, W), mlp__up=("matrix", ff, W),
            mlp__down=("matrix", W, ff), mix__o=("matrix", W, q))
        if family == "sonalorn":
            add(p, ls1=("vector", W), ls2=("vector", W))
            if layer["type"] == "attention":
                add(p + "mix.", q=("matrix", q, W), k=("matrix", kv, W), v=("matrix", kv, W), q__norm=("vector", D),
                    k__norm=("vector", D))
            else:
                add(p + "mix.", q=("matrix", kv, W), k=("matrix", kv, W), v=("matrix", q, W), g=("matrix", q, W),
                    b=("matrix", nq, W), a=("matrix", nq, W), q__conv=("vector", kv, 4), k__conv=("vector", kv, 4),
                    v__conv=("vector", q, 4), A_log=("offset", nq), dt_bias=("offset", nq), norm=("vector", D))
            continue
        for hc in ("hc1.", "hc2."):
            add(p + hc, **{"in": ("average", 4), "out": ("vector", 4), "mix": ("mixing", 4, 4)})
        if layer["type"] == "latent_attention":
            m = layer["mixer"]
            add(p + "mix.", dq=("matrix", m["q_rank"], W), dq__norm=("vector", m["q_rank"]), uq=("matrix", q, m["q_rank"]),
                dkv=("matrix", 128, W), dkv__norm=("vector", 128), uk=("matrix", q, 128), uv=("matrix", q, 128),
                sink=("offset", nq), g=("matrix", q, W))
        elif layer["type"] == "channel_delta":
            add(p + "mix.", q=("matrix", q, W), k=("matrix", q, W), v=("matrix", q, W), b=("matrix", nq, W),
                q__conv=("vector", q, 4), k__conv=("vector", q, 4), v__conv=("vector", q, 4), A_log=("offset", nq),
                dt_bias=("offset", q), a1=("matrix", D, W), a2=("matrix", q, D), g1=("matrix", D, W), g2=("matrix", q, D),
                norm=("vector", D))
        else:
            add(p + "mix.", q=("matrix", q, W), k=("matrix", kv, W), q__b=("offset", q), k__b=("offset", kv),
                q__conv=("vector", q, 4), k__conv=("vector", kv, 4))
    if family == "qwen3":
        add("model.", embed_tokens__weight=("matrix", V, W), norm__weight=("vector", W))
    else:
        add("", embed=("matrix", V, W), final__norm=("vector", W))
        if family == "sonalorn":
            add("", head=("matrix", V, W), pos=("matrix", MAX_SEQ, W), embed__norm=("vector", W))
    return out


def weights(model):
    """The model's tensors: N(0, 0.02^2) matrices, norms around one, offsets around zero, rounded to bfloat16.  What
    writes to the residual stream is scaled down by the root of the number of sublayers, as is usual, and a table that
    starts the stream unscaled is wide enough for it: a stream that every layer overwrote would double each
    rounding a few layers later, as no trained model's does, and nothing could be compared in 16 bits."""
    out, writes = {}, (2 * SIZES[model.split("-")[1]][5]) ** -0.5
    for name, (shape, kind) in shapes(model).items():
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int.from_bytes(hashlib.sha256((model + ":" + name).encode()).digest()[:6], "little"))
        x = torch.randn(shape, generator=gen, device="cuda")
        if kind == "matrix":
            x = (0.3 if name == "model.embed_tokens.weight" else 0.02) * x
        elif kind == "vector":
            x = 1.0 + 0.1 * x
        elif kind == "mixing":
            x = torch.eye(*shape, device="cuda") + 0.1 * x
        else:
            x = 0.1 * x
            if kind == "average":
                x[-1] += 1.0
        if name.endswith(("o_proj.weight", "down_proj.weight", "mix.o", "mlp.down", ".ls1", ".ls2")):
            x = writes * x
        out[name] = x.to(torch.bfloat16)
    return out


_LOADED = {}     # the one engine a program of this kind holds: (model, dtype) -> Engine


def engine_for(model, dtype):
    if (model, dtype) not in _LOADED:
        _LOADED.clear()
        _LOADED[model, dtype] = Engine.from_tensors(config(model), weights(model), dtype, max_tokens=MAX_TOKENS,
                                                    max_batch=MAX_BATCH, max_seq_len=MAX_SEQ)
    return _LOADED[model, dtype]


# -- a pass -----------------------------------------------------------------
#: What requests ask for: the usual defaults of a chat model, plain sampling, a nucleus, a short list.
ASKED = ((0.6, 20, 0.95), (1.0, 0, 1.0), (0.8, 0, 0.9), (0.7, 50, 1.0))


def prepare(case, seed):
    if case["kind"] == "sample":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        # a model's logits: a wide bulk and a few tokens well above it
        logits = 2.0 * torch.randn((case["rows"], case["vocab"]), generator=gen, device="cuda")
        logits += 8.0 * (torch.rand(logits.shape, generator=gen, device="cuda") < 16.0 / case["vocab"])
        rs = np.random.RandomState(seed % (1 << 31))
        params = [SamplingParams(True, t, k, p).normalised()
                  for t, k, p in (ASKED[i % len(ASKED)] for i in range(case["rows"]))]
        return dict(case=case, sampler=DeviceSampler("cuda:0"), logits=logits, params=params,
                    draws=[float(np.float32(u)) for u in rs.random_sample(case["rows"])])
    tokens = tokens_of(case, seed)
    steps = [([(i, tokens[i][at:at + n]) for i, at, n, _w in step], [[n - 1] if w else [] for _i, _at, n, w in step])
             for step in plan(case)]
    return dict(case=case, engine=engine_for(case["model"], case["dtype"]), steps=steps)


def run(state):
    if state["case"]["kind"] == "sample":
        return state["sampler"].choose(state["logits"], state["params"], state["draws"])
    engine = state["engine"]
    slots = [engine.open_sequence() for _ in range(state["case"]["seqs"])]
    out = []
    for entries, want in state["steps"]:
        logits = engine.step([(slots[i], toks) for i, toks in entries], want)
        if logits is not None:
            out.append(logits)
    for slot in slots:
        engine.close_sequence(slot)
    return out


# -- what a pass cannot do without ------------------------------------------
def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4 * case["rows"] * (case["vocab"] + 5), "flops": 0}
    cfg = config(case["model"])
    W, nq, nkv, D, _ff, n, V = SIZES[case["model"].split("-")[1]]
    size = 4 if case["dtype"] == "float32" else 2
    family, table = case["model"].split("-")[0], {"qwen3": "model.embed_tokens.weight"}.get(case["model"].split("-")[0], "embed")
    kinds = [None if family == "qwen3" else layer["type"] for layer in cfg["layers"]] if family != "qwen3" else ["attention"] * n
    held = sum(math.prod(s) for name, (s, _k) in shapes(case["model"]).items() if name not in (table, "head", "pos"))
    bytes_, flops = 0.0, 0.0
    for step in plan(case):
        rows, wanted = sum(k for _i, _at, k, _w in step), sum(w for _i, _at, _k, w in step)
        bytes_ += size * (held + rows * W) + (size * V * W if wanted else 0) + 4 * wanted * V
        flops += 2.0 * rows * held + 2.0 * wanted * V * W
        for kind in kinds:
            for _i, at, k, _w in step:
                if kind in ("delta", "channel_delta"):       # a state read and written, two products a row
                    bytes_ += (8 if at else 4) * nq * D * D
                    flops += 6.0 * k * nq * D * D
                    continue
                seen = 1024 if family == "keralix" and kind == "attention" else at + k
                row = D if kind == "latent_attention" else nkv * D * (1 if kind == "attention" and family == "keralix" else 2)
                bytes_ += size * row * (min(at + k, seen + k - 1) + k)
                flops += 4.0 * nq * D * sum(min(p + 1, seen) for p in range(at, at + k))
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    # measured against exact(): 6e-7 in 32 bits, 0.004 to 0.01 in bfloat16; two correct runs are both off by that
    return {"rel": 3e-6, "max": 5e-5} if case["dtype"] == "float32" else {"rel": 0.025, "max": 0.2}


# -- the same in 64 bits ----------------------------------------------------
F = torch.float64


def rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def conv(x, w):
    """Causal, per channel: w[c, -1] meets the row itself."""
    y = torch.zeros_like(x)
    for j in range(w.shape[1]):
        m = w.shape[1] - 1 - j
        y[m:] += w[:, j] * x[:x.shape[0] - m]
    return y


def unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def rotate(x, theta):
    """Halves of a head turn by position times a frequency, both and their product rounded to 32 bits once."""
    half = x.shape[-1] // 2
    i = np.arange(0, 2 * half, 2, dtype=np.float32) / np.float32(2 * half)
    inv = (np.float32(1.0) / np.power(np.float32(theta), i, dtype=np.float32)).astype(np.float32)
    angle = np.arange(x.shape[0], dtype=np.float32)[:, None] * inv
    a = torch.from_numpy(angle.astype(np.float64)).to(x.device)[:, None]
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)


def attend(q, k, v, scale, window=None, cap=None, sink=None):
    T, nq, out = q.shape[0], q.shape[1], []
    i = torch.arange(T, device=q.device)
    hidden = i[None] > i[:, None]
    if window:
        hidden = hidden | (i[None] <= i[:, None] - window)
    for h in range(nq):
        g = h // (nq // k.shape[1])
        s = q[:, h] @ k[:, g].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, 1)[:, :T] @ v[:, g])
    return torch.stack(out, 1).reshape(T, -1)


def delta(q, k, v, beta, decay):
    """Rows of every head at once: the state fades, the key's value moves towards v by beta, q reads."""
    T, H, D = k.shape
    S, out = torch.zeros(H, D, v.shape[2], dtype=F, device=k.device), torch.empty_like(v)
    for t in range(T):
        S = S * decay[t][..., None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out


def silu(x):
    return x * torch.sigmoid(x)


def mixer(model, layer, t, h, D):
    """A layer's mixer on the rows h of one whole sequence; t(name): the layer's tensor."""
    T = h.shape[0]
    heads = lambda x: x.view(T, -1, D)  # noqa: E731
    if model.startswith("qwen3"):
        q, k = (rotate(rms(heads(h @ t(n + "_proj.weight").T), t(n + "_norm.weight"), 1e-6), 1e6) for n in "qk")
        return attend(q, k, heads(h @ t("v_proj.weight").T), D ** -0.5) @ t("o_proj.weight").T
    m, kind = layer["mixer"], layer["type"]
    if model.startswith("sonalorn") and kind == "attention":
        q, k = (rms(heads(h @ t(n).T), t(n + ".norm"), 1e-6) for n in "qk")
        p = torch.arange(T, device=h.device)
        q = q * (1.0 + m["q_temp"]["coef"] * torch.log(((p + 1) // m["q_temp"]["every"] + 1).to(F)))[:, None, None]
        return attend(q, k, heads(h @ t("v").T), m["scale"], sink=torch.zeros(m["heads"], dtype=F, device=h.device)) @ t("o").T
    if kind == "attention":
        q, k = (heads(conv(h @ t(n).T + t(n + ".b"), t(n + ".conv"))) for n in "qk")
        return attend(rotate(q, 1e6), rotate(k, 1e6), k, m["scale"], m["mask"]["size"], m["softcap"]) @ t("o").T
    if kind == "latent_attention":
        q = heads(rms(h @ t("dq").T, t("dq.norm"), 1e-6) @ t("uq").T)
        c = rms(h @ t("dkv").T, t("dkv.norm"), 1e-6)
        o = attend(q, heads(c @ t("uk").T), heads(c @ t("uv").T), m["scale"], sink=t("sink"))
        return (o * torch.sigmoid(h @ t("g").T)) @ t("o").T
    q, k, v = (heads(silu(conv(h @ t(n).T, t(n + ".conv")))) for n in "qkv")
    q, k, beta = unit(q) * D ** -0.5, unit(k), torch.sigmoid(h @ t("b").T)
    if kind == "delta":
        decay = torch.exp(-torch.exp(t("A_log")) * torch.nn.functional.softplus(h @ t("a").T + t("dt_bias")))[..., None]
        gate = silu(h @ t("g").T)
    else:
        a = heads(torch.nn.functional.softplus(h @ t("a1").T @ t("a2").T + t("dt_bias")))
        decay, gate = torch.exp(-torch.exp(t("A_log"))[:, None] * a), torch.sigmoid(h @ t("g1").T @ t("g2").T)
    q, k = (x.repeat_interleave(v.shape[1] // x.shape[1], 1) for x in (q, k))
    return (rms(delta(q, k, v, beta, decay), t("norm"), 1e-6) * heads(gate)).reshape(T, -1) @ t("o").T


def exact(case, seed):
    if case["kind"] == "sample":
        return exact_sample(case, seed)
    model = case["model"]
    cfg, w = config(model), weights(model)
    W, _nq, _nkv, D, _ff, n, _V = SIZES[model.split("-")[1]]
    qwen, sona = model.startswith("qwen3"), model.startswith("sonalorn")
    tokens = tokens_of(case, seed)
    seqs = [torch.tensor(t, device="cuda") for t in tokens]
    ends = torch.tensor(np.cumsum([0] + [len(t) for t in tokens]))
    parts = [slice(int(a), int(b)) for a, b in zip(ends[:-1], ends[1:])]
    x = torch.cat([w["model.embed_tokens.weight" if qwen else "embed"][t] for t in seqs]).to(F)
    if sona:
        x = rms(x + torch.cat([w["pos"][:len(t)] for t in seqs]).to(F), w["embed.norm"].to(F), 1e-6)
    elif not qwen:
        x = x * float(W) ** 0.5
        streams = [x] * 4
    for i in range(n):
        layer = None if qwen else cfg["layers"][i]
        p = f"model.layers.{i}." if qwen else f"l{i}."
        t = lambda name: w[p + name].to(F)  # noqa: B023, E731
        mt = lambda name: t(("self_attn." if qwen else "mix.") + name)  # noqa: B023, E731

        def mix(h):
            return torch.cat([mixer(model, layer, mt, h[part], D) for part in parts])  # noqa: B023

        def feed(h):
            g, u, d = ((f"mlp.{k}_proj.weight" if qwen else f"mlp.{k}") for k in ("gate", "up", "down"))
            a = h @ t(g).T  # noqa: B023
            a = torch.nn.functional.gelu(a, approximate="tanh") if sona else silu(a)
            return (a * (h @ t(u).T)) @ t(d).T  # noqa: B023

        if qwen:
            x = x + mix(rms(x, t("input_layernorm.weight"), 1e-6))
            x = x + feed(rms(x, t("post_attention_layernorm.weight"), 1e-6))
        elif sona:
            x = x + t("ls1") * rms(mix(x), t("norm1"), 1e-6)
            x = x + t("ls2") * rms(feed(x), t("norm2"), 1e-6)
        else:
            for k, sub in ((1, mix), (2, feed)):
                a, b, M = t(f"hc{k}.in"), t(f"hc{k}.out"), t(f"hc{k}.mix")
                y = sub(rms(sum(a[s] * streams[s] for s in range(4)), t(f"norm{k}"), 1e-6))
                streams = [sum(M[s, r] * streams[s] for s in range(4)) + b[r] * y for r in range(4)]
    if not qwen and not sona:
        x = sum(streams)
    x = rms(x, w["model.norm.weight" if qwen else "final.norm"].to(F), 1e-6)
    head = w["head" if sona else "model.embed_tokens.weight" if qwen else "embed"].to(F)
    out = []
    for step in plan(case):
        rows = [int(ends[i]) + at + k - 1 for i, at, k, wanted in step if wanted]
        if rows:
            out.append(x[rows] @ head.T)
    return out


def exact_sample(case, seed):
    """The kept set of a row is its top_k largest scores, of these the shortest prefix whose mass reaches top_p; the
    draw walks the kept set in the order of the vocabulary."""
    state = prepare(case, seed)
    out = []
    for row, p, u in zip(state["logits"].double().cpu().numpy(), state["params"], state["draws"]):
        s = row / p.temperature
        order = np.argsort(-s, kind="stable")[:p.top_k or None]
        mass = np.exp(s[order] - s[order[0]])
        kept = order[:int(np.searchsorted(np.cumsum(mass), p.top_p * mass.sum())) + 1] if p.top_p < 1.0 else order
        kept = np.sort(kept)
        walk = np.cumsum(np.exp(s[kept] - s.max()))
        out.append(int(kept[min(int(np.searchsorted(walk, u * walk[-1])), len(kept) - 1)]))
    return torch.tensor(out, dtype=torch.int32)
