"""The work this framework is timed on: calls of its public entry points over the range of sizes it serves.

A case names what is called and how much it is given:

- ``decode``: one step of an LFM3 model cut to eight layers, one token per request behind a cache, logits of every row; recorded as a CUDA
  graph like every step the engine serves;
- ``prompt``: one prompt through ``StepFunction.run``, layout and upload included, logits of its last token;
- ``ffn``, ``attention``, ``moe``, ``ssm``, ``delta``: one part of a model (``part.forward``) on the rows of a step. Steps of up to
  256 tokens are recorded as the engine records them; longer ones are called directly.

Widths are those of the LFM3 1.2B-, 350M- and 2.6B-size configurations and of the other decoders' 2,048- and 1,024-wide
benchmark sizes; weights are random, as in the benchmark.
"""

from __future__ import annotations

import gc
import math

import torch

from tokenomos_b200 import models
from tokenomos_b200.cache.manager import CacheManager
from tokenomos_b200.engine.step import StepEntry, StepFunction
from tokenomos_b200.parts.spec import ROLE_EMBEDDING, ROLE_MATRIX
from tokenomos_b200.weights.random_init import random_tensors

DEVICE = "cuda"
PAGE = 16
RECORD_ROWS = 256                # steps of up to so many tokens are replayed, as the engine does
# the first eight layers: over all sixteen, two correct 16-bit implementations drift 3 to 4 % apart (1.5 to 2 % over eight)
LAYERS = 8
ATTENTION_AT = (2, 5)
EPS = 1e-5
THETA = 1000000.0

LFM3 = {
    "1.2B": dict(hidden_size=2048, num_attention_heads=32, intermediate_size=8192, attention_gate=True),
    "350M": dict(hidden_size=1024, num_attention_heads=16, intermediate_size=4608, attention_gate=False),
    "2.6B": dict(hidden_size=2048, num_attention_heads=32, intermediate_size=10752, attention_gate=False),
}
KV_HEADS, HEAD = 8, 64
# width, experts, chosen, expert's and shared expert's inner size; state-space heads, groups; delta rule's head size
OTHER = {
    "w2048": dict(width=2048, experts=32, top=4, ff=1536, shared=2048, ssm_heads=64, ssm_groups=8, dim=128),
    "w1024": dict(width=1024, experts=16, top=2, ff=1536, shared=1536, ssm_heads=32, ssm_groups=4, dim=64),
}
SSM_STATE, SSM_DIM, TAPS = 128, 64, 4
DELTA_HEADS, DELTA_KV = 16, 8


def listed() -> list[dict]:
    return [
        # serving a few users: the step whose time is the time between two tokens
        dict(name="decode 1.2B b8", kind="decode", size="1.2B", dtype="bf16", seqs=8, new=1, ctx=2048),
        # the time to the first token of one prompt
        dict(name="prompt 1.2B 2048", kind="prompt", size="1.2B", dtype="bf16", seqs=1, new=2048, ctx=0),
        # a short, odd prompt on the small model: launches and small products
        dict(name="prompt 350M 77", kind="prompt", size="350M", dtype="bf16", seqs=1, new=77, ctx=0),
        # a busy server's decode step: 64 requests, contexts of unequal length
        dict(name="attention decode b64", kind="attention", size="1.2B", dtype="bf16", seqs=64, new=1, ctx=3000),
        # chunked prefill far into a long prompt
        dict(name="attention chunk 512@8k", kind="attention", size="2.6B", dtype="bf16", seqs=1, new=512, ctx=8192),
        # the true 32-bit model reading a prompt: its feed-forward and its attention
        dict(name="ffn fp32 2048", kind="ffn", size="1.2B", dtype="fp32", rows=2048),
        dict(name="attention fp32 1000", kind="attention", size="350M", dtype="fp32", seqs=1, new=1000, ctx=0),
        # the 32-bit model decoding for one user: the smallest call
        dict(name="ffn fp32 1", kind="ffn", size="350M", dtype="fp32", rows=1),
        # experts on a prompt, and on a small decode batch
        dict(name="moe 2048", kind="moe", size="w2048", dtype="bf16", rows=2048),
        dict(name="moe decode 16", kind="moe", size="w2048", dtype="bf16", rows=16),
        # the state-space mixer on one prompt
        dict(name="ssm 2048", kind="ssm", size="w1024", dtype="bf16", seqs=1, new=2048, ctx=0),
        # the gated delta rule on two prompts of unequal length side by side
        dict(name="delta 2x1500", kind="delta", size="w2048", dtype="bf16", seqs=2, new=1500, ctx=0),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("decode", "prompt", "ffn", "ffn", "attention", "attention", "attention", "moe", "ssm", "delta"))
    if kind == "decode":
        return dict(kind=kind, size=rng.choice(("1.2B", "350M")), dtype="bf16", seqs=rng.randint(1, 8), new=1,
                    ctx=_log(rng, 200, 2048))
    if kind == "prompt":
        return dict(kind=kind, size=rng.choice(("1.2B", "350M")), dtype="bf16", seqs=1, new=_log(rng, 20, 2048), ctx=0)
    if kind == "ffn":
        dtype = rng.choice(("fp32", "fp32", "bf16"))
        return dict(kind=kind, size=rng.choice(tuple(LFM3)), dtype=dtype, rows=_log(rng, 1, 1500))
    if kind == "attention":
        size, dtype = rng.choice(tuple(LFM3)), rng.choice(("bf16", "bf16", "fp32"))
        if rng.random() < 0.4:
            return dict(kind=kind, size=size, dtype=dtype, seqs=_log(rng, 1, 64), new=1, ctx=_log(rng, 100, 3000))
        return dict(kind=kind, size=size, dtype=dtype, seqs=rng.randint(1, 3), new=_log(rng, 16, 700), ctx=_log(rng, 16, 2500))
    if kind == "moe":
        return dict(kind=kind, size=rng.choice(tuple(OTHER)), dtype="bf16", rows=_log(rng, 1, 2000))
    return dict(kind=kind, size=rng.choice(tuple(OTHER)), dtype="bf16", seqs=rng.randint(1, 4), new=_log(rng, 20, 700), ctx=0)


# ---- sizes ----

def _spread(mean: int, seqs: int) -> list[int]:
    """Lengths of unequal requests around ``mean`` (half to one and a half of it)."""
    if seqs == 1 or mean <= 1:
        return [mean] * seqs
    return [max(1, int(mean * (0.5 + i / (seqs - 1)))) for i in range(seqs)]


def _lengths(case: dict) -> tuple[list[int], list[int]]:
    """(new tokens, cached tokens) of each request."""
    if case["kind"] == "decode":
        return [1] * case["seqs"], [case["ctx"]] * case["seqs"]
    return _spread(case["new"], case["seqs"]), _spread(case["ctx"], case["seqs"])


def _dtype(case: dict) -> torch.dtype:
    return torch.float32 if case["dtype"] == "fp32" else torch.bfloat16


def _config(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("decode", "prompt", "ffn", "attention"):
        whole = kind in ("decode", "prompt")
        types = ["full_attention" if i in ATTENTION_AT else "conv" for i in range(LAYERS)] if whole else ["full_attention"]
        return {"architectures": ["Lfm3ForCausalLM"], "num_hidden_layers": len(types), "layer_types": types,
                "num_key_value_heads": KV_HEADS, "head_dim": HEAD, "vocab_size": 65536 if whole else 1024,
                "rope_theta": THETA, "norm_eps": EPS, "conv_L_cache": 3, "conv_bias": False, "tie_embedding": True,
                **LFM3[case["size"]]}
    z = OTHER[case["size"]]
    if kind == "delta":
        mixer = {"heads": DELTA_HEADS, "kv_heads": DELTA_KV, "dim": z["dim"], "vdim": z["dim"], "conv": TAPS}
        return {"architecture": "Tifisun", "vocab": 1024, "width": z["width"], "norm": {"eps": 1e-6}, "residual_mult": 0.5,
                "embedding": {"scale": 3.0},
                "layers": [{"type": "delta", "mixer": mixer, "mlp": {"kind": "dense", "ff": 256}}]}
    mixer = {"heads": z["ssm_heads"], "vdim": SSM_DIM, "state": SSM_STATE, "groups": z["ssm_groups"], "conv": TAPS,
             "norm_groups": z["ssm_groups"]}
    mlp = {"kind": "dense", "ff": 256}
    if kind == "moe":
        mlp = {"kind": "moe", "expert": {"ff": z["ff"]}, "router": {"experts": z["experts"], "top": z["top"]},
               "shared": {"ff": z["shared"]}}
    return {"architecture": "Fakelorn", "vocab": 1024, "width": z["width"], "norm": {"eps": 1e-6, "groups": 4},
            "logit_scale": 0.5, "logit_softcap": 30.0, "layers": [{"type": "mamba2", "mixer": mixer, "mlp": mlp}]}


def _weights(case: dict, seed: int):
    """The architecture configured, and its tensors kept as the weight loader keeps them."""
    raw, dtype = _config(case), _dtype(case)
    arch = models.architecture_of(raw)
    conf = models.Configured(arch, arch.config_class.from_dict(raw), dtype)
    decls = arch.declare(conf.config).tensor_decls()
    drawn = random_tensors(decls, seed, 0.02, 0.0, dtype, DEVICE)
    roles = {d.name: d.role for d in decls}
    tensors = {n: t if roles[n] in (ROLE_MATRIX, ROLE_EMBEDDING) else t.float() for n, t in drawn.items()}
    g = torch.Generator(device=DEVICE).manual_seed(seed + 1)
    for name, t in tensors.items():
        # recurrences start from the ranges their published initialisations use: steps of 0.001 to 0.1, decay rates of 1 to 16
        if name.endswith("dt_bias"):
            dt = torch.exp(torch.rand(t.shape, generator=g, device=DEVICE) * math.log(100.0) + math.log(1e-3))
            t.copy_(dt + torch.log(-torch.expm1(-dt)))
        elif name.endswith("A_log"):
            t.copy_(torch.log(1.0 + 15.0 * torch.rand(t.shape, generator=g, device=DEVICE)))
        elif name.endswith("mix.D"):
            t.fill_(1.0)
        elif name.endswith(".conv"):
            t.uniform_(-0.5, 0.5, generator=g)
    return conf, tensors


# ---- what a program has in hand, and one pass ----

class State:
    pass


def prepare(case: dict, seed: int) -> State:
    s = State()
    s.kind = case["kind"]
    dtype = _dtype(case)
    conf, s.tensors = _weights(case, seed)
    s.model = models.from_tensors(conf, s.tensors, DEVICE)
    g = torch.Generator(device=DEVICE).manual_seed(seed + 2)
    if s.kind in ("ffn", "moe"):
        s.x = torch.randn(case["rows"], s.model.width, generator=g, device=DEVICE).to(dtype)
        ffn = s.model.blocks[0].ffn
        s.body = lambda: ffn.forward(s.x)
        rows = case["rows"]
    else:
        new, ctx = _lengths(case)
        rows = sum(new)
        pages = 2 + sum(-(-(n + c) // PAGE) for n, c in zip(new, ctx))
        s.cache = CacheManager(s.model.state_specs(), PAGE, pages, len(new), dtype, DEVICE,
                               max_len=max(n + c for n, c in zip(new, ctx)))
        for key, t in s.cache.states.items():
            if any(ctx):
                # keys and values as normed projections leave them; a convolution's rows of products
                t.normal_(0.0, 1.0 if key[1] == "kv" else 0.5, generator=g)
        for i, c in enumerate(ctx):
            s.cache.admit(i)
            if c:
                s.cache.extend(i, c)
                s.cache.commit(i, c)
        s.steps = StepFunction(s.model, s.cache)
        ids = torch.randint(0, s.model.vocab, (rows,), generator=g, device=DEVICE).tolist()
        s.entries, o = [], 0
        for i, n in enumerate(new):
            s.entries.append(StepEntry(i, ids[o:o + n], [n - 1]))
            o += n
        s.ids = ids
        if s.kind != "prompt":
            s.ctx, s.ids_dev, _ = s.steps.layout(s.entries)
        if s.kind == "decode":
            # the step is run again and again from the same cache: what it does to the rows of the convolutions is undone first
            live = [t for key, t in s.cache.states.items() if key[1] == "conv"]
            s.before = [t.clone() for t in live]

            def step():
                torch._foreach_copy_(live, s.before)
                s.ctx.scratch.clear()
                out = s.model.forward(s.model.embed(s.ids_dev, s.ctx), s.ctx)
                return [s.model.logits(out, None), *live]

            s.body = step
        elif s.kind != "prompt":
            s.x = torch.randn(rows, s.model.width, generator=g, device=DEVICE).to(dtype)
            mixer = s.model.blocks[0].mixer

            def part():
                s.ctx.scratch.clear()
                return mixer.forward(s.x, s.ctx, 0)

            s.body = part
    s.graph = None
    if s.kind != "prompt" and rows <= RECORD_ROWS:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.no_grad(), torch.cuda.stream(side):
            s.body()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        gc.collect()
        gc.disable()
        try:
            s.graph = torch.cuda.CUDAGraph()
            with torch.no_grad(), torch.cuda.graph(s.graph):
                s.out = s.body()
        finally:
            gc.enable()
    return s


def run(s: State):
    if s.kind == "prompt":
        logits = s.steps.run(s.entries, commit=False)
        return [logits, *(t for key, t in s.cache.states.items() if key[1] == "conv")]
    if s.graph is not None:
        s.graph.replay()
        return s.out
    with torch.no_grad():
        out = s.body()
    if s.kind in ("ssm", "delta"):           # the memory the prompt leaves behind
        return [out, s.cache.states[(0, "S")]]
    return out


# ---- the bytes and operations a pass cannot do without ----

def _pairs(new, ctx) -> float:
    return float(sum(n * c + n * (n + 1) / 2 for n, c in zip(new, ctx)))


def work(case: dict) -> dict:
    es = 4 if case["dtype"] == "fp32" else 2
    kind = case["kind"]
    if kind in ("moe", "ffn"):
        rows = case["rows"]
        if kind == "ffn":
            z = LFM3[case["size"]]
            d, weights = z["hidden_size"], 3 * z["hidden_size"] * z["intermediate_size"]
            return {"bytes": es * (weights + 2 * rows * d), "flops": 2.0 * rows * weights}
        z = OTHER[case["size"]]
        d, one = z["width"], 3 * z["width"] * z["ff"]
        shared = 3 * d * z["shared"] + d * z["experts"]
        used = z["experts"] * (1.0 - (1.0 - z["top"] / z["experts"]) ** rows)       # experts that some row chooses
        return {"bytes": es * (used * one + shared + 2 * rows * d), "flops": 2.0 * rows * (z["top"] * one + shared)}
    new, ctx = _lengths(case)
    T = sum(new)
    if kind in ("decode", "prompt", "attention"):
        z = LFM3[case["size"]]
        d, H, I = z["hidden_size"], z["num_attention_heads"], z["intermediate_size"]
        att = d * (2 * H * HEAD + 2 * KV_HEADS * HEAD + (H if z["attention_gate"] else 0))
        kv = 2 * KV_HEADS * HEAD * sum(n + c for n, c in zip(new, ctx))
        scores = 4.0 * _pairs(new, ctx) * H * HEAD
        if kind == "attention":
            return {"bytes": es * (att + kv + 2 * T * d), "flops": 2.0 * T * att + scores}
        A = len(ATTENTION_AT)
        layers = A * att + (LAYERS - A) * 4 * d * d + LAYERS * 3 * d * I
        head = 65536 * d
        wanted = case["seqs"]
        return {"bytes": es * (layers + head + A * kv + T * d) + 4 * wanted * 65536,
                "flops": 2.0 * T * layers + A * scores + 2.0 * wanted * head}
    z = OTHER[case["size"]]
    d = z["width"]
    if kind == "ssm":
        H, G = z["ssm_heads"], z["ssm_groups"]
        weights = d * (3 * H * SSM_DIM + 2 * G * SSM_STATE + H)
        cells, passes = H * SSM_STATE * SSM_DIM, 2
    else:
        D = z["dim"]
        weights = d * (2 * DELTA_KV * D + 3 * DELTA_HEADS * D + 2 * DELTA_HEADS)
        cells, passes = DELTA_HEADS * D * D, 3
    return {"bytes": es * (weights + 2 * T * d) + 4.0 * len(new) * cells, "flops": 2.0 * T * (weights + passes * cells)}


def tolerance(case: dict) -> dict:
    """Relative errors that another order of sums and of 16-bit roundings shows."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.03 if case["kind"] in ("decode", "prompt") else 0.012, "max": 0.4}


# ---- the same in 64 bits ----

F64 = torch.float64


def _norm(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _swiglu(x, W, gate, up, down):
    return (_silu(x @ W(gate).T) * (x @ W(up).T)) @ W(down).T


def _rotate(x, pos):
    """Rotate-half over the whole head; the angle is a 32-bit product, as the model defines it."""
    inv = 1.0 / (THETA ** (torch.arange(0, HEAD, 2, dtype=torch.float32) / HEAD))
    ang = (pos.to(torch.float32)[:, None] * inv.to(pos.device)[None, :]).to(F64)
    cos, sin = (torch.cat((f(ang), f(ang)), -1)[:, None, :] for f in (torch.cos, torch.sin))
    half = HEAD // 2
    return x * cos + torch.cat((-x[..., half:], x[..., :half]), -1) * sin


def _attention(x, W, p, s, key, new, ctx, heads):
    T = x.shape[0]
    q = (x @ W(p + "q_proj.weight").T).view(T, heads, HEAD)
    k = (x @ W(p + "k_proj.weight").T).view(T, KV_HEADS, HEAD)
    v = (x @ W(p + "v_proj.weight").T).view(T, KV_HEADS, HEAD)
    q, k = _norm(q, EPS), _norm(k, EPS)
    out, o, G = torch.empty(T, heads, HEAD, dtype=F64, device=x.device), 0, heads // KV_HEADS
    for i, (n, c) in enumerate(zip(new, ctx)):
        pos = torch.arange(c, c + n, device=x.device)
        qi, ki, vi = _rotate(q[o:o + n], pos), _rotate(k[o:o + n], pos), v[o:o + n]
        if c:
            pool = s.cache.states[key][s.cache.block_table(i, s.cache.state_groups[key])].to(F64)    # [blocks, 2, Hkv, P, D]
            old = pool.permute(1, 0, 3, 2, 4).reshape(2, -1, KV_HEADS, HEAD)[:, :c]
            ki, vi = torch.cat((old[0], ki)), torch.cat((old[1], vi))
        unseen = torch.arange(c + n, device=x.device)[None, :] > pos[:, None]
        for h in range(heads):
            sc = (qi[:, h] @ ki[:, h // G].T * HEAD ** -0.5).masked_fill(unseen, -math.inf)
            out[o:o + n, h] = torch.softmax(sc, -1) @ vi[:, h // G]
        o += n
    if p + "gate_proj.weight" in s.tensors:
        out = out * torch.sigmoid(x @ W(p + "gate_proj.weight").T)[:, :, None]
    return out.reshape(T, heads * HEAD) @ W(p + "o_proj.weight").T


def _conv(x, W, p, state, new, ctx):
    """The gated short convolution of each request, behind the inputs its row of ``state`` holds; with it the rows it leaves."""
    B, C, X = (x @ W(p + "in_proj.weight").T).chunk(3, -1)
    u, taps = B * X, W(p + "conv.weight")[:, 0]
    K = taps.shape[1]
    after, ys, o = state.to(F64), [], 0
    for i, (n, c) in enumerate(zip(new, ctx)):
        before = after[i + 1] if c else torch.zeros(K - 1, u.shape[1], dtype=F64, device=u.device)
        pad = torch.cat((before, u[o:o + n]))
        ys.append(sum(pad[j:j + n] * taps[:, j] for j in range(K)))
        after[i + 1] = pad[-(K - 1):]
        o += n
    return (C * torch.cat(ys)) @ W(p + "out_proj.weight").T, after


def _causal(u, taps, new):
    """A causal convolution of each request from nothing, through silu."""
    K, out = taps.shape[1], []
    for part in u.split(new):
        pad = torch.cat((torch.zeros(K - 1, u.shape[1], dtype=F64, device=u.device), part))
        out.append(sum(pad[j:j + part.shape[0]] * taps[:, j] for j in range(K)))
    return torch.cat(out)


def exact(case: dict, seed: int):
    s = prepare(case, seed)
    W = lambda name: s.tensors[name].to(F64)  # noqa: E731
    kind = case["kind"]
    with torch.no_grad():
        if kind == "ffn":
            f = "model.layers.0.feed_forward."
            return _swiglu(s.x.to(F64), W, f + "w1.weight", f + "w3.weight", f + "w2.weight")
        if kind == "moe":
            x, z = s.x.to(F64), OTHER[case["size"]]
            # (the router's rows are kept in the storage type)
            val, idx = torch.topk(x @ s.tensors["l0.mlp.router"].to(s.x.dtype).to(F64).T, z["top"], -1)
            w, out = torch.softmax(val, -1), _swiglu(x, W, *(f"l0.mlp.shared.{n}" for n in ("gate", "up", "down")))
            for e in range(z["experts"]):
                at, j = (idx == e).nonzero(as_tuple=True)
                if at.numel():
                    out[at] += w[at, j][:, None] * _swiglu(x[at], W, *(f"l0.mlp.e{e}.{n}" for n in ("gate", "up", "down")))
            return out
        new, ctx = _lengths(case)
        if kind == "attention":
            return _attention(s.x.to(F64), W, "model.layers.0.self_attn.", s, (0, "kv"), new, ctx,
                              LFM3[case["size"]]["num_attention_heads"])
        if kind in ("decode", "prompt"):
            x = s.tensors["model.embed_tokens.weight"][torch.tensor(s.ids, device=DEVICE)].to(F64)
            states = dict(zip((k for k in s.cache.states if k[1] == "conv"), s.before)) if kind == "decode" else s.cache.states
            rows = []
            for i in range(LAYERS):
                p = f"model.layers.{i}."
                h = _norm(x, EPS)
                if i in ATTENTION_AT:
                    y = _attention(h, W, p + "self_attn.", s, (i, "kv"), new, ctx, LFM3[case["size"]]["num_attention_heads"])
                else:
                    y, after = _conv(h, W, p + "conv.", states[(i, "conv")], new, ctx)
                    rows.append(after)
                x = x + y
                f = p + "feed_forward."
                x = x + _swiglu(_norm(x, EPS), W, f + "w1.weight", f + "w3.weight", f + "w2.weight")
            if kind == "prompt":
                x = x[-1:]
            return [_norm(x, EPS) @ W("model.embed_tokens.weight").T, *rows]
        z, x, p = OTHER[case["size"]], s.x.to(F64), "l0.mix."
        T = x.shape[0]
        if kind == "ssm":
            H, G, V, N = z["ssm_heads"], z["ssm_groups"], SSM_DIM, SSM_STATE
            inner = H * V
            proj = x @ W(p + "in").T
            gate, xbc, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * G * N], proj[:, 2 * inner + 2 * G * N:]
            xbc = _silu(_causal(xbc, W(p + "conv"), new) + W(p + "conv.b"))
            u = xbc[:, :inner].view(T, H, V)
            B = xbc[:, inner:inner + G * N].view(T, G, N).repeat_interleave(H // G, 1)
            C = xbc[:, inner + G * N:].view(T, G, N).repeat_interleave(H // G, 1)
            dt = torch.nn.functional.softplus(dt + W(p + "dt_bias"))
            decay = torch.exp(-torch.exp(W(p + "A_log")) * dt)
            last = torch.zeros(len(new) + 1, H, N, V, dtype=F64, device=DEVICE)
            ys, o = [], 0
            for i, n in enumerate(new):
                S = last[i + 1]
                for t in range(o, o + n):
                    S.mul_(decay[t, :, None, None]).add_((dt[t, :, None] * B[t])[:, :, None] * u[t][:, None, :])
                    ys.append(torch.bmm(C[t][:, None, :], S)[:, 0])
                o += n
            y = (torch.stack(ys) + W(p + "D")[:, None] * u).reshape(T, inner) * _silu(gate)
            y = _norm(y.view(T, G, inner // G), 1e-6).reshape(T, inner) * W(p + "norm")
            out = y @ W(p + "o").T
            return [out, last] if sum(new) > RECORD_ROWS else out
        H, K, D = DELTA_HEADS, DELTA_KV, z["dim"]
        u = {n: _silu(_causal(x @ W(p + n).T, W(p + n + ".conv"), new)) for n in ("q", "k", "v")}
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q = (unit(u["q"].view(T, K, D)) * D ** -0.5).repeat_interleave(H // K, 1)
        k = unit(u["k"].view(T, K, D)).repeat_interleave(H // K, 1)
        v, beta = u["v"].view(T, H, D), torch.sigmoid(x @ W(p + "b").T)
        decay = torch.exp(-torch.exp(W(p + "A_log")) * torch.nn.functional.softplus(x @ W(p + "a").T + W(p + "dt_bias")))
        last = torch.zeros(len(new) + 1, H, D, D, dtype=F64, device=DEVICE)         # [head, value column, key row]
        ys, o = [], 0
        for i, n in enumerate(new):
            S = last[i + 1]
            for t in range(o, o + n):
                S.mul_(decay[t, :, None, None])
                w = beta[t, :, None] * (v[t] - torch.bmm(S, k[t][:, :, None])[..., 0])
                S.add_(w[:, :, None] * k[t][:, None, :])
                ys.append(torch.bmm(S, q[t][:, :, None])[..., 0])
            o += n
        y = _norm(torch.stack(ys), 1e-6) * W(p + "norm")
        out = (y.reshape(T, H * D) * _silu(x @ W(p + "g").T)) @ W(p + "o").T
        return [out, last] if sum(new) > RECORD_ROWS else out
