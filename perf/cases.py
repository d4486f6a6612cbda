"""Cases on which the speed of the framework's main paths is measured.

What a program that serves or scores with a decoder has it do: whole steps of the step function (single-stream
decoding, a decode batch, a mixed batch under a token budget), and its layers one by one through their parts
(grouped-query attention over the paged cache, the gated feed-forward, the routed feed-forward, the head with the
sampler), in both precisions.  Sizes are those of the framework's own benchmark shapes; ``draw`` gives more of the
same ranges, odd ones among them.

A part adds its output into the float32 residual stream in place, so a pass begins by putting the stream's rows
where the layer expects them.  A step grows its requests, so a pass of a step runs on forks of requests that keep
their contexts: the fork shares the context's pages, gets its new tokens, and gives everything back.
"""
import math
import random
import zlib

import torch

from bitwise_b200 import LlamaConfig, Model
from bitwise_b200.cache.storage import build_cache
from bitwise_b200.engine.step import StepEntry, Stepper
from bitwise_b200.kernels.ops import get_ops
from bitwise_b200.parts.base import StepContext, Workspace
from bitwise_b200.parts.embedding import OutputHead
from bitwise_b200.parts.mlp import SwiGLU
from bitwise_b200.parts.norm import RMSNorm
from bitwise_b200.parts.routed_ffn import ClampedGLU, RoutedFFN

DEVICE = "cuda:0"
PAGE = 16
EPS = 1e-5
THETA = 130000.0
GLU_ALPHA, GLU_LIMIT = 1.702, 7.0

# hidden size, heads, key/value heads, head size, inner size of the feed-forward
S360M = dict(hidden=960, heads=15, kv_heads=5, head_dim=64, inner=2560)
S1B7 = dict(hidden=2048, heads=32, kv_heads=32, head_dim=64, inner=8192)
S8B = dict(hidden=4096, heads=32, kv_heads=8, head_dim=128, inner=14336)


def _attn(s):
    return {k: s[k] for k in ("hidden", "heads", "kv_heads", "head_dim")}


def _ffn(s):
    return {k: s[k] for k in ("hidden", "inner")}


def listed():
    return [
        # one user's stream: a token at a time through a whole small model, where launches and latency count
        dict(name="step_decode_1_360m", kind="step", dtype="bfloat16", layers=32, vocab=49152, **S360M,
             decode=1, ctx_lo=700, ctx_hi=700, prompt=0, start=0),
        # the benchmark's decode step: 8 requests with 2,048-token contexts through the whole model
        dict(name="step_decode_8_1b7", kind="step", dtype="bfloat16", layers=24, vocab=49152, **S1B7,
             decode=8, ctx_lo=2047, ctx_hi=2047, prompt=0, start=0),
        # continuous batching under a 512-token budget: single tokens of running requests beside a portion of a prompt
        dict(name="step_mixed_512_360m", kind="step", dtype="bfloat16", layers=32, vocab=49152, **S360M,
             decode=24, ctx_lo=20, ctx_hi=1270, prompt=488, start=512),
        # a layer's attention on a whole prompt, its length no round number
        dict(name="attn_prefill_2047_1b7", kind="attention", dtype="bfloat16", **_attn(S1B7),
             decode=0, ctx_lo=0, ctx_hi=0, prompt=2047, start=0),
        # the second portion of a longer prompt, grouped heads of size 128
        dict(name="attn_prefill_1200_8b", kind="attention", dtype="bfloat16", **_attn(S8B),
             decode=0, ctx_lo=0, ctx_hi=0, prompt=1200, start=848),
        # a large decode batch of ragged contexts, grouped heads of size 128
        dict(name="attn_decode_64_8b", kind="attention", dtype="bfloat16", **_attn(S8B),
             decode=64, ctx_lo=900, ctx_hi=4090, prompt=0, start=0),
        # the feed-forward of an ordinary decode batch
        dict(name="mlp_48_1b7", kind="mlp", dtype="bfloat16", rows=48, **_ffn(S1B7)),
        # the feed-forward of a prompt, the largest products
        dict(name="mlp_2048_8b", kind="mlp", dtype="bfloat16", rows=2048, **_ffn(S8B)),
        # the end of a decode step: last norm, head and sampler over a large vocabulary
        dict(name="head_64_8b", kind="head", dtype="bfloat16", rows=64, hidden=4096, vocab=128256),
        # the exact 32-bit path: a prompt's feed-forward, and a decode batch's attention
        dict(name="mlp_2048_1b7_f32", kind="mlp", dtype="float32", rows=2048, **_ffn(S1B7)),
        dict(name="attn_decode_8_1b7_f32", kind="attention", dtype="float32", **_attn(S1B7),
             decode=8, ctx_lo=2047, ctx_hi=2047, prompt=0, start=0),
        # routed experts with a shared one, in a decode batch
        dict(name="routed_8", kind="routed", dtype="bfloat16", rows=8, hidden=2048, experts=64, groups=8, keep=4, top=6,
             inner=1408, shared=2816),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    kind = rng.choice(["step", "step", "attention", "attention", "attention", "mlp", "mlp", "mlp", "head", "routed"])
    dtype = "float32" if kind in ("attention", "mlp") and rng.random() < 0.3 else "bfloat16"
    head_dim = rng.choice([64, 64, 128])
    group = rng.choice([1, 2, 3, 4, 8])
    kv = rng.choice([1, 2, 3, 4, 5, 8, 16])
    heads = kv * group
    hidden = rng.choice([heads * head_dim, 64 * rng.randint(8, 64)])
    shape = dict(hidden=hidden, heads=heads, kv_heads=kv, head_dim=head_dim)
    if kind == "step":
        prompt = rng.choice([0, 0, rng.randint(1, 512)])
        decode = _log_int(rng, 1, 64)
        lo = _log_int(rng, 8, 2048)
        return dict(kind=kind, dtype=dtype, layers=rng.randint(2, 32), vocab=rng.choice([32000, 49152]), **shape,
                    inner=8 * rng.randint(64, 1024), decode=decode, ctx_lo=lo, ctx_hi=rng.randint(lo, 2048),
                    prompt=prompt, start=rng.choice([0, rng.randint(1, 1024)]) if prompt else 0)
    if kind == "attention":
        if rng.random() < 0.5:
            lo = _log_int(rng, 8, 4096)
            return dict(kind=kind, dtype=dtype, **shape, decode=_log_int(rng, 1, 64), ctx_lo=lo, ctx_hi=rng.randint(lo, 4096),
                        prompt=0, start=0)
        return dict(kind=kind, dtype=dtype, **shape, decode=0, ctx_lo=0, ctx_hi=0, prompt=_log_int(rng, 16, 2048),
                    start=rng.choice([0, rng.randint(1, 2048)]))
    if kind == "mlp":
        return dict(kind=kind, dtype=dtype, rows=_log_int(rng, 1, 2048), hidden=8 * rng.randint(32, 512), inner=8 * rng.randint(64, 1792))
    if kind == "head":
        return dict(kind=kind, dtype=dtype, rows=_log_int(rng, 1, 64), hidden=64 * rng.randint(8, 64), vocab=_log_int(rng, 16000, 130000))
    groups = rng.choice([1, 4, 8])
    experts = groups * rng.choice([4, 8])
    keep = max(1, groups // 2)
    return dict(kind=kind, dtype=dtype, rows=_log_int(rng, 1, 2048), hidden=64 * rng.randint(8, 32), experts=experts, groups=groups,
                keep=keep, top=min(rng.randint(1, 8), keep * (experts // groups)), inner=64 * rng.randint(4, 22), shared=64 * rng.randint(8, 44))


def _cost(case):
    """Seconds that the work takes at rough rates of the device: for keeping drawn cases within the listed ones."""
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / (70e12 if case["dtype"] == "float32" else 1.6e15))


def draw(rng):
    limit = {d: max(_cost(c) for c in listed() if c["dtype"] == d) for d in ("bfloat16", "float32")}
    while True:
        case = _draw_once(rng)
        if case.get("heads", 0) * case.get("head_dim", 0) <= 4096 and _cost(case) <= limit[case["dtype"]]:
            return case


# -- sizes ------------------------------------------------------------------------------------------

def _lengths(case):
    """Contexts of the decoding requests: spread evenly over ctx_lo .. ctx_hi, in a mixed order."""
    n, lo, hi = case["decode"], case["ctx_lo"], case["ctx_hi"]
    spread = [lo + (hi - lo) * i // max(n - 1, 1) for i in range(n)]
    random.Random(n).shuffle(spread)
    return spread


def _sequences(case):
    """(tokens in the cache, new tokens) of every request of a step."""
    seqs = [(c, 1) for c in _lengths(case)]
    if case["prompt"]:
        seqs.append((case["start"], case["prompt"]))
    return seqs


def work(case):
    e = 4 if case["dtype"] == "float32" else 2
    kind, h = case["kind"], case["hidden"]
    if kind == "mlp":
        w = 3 * h * case["inner"]
        return {"bytes": w * e + case["rows"] * h * (e + 8), "flops": 2 * case["rows"] * w}
    if kind == "head":
        w = h * case["vocab"]
        return {"bytes": w * e + case["rows"] * (4 * h + 4 * case["vocab"]), "flops": 2 * case["rows"] * w}
    if kind == "routed":
        pairs = case["rows"] * case["top"]
        # experts that a step of that many choices touches, if they fall evenly
        used = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** case["rows"])
        one, shared = 3 * h * case["inner"], 3 * h * case["shared"] + h * case["experts"]
        return {"bytes": (used * one + shared) * e + case["rows"] * h * (e + 8), "flops": 2 * (pairs * one + case["rows"] * shared)}
    q, kv = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    seqs = _sequences(case)
    rows = sum(n for _, n in seqs)
    w = h * (2 * q + 2 * kv)
    cached = sum(c + n for c, n in seqs)
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in seqs)
    layer = {"bytes": w * e + 2 * kv * e * cached, "flops": 2 * rows * w + 4 * q * pairs}
    if kind == "attention":
        return {"bytes": layer["bytes"] + rows * h * (e + 8), "flops": layer["flops"]}
    mlp = 3 * h * case["inner"]
    head, out = h * case["vocab"], len(seqs)
    return {"bytes": case["layers"] * (layer["bytes"] + mlp * e) + head * e + out * 4 * case["vocab"],
            "flops": case["layers"] * (layer["flops"] + 2 * rows * mlp) + 2 * out * head}


def tolerance(case):
    """About four times what the path is off from 64 bits: 2e-6 for the 32-bit feed-forward, 1.1e-5 for the 32-bit attention
    (angles of thousands of radians in 32 bits), 0.0017 to 0.0048 for a layer in bfloat16, 0.005 to 0.013 for a whole model."""
    if case["dtype"] == "float32":
        return {"rel": 8e-6, "max": 2e-4} if case["kind"] == "mlp" else {"rel": 4e-5, "max": 1e-3}
    if case["kind"] == "step":
        return {"rel": 0.03, "max": 0.3}
    if case["kind"] == "head":  # tokens are drawn from the logits: a draw on the edge of two may fall either way
        return {"rel": 0.007, "max": 0.07, "differ": 0.01}
    return {"rel": 0.016, "max": 0.16}


# -- inputs, from the seed alone ----------------------------------------------------------------------

def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _normal(name, shape, seed, std, dtype=torch.float32):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
    return (torch.randn(shape, generator=gen, device=DEVICE) * std).to(dtype)


def _norm_weight(name, width, seed):
    return 1.0 + _normal(name, (width,), seed, 0.1)


def _layer_tensors(case, seed, i):
    """The tensors of decoder layer i (attention layers alone keep a feed-forward of no consequence)."""
    dt, h, p = _dtype(case), case["hidden"], f"model.layers.{i}"
    q, kv = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    inner = case.get("inner", 64)
    shapes = {"self_attn.q_proj": (q, h), "self_attn.k_proj": (kv, h), "self_attn.v_proj": (kv, h), "self_attn.o_proj": (h, q),
              "mlp.gate_proj": (inner, h), "mlp.up_proj": (inner, h), "mlp.down_proj": (h, inner)}
    out = {f"{p}.{k}.weight": _normal(f"{p}.{k}", s, seed, 0.02, dt) for k, s in shapes.items()}
    for k in ("input_layernorm", "post_attention_layernorm"):
        out[f"{p}.{k}.weight"] = _norm_weight(f"{p}.{k}", h, seed)
    return out


def _outer_tensors(case, seed):
    h = case["hidden"]
    # (entries of size 1: a stream that its layers add to, as in a trained model, rather than one that they drown)
    return {"model.embed_tokens.weight": _normal("embed", (case.get("vocab", 256), h), seed, 1.0, _dtype(case)),
            "model.norm.weight": _norm_weight("norm", h, seed)}


def _cached(case, seed, layer):
    """Keys and values of every request's cached positions: [pages, PAGE, kv heads, head size], request after request."""
    pages = sum((c + PAGE - 1) // PAGE for c, _ in _sequences(case))
    shape = (pages, PAGE, case["kv_heads"], case["head_dim"])
    std = 0.02 * math.sqrt(case["hidden"])  # what the projections of normed rows give
    return _normal(f"k{layer}", shape, seed, std, _dtype(case)), _normal(f"v{layer}", shape, seed, std, _dtype(case))


def _tokens(case, seed):
    r = random.Random(seed)
    return [[r.randrange(case.get("vocab", 256)) for _ in range(n)] for _, n in _sequences(case)]


def _rows(case, seed, n):
    """Normed rows in the activation type, and the rows of the residual stream that the output is added to."""
    return _normal("xn", (n, case["hidden"]), seed, 1.0, _dtype(case)), _normal("x", (n, case["hidden"]), seed, 0.02)


def _serving_state(case, seed):
    """A decoder of the case's layers, its cache filled with the requests' contexts, and a step function."""
    layers, seqs = case.get("layers", 1), _sequences(case)
    tensors = _outer_tensors(case, seed)
    for i in range(layers):
        tensors.update(_layer_tensors(case, seed, i))
    top = max(c + n for c, n in seqs)
    cfg = LlamaConfig(vocab_size=case.get("vocab", 256), hidden_size=case["hidden"], num_hidden_layers=layers,
                      num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], head_dim=case["head_dim"],
                      intermediate_size=case.get("inner", 64), rope_theta=THETA, rms_norm_eps=EPS, tie_word_embeddings=True,
                      max_position_embeddings=(top + 255) // 256 * 256)
    model = Model.from_tensors(cfg, tensors, dtype=case["dtype"], device=DEVICE)
    del tensors
    # pages for the contexts, and for what a pass adds to its forks
    pages = sum((c + PAGE - 1) // PAGE + (n + PAGE - 1) // PAGE + 1 for c, n in seqs)
    manager, storage = build_cache(model.decoder, pages, PAGE, 2 * len(seqs), _dtype(case), DEVICE)
    ids = []
    for s, (c, _) in enumerate(seqs):
        manager.begin(("kept", s))
        if c:
            assert manager.ensure(("kept", s), c)
            manager.advance(("kept", s), c)
            ids += manager.get(("kept", s)).tables[0]
    if ids:
        at = torch.tensor(ids, device=DEVICE)
        for i in range(layers):
            k, v = _cached(case, seed, i)
            storage.k[i][at], storage.v[i][at] = k.transpose(1, 2), v.transpose(1, 2)
    stepper = Stepper(model.decoder, manager, storage, model.ops, max_rows=sum(n for _, n in seqs), max_seqs=len(seqs),
                      max_tokens_per_request=(top + PAGE) // PAGE * PAGE)
    return model, manager, stepper


def _context(ops, n, rows=None):
    """What a step hands to parts that look at nothing but its rows."""
    return StepContext(ops=ops, workspace=Workspace(DEVICE, n), n=n, num_seqs=1, tokens=None, pos=None, row_seq=None, seq_row0=None,
                       seq_pos0=None, seq_slot=None, logit_rows=rows, num_logit_rows=n if rows is not None else 0, max_keys=n)


def _mlp_tensors(case, seed, prefix="mlp", names=("gate_proj.weight", "up_proj.weight", "down_proj.weight"), inner=None):
    h, inner = case["hidden"], inner or case["inner"]
    shapes = ((inner, h), (inner, h), (h, inner))
    return {f"{prefix}.{n}": _normal(f"{prefix}.{n}", s, seed, 0.02, _dtype(case)) for n, s in zip(names, shapes)}


def _routed_tensors(case, seed):
    out = {}
    for e in range(case["experts"]):
        out.update(_mlp_tensors(case, seed, f"ffn.e{e}", ("gate", "up", "down")))
    out.update(_mlp_tensors(case, seed, "ffn.shared", ("gate", "up", "down"), case["shared"]))
    out["ffn.router"] = _normal("router", (case["experts"], case["hidden"]), seed, 0.02, _dtype(case))
    out["ffn.correction"] = _normal("correction", (case["experts"],), seed, 0.1)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        model, manager, stepper = _serving_state(case, seed)
        return dict(kind=kind, model=model, manager=manager, stepper=stepper, tokens=_tokens(case, seed))
    if kind == "attention":
        model, manager, stepper = _serving_state(case, seed)
        entries = [StepEntry(("kept", s), t, []) for s, t in enumerate(_tokens(case, seed))]
        ctx, _ = stepper.prepare(entries)
        n = sum(n for _, n in _sequences(case))
        # (the step function fills a decode batch up to a round size with rows of no request)
        xn, x0 = (torch.cat([t, t.new_zeros(ctx.n - n, t.shape[1])]) for t in _rows(case, seed, n))
        return dict(kind=kind, part=model.decoder.blocks[0].mixer, ctx=ctx, view=ctx.cache_views[0], xn=xn, x0=x0, x=torch.empty_like(x0),
                    rows=n, keep=(model, manager, stepper))
    ops = get_ops(case["dtype"])
    n = case["rows"]
    if kind == "head":
        norm = RMSNorm(case["hidden"], EPS)
        head = OutputHead(case["vocab"], case["hidden"], norm)
        head.load_params({"model.norm.weight": _norm_weight("norm", case["hidden"], seed),
                          "lm_head.weight": _normal("lm_head", (case["vocab"], case["hidden"]), seed, 0.02, _dtype(case))})
        r = random.Random(seed)
        rows = torch.arange(n, dtype=torch.int32, device=DEVICE)
        return dict(kind=kind, part=head, ctx=_context(ops, n, rows), ops=ops, x=_normal("x", (n, case["hidden"]), seed, 1.0),
                    # every other request is greedy, the others sample at an ordinary temperature
                    temperature=torch.tensor([0.8 * (i % 2) for i in range(n)], device=DEVICE),
                    uniform=torch.tensor([r.random() for _ in range(n)], dtype=torch.float64, device=DEVICE),
                    tokens=torch.zeros(n, dtype=torch.int32, device=DEVICE))
    if kind == "mlp":
        part = SwiGLU(case["hidden"], case["inner"])
        part.load_params(_mlp_tensors(case, seed), "mlp")
        part.prepare(ops)
    else:
        part = RoutedFFN(case["hidden"], case["experts"], case["top"], case["inner"], GLU_LIMIT, GLU_ALPHA, 1.0, case["groups"], case["keep"],
                         shared=ClampedGLU(case["hidden"], case["shared"], GLU_LIMIT, GLU_ALPHA))
        part.load_params(_routed_tensors(case, seed), "ffn")
        part.prepare(ops)
    xn, x0 = _rows(case, seed, n)
    return dict(kind=kind, part=part, ctx=_context(ops, n), xn=xn, x0=x0, x=torch.empty_like(x0))


def run(state):
    kind = state["kind"]
    if kind == "step":
        manager, stepper = state["manager"], state["stepper"]
        entries = []
        for s, tokens in enumerate(state["tokens"]):
            manager.fork(("kept", s), ("pass", s))
            entries.append(StepEntry(("pass", s), tokens, [len(tokens) - 1]))
        logits = stepper.run(entries)
        for e in entries:
            stepper.finish(e.rid)
        return logits
    if kind == "head":
        logits = state["part"].forward(state["ctx"], state["x"])
        state["ops"].sample_rows(logits, state["temperature"], state["uniform"], state["tokens"])
        return logits, state["tokens"]
    state["x"].copy_(state["x0"])
    if kind == "attention":
        state["part"].forward(state["ctx"], state["xn"], state["x"], state["view"])
        # the rows, and the cache with the rows' keys and values stored in it
        return state["x"][:state["rows"]], state["view"].k, state["view"].v
    state["part"].forward(state["ctx"], state["xn"], state["x"])
    return state["x"]


# -- the same in 64 bits -------------------------------------------------------------------------------

def _d(t):
    return t.to(torch.float64)


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * _d(w)


def _rotate(x, pos, head_dim):
    """x [rows, heads, head size]; entries i and i + head size / 2 turn together."""
    half = head_dim // 2
    freq = THETA ** (-torch.arange(half, dtype=torch.float64, device=DEVICE) * 2 / head_dim)
    ang = pos.to(torch.float64)[:, None] * freq[None, :]
    c, s = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attention_exact(case, seed, layer, t, xn):
    """The attention layer's output for the normed rows of all requests, request after request."""
    heads, kvh, hd = case["heads"], case["kv_heads"], case["head_dim"]
    p = f"model.layers.{layer}.self_attn"
    k_all, v_all = _cached(case, seed, layer)
    out, row, page = [], 0, 0
    for c, n in _sequences(case):
        xs = xn[row:row + n]
        pos = torch.arange(c, c + n, device=DEVICE)
        q = _rotate((xs @ _d(t[f"{p}.q_proj.weight"]).T).view(n, heads, hd), pos, hd)
        k = _rotate((xs @ _d(t[f"{p}.k_proj.weight"]).T).view(n, kvh, hd), pos, hd)
        v = (xs @ _d(t[f"{p}.v_proj.weight"]).T).view(n, kvh, hd)
        pages = (c + PAGE - 1) // PAGE
        k = torch.cat([_d(k_all[page:page + pages]).reshape(-1, kvh, hd)[:c], k])
        v = torch.cat([_d(v_all[page:page + pages]).reshape(-1, kvh, hd)[:c], v])
        seen = torch.arange(c + n, device=DEVICE)[None, :] <= pos[:, None]
        o = torch.empty(n, heads, hd, dtype=torch.float64, device=DEVICE)
        for h in range(heads):
            g = h // (heads // kvh)
            s = (q[:, h] @ k[:, g].T) / math.sqrt(hd)
            o[:, h] = torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, g]
        out.append(o.reshape(n, -1))
        row, page = row + n, page + pages
    return torch.cat(out) @ _d(t[f"{p}.o_proj.weight"]).T


def _glu(t, p, xn, names, act):
    g, u, d = (_d(t[f"{p}.{n}"]) for n in names)
    return act(xn @ g.T, xn @ u.T) @ d.T


def _swiglu(g, u):
    return torch.nn.functional.silu(g) * u


def _clamped(g, u):
    g, u = g.clamp(max=GLU_LIMIT), u.clamp(-GLU_LIMIT, GLU_LIMIT)
    return g * torch.sigmoid(GLU_ALPHA * g) * (u + 1)


def _routed_exact(case, seed, xn):
    t = _routed_tensors(case, seed)
    score = torch.sigmoid(xn @ _d(t["ffn.router"]).T)
    choice = score + _d(t["ffn.correction"])
    per = case["experts"] // case["groups"]
    grouped = choice.view(-1, case["groups"], per)
    kept = grouped.topk(min(2, per), -1).values.sum(-1).topk(case["keep"], -1).indices
    mask = torch.zeros(choice.shape[0], case["groups"], dtype=torch.bool, device=DEVICE).scatter_(1, kept, True)
    chosen = grouped.masked_fill(~mask[:, :, None], -math.inf).reshape(choice.shape).topk(case["top"], -1).indices
    names = ("gate", "up", "down")
    out = _glu(t, "ffn.shared", xn, names, _clamped)
    for e in range(case["experts"]):
        rows = (chosen == e).any(-1).nonzero()[:, 0]
        if rows.numel():
            out[rows] += score[rows, e, None] * _glu(t, f"ffn.e{e}", xn[rows], names, _clamped)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        outer = _outer_tensors(case, seed)
        table = _d(outer["model.embed_tokens.weight"])
        tokens = _tokens(case, seed)
        x = table[torch.tensor([t for ts in tokens for t in ts], device=DEVICE)]
        for i in range(case["layers"]):
            t, p = _layer_tensors(case, seed, i), f"model.layers.{i}"
            x = x + _attention_exact(case, seed, i, t, _rms(x, t[f"{p}.input_layernorm.weight"]))
            xn = _rms(x, t[f"{p}.post_attention_layernorm.weight"])
            x = x + _glu(t, f"{p}.mlp", xn, ("gate_proj.weight", "up_proj.weight", "down_proj.weight"), _swiglu)
        last = torch.tensor([len(ts) for ts in tokens], device=DEVICE).cumsum(0) - 1
        return _rms(x[last], outer["model.norm.weight"]) @ table.T
    if kind == "head":
        x = _d(_normal("x", (case["rows"], case["hidden"]), seed, 1.0))
        w = _d(_normal("lm_head", (case["vocab"], case["hidden"]), seed, 0.02, _dtype(case)))
        return _rms(x, _norm_weight("norm", case["hidden"], seed)) @ w.T, None
    n = case["rows"] if kind in ("mlp", "routed") else sum(n for _, n in _sequences(case))
    xn, x0 = (_d(t) for t in _rows(case, seed, n))
    if kind == "attention":
        return x0 + _attention_exact(case, seed, 0, _layer_tensors(case, seed, 0), xn), None, None
    if kind == "mlp":
        return x0 + _glu(_mlp_tensors(case, seed), "mlp", xn, ("gate_proj.weight", "up_proj.weight", "down_proj.weight"), _swiglu)
    return x0 + _routed_exact(case, seed, xn)
