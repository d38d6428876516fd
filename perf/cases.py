"""The work that a program has this engine do, as cases to time and to compare.

Most cases are one layer's own work through the function that the layers themselves come through: attention over the
paged cache (``attend_over_pages``), the matrix memories' recurrences, the routed experts' layer, the residual stream's
norms. Two are whole calls of ``Engine.step``: a prompt, and a generation (prompts, then one token a step).

A case is a dict of plain values; ``portions`` is a text "new@cached,new@cached,...": what every request of the step
brings and what the cache holds of it already.
"""
import math
import random

import torch

from hi_b200.engine.core import Engine, StepEntry
from hi_b200.kernels import ops
from hi_b200.parts import feed_forward  # noqa: F401  (registers the experts' layer)
from hi_b200.parts.attention import attend_over_pages
from hi_b200.parts.context import StepContext
from hi_b200.parts.registry import BuildEnv, build
from hi_b200.parts.spec import PartSpec

DEV = "cuda:0"
PAGE = 64
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def listed():
    return [
        # a chat's next token: one request, a thousand keys; launches and latency
        dict(name="attention_decode_1x1000", op="attention", dtype="bfloat16", heads=40, kv_heads=8, dim=128, chunk=0,
             window=0, portions="1@999"),
        # a full serving batch's next tokens, contexts as uneven as requests are
        dict(name="attention_decode_64_ragged", op="attention", dtype="bfloat16", heads=40, kv_heads=8, dim=128, chunk=0,
             window=0, portions=",".join(f"1@{200 + (i * 2477) % 3801}" for i in range(64))),
        # a prompt in one portion
        dict(name="attention_prompt_2048", op="attention", dtype="bfloat16", heads=40, kv_heads=8, dim=128, chunk=0,
             window=0, portions="2048@0"),
        # a mixed step on a layer of 8,192-token chunks: later portions of long prompts beside decoding requests
        dict(name="attention_mixed_chunked", op="attention", dtype="bfloat16", heads=40, kv_heads=8, dim=128, chunk=8192,
             window=0, portions="513@7000,1@8190,200@1234,1@500,1@3000,129@0,1@12000"),
        # the true 32-bit path: a prompt's second portion
        dict(name="attention_prompt_f32_600", op="attention", dtype="float32", heads=16, kv_heads=4, dim=128, chunk=0,
             window=0, portions="600@301"),
        # the gated delta rule, decay per key channel: a prompt in one portion
        dict(name="memory_delta_2048", op="memory", kind="delta", heads=16, kv_heads=16, dim=128, vdim=128,
             portions="2048@0"),
        # the mLSTM's matrix memory: ragged portions of two prompts beside single tokens
        dict(name="memory_mlstm_ragged", op="memory", kind="mlstm", heads=16, kv_heads=16, dim=128, vdim=128,
             portions="1101@0,1@77,467@512,1@2000"),
        # Mamba-2: 32 decoding requests, every state read and written once
        dict(name="memory_mamba2_decode_32", op="memory", kind="mamba2", heads=32, kv_heads=8, dim=128, vdim=128,
             portions=",".join("1@100" for _ in range(32))),
        # decoding: 8 tokens through 16 experts of 8,192 with a shared one, top 1 (weights are what moves)
        dict(name="experts_8_tokens", op="experts", hidden=5120, inter=8192, experts=16, top_k=1, tokens=8, shared=True,
             output_scale=False),
        # a prompt's experts: 2 of 8 experts of 4,096 a token, scores on the outputs
        dict(name="experts_2048_tokens", op="experts", hidden=2048, inter=4096, experts=8, top_k=2, tokens=2048,
             shared=False, output_scale=True),
        # a prompt through a layer's residual stream: embedding, norm, sum + norm (with the router's copy), sum with
        # routed rows + norm
        dict(name="stream_2048", op="stream", hidden=5120, tokens=2048, top_k=1, vocab=32000),
        # whole calls, prompt and decoding: five requests of uneven prompts, then a token a step
        dict(name="engine_generate", op="engine", model="vinurax", width=2048, heads=16, ff=8192, layers=3,
             portions="37@0,300@0,511@0,128@0,990@0", steps=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    op = rng.choice(["decode", "decode", "prompt", "prompt", "memory", "memory", "memory", "experts", "experts", "stream",
                     "engine"])
    if op in ("decode", "prompt"):
        heads, kv = rng.choice([(40, 8), (16, 4), (32, 8), (8, 2), (24, 24)])
        dim = rng.choice([64, 128, 128, 192])
        mask = rng.choice(["", "", "chunk", "window"])
        case = dict(op="attention", dtype="bfloat16", heads=heads, kv_heads=kv, dim=dim, chunk=8192 if mask == "chunk" else 0,
                    window=rng.choice([1024, 4096]) if mask == "window" else 0)
        if op == "decode":
            n, longest = _log(rng, 1, 64), _log(rng, 64, 16384)
            if n * longest > 160000:
                longest = 160000 // n
            case["portions"] = ",".join(f"1@{rng.randint(longest // 3, longest)}" for _ in range(n))
            return case
        if rng.random() < 0.2:                     # the 32-bit path
            case.update(dtype="float32", heads=8, kv_heads=2, dim=rng.choice([64, 128, 80]))
            case["portions"] = f"{_log(rng, 2, 600)}@{_log(rng, 1, 600) - 1}"
            return case
        parts, left = [], 2048
        for _ in range(rng.choice([1, 1, 2, 3])):
            new = min(_log(rng, 2, 2048), left)
            if new < 2:
                break
            left -= new
            parts.append(f"{new}@{rng.choice([0, _log(rng, 1, 16384 if new < 1024 else 2048)])}")
        parts += [f"1@{_log(rng, 16, 8192)}" for _ in range(rng.choice([0, 0, 2, 5]))]
        case["portions"] = ",".join(parts)
        return case
    if op == "memory":
        kind = rng.choice(["delta", "delta_head", "gla", "mamba2", "mlstm"])
        heads = rng.choice([4, 8, 16, 32])
        case = dict(op="memory", kind=kind, heads=heads, kv_heads=heads // rng.choice([1, 2, 4]) if kind != "mlstm" else heads,
                    dim=rng.choice([64, 96, 128, 128]), vdim=rng.choice([64, 80, 128, 128]))
        if rng.random() < 0.4:
            case["portions"] = ",".join("1@9" for _ in range(_log(rng, 1, 64)))
        else:
            left = _log(rng, 16, 2048)
            parts = []
            while left > 0 and len(parts) < 4:
                n = left if len(parts) == 3 else rng.randint(1, left)
                parts.append(f"{n}@{rng.choice([0, 100])}")
                left -= n
            case["portions"] = ",".join(parts)
        return case
    if op == "experts":
        hidden, inter, experts, top_k = rng.choice([(2048, 4096, 8, 2), (1024, 2048, 16, 4), (2048, 8192, 16, 1), (5120, 8192, 16, 1)])
        return dict(op="experts", hidden=hidden, inter=inter, experts=experts, top_k=top_k,
                    tokens=_log(rng, 1, 2048 if hidden * inter < 2e7 else 256), shared=rng.random() < 0.5,
                    output_scale=rng.random() < 0.5)
    if op == "stream":
        return dict(op="stream", hidden=rng.choice([1024, 2048, 4096, 5120]), tokens=_log(rng, 1, 2048),
                    top_k=rng.choice([1, 2, 4]), vocab=32000)
    model = rng.choice(["vinurax", "surinex", "dense"])
    return dict(op="engine", model=model, width=rng.choice([1024, 2048]), heads=8, ff=4096, layers=3,
                portions=",".join(f"{_log(rng, 4, 500)}@0" for _ in range(rng.randint(1, 4))), steps=rng.randint(2, 12))


# --------------------------------------------------------------------------- inputs
def _portions(case):
    return [tuple(int(v) for v in p.split("@")) for p in case["portions"].split(",")]


def _context(portions, generator, pages=True):
    """The step's tables, as the engine lays them out: pages of a request anywhere in the pool."""
    n_new, start = [n for n, _c in portions], [c for _n, c in portions]
    cu = [0]
    for n in n_new:
        cu.append(cu[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    positions = torch.cat([torch.arange(c, c + n) for n, c in portions]).to(torch.int32).to(DEV)
    seq = torch.repeat_interleave(torch.arange(len(portions)), torch.tensor(n_new)).to(torch.int32).to(DEV)
    ctx = StepContext(n_tokens=cu[-1], n_seqs=len(portions), tokens=torch.zeros(cu[-1], dtype=torch.int32, device=DEV),
                      positions=positions, seq_of_token=seq, cu_seqlens=i32(cu), slots=i32(list(range(len(portions)))),
                      start_pos=start, n_new=n_new, slot_ids=list(range(len(portions))), page_size=PAGE,
                      max_context=max(n + c for n, c in portions))
    singles = [i for i, n in enumerate(n_new) if n == 1]
    if singles and len(singles) < len(n_new):
        ctx.decode_rows = torch.tensor([cu[i] for i in singles], dtype=torch.int64, device=DEV)
        ctx.decode_max_context = max(start[i] + 1 for i in singles)
    if not pages:
        return ctx, None
    need = [-(-(n + c) // PAGE) for n, c in portions]
    order = torch.randperm(sum(need), device=DEV, generator=generator).to(torch.int32)
    table = torch.zeros((len(portions), max(need)), dtype=torch.int32, device=DEV)
    at = 0
    for s, k in enumerate(need):
        table[s, :k] = order[at: at + k]
        at += k
    return ctx, table


def _attention_state(case, g):
    dtype = BF16 if case["dtype"] == "bfloat16" else F32
    nh, nkv, hd = case["heads"], case["kv_heads"], case["dim"]
    ctx, table = _context(_portions(case), g)
    n_pages = int(sum(-(-(n + c) // PAGE) for n, c in _portions(case)))
    rnd = lambda *shape: torch.randn(*shape, device=DEV, generator=g)
    return dict(q=rnd(ctx.n_tokens, nh, hd).to(dtype), k=rnd(n_pages, nkv, PAGE, hd).to(dtype),
                v=rnd(n_pages, nkv, PAGE, hd).to(dtype), table=table, ctx=ctx)


def _memory_state(case, g):
    h, kvh, d, vd, kind = case["heads"], case["kv_heads"], case["dim"], case["vdim"], case["kind"]
    portions = _portions(case)
    ctx, _ = _context(portions, g, pages=False)
    n, s = ctx.n_tokens, ctx.n_seqs
    rnd = lambda *shape: torch.randn(*shape, device=DEV, generator=g)
    soft = torch.nn.functional.softplus
    fresh = torch.tensor([0.0 if c == 0 else 1.0 for _n, c in portions], device=DEV).view(-1, 1)   # a prompt starts at zero
    if kind == "mlstm":
        proj = (0.5 * rnd(n, h * (2 * d + vd))).to(BF16)
        z = rnd(n, 2 * h)
        z[:, h:] += 3.0                                         # forget gates near one, as they are set up
        floats = ops.mlstm_state_floats(h, d, vd)
        return dict(ctx=ctx, proj=proj, z=z, initial=0.3 * rnd(s, floats) * fresh, state=torch.empty(s, floats, device=DEV))
    st = dict(ctx=ctx, initial=0.1 * rnd(s, h * d * vd) * fresh, state=torch.empty(s, h * d * vd, device=DEV))
    unit = lambda t: torch.nn.functional.normalize(t.view(n, kvh, d), dim=-1).reshape(n, kvh * d).contiguous()
    silu = torch.nn.functional.silu
    st["beta"] = None
    if kind in ("delta", "delta_head"):
        st["q"], st["k"] = unit(silu(rnd(n, kvh * d))) * d ** -0.5, unit(silu(rnd(n, kvh * d)))
        st["v"], st["beta"] = silu(rnd(n, h * vd)), torch.sigmoid(rnd(n, h))
        rate = torch.exp(1.5 * torch.rand(h, 1, device=DEV, generator=g))
        per = rnd(n, h, d if kind == "delta" else 1)
        st["decay"] = torch.exp(-rate * soft(per - 4.0)).expand(n, h, d).reshape(n, h * d).contiguous()
    elif kind == "gla":
        st["q"], st["k"], st["v"] = rnd(n, kvh * d) * d ** -0.5, rnd(n, kvh * d), rnd(n, h * vd)
        st["decay"] = torch.sigmoid(rnd(n, h * d)) ** (1.0 / 16.0)
    else:
        st["q"], st["k"] = silu(rnd(n, kvh * d)), silu(rnd(n, kvh * d))
        dt = soft(rnd(n, h) - 3.0)
        st["v"] = (silu(rnd(n, h, vd)) * dt.unsqueeze(-1)).reshape(n, h * vd).contiguous()
        rate = 1.0 + 15.0 * torch.rand(h, device=DEV, generator=g)
        st["decay"] = torch.exp(-rate * dt).unsqueeze(-1).expand(n, h, d).reshape(n, h * d).contiguous()
    return st


def _expert_tensors(case, g):
    e, i, h = case["experts"], case["inter"], case["hidden"]
    names = {"m.router.weight": (e, h), "m.experts.gate_proj.weight": (e, i, h), "m.experts.up_proj.weight": (e, i, h),
             "m.experts.down_proj.weight": (e, h, i)}
    if case["shared"]:
        names.update({"m.shared_expert.gate_proj.weight": (i, h), "m.shared_expert.up_proj.weight": (i, h),
                      "m.shared_expert.down_proj.weight": (h, i)})
    out = {}
    for name, shape in names.items():
        t = torch.empty(shape, dtype=BF16, device=DEV)
        out[name] = t.normal_(0.0, 0.02, generator=g)
    x = torch.randn(case["tokens"], h, device=DEV, generator=g)
    return out, x


def _experts_state(case, g):
    tensors, x = _expert_tensors(case, g)
    part = build("feed_forward", PartSpec("routed_experts", {
        "hidden_size": case["hidden"], "num_experts": case["experts"], "top_k": case["top_k"],
        "intermediate_size": case["inter"], "shared_expert": case["shared"],
        "scale": "output" if case["output_scale"] else "input"}), BuildEnv(BF16, torch.device(DEV), case["hidden"]), "m")
    part.load(lambda name: tensors[name])
    ctx, _ = _context([(case["tokens"], 0)], g, pages=False)
    return dict(part=part, ctx=ctx, x=x.to(BF16), x32=x)


def _stream_state(case, g):
    n, h, k = case["tokens"], case["hidden"], case["top_k"]
    rnd = lambda *shape: torch.randn(*shape, device=DEV, generator=g)
    return dict(table=rnd(case["vocab"], h).to(BF16), stream=torch.empty(n, h, device=DEV),
                tokens=torch.randint(0, case["vocab"], (n,), device=DEV, generator=g).to(torch.int32),
                w=[(1.0 + 0.1 * rnd(h)).to(BF16) for _ in range(3)], mixed=rnd(n, h).to(BF16), shared=rnd(n, h).to(BF16),
                routed=rnd(n * k, h), slot=torch.randperm(n * k, device=DEV, generator=g).to(torch.int32), k=k)


def _engine_config(case):
    w, heads, ff, layers = case["width"], case["heads"], case["ff"], case["layers"]
    kv = max(1, heads // 4)
    mlp = {"kind": "dense", "ff": ff}
    if case["model"] == "dense":
        return {"architectures": ["Llama4ForCausalLM"], "model_type": "llama4_text", "vocab_size": 32000, "hidden_size": w,
                "num_hidden_layers": layers, "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": 128,
                "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "rope_scaling": None, "attention_chunk_size": 1 << 20,
                "nope_layer_interval": 0, "use_qk_norm": False, "attn_temperature_tuning": False,
                "interleave_moe_layer_step": 0, "num_local_experts": 1, "num_experts_per_tok": 1, "intermediate_size": 8,
                "intermediate_size_mlp": ff, "tie_word_embeddings": True, "max_position_embeddings": 1 << 20}
    if case["model"] == "vinurax":
        latent = {"type": "latent_attention", "mlp": mlp,
                  "mixer": {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": 128, "scale": 128 ** -0.5}}
        delta = {"type": "channel_delta", "mlp": mlp, "mixer": {
            "heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}}
        return {"architecture": "Vinurax", "vocab": 32000, "width": w, "norm": {"eps": 1e-5},
                "layers": [(latent, delta)[i % 2] for i in range(layers)]}
    gla = {"type": "gla", "mixer": {"heads": heads, "dim": 128, "vdim": 128, "tau": 16.0, "decay_rank": 64}, "mlp": mlp}
    pair = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                 "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}},
        "right": {"heads": max(1, heads // 2), "kv_heads": kv, "dim": 128, "vdim": 128, "conv": 4}}}
    latent = {"type": "latent_attention", "mlp": mlp, "mixer": {
        "heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 128, "q_rank": w // 2, "scale": 192 ** -0.5,
        "rot": {"base": 500000.0, "dims": 64}}}
    return {"architecture": "Surinex", "vocab": 32000, "width": w, "norm": {"eps": 1e-5}, "canon": {"taps": 4},
            "layers": [(gla, pair, latent)[i % 3] for i in range(layers)], "loop": {"start": 0, "stop": min(2, layers), "times": 2}}


def _engine_state(case, g, seed):
    portions = _portions(case)
    tokens = sum(-(-(n + case["steps"]) // PAGE) * PAGE for n, _c in portions)
    engine = Engine.from_config(_engine_config(case), seed=seed, std=0.02, dtype="bfloat16", device=DEV, kv_page_size=PAGE,
                                kv_cache_tokens=tokens + PAGE, max_active_requests=len(portions))
    rng = random.Random(seed)
    word = lambda n: [rng.randrange(engine.vocab_size) for _ in range(n)]
    return dict(engine=engine, prompts=[word(n) for n, _c in portions],
                later=[word(len(portions)) for _ in range(case["steps"])])


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    make = {"attention": _attention_state, "memory": _memory_state, "experts": _experts_state, "stream": _stream_state}
    state = _engine_state(case, g, seed) if case["op"] == "engine" else make[case["op"]](case, g)
    state["case"] = case
    return state


# --------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "attention":
        return attend_over_pages(state["q"], state["k"], state["v"], state["table"], state["ctx"], case["heads"],
                                 case["kv_heads"], case["dim"], case["chunk"], case["window"], case["dim"] ** -0.5)
    if op == "memory":
        ctx, st, h, d, vd = state["ctx"], state["state"], case["heads"], case["dim"], case["vdim"]
        st.copy_(state["initial"])                     # the requests' states as the step finds them
        if case["kind"] == "mlstm":
            keep, take, floor = ops.mlstm_gates(state["z"], None, None, 15.0, st, ctx.cu_seqlens, ctx.slots, h, d, vd)
            o, nq = ops.mlstm_recurrence(state["proj"], 0, h * d, 2 * h * d, d ** -0.5, keep, take, st, ctx.cu_seqlens,
                                         ctx.slots, h, d, vd)
            return o, nq, floor, st
        o = ops.delta_recurrence(state["q"], state["k"], state["v"], state["beta"], state["decay"], st, ctx.cu_seqlens,
                                 ctx.slots, h, case["kv_heads"], d, vd, single_tokens=ctx.max_new == 1,
                                 plain=state["beta"] is None)
        return o, st
    if op == "experts":
        return state["part"].forward(state["x"], state["ctx"], state["x32"]).materialize(case["tokens"])
    if op == "stream":
        x = ops.embed_gather(state["table"], state["tokens"], out=state["stream"])
        w = state["w"]
        a = ops.add_rmsnorm(x, None, w[0], 1e-5, BF16)
        b, b32 = ops.add_rmsnorm(x, state["mixed"], w[1], 1e-5, BF16, also_f32=True)
        c = ops.add_rmsnorm(x, state["shared"], w[2], 1e-5, BF16, routed=state["routed"], slot_of_entry=state["slot"],
                            top_k=state["k"])
        return x, a, b, b32, c
    engine, prompts = state["engine"], state["prompts"]
    logits = [engine.step([StepEntry(i, p, [len(p) - 1]) for i, p in enumerate(prompts)])]
    for row in state["later"]:
        logits.append(engine.step([StepEntry(i, [t], [0]) for i, t in enumerate(row)]))
    for i in range(len(prompts)):
        engine.finish(i)
    return logits


# --------------------------------------------------------------------------- what a pass cannot do without
def _visible(case):
    """Per request, the keys that its new tokens read in all, and the distinct ones among them."""
    pairs = distinct = 0
    for n, c in _portions(case):
        lo = c + n
        for p in range(c, c + n):
            first = 0
            if case["chunk"]:
                first = p // case["chunk"] * case["chunk"]
            if case["window"]:
                first = max(first, p - case["window"] + 1)
            pairs += p + 1 - first
            lo = min(lo, first)
        distinct += c + n - lo
    return pairs, distinct


def work(case):
    op = case["op"]
    if op == "attention":
        size = 2 if case["dtype"] == "bfloat16" else 4
        pairs, distinct = _visible(case)
        n = sum(p for p, _c in _portions(case))
        return {"bytes": size * (2 * n * case["heads"] + 2 * distinct * case["kv_heads"]) * case["dim"],
                "flops": 4.0 * pairs * case["heads"] * case["dim"]}
    if op == "memory":
        h, d, vd = case["heads"], case["dim"], case["vdim"]
        n, s = sum(p for p, _c in _portions(case)), len(_portions(case))
        if case["kind"] == "mlstm":
            return {"bytes": 2 * n * h * (2 * d + vd) + 4 * n * h * (vd + 4) + 8 * s * h * (vd + 1) * d,
                    "flops": 5.0 * n * h * d * (vd + 1)}
        inputs = n * (2 * case["kv_heads"] * d + h * (d + vd)) + (n * h if case["kind"].startswith("delta") else 0)
        return {"bytes": 4 * (inputs + n * h * vd) + 8 * s * h * d * vd,
                "flops": (8.0 if case["kind"].startswith("delta") else 5.0) * n * h * d * vd}
    if op == "experts":
        n, h, i, e, k = case["tokens"], case["hidden"], case["inter"], case["experts"], case["top_k"]
        touched = e * (1.0 - (1.0 - k / e) ** n)
        each = touched + (1 if case["shared"] else 0)
        return {"bytes": 2 * 3 * each * h * i + 2 * e * h + n * h * (2 + 4 + 4),
                "flops": 6.0 * n * (k + (1 if case["shared"] else 0)) * h * i}
    if op == "stream":
        n, h, k = case["tokens"], case["hidden"], case["top_k"]
        # rows in: embedding, two results, k routed; rows out: the stream, three normed, one of them in 32 bits too
        return {"bytes": n * h * (3 * 2 + 4 * k + 4 + 3 * 2 + 4), "flops": n * h * (20.0 + k)}
    w, ff, layers = case["width"], case["ff"], case["layers"]
    runs = layers + (min(2, layers) if case["model"] == "surinex" else 0)
    per_layer = (6 if case["model"] == "vinurax" else 4) * w * case["heads"] * 128 + (2 if case["model"] == "vinurax" else 3) * w * ff
    prompt = sum(n for n, _c in _portions(case))
    rows = case["steps"] * len(_portions(case))
    weights = 2 * (layers * per_layer + 32000 * w)
    return {"bytes": weights * (1 + case["steps"]) + 4 * 32000 * (rows + len(_portions(case))),
            "flops": 2.0 * (prompt + rows) * runs * per_layer + 2.0 * 32000 * w * (rows + len(_portions(case)))}


def tolerance(case):
    """About four times the distance between this path and the same in 64 bits (the whole calls: and the same prompts
    cut elsewhere)."""
    op = case["op"]
    if op == "attention":
        return {"rel": 8e-3, "max": 0.18} if case["dtype"] == "bfloat16" else {"rel": 2e-6, "max": 3e-5}
    if op == "memory":
        return {"rel": 1e-6, "max": 1.5e-5}
    if op == "experts":
        return {"rel": 1.2e-2, "max": 0.06}
    if op == "stream":
        return {"rel": 7e-3, "max": 1.6e-2}
    return {"rel": 1e-2, "max": 0.1}


# --------------------------------------------------------------------------- the same in 64 bits
def _exact_attention(case, st):
    nh, nkv, hd = case["heads"], case["kv_heads"], case["dim"]
    out = torch.empty((st["ctx"].n_tokens, nh, hd), dtype=F64, device=DEV)
    at = 0
    for s, (n, c) in enumerate(_portions(case)):
        pages = st["table"][s, : -(-(n + c) // PAGE)].long()
        rows = lambda t, h: t[pages, h].reshape(-1, hd)[: n + c].to(F64)
        p = torch.arange(c, c + n, device=DEV).view(-1, 1)
        j = torch.arange(n + c, device=DEV).view(1, -1)
        hidden = j > p
        if case["chunk"]:
            hidden |= j < p // case["chunk"] * case["chunk"]
        if case["window"]:
            hidden |= j <= p - case["window"]
        for h in range(nkv):
            k, v = rows(st["k"], h), rows(st["v"], h)
            for a in range(h * (nh // nkv), (h + 1) * (nh // nkv)):
                scores = st["q"][at: at + n, a].to(F64) @ k.t() * hd ** -0.5
                out[at: at + n, a] = torch.softmax(scores.masked_fill_(hidden, float("-inf")), dim=1) @ v
        at += n
    return out


def _exact_mlstm(case, st):
    h, d, vd = case["heads"], case["dim"], case["vdim"]
    proj, z = st["proj"].to(F64), st["z"].to(F64)
    n = proj.shape[0]
    q, k = (proj[:, i * h * d: (i + 1) * h * d].view(n, h, d) for i in (0, 1))
    v = proj[:, 2 * h * d:].view(n, h, vd)
    gi, gf = (15.0 * torch.tanh(z[:, i * h: (i + 1) * h] / 15.0) for i in (0, 1))
    gf = torch.nn.functional.logsigmoid(gf)
    final = st["initial"].to(F64).clone()
    o, nq, floor = (torch.empty(s, dtype=F64, device=DEV) for s in ((n, h, vd), (n, h), (n, h)))
    at = 0
    for s, (count, _c) in enumerate(_portions(case)):
        S = final[s, : h * (vd + 1) * d].view(h, vd + 1, d)
        m = final[s, h * (vd + 1) * d:]
        for t in range(at, at + count):
            now = torch.maximum(gf[t] + m, gi[t])
            keep, take = torch.exp(gf[t] + m - now), torch.exp(gi[t] - now)
            vt = torch.cat([v[t], torch.ones(h, 1, dtype=F64, device=DEV)], dim=1)
            S = keep.view(h, 1, 1) * S + (take.view(h, 1) * vt).unsqueeze(2) * k[t].unsqueeze(1)
            out = torch.einsum("hcd,hd->hc", S, q[t]) * d ** -0.5
            o[t], nq[t], floor[t], m = out[:, :vd], out[:, vd], torch.exp(-now), now
        final[s] = torch.cat([S.reshape(-1), m])
        at += count
    return o, nq, floor, final


def _exact_memory(case, st):
    if case["kind"] == "mlstm":
        return _exact_mlstm(case, st)
    h, kvh, d, vd = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
    n = st["q"].shape[0]
    wide = lambda t: t.to(F64).view(n, kvh, d).repeat_interleave(h // kvh, dim=1)
    q, k, v, g = wide(st["q"]), wide(st["k"]), st["v"].to(F64).view(n, h, vd), st["decay"].to(F64).view(n, h, d)
    beta = None if st["beta"] is None else st["beta"].to(F64)
    final = st["initial"].to(F64).clone()
    out = torch.empty((n, h * vd), dtype=F64, device=DEV)
    at = 0
    for s, (count, _c) in enumerate(_portions(case)):
        S = final[s].view(h, d, vd)
        for t in range(at, at + count):
            S = S * g[t].unsqueeze(2)
            u = v[t] if beta is None else beta[t].unsqueeze(1) * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t].unsqueeze(2) * u.unsqueeze(1)
            out[t] = torch.einsum("hdv,hd->hv", S, q[t]).reshape(-1)
        final[s] = S.reshape(-1)
        at += count
    return out, final


def _exact_experts(case, st, g):
    w, x32 = _expert_tensors(case, g)
    x = x32.to(BF16).to(F64)
    silu = torch.nn.functional.silu
    logits = x32.to(F64) @ w["m.router.weight"].to(F64).t()
    top, ids = torch.topk(logits, case["top_k"], dim=1)
    score = torch.sigmoid(top)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        rows, rank = (ids == e).nonzero(as_tuple=True)
        if not rows.numel():
            continue
        s = score[rows, rank].unsqueeze(1)
        xe = x[rows] if case["output_scale"] else x[rows] * s
        gate, up, down = (w[f"m.experts.{n}_proj.weight"][e].to(F64) for n in ("gate", "up", "down"))
        y = (silu(xe @ gate.t()) * (xe @ up.t())) @ down.t()
        out.index_add_(0, rows, y * s if case["output_scale"] else y)
    if case["shared"]:
        gate, up, down = (w[f"m.shared_expert.{n}_proj.weight"].to(F64) for n in ("gate", "up", "down"))
        out += (silu(x @ gate.t()) * (x @ up.t())) @ down.t()
    return out


def _exact_stream(case, st):
    norm = lambda x, w: x / torch.sqrt((x * x).mean(dim=1, keepdim=True) + 1e-5) * w.to(F64)
    x = st["table"].to(F64)[st["tokens"].long()]
    a = norm(x, st["w"][0])
    x = x + st["mixed"].to(F64)
    b = norm(x, st["w"][1])
    x = x + st["shared"].to(F64) + st["routed"].to(F64)[st["slot"].long()].view(case["tokens"], case["top_k"], -1).sum(dim=1)
    return x, a, b, b, norm(x, st["w"][2])


def exact(case, seed):
    if case["op"] == "engine":
        return None
    g = torch.Generator(device=DEV).manual_seed(seed)
    if case["op"] == "experts":
        return _exact_experts(case, None, g)
    st = {"attention": _attention_state, "memory": _memory_state, "stream": _stream_state}[case["op"]](case, g)
    return {"attention": _exact_attention, "memory": _exact_memory, "stream": _exact_stream}[case["op"]](case, st)
