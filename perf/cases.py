"""What is measured of this framework: the work that its users have it do, through its public entry points.

Four kinds of case, each over the range of sizes that `draw` spans:

  attention   paged decode attention as a plug-in of another engine calls it (`ops.paged_attention_decode_batch`)
  projection  a packed projection as such a plug-in calls it (`quantization.quantized_matmul`)
  decode      one step of a batch of running requests (`run_decode_batch`), for every model family
  prompt      prompts of new requests: all logits of Llama-shaped models (`run_prefill_batch`), the last one's of the other families
              (`run_step_batch`) and, as those keep recurrent states, the logits of the token behind it

Models have random weights of the shapes that `bench.py` and `bench_hybrid.py` measure (width 4096: ff 14336, 32 heads; width 2048:
ff 5632, 16 heads; 8 key/value heads, vocabulary 32768), cut to a few layers: deeper ones repeat the same layers. `exact` restates
every family in float64.
"""
from __future__ import annotations

import math
import zlib

import torch

DEV = "cuda"
VOCAB = 32768
SHAPES = {4096: dict(ff=14336, heads=32, kv=8, dim=128, rank=512, rot=64, window=4096, side=256, experts=32, top=4, expert_ff=1792, shared_ff=7168),
          2048: dict(ff=5632, heads=16, kv=8, dim=128, rank=256, rot=64, window=1024, side=128, experts=32, top=4, expert_ff=704, shared_ff=2816)}
# (rows, columns) of projections: those of the two widths, and the shards of an 8-way split of a width of 8192
PROJECTIONS = ((6144, 4096), (4096, 4096), (14336, 4096), (4096, 14336), (4096, 2048), (5632, 2048), (2048, 5632), (1280, 8192), (7168, 8192), (8192, 3584))
ROOM = 512          # tokens that a decoding batch appends before its requests end and as many others take their place


def listed():
    return [
        # the attention of one request with a short context: four layers' launches, nothing but latency
        dict(name="attention one request", kind="attention", batch=1, ctx_min=333, ctx_max=333, dtype="float16", kv="same", layers=4),
        # 64 requests of very different contexts in one launch: the cache streams
        dict(name="attention ragged batch", kind="attention", batch=64, ctx_min=512, ctx_max=8192, dtype="float16", kv="same", layers=1),
        # one request's gate projection in group-wise int4: the weights stream once for a single row
        dict(name="projection int4 1 row", kind="projection", rows=1, n=14336, k=4096, quant="int4_g128", tiled=False, layers=8),
        # the same weights for a batch, in the tile order that the runtime keeps them in
        dict(name="projection int4 32 rows", kind="projection", rows=32, n=14336, k=4096, quant="int4_g128", tiled=True, layers=8),
        # a chat of one user on a small model: every launch is short
        dict(name="decode llama 1", kind="decode", family="llama", width=2048, layers=4, quant="int4_awq", kv="same", batch=1, ctx=499),
        # a server's steady state: 32 requests with 2048 cached tokens each, int8 weights
        dict(name="decode llama 32", kind="decode", family="llama", width=4096, layers=4, quant="int8", kv="same", batch=32, ctx=2048),
        # a few short questions that arrive together
        dict(name="prompt llama short", kind="prompt", family="llama", width=2048, layers=4, quant="int8", prompts="61,17,140,33"),
        # a long prompt
        dict(name="prompt llama long", kind="prompt", family="llama", width=4096, layers=4, quant="int8", prompts="2048"),
        # the other families: two prompts in one step, a server's batch, one prompt of odd length, a small batch
        dict(name="prompt gutorax", kind="prompt", family="gutorax", width=4096, layers=4, prompts="1500,548"),
        dict(name="decode topunex", kind="decode", family="topunex", width=2048, layers=4, batch=32, ctx=1024),
        dict(name="prompt rekodra", kind="prompt", family="rekodra", width=2048, layers=4, prompts="1001"),
        dict(name="decode zimorax", kind="decode", family="zimorax", width=2048, layers=6, batch=8, ctx=700),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Kinds in the shares that the listed cases have; sizes over their whole range."""
    kind = rng.choice(["attention"] * 2 + ["projection"] * 2 + ["llama decode"] * 2 + ["llama prompt"] * 2 + ["family decode"] * 2 + ["family prompt"] * 2)
    if kind == "attention":
        batch, top = _log(rng, 1, 64), _log(rng, 64, 8192)
        return dict(kind="attention", batch=batch, ctx_min=max(1, top // rng.choice([1, 4, 16])), ctx_max=top, dtype=rng.choice(["float16", "float16", "bfloat16"]),
                    kv="same", layers=1 if batch * top > 60000 else 4) if rng.random() < 0.75 else \
            dict(kind="attention", batch=batch, ctx_min=max(1, top // 4), ctx_max=top, dtype="float16", kv="int8", layers=1 if batch * top > 60000 else 4)
    if kind == "projection":
        n, k = rng.choice(PROJECTIONS)
        rows, quant = _log(rng, 1, 128), rng.choice(["int4_g128", "int4_awq", "int8"])
        return dict(kind="projection", rows=rows, n=n, k=k, quant=quant, tiled=rows > 8 or rng.random() < 0.5, layers=8)
    family = "llama" if kind.startswith("llama") else rng.choice(["gutorax", "topunex", "rekodra", "zimorax"])
    width = rng.choice([2048, 4096])
    case = dict(kind=kind.split()[1], family=family, width=width, layers=6 if family == "zimorax" else 4)
    if family == "llama":
        case["quant"] = rng.choice(["int8", "int8", "int4_awq", "int4_g128"])
    if case["kind"] == "decode":
        batch = _log(rng, 1, 32)
        case.update(batch=batch, ctx=_log(rng, 64, 2048 if family == "llama" or batch <= 8 else 1024))
        if family == "llama":
            case["kv"] = rng.choice(["same", "same", "int8"])
    else:
        count, total = rng.choice([1, 1, 2, 5]), _log(rng, 40, 2048)
        cuts = sorted(rng.sample(range(1, total), count - 1))
        case["prompts"] = ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))
    return case


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed, name):
    return torch.Generator(device=DEV).manual_seed(zlib.crc32(name.encode()) ^ (seed * 7919 & 0x7FFFFFFF))


def _randn(seed, name, *shape):
    return torch.randn(shape, device=DEV, generator=_gen(seed, name))


def _weight(seed, name, shape):
    """A model's parameter: what `bench_hybrid.py` gives it, matrices as bfloat16 numbers in float32."""
    if len(shape) <= 1:
        if name.endswith("mix.right.f.b"):
            return torch.full(shape, 4.0, device=DEV)
        if name.endswith(("dt_bias", "A_log")):
            return torch.full(shape, -2.0, device=DEV) + 0.2 * _randn(seed, name, *shape)
        if name.endswith((".b", "correction")):
            return 0.02 * _randn(seed, name, *shape)
        return (0.6 if name.endswith("alpha") else 1.0) + 0.1 * _randn(seed, name, *shape)
    if name.endswith(".talk"):
        return torch.eye(shape[0], device=DEV) + 0.02 * _randn(seed, name, *shape)
    if name.endswith("conv"):
        return 0.5 * _randn(seed, name, *shape)
    return (0.02 * _randn(seed, name, *shape)).to(torch.bfloat16).float()


def _tokens(seed, name, count):
    return torch.randint(0, VOCAB, (count,), device=DEV, generator=_gen(seed, name)).tolist()


def _prompts(case, seed):
    return [_tokens(seed, f"prompt{i}", int(n)) for i, n in enumerate(case["prompts"].split(","))]


def _contexts(case, seed):
    """Cached tokens and the next one of every decoding request."""
    return [_tokens(seed, f"context{i}", case["ctx"] + 1) for i in range(case["batch"])]


def _attention_inputs(case, seed):
    heads, kv, dim, page = 32, 8, 128, 16
    dtype = getattr(torch, case["dtype"])
    span = case["ctx_max"] - case["ctx_min"] + 1
    lens = case["ctx_min"] + torch.randint(0, span, (case["batch"],), device=DEV, generator=_gen(seed, "lens")) if span > 1 else \
        torch.full((case["batch"],), case["ctx_max"], device=DEV)
    pages = (lens + page - 1) // page
    ends = pages.cumsum(0)
    slots = torch.randperm(int(ends[-1]), device=DEV, generator=_gen(seed, "slots"))
    at = torch.arange((case["ctx_max"] + page - 1) // page, device=DEV)[None, :]
    table = torch.where(at < pages[:, None], slots[((ends - pages)[:, None] + at).clamp_max(len(slots) - 1)], 0).int()
    layers = []
    for i in range(case["layers"]):
        shape = (len(slots), kv, page, dim)
        layer = {"q": _randn(seed, f"q{i}", case["batch"], heads, dim).to(dtype), "scales": None}
        for name in ("k", "v"):
            layer[name] = torch.randn(shape, device=DEV, dtype=dtype, generator=_gen(seed, f"{name}{i}"))
        if case["kv"] == "int8":
            both = torch.stack([layer["k"], layer["v"]], dim=2).float()
            layer["scales"] = (both.abs().amax(dim=-1) / 127.0).half()
            codes = (torch.round(both / layer["scales"].float().unsqueeze(-1)) + 128.0).clamp(1, 255).to(torch.uint8)
            layer["k"], layer["v"] = codes[:, :, 0].contiguous(), codes[:, :, 1].contiguous()
        layers.append(layer)
    return layers, table, lens.int()


def _projection_inputs(case, seed, i):
    x = _randn(seed, f"x{i}", case["rows"], case["k"]).half()
    return x, 0.02 * _randn(seed, f"w{i}", case["n"], case["k"])


# ---- models ----------------------------------------------------------------------------------------------------------
def _family_config(family, width, count):
    s = dict(SHAPES[width], width=width)
    heads, kv, dim = s["heads"], s["kv"], s["dim"]
    layers = []
    for i in range(count):
        if family == "gutorax":        # latent attention, recurrence, latent attention on the first one's cache, recurrence
            if i % 2:
                kind, m = "lightning", dict(heads=heads, dim=dim, vdim=dim, decay=[1 - 2.0 ** -(2 + h * 8 / heads) for h in range(heads)])
            else:
                kind, m = "latent_attention", dict(heads=heads, dim=dim, rot_dim=s["rot"], vdim=dim, kv_rank=s["rank"], scale=(dim + s["rot"]) ** -0.5,
                                                   mask={"size": s["window"]}, rot={"base": 500000.0, "dims": s["rot"]})
                if i % 4 == 2:
                    m["kv_from"] = i - 2
            mlp = {"kind": "dense", "ff": s["ff"]}
        elif family == "topunex":      # feed-forward layers and mixtures of experts in turn
            kind = "attention"
            m = dict(heads=heads, kv_heads=kv, dim=dim, vdim=dim, scale=dim ** -0.5, softcap=30.0, mask={"size": s["window"], "keep_first": 4},
                     rot={"base": 500000.0, "dims": s["rot"], "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}})
            moe = {"kind": "moe", "expert": {"ff": s["expert_ff"], "limit": 7.0}, "shared": {"ff": s["shared_ff"], "limit": 7.0},
                   "router": {"experts": s["experts"], "top": s["top"], "scale": 2.0}}
            mlp = moe if i % 2 else {"kind": "dense", "ff": s["ff"]}
        elif family == "rekodra":      # attention over all tokens, and window attention beside matrix memory, in turn
            half = heads // 2
            if i % 2:
                kind = "parallel"
                m = {"left": dict(heads=half, kv_heads=kv, dim=dim, vdim=dim, scale=dim ** -0.5, mask={"size": s["window"]}),
                     "right": dict(heads=half, dim=dim, vdim=dim, gate_cap=15.0)}
            else:
                kind, m = "attention", dict(heads=heads, kv_heads=kv, dim=dim, vdim=dim, scale=dim ** -0.5, rot={"base": 500000.0, "dims": s["rot"]})
            mlp = {"kind": "moe", "expert": {"ff": s["expert_ff"]}, "shared": {"ff": s["shared_ff"]},
                   "router": {"experts": s["experts"] * 7 // 8, "identity": s["experts"] // 8, "top": s["top"], "groups": {"count": 4, "keep": 2}}}
        else:                          # zimorax: talking-heads attention, a state space, a delta rule, in turn
            kind = ("attention", "mamba2", "delta")[i % 3]
            m = (dict(heads=heads, kv_heads=kv, dim=dim, vdim=dim, scale=dim ** -0.5, mask={"size": s["window"]},
                      rot={"base": 500000.0, "dims": s["rot"], "scaling": {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}}),
                 dict(heads=2 * width // 64, vdim=64, state=128, groups=8, norm_groups=8, conv=4),
                 dict(heads=heads, kv_heads=heads // 2, dim=dim, vdim=dim, conv=4))[i % 3]
            mlp = {"kind": "dense", "ff": s["ff"] * 3 // 2}
        layers.append({"type": kind, "mixer": m, "mlp": mlp})
    cfg = {"architecture": family.capitalize(), "width": width, "vocab": VOCAB, "norm": {"eps": 1e-5 if family == "gutorax" else 1e-6}, "layers": layers}
    if family == "gutorax":
        cfg.update(embedding={"scale": width ** 0.5}, token_side={"dim": s["side"]})
    if family == "rekodra":
        cfg.update(embedding={"scale": 1.0}, logit_scale=1.0)
    return cfg


def _artifact(case):
    import cacheir_b200 as C
    s = SHAPES[case["width"]]
    if case["family"] == "llama":
        return C.build_decoder_artifact(C.ModelConfig(
            architecture="LlamaForCausalLM", hidden_size=case["width"], intermediate_size=s["ff"], num_layers=case["layers"], num_attention_heads=s["heads"],
            num_key_value_heads=s["kv"], vocab_size=VOCAB, max_position_embeddings=8192, rope_theta=500000.0, rms_norm_eps=1e-5, dtype="float16"),
            quant=case["quant"], modes=("decode",))
    config, build = {"gutorax": (C.GutoraxConfig, C.build_gutorax_artifact), "topunex": (C.TopunexConfig, C.build_topunex_artifact),
                     "rekodra": (C.RekodraConfig, C.build_rekodra_artifact), "zimorax": (C.ZimoraxConfig, C.build_zimorax_artifact)}[case["family"]]
    return build(config.from_dict(_family_config(case["family"], case["width"], case["layers"])))


def _runtime(case, seed, sequences, tokens):
    import cacheir_b200 as C
    page = 16 if case["family"] == "llama" else 64
    alloc = C.B200KVPageAllocator(page_size=page, initial_slots=sequences * ((tokens + page - 1) // page) + 1, initial_states=sequences)
    options = {"kv_dtype": case.get("kv", "same")} if case["family"] == "llama" else {}
    return C.B200DecodeRuntime(_artifact(case), dtype="float16" if case["family"] == "llama" else "bfloat16", kv_allocator=alloc, max_seq_len=tokens,
                               tensor_source=lambda key, shape: _weight(seed, key, tuple(shape)), **options)


# ---- what a program has in hand, and one pass ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "attention":
        from cacheir_b200 import ops
        layers, table, lens = _attention_inputs(case, seed)
        outs = [torch.empty_like(layer["q"]) for layer in layers]
        batch, heads, dim = outs[0].shape
        splits = ops.attention_auto_splits(batch, heads, 8, int(table.shape[1]), 16, dim)
        scratch = torch.empty(max(1, ops.attention_workspace_bytes(batch, heads, dim, splits) // 4), device=DEV)

        def step():
            for layer, out in zip(layers, outs):
                ops.paged_attention_decode_batch(layer["q"], layer["k"], layer["v"], table, lens, out=out, num_splits=splits, workspace=scratch,
                                                 kv_scales=layer["scales"])
        return _captured(step, outs)
    if case["kind"] == "projection":
        from cacheir_b200 import ops
        from cacheir_b200.quantization import pack_weight_device, quantized_matmul, to_tiled
        work = []
        for i in range(case["layers"]):
            x, dense = _projection_inputs(case, seed, i)
            packed = pack_weight_device(dense, case["quant"])
            work.append((x, to_tiled(packed) if case["tiled"] else packed, torch.empty((case["rows"], case["n"]), device=DEV, dtype=torch.float16)))
        scratch = torch.zeros(ops.qgemv_workspace_bytes(case["rows"], case["k"]), device=DEV, dtype=torch.uint8)

        def step():
            for x, w, out in work:
                quantized_matmul(x, w, out=out, workspace=scratch)
        return _captured(step, [out for _, _, out in work])
    if case["kind"] == "decode":
        rows = _contexts(case, seed)
        rt = _runtime(case, seed, len(rows), case["ctx"] + ROOM + 64)
        sessions = [rt.fork() for _ in rows]
        rt.run_step_batch(sessions, [r[:-3] for r in rows], [[] for _ in rows])
        for back in (3, 2):            # a server is under way: its plan for this batch exists
            rt.run_decode_batch(sessions, [r[-back] for r in rows])
        return {"case": case, "rt": rt, "sessions": sessions, "tokens": [r[-1] for r in rows]}
    prompts = _prompts(case, seed)
    rt = _runtime(case, seed, len(prompts), max(map(len, prompts)) + 1)
    state = {"case": case, "rt": rt, "sessions": [rt.fork() for _ in prompts], "prompts": [p[::-1] for p in prompts], "tokens": _tokens(seed, "next", len(prompts))}
    for _ in range(2):                 # it has served prompts of these lengths before
        run(state)
    return dict(state, prompts=prompts)


def _captured(step, outs):
    """The calls of one decode step as a CUDA graph, the way an engine issues them."""
    for _ in range(2):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    return {"case": None, "graph": graph, "step": step, "outs": outs}


def run(state):
    if state["case"] is None:
        state["graph"].replay()
        return state["outs"]
    case, rt, sessions = state["case"], state["rt"], state["sessions"]
    if case["kind"] == "decode":
        if sessions[0].kv_cache.tokens >= case["ctx"] + ROOM:
            for s in sessions:
                s.kv_cache.clear()
                s.kv_cache.extend(case["ctx"])
        return rt.run_decode_batch(sessions, state["tokens"])
    if case["family"] == "llama":
        return rt.run_prefill_batch(sessions, state["prompts"])
    for s in sessions:
        s.kv_cache.clear()
    return [rt.run_step_batch(sessions, state["prompts"]), rt.run_decode_batch(sessions, state["tokens"])]


# ---- bytes and operations of one pass -----------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "attention":
        keys = case["batch"] * (case["ctx_min"] + case["ctx_max"]) / 2
        row = 128 * 2 if case["kv"] == "same" else 128 + 2
        return {"bytes": case["layers"] * (keys * 8 * 2 * row + 2 * case["batch"] * 32 * 128 * 2), "flops": case["layers"] * 4.0 * keys * 32 * 128}
    if case["kind"] == "projection":
        n, k, m = case["n"], case["k"], case["rows"]
        scales = n * k / 128 * 2 if case["quant"] == "int4_g128" else 8 * n
        return {"bytes": case["layers"] * (n * k * (1 if case["quant"] == "int8" else 0.5) + scales + 2.0 * m * (n + k)), "flops": case["layers"] * 2.0 * m * n * k}
    if case["kind"] == "decode":
        rows, logits, cached, pairs = case["batch"], case["batch"], case["batch"] * case["ctx"], case["batch"] * (case["ctx"] + 1)
    else:
        lens = [int(n) for n in case["prompts"].split(",")]
        rows, cached, pairs = sum(lens), 0, sum(n * (n + 1) / 2 for n in lens)
        logits = rows if case["family"] == "llama" else 2 * len(lens)
    s, width = SHAPES[case["width"]], case["width"]
    h, g, d, rot, rank = s["heads"], s["kv"], s["dim"], s["rot"], s["rank"]
    held = flops = traffic = 0.0           # weights read, operations, cache and state bytes
    each = {"int8": 1.0, "int4_awq": 0.5, "int4_g128": 0.5 + 2 / 128}.get(case.get("quant"), 2.0)

    def matrix(n, k, share=1.0, touched=1.0, t=rows):
        nonlocal held, flops
        held += touched * n * k * each
        flops += 2.0 * t * share * n * k

    def attention(key, value, heads, cache_row):
        nonlocal flops, traffic
        flops += 2.0 * pairs * heads * (key + value)
        traffic += (cached + rows) * cache_row

    def experts(count, top, shared=True):
        touched = count * (1 - (1 - top / s["experts"]) ** rows)
        matrix(3 * s["expert_ff"], width, top, touched)
        if shared:
            matrix(3 * s["shared_ff"], width)

    cfg = None if case["family"] == "llama" else _family_config(case["family"], width, case["layers"])
    for i in range(case["layers"]):
        kind, m = ("llama", {}) if cfg is None else (cfg["layers"][i]["type"], cfg["layers"][i]["mixer"])
        if cfg is None:
            matrix((2 * h + 2 * g) * d, width)
            attention(d, d, h, 2 * g * (d * 2 if case.get("kv", "same") == "same" else d + 2))
            matrix(3 * s["ff"], width)
        elif case["family"] == "gutorax":
            if kind == "lightning":
                matrix(5 * h * d, width)
                traffic += (len(case["prompts"].split(",")) if case["kind"] == "prompt" else 2 * rows) * h * d * d * 4
                flops += 4.0 * rows * h * d * d
            else:
                matrix(h * (3 * d + rot) + (0 if "kv_from" in m else rank + rot), width)
                matrix(2 * h * d, rank)
                attention(rank + rot, rank, h, 2 * (rank + rot))
            matrix(3 * s["ff"] + 2 * s["side"], width)
        elif case["family"] == "topunex":
            matrix((3 * h + g) * d, width)
            attention(d, d, h, g * (2 * (d + rot) + 4))
            if i % 2:
                experts(s["experts"], s["top"])
            else:
                matrix(3 * s["ff"], width)
        elif case["family"] == "rekodra":
            if kind == "attention":
                matrix((2 * h + g) * d, width)
                attention(d, d, h, g * (2 * (d + rot) + 4))
            else:
                matrix(h // 2 * d * 7 + 2 * g * d, width)
                attention(d, d, h // 2, g * (4 * d + 4))
                traffic += (len(case["prompts"].split(",")) if case["kind"] == "prompt" else 2 * rows) * h // 2 * d * (d + 1) * 4
                flops += 4.0 * rows * h // 2 * d * d
            experts(s["experts"] * 7 // 8, s["top"] * 7 / 8)
        else:
            seqs = len(case["prompts"].split(",")) if case["kind"] == "prompt" else 2 * rows
            if kind == "attention":
                matrix((2 * h + 2 * g) * d, width)
                attention(d, d, h, 4 * g * d)
                flops += 2.0 * pairs * h * h
            elif kind == "mamba2":
                inner = 2 * width
                matrix(3 * inner + 2 * 8 * 128 + inner // 64, width)
                traffic += seqs * inner * 128 * 4
                flops += 4.0 * rows * inner * 128
            else:
                matrix((2 * h // 2 + 3 * h) * d + 2 * h, width)
                traffic += seqs * h * d * d * 4
                flops += 6.0 * rows * h * d * d
            matrix(3 * s["ff"], width)
    matrix(VOCAB, width, t=logits)
    return {"bytes": held + traffic + rows * width * 2 + logits * VOCAB * (2 if cfg is None else 4), "flops": flops}


def tolerance(case):
    """About four times the distance from `exact` that the entry points show: one rounding of float16 outputs for the operators,
    the roundings of a few layers' activations for the models. A mixture's choices may differ where two experts score alike."""
    if case["kind"] == "attention":
        return {"rel": 8e-3, "max": 0.1} if case["dtype"] == "bfloat16" else {"rel": 1e-3, "max": 0.02}
    if case["kind"] == "projection":
        return {"rel": 1e-3, "max": 0.02}
    return {"rel": {"llama": 1e-2, "gutorax": 2e-2, "topunex": 2e-2}.get(case["family"], 3e-2), "max": 0.5}


# ---- the same in float64, from the definitions ----------------------------------------------------------------------------
def _unpacked(w, quant):
    """What a packed weight stands for: per row affine codes, or groups of 128 symmetric ones with float16 scales."""
    if quant == "int4_g128":
        groups = w.view(w.shape[0], -1, 128)
        scale = (groups.abs().amax(dim=2) / 7.0).clamp_min(1e-8).half().float().unsqueeze(2)
        return ((torch.round(groups / scale) + 8.0).clamp(0.0, 15.0).double() - 8.0).mul(scale.double()).view(w.shape)
    top = 255 if quant == "int8" else 15
    span = w.amax(dim=1) - w.amin(dim=1)
    scale = (span / torch.full_like(span, top)).clamp_min(1e-8)        # (divided by a number it would be multiplied by the reciprocal)
    zero = torch.round(-w.amin(dim=1) / scale)
    codes = torch.round((w / scale[:, None]).double() + zero.double()[:, None]).clamp(0, top)
    return (codes - zero.double()[:, None]) * scale.double()[:, None]


def _rms(x, eps):
    return x / (x.square().mean(dim=-1, keepdim=True) + eps).sqrt()


def _turned(x, freq, factor=1.0):
    """Entry i of x [tokens, heads, d] turns with entry i + len(freq) by position times freq[i]."""
    half = len(freq)
    angle = (torch.arange(x.shape[0], device=DEV, dtype=torch.float64)[:, None] * freq)[:, None, :]
    c, s = angle.cos() * factor, angle.sin() * factor
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], dim=-1)


def _freq(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=torch.float64) / dims)


def _seen(n, size=None, keep_first=0):
    i = torch.arange(n, device=DEV)
    gap = i[:, None] - i[None, :]
    return (gap >= 0) & ((gap < (size or n)) | (i[None, :] < keep_first))


def _attend(q, k, v, scale, mask, sink=None, cap=None):
    """q [n, H, d], k [n, G, d], v [n, G, e]; with a sink one more exp(sink[h]) in the denominator."""
    out, share = [], q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        z = q[:, h] @ k[:, h // share].T * scale
        z = z if cap is None else cap * torch.tanh(z / cap)
        z = z.masked_fill(~mask, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink[h].expand(len(z), 1)], dim=1)
        p = z.softmax(dim=1)
        out.append(p[:, : len(mask)] @ v[:, h // share])
    return torch.stack(out, dim=1)


class _Params:
    """Parameters of one model in float64, by name; shapes come from the caller."""

    def __init__(self, seed, quant=None):
        self.seed, self.quant, self.kept = seed, quant, {}

    def __call__(self, name, *shape):
        if name not in self.kept:
            w = _weight(self.seed, name, shape)
            if self.quant is not None:
                w = (_unpacked(w, self.quant) if len(shape) == 2 else w.half()).double()
                w = w.half().double() if "embed" in name else w
            self.kept[name] = w.double()
        return self.kept[name]


def _llama(case, w, tokens):
    width, s = case["width"], SHAPES[case["width"]]
    n, h, g, d = len(tokens), s["heads"], s["kv"], s["dim"]
    angle = torch.arange(n, device=DEV, dtype=torch.float64)[:, None, None] * _freq(d, 500000.0)
    c, sn = angle.cos(), angle.sin()

    def rope(t):
        a, b = t[..., 0::2], t[..., 1::2]
        return torch.stack([a * c - b * sn, a * sn + b * c], dim=-1).flatten(-2)
    x = w("model.embed_tokens.weight", VOCAB, width)[tokens]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        y = _rms(x, 1e-5) * w(p + "input_layernorm.weight", width)
        q, k, v = ((y @ w(f"{p}self_attn.{name}_proj.weight", heads * d, width).T).view(n, heads, d) for name, heads in (("q", h), ("k", g), ("v", g)))
        y = _attend(rope(q), rope(k), v, d ** -0.5, _seen(n)).flatten(1)
        x = x + y @ w(p + "self_attn.o_proj.weight", width, width).T
        y = _rms(x, 1e-5) * w(p + "post_attention_layernorm.weight", width)
        gate, up = (y @ w(f"{p}mlp.{name}_proj.weight", s["ff"], width).T for name in ("gate", "up"))
        x = x + (torch.nn.functional.silu(gate) * up) @ w(p + "mlp.down_proj.weight", width, s["ff"]).T
    return lambda rows: (_rms(x[rows], 1e-5) * w("model.norm.weight", width)) @ w("lm_head.weight", VOCAB, width).T


def _gelu(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


def _gutorax(cfg, w, tokens):
    width, eps, n, side = cfg["width"], cfg["norm"]["eps"], len(tokens), cfg["token_side"]["dim"]

    def squash(x, name):
        return torch.tanh(w(name + ".alpha") * x) * w(name, width) + w(name + ".b", width)
    x, caches = w("embed", VOCAB, width)[tokens] * cfg["embedding"]["scale"], {}
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        y, hd = squash(x, p + "norm1"), m["heads"] * m["dim"]
        if layer["type"] == "lightning":
            q, k, v = (torch.nn.functional.silu(y @ w(p + "mix." + name, hd, width).T).view(n, m["heads"], m["dim"]) for name in "qkv")
            gap = torch.arange(n, device=DEV)[:, None] - torch.arange(n, device=DEV)[None, :]
            o = torch.stack([(q[:, h] @ k[:, h].T * torch.where(gap >= 0, float(m["decay"][h]) ** gap.clamp_min(0).double(), 0.0)) @ v[:, h]
                             for h in range(m["heads"])], dim=1)
            o = _rms(o.flatten(1), eps) * w(p + "mix.norm", hd)
        else:
            rot, rank = m["rot_dim"], m["kv_rank"]
            freq = _freq(m["rot"]["dims"], m["rot"]["base"])
            source = m.get("kv_from", i)
            if source == i:
                down = y @ w(p + "mix.dkv", rank + rot, width).T
                caches[i] = (_rms(down[:, :rank], eps) * w(p + "mix.dkv.norm", rank), _turned(down[:, None, rank:], freq))
            latent, turned = caches[source]
            q = (y @ w(p + "mix.q", m["heads"] * (m["dim"] + rot), width).T).view(n, m["heads"], -1)
            q = torch.cat([q[..., : m["dim"]], _turned(q[..., m["dim"]:], freq)], dim=-1)
            k, v = ((latent @ w(p + "mix." + name, hd, rank).T).view(n, m["heads"], m["dim"]) for name in ("uk", "uv"))
            k = torch.cat([k, turned.expand(n, m["heads"], rot)], dim=-1)
            o = _attend(q, k, v, m["scale"], _seen(n, m["mask"]["size"]), w(p + "mix.sink", m["heads"])).flatten(1)
        o = (o * torch.sigmoid(y @ w(p + "mix.g", hd, width).T)) @ w(p + "mix.o", width, hd).T
        x = x + squash(o, p + "norm1b")
        y = squash(x, p + "norm2")
        y = (_gelu(y @ w(p + "mlp.gate", ff, width).T) * (y @ w(p + "mlp.up", ff, width).T)) @ w(p + "mlp.down", width, ff).T
        x = x + squash(y, p + "norm2b")
        e = w("side.embed", VOCAB, side * len(cfg["layers"]))[tokens, i * side:(i + 1) * side]
        y = (_gelu(x @ w(p + "side.gate", side, width).T) * e) @ w(p + "side.proj", width, side).T
        x = x + _rms(y, eps) * w(p + "side.norm", width)
    return lambda rows: squash(x[rows], "final.norm") @ w("head", VOCAB, width).T


def _mixture(y, chosen, weight, expert, count):
    out = torch.zeros_like(y)
    for e in range(count):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            out[rows] += weight[rows, place].unsqueeze(1) * expert(y[rows], e)
    return out


def _topunex(cfg, w, tokens):
    width, eps, n = cfg["width"], cfg["norm"]["eps"], len(tokens)

    def clamped(y, p, ff, limit):
        g = (y @ w(p + "gate", ff, width).T).clamp_max(limit)
        u = (y @ w(p + "up", ff, width).T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + "down", width, ff).T
    x = w("embed", VOCAB, width)[tokens]
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        h, g, d, sc = m["heads"], m["kv_heads"], m["dim"], m["rot"]["scaling"]
        freq = _freq(m["rot"]["dims"], m["rot"]["base"])
        length = 2 * math.pi / freq
        keep = ((sc["original"] / length - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)
        freq = (1.0 - keep) * freq / sc["factor"] + keep * freq
        q = (x @ w(p + "mix.q", h * d, width).T + w(p + "mix.q.b", h * d)).view(n, h, d)
        v = (x @ w(p + "mix.k", g * d, width).T + w(p + "mix.k.b", g * d)).view(n, g, d)
        o = _attend(_rms(_turned(q, freq), eps), _rms(_turned(v, freq), eps), v, m["scale"], _seen(n, m["mask"]["size"], m["mask"]["keep_first"]),
                    w(p + "mix.sink", h), m["softcap"]).flatten(1)
        o = (o * torch.sigmoid(x @ w(p + "mix.g", h * d, width).T)) @ w(p + "mix.o", width, h * d).T + w(p + "mix.o.b", width)
        x = x + _rms(o, eps) * w(p + "norm1", width)
        p += "mlp."
        if mlp["kind"] == "dense":
            ff = mlp["ff"]
            a = x @ w(p + "gate", ff, width).T + w(p + "gate.b", ff)
            y = (torch.nn.functional.silu(a) * (x @ w(p + "up", ff, width).T + w(p + "up.b", ff))) @ w(p + "down", width, ff).T + w(p + "down.b", width)
        else:
            r, ff, limit = mlp["router"], mlp["expert"]["ff"], mlp["expert"]["limit"]
            z, chosen = (x @ w(p + "router", r["experts"], width).T).topk(r["top"], dim=1)
            y = _mixture(x, chosen, torch.sigmoid(z) * r["scale"], lambda t, e: clamped(t, f"{p}e{e}.", ff, limit), r["experts"])
            y = y + clamped(x, p + "shared.", mlp["shared"]["ff"], mlp["shared"]["limit"])
        x = x + _rms(y, eps) * w(f"l{i}.norm2", width)
    return lambda rows: (_rms(x[rows], eps) * w("final.norm", width)) @ w("head", VOCAB, width).T


def _rekodra(cfg, w, tokens):
    width, eps, n = cfg["width"], cfg["norm"]["eps"], len(tokens)

    def swiglu(y, p, ff):
        return (torch.nn.functional.silu(y @ w(p + "gate", ff, width).T) * (y @ w(p + "up", ff, width).T)) @ w(p + "down", width, ff).T

    def memory(y, m, p):
        h, d = m["heads"], m["dim"]
        q, k, v = ((y @ w(p + name, h * d, width).T).view(n, h, d) for name in "qkv")
        gi = m["gate_cap"] * torch.tanh((y @ w(p + "i", h, width).T + w(p + "i.b", h)) / m["gate_cap"])
        gf = torch.nn.functional.logsigmoid(m["gate_cap"] * torch.tanh((y @ w(p + "f", h, width).T + w(p + "f.b", h)) / m["gate_cap"]))
        total = gf.cumsum(0)                                   # a token's share decays by exp(total[t] - total[s])
        top = total + (gi - total).cummax(0).values.clamp_min(0.0)
        out = []
        for j in range(h):
            share = (total[:, j, None] - total[None, :, j] + gi[None, :, j] - top[:, j, None]).masked_fill(~_seen(n), -math.inf).exp()
            a = (q[:, j] * d ** -0.5) @ k[:, j].T * share
            out.append((a @ v[:, j]) / (torch.maximum(a.sum(1).abs(), torch.exp(-top[:, j])) + 1e-6)[:, None])
        o = _rms(torch.stack(out, dim=1), eps).flatten(1) * w(p + "norm", h * d)
        return (o * torch.sigmoid(y @ w(p + "g", h * d, width).T)) @ w(p + "o", width, h * d).T

    x = w("embed", VOCAB, width)[tokens] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        y = _rms(x, eps) * w(f"l{i}.norm1", width)
        if layer["type"] == "attention":
            h, g, d = m["heads"], m["kv_heads"], m["dim"]
            freq = _freq(m["rot"]["dims"], m["rot"]["base"])
            q, k = y @ w(p + "q", h * d, width).T, y @ w(p + "k", g * d, width).T
            qn, kn = ((_rms(t, eps) * w(p + name, heads * d)).view(n, heads, d) for t, name, heads in ((q, "q.norm", h), (k, "k.norm", g)))
            o = _attend(_turned(qn, freq), _turned(kn, freq), k.view(n, g, d), m["scale"], _seen(n), w(p + "sink", h)).flatten(1)
            x = x + o @ w(p + "o", width, h * d).T
        else:
            a, h, g, d = m["left"], m["left"]["heads"], m["left"]["kv_heads"], m["left"]["dim"]
            q = _rms((y @ w(p + "left.q", h * d, width).T).view(n, h, d), eps) * w(p + "left.q.norm", d)
            k = _rms((y @ w(p + "left.k", g * d, width).T).view(n, g, d), eps) * w(p + "left.k.norm", d)
            v = (y @ w(p + "left.v", g * d, width).T).view(n, g, d)
            left = _attend(q, k, v, a["scale"], _seen(n, a["mask"]["size"])).flatten(1) @ w(p + "left.o", width, h * d).T
            right = memory(y, m["right"], p + "right.")
            x = x + 0.5 * (_rms(left, eps) * w(p + "left.out", width) + _rms(right, eps) * w(p + "right.out", width))
        p = f"l{i}.mlp."
        y, r, ff = _rms(x, eps) * w(f"l{i}.norm2", width), mlp["router"], mlp["expert"]["ff"]
        scored, groups = r["experts"] + r["identity"], r["groups"]
        score = (y @ w(p + "router", scored, width).T).softmax(dim=1)
        choice = (score + w(p + "correction", scored)).view(n, groups["count"], -1)
        kept = torch.zeros((n, groups["count"]), device=DEV, dtype=torch.bool).scatter_(1, choice.amax(dim=2).topk(groups["keep"], dim=1).indices, True)
        chosen = choice.masked_fill(~kept[:, :, None], -math.inf).flatten(1).topk(r["top"], dim=1).indices
        out = _mixture(y, chosen, score.gather(1, chosen), lambda t, e: t if e >= r["experts"] else swiglu(t, f"{p}e{e}.", ff), scored)
        x = x + out + swiglu(y, p + "shared.", mlp["shared"]["ff"]) * torch.sigmoid(y @ w(p + "shared.sg", 1, width).T)
    return lambda rows: (_rms(x[rows], eps) * w("final.norm", width)) @ w("embed", VOCAB, width).T * cfg["logit_scale"]


def _zimorax(cfg, w, tokens):
    width, eps, n = cfg["width"], cfg["norm"]["eps"], len(tokens)
    silu, softplus = torch.nn.functional.silu, torch.nn.functional.softplus

    def norm(x, name):
        return _rms(x - x.mean(dim=-1, keepdim=True), eps) * w(name, width)

    def conv(x, taps, bias=None):
        count = taps.shape[1]
        y = sum(taps[:, j] * torch.nn.functional.pad(x, (0, 0, count - 1 - j, 0))[:n] for j in range(count))
        return silu(y if bias is None else y + bias)

    def attention(y, m, p):
        h, g, d, sc = m["heads"], m["kv_heads"], m["dim"], m["rot"]["scaling"]
        dims, base = m["rot"]["dims"], m["rot"]["base"]
        q = (y @ w(p + "q", h * d, width).T + w(p + "q.b", h * d)).view(n, h, d)
        k = (y @ w(p + "k", g * d, width).T + w(p + "k.b", g * d)).view(n, g, d)
        v = _rms((y @ w(p + "v", g * d, width).T + w(p + "v.b", g * d)).view(n, g, d), eps)
        lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base)) for turns in (sc["fast"], sc["slow"]))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = ((torch.arange(dims // 2, device=DEV, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        freq = _freq(dims, base) / sc["factor"] * ramp + _freq(dims, base) * (1.0 - ramp)
        factor = 0.1 * math.log(sc["factor"]) + 1.0
        q, k = _turned(q, freq, factor), _turned(k, freq, factor).repeat_interleave(h // g, dim=1)
        z = torch.einsum("hg,gnm->hnm", w(p + "talk", h, h), torch.einsum("nhd,mhd->hnm", q, k) * m["scale"]).masked_fill_(~_seen(n, m["mask"]["size"]), -math.inf)
        prob = torch.cat([z, torch.zeros((h, n, 1), device=DEV, dtype=torch.float64)], dim=2).softmax(dim=2)[:, :, :n]
        return torch.einsum("hnm,mhe->nhe", prob, v.repeat_interleave(h // g, dim=1)).flatten(1), h * d

    def state_space(y, m, p):
        h, e, d, g = m["heads"], m["vdim"], m["state"], m["groups"]
        inner, channels = h * e, h * e + 2 * g * d
        z, xbc, dt = (y @ w(p + "in", inner + channels + h, width).T).split([inner, channels, h], dim=1)
        xs, b, c = conv(xbc, w(p + "conv", channels, m["conv"]), w(p + "conv.b", channels)).split([inner, g * d, g * d], dim=1)
        xs, b, c = xs.reshape(n, h, e), b.reshape(n, g, d), c.reshape(n, g, d)
        dt = softplus(dt + w(p + "dt_bias", h))
        total = (-torch.exp(w(p + "A_log", h)) * dt).cumsum(0)
        out = []
        for j in range(h):
            share = (total[:, j, None] - total[None, :, j]).masked_fill(~_seen(n), -math.inf).exp() * dt[None, :, j]
            out.append((c[:, j * g // h] @ b[:, j * g // h].T * share) @ xs[:, j] + w(p + "D", h)[j] * xs[:, j])
        o = (torch.stack(out, dim=1).flatten(1) * silu(z)).view(n, m["norm_groups"], -1)
        return _rms(o, eps).flatten(1) * w(p + "norm", inner), inner

    def delta(y, m, p):
        h, g, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (conv(y @ w(p + name, size, width).T, w(f"{p}{name}.conv", size, m["conv"])) for name, size in (("q", g * d), ("k", g * d), ("v", h * e)))
        q, k = (t / (t.square().sum(dim=-1, keepdim=True) + 1e-6).sqrt() for t in (q.view(n, g, d), k.view(n, g, d)))
        q, k, v = (q * d ** -0.5).repeat_interleave(h // g, dim=1), k.repeat_interleave(h // g, dim=1), v.view(n, h, e)
        beta = torch.sigmoid(y @ w(p + "b", h, width).T)
        decay = torch.exp(-torch.exp(w(p + "A_log", h)) * softplus(y @ w(p + "a", h, width).T + w(p + "dt_bias", h)))
        state, out = torch.zeros((h, d, e), device=DEV, dtype=torch.float64), []
        for t in range(n):
            state = decay[t, :, None, None] * state
            u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None, :], state)[:, 0])
            state = torch.baddbmm(state, k[t, :, :, None], u[:, None, :])
            out.append(torch.bmm(q[t, :, None, :], state)[:, 0])
        o = _rms(torch.stack(out), eps) * w(p + "norm", e)
        return (o * silu(y @ w(p + "g", h * e, width).T).view(n, h, e)).flatten(1), h * e

    x = w("embed", VOCAB, width)[tokens]
    for i, layer in enumerate(cfg["layers"]):
        p, ff = f"l{i}.", layer["mlp"]["ff"]
        y, cols = {"attention": attention, "mamba2": state_space, "delta": delta}[layer["type"]](norm(x, p + "norm1"), layer["mixer"], p + "mix.")
        x = x + (y @ w(p + "mix.o", width, cols).T) * w(p + "ls1", width)
        y = torch.relu(norm(x, p + "norm2") @ w(p + "mlp.up", ff, width).T + w(p + "mlp.up.b", ff)).square()
        x = x + (y @ w(p + "mlp.down", width, ff).T + w(p + "mlp.down.b", width)) * w(p + "ls2", width)
    return lambda rows: norm(x[rows], "final.norm") @ w("head", VOCAB, width).T


def exact(case, seed):
    if case["kind"] == "attention":
        layers, table, lens = _attention_inputs(case, seed)
        outs = []
        for layer in layers:
            out = torch.empty(layer["q"].shape, device=DEV, dtype=torch.float64)
            for b, n in enumerate(lens.tolist()):
                pages = table[b, : (n + 15) // 16].long()
                k, v = (layer[name][pages].double() for name in ("k", "v"))
                if layer["scales"] is not None:
                    scale = layer["scales"][pages].double().unsqueeze(-1)
                    k, v = (k - 128.0) * scale[:, :, 0], (v - 128.0) * scale[:, :, 1]
                k, v = (t.transpose(0, 1).flatten(1, 2)[:, :n] for t in (k, v))
                q = layer["q"][b].double().view(8, 4, 128)
                out[b] = (torch.bmm(q, k.transpose(1, 2)) * 128 ** -0.5).softmax(dim=2).bmm(v).view(32, 128)
            outs.append(out)
        return outs
    if case["kind"] == "projection":
        outs = []
        for i in range(case["layers"]):
            x, dense = _projection_inputs(case, seed, i)
            outs.append(x.double() @ _unpacked(dense, case["quant"]).T)
        return outs
    w = _Params(seed, case.get("quant"))
    cfg = None if case["family"] == "llama" else _family_config(case["family"], case["width"], case["layers"])

    def model(tokens):
        tokens = torch.tensor(tokens, device=DEV)
        return _llama(case, w, tokens) if cfg is None else {"gutorax": _gutorax, "topunex": _topunex, "rekodra": _rekodra, "zimorax": _zimorax}[case["family"]](cfg, w, tokens)
    if case["kind"] == "decode":
        return torch.cat([model(r)(slice(-1, None)) for r in _contexts(case, seed)]).unsqueeze(1)
    prompts = _prompts(case, seed)
    if cfg is None:
        out = torch.zeros((len(prompts), max(map(len, prompts)), VOCAB), device=DEV, dtype=torch.float64)
        for i, p in enumerate(prompts):
            out[i, : len(p)] = model(p)(slice(None))
        return out
    both = [model(p + [t])(slice(-2, None)) for p, t in zip(prompts, _tokens(seed, "next", len(prompts)))]
    return [torch.stack([b[0] for b in both]), torch.stack([b[1] for b in both]).unsqueeze(1)]
