"""The kernels of prompt passes (more than 64 rows of several sequences) against the 64-row kernels they extend."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _status():
    from cacheir_b200 import _lib
    return int(_lib.load().cacheir_b200_device_status(1))


# edges: one row past the 64-row kernels, whole and ragged blocks of 128, an odd number of weight tiles (half a pair), a last tile
# that is not full, a single k block, more tiles than CTA pairs, K split over two and four pairs (evenly and not),
# few tiles and a long K (int4: passes)
@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m, n, k, epilogue", [(65, 128, 128, 0), (128, 384, 256, 1), (129, 320, 1024, 0), (300, 1280, 2048, 1), (192, 256, 640, 2),
                                               (257, 640, 1152, 2), (1024, 4096, 512, 0), (192, 256, 2048, 2), (200, 2304, 1024, 2), (128, 384, 1152, 1),
                                               (129, 320, 2176, 0), (70, 512, 9216, 0)])
def test_rows_equal_passes_of_64(bits, m, n, k, epilogue):
    from cacheir_b200 import ops
    from cacheir_b200.quantization import pack_weight_device, to_tiled

    g = torch.Generator(device="cuda").manual_seed(m * 7 + n + k)
    w = to_tiled(pack_weight_device(torch.randn((n, k), device="cuda", generator=g) * 0.02, "int8" if bits == 8 else "int4_awq"), paired=epilogue == 2)
    x = torch.randn((m, k), device="cuda", generator=g).half()
    x[m // 2] = 0.0
    n_out = n // 2 if epilogue == 2 else n
    res = torch.randn((m, n_out), device="cuda", generator=g).half() if epilogue == 1 else None
    kw = dict(bits=bits, n=n, k=k, epilogue=epilogue, paired=w.paired)
    ws = torch.zeros(ops.qgemv_workspace_bytes(64, k), device="cuda", dtype=torch.uint8)
    whole = [torch.cat([t, torch.zeros((-m % 64, t.shape[1]), device="cuda", dtype=t.dtype)]) if t is not None else None for t in (x, res)]
    want = torch.cat([ops.qgemv(whole[0][i:i + 64], w.packed_values, w.scales, w.zero_points, residual=None if res is None else whole[1][i:i + 64],
                                workspace=ws, tiled=True, **kw) for i in range(0, m, 64)])[:m]
    big = torch.full((ops.qgemv_workspace_bytes(m, k),), 255, device="cuda", dtype=torch.uint8)

    def same(a, b):      # the residual may join in one fused rounding or two: a float32 rounding apart, so at most neighbours in fp16
        return torch.equal(a, b) if epilogue != 1 else bool(((a.float() - b.float()).abs() <= 2.0 ** -10 * b.float().abs().clamp_min(2.0 ** -14)).all())
    assert same(ops.qgemv(x, w.packed_values, w.scales, w.zero_points, residual=res, workspace=big, tiled=True, **kw), want)
    real = m - 31                        # only some of the rows are real: the others stay as they were
    out = torch.full((m, n_out), 7.0, device="cuda", dtype=torch.float16)
    ops.qgemm_rows(x, w.packed_values, w.scales, w.zero_points, residual=res, out=out, workspace=big,
                   n_rows=torch.tensor([real], device="cuda", dtype=torch.int32), **kw)
    assert same(out[:real], want[:real]) and bool((out[real:] == 7.0).all())
    assert _status() == 0


@pytest.mark.parametrize("heads, kv_heads, dim", [(32, 8, 128), (6, 2, 64), (16, 1, 128), (3, 3, 128)])
def test_prompt_attention_equals_the_rows_one_by_one(heads, kv_heads, dim):
    """Several sequences, some with tokens in the cache already; each row's output against the decode kernel's, which sees the
    same keys. Both round probabilities to fp16 (2^-11 each, averaged over the keys) and the output once more: rel-L2 5e-4."""
    from cacheir_b200 import ops

    rng = np.random.default_rng(heads)
    parts = [(0, 1), (0, 64), (15, 17), (200, 130), (63, 2), (0, 333)]            # (tokens before, rows)
    group, page = heads // kv_heads, 16
    step = 64 // group
    pages = [(a + n + page - 1) // page for a, n in parts]
    perm = rng.permutation(sum(pages) + 3)
    table = np.zeros((len(parts), max(pages)), dtype=np.int32)
    tiles, row_table, lens, at, row = [], [], [], 0, 0
    for i, (a, n) in enumerate(parts):
        table[i, :pages[i]] = perm[at:at + pages[i]]
        at += pages[i]
        tiles += [(i, row + t, a + t, min(step, n - t)) for t in range(0, n, step)]
        row_table += [i] * n
        lens += range(a + 1, a + n + 1)
        row += n
    g = torch.Generator(device="cuda").manual_seed(dim)
    k, v = (torch.randn((sum(pages) + 3, kv_heads, page, dim), device="cuda", generator=g).half() for _ in range(2))
    wide = torch.randn((row + 5, heads * dim + 64), device="cuda", generator=g).half()      # rows of a wider buffer
    q = wide[:, :heads * dim].as_strided((row + 5, heads, dim), (wide.stride(0), dim, 1))
    listed = torch.zeros((len(tiles) + 9, 4), dtype=torch.int32)
    listed[:len(tiles)] = torch.tensor(tiles, dtype=torch.int32)
    out = torch.full((row + 5, heads, dim), 7.0, device="cuda", dtype=torch.float16)
    ops.paged_attention_prompt(q, k, v, torch.from_numpy(table).cuda(), listed.cuda(), torch.tensor([len(tiles)], dtype=torch.int32, device="cuda"), out)
    want = ops.paged_attention_decode_batch(q[:row], k, v, torch.from_numpy(table[row_table]).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"))
    err = (out[:row].float() - want.float()).norm() / want.float().norm()
    assert float(err) <= 5e-4, float(err)
    assert bool((out[row:] == 7.0).all()) and _status() == 0
    exact, at = [], 0                     # the same against 64-bit arithmetic: one such rounding less
    for i, (a, n) in enumerate(parts):
        slots = torch.from_numpy(table[i, :pages[i]]).long().cuda()
        keys, values = (p[slots].transpose(1, 2).reshape(-1, kv_heads, dim)[:a + n].double().repeat_interleave(group, dim=1) for p in (k, v))
        scores = torch.einsum("thd,shd->hts", q[at:at + n].double(), keys) * dim ** -0.5
        later = torch.arange(a + n, device="cuda")[None, :] > a + torch.arange(n, device="cuda")[:, None]
        exact.append(torch.einsum("hts,shd->thd", scores.masked_fill(later, -torch.inf).softmax(dim=2), values))
        at += n
    exact = torch.cat(exact)
    assert float((out[:row].double() - exact).norm() / exact.norm()) <= 4e-4


def test_rope_append_rows_equals_rope_append():
    from cacheir_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(3)
    q_dim, k_dim, dim, rows = 512, 256, 128, 70
    qkv = torch.randn((rows, q_dim + 2 * k_dim), device="cuda", generator=g).half()
    positions = torch.arange(rows, device="cuda", dtype=torch.int32) + 11
    slots = torch.randperm(8, device="cuda", generator=g).int()
    table = slots.repeat(rows, 1).contiguous()
    pools = [torch.zeros((8, 2, 16, dim), device="cuda", dtype=torch.float16) for _ in range(4)]
    a, b = qkv.clone(), qkv.clone()
    ops.rope_append(a, positions, table, pools[0], pools[1], q_dim=q_dim, k_dim=k_dim, head_dim=dim, theta=10000.0)
    ops.rope_append_rows(b, positions, slots[positions.long() // 16].contiguous(), ops.rope_table(128, dim, 10000.0, torch.device("cuda")), pools[2], pools[3],
                         q_dim=q_dim, k_dim=k_dim, head_dim=dim, n_rows=torch.tensor([rows], device="cuda", dtype=torch.int32))
    assert torch.equal(a[:, :q_dim], b[:, :q_dim]) and torch.equal(pools[0], pools[2]) and torch.equal(pools[1], pools[3])


def _runtime(quant="int8", *, intermediate=768, **kwargs):
    import cacheir_b200 as C

    gen = torch.Generator(device="cuda")

    def source(key, shape):
        gen.manual_seed(len(key) * 131 + sum(map(ord, key)))
        return torch.ones(shape, device="cuda") if len(shape) == 1 else torch.randn(shape, device="cuda", generator=gen) * 0.05

    art = C.build_decoder_artifact(C.ModelConfig(architecture="LlamaForCausalLM", hidden_size=512, intermediate_size=intermediate, num_layers=2,
                                                 num_attention_heads=4, num_key_value_heads=2, vocab_size=640, max_position_embeddings=512,
                                                 rope_theta=10000.0, dtype="float16"),
                                   quant=quant, modes=("decode",))
    return C.B200DecodeRuntime(art, dtype="float16", tensor_source=source, max_seq_len=512, **kwargs)


@pytest.mark.parametrize("chunk", [16, 32, 100, 512])
def test_passes_keep_to_the_prefill_chunk(chunk):
    """A chunk that was set bounds every pass, above 64 rows and below: all tokens reach the cache and have their logits."""
    rt = _runtime()
    want = rt.fork().run([list(range(200))], mode="prefill")
    rt._engine.prefill_chunk = chunk
    assert rt._engine.pass_rows == chunk
    one, many = rt.fork(), [rt.fork(), rt.fork()]
    got = one.run([list(range(200))], mode="prefill")
    assert float((got.float() - want.float()).norm() / want.float().norm()) <= 2e-3
    rt.run_prefill_batch(many, [list(range(150)), [7] * 40])
    steps = rt.run_step_batch([one] + many, [[3] * 40, [5], [6] * 30])
    rt._engine.prefill_chunk = 64
    again, others = rt.fork(), [rt.fork(), rt.fork()]
    again.run([list(range(200))], mode="prefill")
    rt.run_prefill_batch(others, [list(range(150)), [7] * 40])
    want = rt.run_step_batch([again] + others, [[3] * 40, [5], [6] * 30])
    assert float((steps.float() - want.float()).norm() / want.float().norm()) <= 2e-3


@pytest.mark.parametrize("quant", ["int8", "int4_awq", "int4_g128"])
def test_prompt_pass_equals_passes_of_64_rows(quant):
    """Prompts through one pass against 64-row passes of the decode plan: logits and the cached rows that later steps read. The
    products are the same integers (int4_g128: the same fp16 products), only the attention adds in another order."""
    rt = _runtime(quant)
    assert rt._engine.prompt_rows == 2048
    rng = np.random.default_rng(5)
    prompts = [[int(t) for t in rng.integers(0, 640, n)] for n in (5, 200, 1, 70)]
    fast, slow = [rt.fork() for _ in prompts], [rt.fork() for _ in prompts]
    got = [rt.run_prefill_batch(fast, prompts), rt.run_prefill_batch(fast, [p[::-1] for p in prompts]), rt.run_prefill_batch(fast, prompts)][2]   # third: a replay
    follow = rt.run_step_batch(fast, [[3] * n for n in (40, 1, 66, 2)])          # portions behind cached tokens
    assert rt.kernel_counts["b200.paged_attention_prompt"] > 0
    rt._engine.prompt_rows = 0
    want = rt.run_prefill_batch(slow, prompts)
    want_follow = rt.run_step_batch(slow, [[3] * n for n in (40, 1, 66, 2)])
    for a, b in ((got, want), (follow, want_follow)):
        assert float((a.float() - b.float()).norm() / b.float().norm()) <= 2e-3
    for layer in range(2):
        pool = rt.kv_allocator.pool_for_layer(layer)
        for f, s in zip(fast, slow):
            for name in ("keys", "values"):
                a, b = (torch.cat([pool[name][p.page_id][:, :p.length] for p in x.kv_cache.pages], dim=1).float() for x in (f, s))
                assert float((a - b).norm() / b.norm()) <= 2e-3
    rt.check_device_status()


@pytest.mark.parametrize("quant", ["int8", "int4_awq"])
def test_prompt_pass_of_a_very_wide_model(quant):
    """A down projection whose K is beyond the 32-bit sums of the integer products: the pass takes the general product for it, the same one
    that 64-row passes take. Only the attention adds in another order."""
    rt = _runtime(quant, intermediate=32896)
    assert rt._engine.prompt_rows > 0
    prompts = [list(range(100)), [9] * 45]
    got = rt.run_prefill_batch([rt.fork(), rt.fork()], prompts)
    assert rt.kernel_counts["b200.paged_attention_prompt"] > 0
    rt._engine.prompt_rows = 0
    want = rt.run_prefill_batch([rt.fork(), rt.fork()], prompts)
    assert float((got.float() - want.float()).norm() / want.float().norm()) <= 2e-3
    rt.check_device_status()


def test_a_collection_during_a_capture():
    """Graphs of plans that nobody refers to any more are freed whenever the collector runs, which it may while a plan is captured."""
    rt = _runtime()
    session, other = rt.fork(), [rt.fork(), rt.fork()]
    want = rt.run_decode_batch([session], [1]).clone()
    for _ in range(2):                                     # the second step is captured
        rt.run_decode_batch(other, [1, 1])
    dropped = [rt._engine.plans.pop(("decode", 2))]        # (its launch list refers back to it: only the collector frees it)
    enabled = []

    def collect():
        dropped.clear()
        enabled.append(gc.isenabled())
        gc.collect()
    rt._engine.plans[("decode", 1)].program.insert(0, collect)
    session.kv_cache.clear()
    got = rt.run_decode_batch([session], [1])
    assert torch.equal(got, want) and rt._engine.graph_captures == 2
    assert enabled == [True] and gc.isenabled()


def test_prompt_plans_of_every_size_stay():
    """One plan per bucket of rows: lengths in turn make and capture each of them once."""
    rt = _runtime(max_plans=3)
    session, lengths = rt.fork(), (65, 129, 193, 257, 385)
    for _ in range(3):
        for n in lengths:
            rt.run_prefill_batch([session], [[i % 640 for i in range(n)]])
    assert (rt._engine.plans_lowered, rt._engine.graph_captures) == (len(lengths), len(lengths))


def _prefilled(rt, sessions=None):
    prompts = [list(range(200)), [9] * 70]
    sessions = sessions or [rt.fork() for _ in prompts]
    logits = rt.run_prefill_batch(sessions, prompts)
    return torch.cat([logits[i, :len(p)] for i, p in enumerate(prompts)]).float(), rt.run_decode_batch(sessions, [1, 2]).float().clone()


def _near(a, b):
    return all(float((x - y).norm() / y.norm()) <= 2e-3 for x, y in zip(a, b))


def test_prompts_that_leave_no_room_for_long_passes(monkeypatch):
    """Where the buffers of a long pass cannot be had, prompts go through passes of the decode plan, as they do for other models."""
    from cacheir_b200 import runtime

    rt = _runtime()
    want = _prefilled(rt)
    assert rt._engine.prompt_plans
    other = _runtime()

    def refuse(*args):
        raise torch.cuda.OutOfMemoryError("no room")
    monkeypatch.setattr(runtime._PromptPlan, "_make_buffers", refuse)
    assert _near(_prefilled(other), want) and not other._engine.prompt_plans and other.oom_recoveries == 0
    one = other.fork().run([list(range(200))], mode="prefill")[0].float()
    assert float((one - want[0][:200]).norm() / want[0][:200].norm()) <= 2e-3


def test_prompt_memory_under_a_limit():
    """A session's limit counts the buffers of long passes: they are not made where they do not fit, and given back before any session
    loses its tokens."""
    rt = _runtime()
    want = _prefilled(rt)
    held = torch.cuda.memory_allocated()
    rt._recover_from_oom()
    freed = held - torch.cuda.memory_allocated()
    assert not rt._engine.prompt_plans and freed >= 0.9 * rt._engine.prompt_bytes()
    assert _near(_prefilled(rt), want) and rt._engine.prompt_plans          # (made again)
    rt._engine.release_prompt_plans()
    tight = [rt.fork() for _ in range(2)]
    room = torch.cuda.memory_allocated() + rt._engine.prompt_bytes() / 2
    for session in tight:
        session.memory_limit_mb = room / 2 ** 20
    rt.memory_limit_mb = room / 2 ** 20
    assert _near(_prefilled(rt, tight), want) and not rt._engine.prompt_plans
    rt.memory_limit_mb = None
    _prefilled(rt)
    rt.memory_limit_mb = (torch.cuda.memory_allocated() - rt._engine.prompt_bytes() / 4) / 2 ** 20
    before, recovered = [s.kv_cache.tokens for s in tight], rt.oom_recoveries
    rt.run_decode_batch(tight, [3, 4])
    assert not rt._engine.prompt_plans and rt.oom_recoveries == recovered and [s.kv_cache.tokens for s in tight] == [n + 1 for n in before]


def test_more_than_64_prequantized_rows_are_refused():
    """`quantize_activations` fills a workspace for up to 64 rows; more of them are `qgemm_rows`' business, after `rms_norm_quantize_rows`."""
    from cacheir_b200 import _lib, ops

    for bits in (8, 4):
        ops.qgemv_plan(64, 1024, 1024, bits=bits, tiled=True, prequantized=True)
        for rows in (65, 128, 300):
            with pytest.raises(_lib.CacheIRB200Error):
                ops.qgemv_plan(rows, 1024, 1024, bits=bits, tiled=True, prequantized=True)


def test_prompts_as_tensors():
    """Token batches may be anything whose elements `int` reads, a CUDA tensor among them."""
    rt = _runtime()
    prompts = [list(range(90)), [5] * 20]
    want = rt.run_prefill_batch([rt.fork(), rt.fork()], prompts)
    assert rt.kernel_counts["b200.paged_attention_prompt"] > 0
    for form in (lambda p: torch.tensor(p, device="cuda"), lambda p: list(torch.tensor(p, device="cuda")), lambda p: np.array(p), tuple):
        assert torch.equal(rt.run_prefill_batch([rt.fork(), rt.fork()], [form(p) for p in prompts]), want)


@pytest.mark.parametrize("quant, batch", [("int8", 3), ("int8", 70), ("int4_awq", 5), ("int4_awq", 70), ("int4_awq", 130)])
def test_launches_of_a_decode_step(quant, batch):
    """What a plan counts per step is what runs (a product of more than 64 rows: its pre-pass and one kernel, not one per 64 rows)."""
    rt = _runtime(quant)
    sessions = [rt.fork() for _ in range(batch)]
    rt.run_decode_batch(sessions, [1] * batch)
    plan = rt._engine.plans[("decode", batch)]
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
        for fn in plan.program:
            fn()
        torch.cuda.synchronize()
    kernels = [e.name for e in profile.events() if e.device_type == torch.autograd.DeviceType.CUDA and not e.name.startswith("Mem")]
    assert len(kernels) == plan.launches_per_step, kernels


# (intermediate 3072: the gate and up rows are the three million numbers from which up to 128 rows run without a pre-pass)
@pytest.mark.parametrize("batch", [20, 65, 128, 129])
def test_launches_of_an_int4_decode_step_of_wide_products(batch, monkeypatch):
    narrow = _runtime
    monkeypatch.setitem(globals(), "_runtime", lambda quant: narrow(quant, intermediate=3072))
    test_launches_of_a_decode_step("int4_awq", batch)
