"""Dense products of prompts on CTA pairs against 64-bit products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tokens(t, n, k, batch=1):
    """Tokens per tile of the pairs that the product runs on, 0: single CTAs."""
    from cacheir_b200 import _lib
    return _lib.load_group("ragged").cacheir_b200_dense_pair_tokens(t, n, k, batch)


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def _inputs(t, n, k):
    g = torch.Generator(device="cuda").manual_seed(t + n + k)
    x = torch.randn((t, k), device="cuda", generator=g).bfloat16()
    w = (torch.randn((n, k), device="cuda", generator=g) * k ** -0.5).bfloat16()
    return g, x, w, x.double() @ w.double().T


# the fewest tokens that take pairs, ragged token and weight tiles (half a pair, a piece of a tile), a k block that is not full,
# more tiles than pairs with either width of the token tile (three tiles a pair: each accumulator is used again)
SHAPES = [(768, 1544, 520, 128), (1025, 5128, 72, 128), (900, 1288, 1032, 128), (1537, 4096, 136, 128), (2047, 6152, 200, 256), (1793, 6144, 1096, 256)]


@pytest.mark.parametrize("t,n,k,tokens", SHAPES)
def test_dense_pairs(t, n, k, tokens):
    """float32 sums of k products: rel-L2 1e-5; bf16 results round once (2^-9): 3e-3."""
    from cacheir_b200 import hybrid_ops as H

    assert _tokens(t, n, k) == tokens
    _, x, w, want = _inputs(t, n, k)
    f32 = torch.full((t, n), 9.0, device="cuda")
    H.dense_gemm(x, w, f32, epilogue=H.DENSE_F32)
    assert _rel(f32, want) <= 1e-5
    wide = torch.zeros((t, n + 8), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, wide)
    assert _rel(wide[:, :n], want) <= 3e-3 and float(wide[:, n:].abs().max()) == 0.0
    paired = torch.empty((t, n // 2), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, paired, epilogue=H.DENSE_GEGLU)
    assert _rel(paired, torch.nn.functional.gelu(want[:, 0::2], approximate="tanh") * want[:, 1::2]) <= 3e-3


# (a product of the same kind on the other side of the choice: pairs would show their epilogue)
@pytest.mark.parametrize("t,n,k,tokens", [SHAPES[0], SHAPES[4], (1025, 2000, 72, 0)])
def test_dense_pairs_finish_a_sublayer(t, n, k, tokens):
    """Residual (float32: its own rounding and tanhf's, 1e-5), bias, float32 columns behind the others, embedding."""
    from cacheir_b200 import hybrid_ops as H

    assert _tokens(t, n, k) == tokens
    g, x, w, want = _inputs(t, n, k)
    res = torch.randn((t, n), device="cuda", generator=g)
    w1, b1, w2, b2 = (torch.randn(n, device="cuda", generator=g) for _ in range(4))
    sums = res.double() + torch.tanh(0.6 * want) * w1.double() + b1.double()
    nxt = torch.empty((t, n), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, epilogue=H.DENSE_RESIDUAL, residual=res, norm=H.DynamicTanh(w1, b1, 0.6), nx=H.Next(nxt, H.DynamicTanh(w2, b2, 0.4)))
    assert _rel(res, sums) <= 1e-5 and _rel(nxt, torch.tanh(0.4 * sums) * w2.double() + b2.double()) <= 3e-3
    tail = torch.full((t, 12), 9.0, device="cuda")
    out = torch.empty((t, n - 10), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, out, epilogue=H.DENSE_SILU, act_cols=n // 2, bias=b1, tail=tail[:, :10])
    biased = want + b1.double()
    assert _rel(tail[:, :10], biased[:, n - 10:]) <= 1e-5 and bool((tail[:, 10:] == 9.0).all())
    assert _rel(out[:, :n // 2], torch.nn.functional.silu(biased[:, :n // 2])) <= 3e-3 and _rel(out[:, n // 2:], biased[:, n // 2:n - 10]) <= 3e-3
    half = torch.empty((t, (n - 10) // 2), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, half, epilogue=H.DENSE_SWIGLU, tail=tail[:, :10])
    assert _rel(half, torch.nn.functional.silu(want[:, 0:n - 10:2]) * want[:, 1:n - 10:2]) <= 3e-3 and _rel(tail[:, :10], want[:, n - 10:]) <= 1e-5
    table = torch.randn((11, n + 24), device="cuda", generator=g).bfloat16()
    ids = torch.randint(0, 11, (t,), device="cuda", generator=g)
    emb = torch.empty((t, n), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, emb, epilogue=H.DENSE_GELU_EMBED, ids=ids, table=table, table_col=16)
    assert _rel(emb, torch.nn.functional.gelu(want, approximate="tanh") * table[ids, 16:16 + n].double()) <= 3e-3
    assert H.device_status() == 0


# per head, either side of the line between single CTAs and pairs: a long K on pairs; a short K on tiles of 256 and of 128 tokens of single CTAs
@pytest.mark.parametrize("t,batch,n,k,tokens", [(767, 8, 256, 1088, 0), (768, 8, 256, 1088, 128), (1000, 40, 256, 1032, 256), (767, 52, 128, 136, 0), (768, 52, 128, 136, 0)])
def test_products_per_head(t, batch, n, k, tokens):
    from cacheir_b200 import hybrid_ops as H

    assert _tokens(t, n, k, batch) == tokens
    g = torch.Generator(device="cuda").manual_seed(t + batch)
    x = torch.randn((t, batch * (k + 8)), device="cuda", generator=g).bfloat16()
    w = (torch.randn((batch * n, k), device="cuda", generator=g) * k ** -0.5).bfloat16()
    gate = torch.randn((t, batch * n), device="cuda", generator=g).bfloat16()
    want = torch.einsum("tbk,bnk->tbn", x.view(t, batch, k + 8)[:, :, :k].double(), w.view(batch, n, k).double()).reshape(t, -1)
    out = torch.empty((t, batch * n), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, out, epilogue=H.DENSE_GATED, batch=batch, x_batch_cols=k + 8, gate=gate)
    assert _rel(out, want * torch.sigmoid(gate.double())) <= 3e-3
    f32 = torch.empty((t, batch * n), device="cuda")
    H.dense_gemm(x, w, f32, epilogue=H.DENSE_F32, batch=batch, x_batch_cols=k + 8)
    assert _rel(f32, want) <= 1e-5 and H.device_status() == 0
