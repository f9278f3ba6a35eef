"""Dense products of prompts on CTA pairs against 64-bit products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# the fewest tokens that take pairs, ragged token and weight tiles (half a pair, a piece of a tile), a k block that is not full,
# more tiles than pairs with either width of the token tile
@pytest.mark.parametrize("t,n,k", [(768, 1544, 200), (1025, 2000, 72), (900, 1288, 1032), (1537, 4096, 136)])
def test_dense_pairs(t, n, k):
    """float32 sums of k products: rel-L2 1e-5; bf16 results round once (2^-9): 3e-3."""
    from cacheir_b200 import hybrid_ops as H

    g = torch.Generator(device="cuda").manual_seed(t + n + k)
    x = torch.randn((t, k), device="cuda", generator=g).bfloat16()
    w = (torch.randn((n, k), device="cuda", generator=g) * k ** -0.5).bfloat16()
    want = x.double() @ w.double().T

    def rel(a, b):
        return float((a.double() - b).norm() / b.norm())
    f32 = torch.full((t, n), 9.0, device="cuda")
    H.dense_gemm(x, w, f32, epilogue=H.DENSE_F32)
    assert rel(f32, want) <= 1e-5
    wide = torch.zeros((t, n + 8), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, wide)
    assert rel(wide[:, :n], want) <= 3e-3 and float(wide[:, n:].abs().max()) == 0.0
    paired = torch.empty((t, n // 2), device="cuda", dtype=torch.bfloat16)
    H.dense_gemm(x, w, paired, epilogue=H.DENSE_GEGLU)
    assert rel(paired, torch.nn.functional.gelu(want[:, 0::2], approximate="tanh") * want[:, 1::2]) <= 3e-3
