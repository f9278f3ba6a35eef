"""Decode attention whose context splits merge inside a thread-block cluster, against the same launch in one split."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# sequences shorter than a split's share (its CTA has no keys), lengths around the share's edge, one empty sequence, every split count
@pytest.mark.parametrize("dtype, dim, heads, kv_heads, kv8", [(torch.float16, 128, 32, 8, False), (torch.bfloat16, 64, 4, 2, False), (torch.float16, 128, 16, 1, True),
                                                              (torch.float16, 64, 3, 3, False)])
@pytest.mark.parametrize("splits", [2, 3, 5, 8])
def test_cluster_merge(splits, dtype, dim, heads, kv_heads, kv8):
    """Both sum the same products, in shares of other sizes: float32 sums of fp16 (bf16) probabilities, rounded to the output once."""
    from cacheir_b200 import _lib, ops

    rng = np.random.default_rng(splits * heads)
    lens = [1, 17, 0, 333, 640, 511]
    pages = [(n + 15) // 16 for n in lens]
    table = np.zeros((len(lens), 40), dtype=np.int32)
    perm, at = rng.permutation(sum(pages)), 0
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    g = torch.Generator(device="cuda").manual_seed(dim)
    k, v = (torch.randn((sum(pages), kv_heads, 16, dim), device="cuda", generator=g).to(dtype) for _ in range(2))
    scales = None
    if kv8:
        both = torch.stack([k, v], dim=2).float()
        scales = (both.abs().amax(dim=-1) / 127.0).half()
        codes = (torch.round(both / scales.float().unsqueeze(-1)) + 128.0).clamp(1, 255).to(torch.uint8)
        k, v = codes[:, :, 0].contiguous(), codes[:, :, 1].contiguous()
    q = torch.randn((len(lens), heads, dim), device="cuda", generator=g).to(dtype)
    args = (q, k, v, torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"))
    want = ops.paged_attention_decode_batch(*args, num_splits=1, kv_scales=scales)
    got = ops.paged_attention_decode_batch(*args, num_splits=splits, kv_scales=scales)
    assert not bool(got[2].any()) and torch.equal(got, ops.paged_attention_decode_batch(*args, num_splits=splits, kv_scales=scales))
    assert float((got.float() - want.float()).norm() / want.float().norm()) <= (4e-3 if dtype == torch.bfloat16 else 5e-4)
    assert int(_lib.load().cacheir_b200_device_status(1)) == 0


@pytest.mark.parametrize("batch", [1, 3, 4])
def test_scratch_for_the_coarser_choice_is_enough(batch):
    """Left to choose, a call takes the finest split whose partials fit the scratch that it was given."""
    from cacheir_b200 import _lib, ops

    heads, kv_heads, dim, pages = 32, 8, 128, 32
    g = torch.Generator(device="cuda").manual_seed(batch)
    k, v = (torch.randn((batch * pages, kv_heads, 16, dim), device="cuda", generator=g).half() for _ in range(2))
    q = torch.randn((batch, heads, dim), device="cuda", generator=g).half()
    table = torch.arange(batch * pages, device="cuda", dtype=torch.int32).view(batch, pages)
    lens = torch.full((batch,), 16 * pages - 3, device="cuda", dtype=torch.int32)
    want = ops.paged_attention_decode_batch(q, k, v, table, lens, num_splits=1)
    fine = ops.attention_auto_splits(batch, heads, kv_heads, pages, 16, dim)
    assert fine > 2
    for splits in (2, fine):
        ws = torch.empty(ops.attention_workspace_bytes(batch, heads, dim, splits) // 4, device="cuda")
        got = ops.paged_attention_decode_batch(q, k, v, table, lens, workspace=ws)
        assert torch.equal(got, ops.paged_attention_decode_batch(q, k, v, table, lens, num_splits=splits))
        assert float((got.float() - want.float()).norm() / want.float().norm()) <= 5e-4
    with pytest.raises(_lib.CacheIRB200Error):
        ops.paged_attention_decode_batch(q, k, v, table, lens, workspace=ws[:100])


def test_launches_of_a_call():
    """One for a single split or splits of one cluster, two where a kernel of its own merges them (general kernel, many splits)."""
    from cacheir_b200 import ops

    assert ops.attention_launches(1, 32, 8, 32, 16, 128, torch.float16) == 1
    assert ops.attention_launches(1, 32, 8, 16, 16, 128, torch.float32, num_splits=1) == 1
    assert ops.attention_launches(1, 32, 8, 32, 16, 128, torch.float32) == 2
    assert ops.attention_launches(1, 32, 8, 32, 16, 96, torch.float16) == 2
    assert ops.attention_launches(1, 32, 8, 4096, 16, 128, torch.float16) == 2
    assert ops.attention_launches(64, 32, 8, 512, 16, 128, torch.float16, num_splits=2) == 2
    assert ops.attention_launches(2, 16, 2, 64, 16, 128, torch.float16, kv8=True, num_splits=8) == 1
