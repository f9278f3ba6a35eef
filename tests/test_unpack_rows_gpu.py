"""The rows of a shared prompt pass at their places in zero-padded outputs."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype, columns, lens, max_len", [(torch.float16, 8, [1], 1), (torch.float16, 32768, [61, 17, 140, 33], 140), (torch.float32, 516, [3, 1, 2], 5),
                                                           (torch.bfloat16, 16392, [2, 7], 7), (torch.float16, 64, [1 + i % 3 for i in range(130)], 4)])
def test_rows_at_their_places(dtype, columns, lens, max_len):
    """More than one vector per thread and a ragged last one, more parts than one launch takes, sequences cut between two passes."""
    from cacheir_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(columns)
    rows = torch.randn((sum(lens) + 2, columns), device="cuda", generator=g).to(dtype)
    out = torch.full((len(lens), max_len, columns), float("nan"), device="cuda", dtype=dtype)
    want = torch.zeros_like(out)
    first, second, at = [], [], 0
    for i, n in enumerate(lens):
        want[i, :n] = rows[at:at + n]
        at += n
        cut = n // 2 if i + 1 == len(lens) else n           # the last sequence goes on in a second pass
        first.append((i, 0, cut, max_len if cut == n else cut))
        if cut < n:
            second.append((i, cut, n, max_len))
    ops.unpack_rows(rows, out, first)
    if second:
        ops.unpack_rows(rows[at - (second[0][2] - second[0][1]):], out, second)
    assert torch.equal(out, want)


@pytest.mark.gpu
def test_parts_outside_the_output_are_refused():
    from cacheir_b200 import ops
    from cacheir_b200._lib import CacheIRB200Error

    rows, out = torch.zeros((4, 8), device="cuda", dtype=torch.float16), torch.zeros((2, 3, 8), device="cuda", dtype=torch.float16)
    for part in [(2, 0, 1, 1), (-1, 0, 1, 1), (0, 2, 4, 4), (0, 1, 0, 0), (0, 0, 1, 4), (0, 0, 2, 1)]:
        with pytest.raises(CacheIRB200Error):
            ops.unpack_rows(rows, out, [part])
    with pytest.raises(ValueError):
        ops.unpack_rows(rows, out, [(0, 0, 3, 3), (1, 0, 2, 3)])
