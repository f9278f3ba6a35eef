"""Kernels take their places, and ask for their weights, while the kernel before them is at work: what that one writes must arrive all the same."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _same_as_waiting(step, outs):
    """The calls of `step` eagerly with a wait behind each, back to back, and as a graph: the same bits."""
    step(torch.cuda.synchronize)
    want = [o.clone() for o in outs]
    for run in ("eager", "graph"):
        for o in outs:
            o.fill_(float("nan"))
        if run == "eager":
            step(lambda: None)
        else:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                step(lambda: None)
            graph.replay()
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert torch.equal(o, w), run


# the second product's weights are the first one's output: decode kernels, K split over a cluster, pairs of CTAs
@pytest.mark.parametrize("t, k, rows", [(128, 512, 8), (2048, 2048, 16), (1024, 4096, 100), (2048, 1024, 1024)])
def test_weights_written_by_the_kernel_before(t, k, rows):
    from cacheir_b200 import hybrid_ops as H

    g = torch.Generator(device="cuda").manual_seed(t + k)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g).bfloat16()
    n, steps = 1024, 6
    xs, w, qs = [rand(t, k) for _ in range(steps)], rand(n, k), rand(rows, n)
    mid = torch.empty((t, n), device="cuda", dtype=torch.bfloat16)             # written again and again
    outs = [torch.empty((rows, t), device="cuda", dtype=torch.bfloat16) for _ in range(steps)]

    def step(wait):
        for x, out in zip(xs, outs):
            H.dense_gemm(x, w, mid)
            wait()
            H.dense_gemm(qs, mid, out)
            wait()
    _same_as_waiting(step, outs)


# codes that a copy (another library's kernel) or this library's own relayout has just written
@pytest.mark.parametrize("quant", ["int4_g128", "int4_awq", "int8"])
@pytest.mark.parametrize("m", [1, 24, 100])
def test_codes_written_by_the_kernel_before(quant, m):
    from cacheir_b200 import ops
    from cacheir_b200.quantization import pack_weight_device, quantized_matmul, to_tiled

    g = torch.Generator(device="cuda").manual_seed(m)
    n, k, steps = 4096, 2048, 4
    packs = [pack_weight_device(torch.randn((n, k), device="cuda", generator=g) * 0.02, quant) for _ in range(steps)]
    tiled = [to_tiled(p) for p in packs]
    x = torch.randn((m, k), device="cuda", generator=g).half()
    scratch = torch.zeros(ops.qgemv_workspace_bytes(m, k), device="cuda", dtype=torch.uint8)
    rows, lines = (make(pack_weight_device(torch.zeros((n, k), device="cuda"), quant)) for make in (lambda w: w, to_tiled))      # (scales of their own)
    outs = [torch.empty((m, n), device="cuda", dtype=torch.float16) for _ in range(2 * steps)]

    def step(wait):
        for i in range(steps):
            for w, source, out in ((rows, packs[i], outs[2 * i]), (lines, tiled[i], outs[2 * i + 1])):
                w.packed_values.copy_(source.packed_values)
                w.scales.copy_(source.scales)
                if w.zero_points is not None:
                    w.zero_points.copy_(source.zero_points)
                wait()
                quantized_matmul(x, w, out=out, workspace=scratch)
                wait()
    _same_as_waiting(step, outs)
