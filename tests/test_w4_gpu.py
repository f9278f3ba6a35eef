"""The int4 product with the weights in tensor memory (up to 128 rows) against float64 products of the dequantised weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# edges: one row more and one less than each tile of activation rows, a full tile (another copy of x), fewer weight rows than the last band
# holds, k blocks that no ring is a multiple of, every number of CTAs along K, groups of two k blocks
@pytest.mark.parametrize("tiled", [True, False])
@pytest.mark.parametrize("m, n, k, split", [(9, 2048, 2048, 4), (16, 5100, 640, 1), (17, 1280, 8192, 8), (31, 2048, 5632, 6), (32, 3072, 2176, 4),
                                            (33, 5120, 1536, 3), (64, 6400, 3584, 2), (65, 3648, 896, 1), (127, 4096, 1280, 2), (128, 19200, 1152, 1)])
def test_weights_in_tensor_memory(m, n, k, split, tiled):
    """Products of exact fp16 integers are summed in float32 (2^-24 each) and rounded to fp16 once: 2^-11 / sqrt(3) of the result's
    root mean square is 2.8e-4."""
    from cacheir_b200 import _lib, ops
    from cacheir_b200.quantization import dequantize_device, pack_weight_device, to_tiled

    g = torch.Generator(device="cuda").manual_seed(m * 31 + n + k)
    dense = torch.randn((n, k), device="cuda", generator=g) * 0.02
    x = torch.randn((m, k + 8), device="cuda", generator=g).half()[:, :k]            # rows of a wider buffer
    for quant in ("int4_g128", "int4_g256", "int4_awq"):
        if quant == "int4_g256" and k % 256:
            continue
        for odd_zero in (False, True) if quant == "int4_awq" else (False,):
            w = pack_weight_device(dense, quant)
            if odd_zero:                                   # zero points that are no small integers
                w.zero_points[::3] += 0.25
                w.zero_points[1] = -1500.0
            full = dequantize_device(w, torch.float32).double() if not odd_zero else \
                (torch.stack([w.packed_values & 15, w.packed_values >> 4], dim=2).view(n, k).double() - w.zero_points.double()[:, None]) * w.scales.double()[:, None]
            for epilogue in (0, 1, 2):
                paired = tiled and epilogue == 2 and quant == "int4_awq"
                if epilogue == 2 and n % 128:
                    continue
                v = to_tiled(w, paired=paired) if tiled else w
                n_out = n // 2 if epilogue == 2 else n
                res = torch.randn((m, n_out), device="cuda", generator=g).half() if epilogue == 1 else None
                kw = dict(bits=4, group_size=v.group_size or 0, epilogue=epilogue, tiled=tiled, paired=paired)
                plan = ops.qgemv_plan(m, n, k, workspace=False, **kw)
                if quant != "int4_awq" and not plan.get("tensor_memory"):
                    continue                               # (the streaming kernel's, of up to 32 rows and fewer than 6 M numbers)
                assert plan["tensor_memory"] and (epilogue == 2 or plan["split"] == split), plan
                y = ops.qgemv(x, v.packed_values, v.scales, v.zero_points, n=n, k=k, residual=res, **kw)
                want = x.double() @ full.T
                if epilogue == 2:
                    want = torch.nn.functional.silu(want[:, :n_out]) * want[:, n_out:]
                if epilogue == 1:
                    want = want + res.double()
                err = float((y.double() - want).norm() / want.norm())
                # (a zero point of -1500 makes its row outweigh all others: then a single rounding counts, at most 2^-11)
                assert err <= (2.0 ** -11 if odd_zero else 2.8e-4), (quant, epilogue, odd_zero, err)
                again = ops.qgemv(x, v.packed_values, v.scales, v.zero_points, n=n, k=k, residual=res, **kw)
                assert torch.equal(again, y)
    assert int(_lib.load().cacheir_b200_device_status(1)) == 0


# batches that run as chunks of 128 rows, the last one a few rows, a share, or all of them
@pytest.mark.parametrize("tiled", [True, False])
@pytest.mark.parametrize("m", [129, 150, 177, 256])
def test_taller_batches_in_chunks(m, tiled):
    """The plan names the kernel that the first chunk takes, and every chunk has the bits of a call of its own."""
    from cacheir_b200 import _lib, ops
    from cacheir_b200.quantization import dequantize_device, pack_weight_device, quantized_matmul, to_tiled

    n, k = 2048, 1024
    g = torch.Generator(device="cuda").manual_seed(m)
    w = pack_weight_device(torch.randn((n, k), device="cuda", generator=g) * 0.02, "int4_g128")
    x, res = torch.randn((m, k), device="cuda", generator=g).half(), torch.randn((m, n), device="cuda", generator=g).half()
    v = to_tiled(w) if tiled else w
    kw = dict(bits=4, group_size=128, tiled=tiled, workspace=False)
    assert ops.qgemv_plan(m, n, k, **kw) == ops.qgemv_plan(128, n, k, **kw)
    assert ops.qgemv_plan(m, n, k, **kw)["tensor_memory"]
    want = x.double() @ dequantize_device(w, torch.float32).double().T
    for epilogue, residual in ((ops.EPI_NONE, None), (ops.EPI_RESIDUAL, res)):
        y = quantized_matmul(x, v, epilogue=epilogue, residual=residual)
        full = want if residual is None else want + residual.double()
        assert float((y.double() - full).norm() / full.norm()) <= 2.8e-4
        tail = quantized_matmul(x[128:], v, epilogue=epilogue, residual=None if residual is None else residual[128:])
        assert torch.equal(y[128:], tail)
    assert ops.qgemv_plan(150, 384, 512, **kw)["family"] == "f16"            # (fewer than a million numbers)
    assert int(_lib.load().cacheir_b200_device_status(1)) == 0


# group scales at the row counts where the two-CTA tile of 16 rows starts and ends, and one row beside it: groups of one and two k blocks, scales
# of both types, k blocks that its three accumulators do not divide, every epilogue
@pytest.mark.parametrize("tiled", [True, False])
@pytest.mark.parametrize("m, n, k", [(4, 6272, 1024), (5, 3328, 2048), (8, 1536, 4352), (9, 5120, 1280), (15, 5100, 1280), (16, 2176, 3072), (17, 8960, 768)])
def test_group_scales_with_weights_in_tensor_memory(m, n, k, tiled):
    """Exact fp16 products, float32 sums, one rounding to fp16: as above. (int4_g128 and int4_g256 differ in their scales alone.)"""
    from cacheir_b200 import _lib, ops
    from cacheir_b200.quantization import dequantize_device, pack_weight_device, to_tiled

    g = torch.Generator(device="cuda").manual_seed(m * 31 + n + k)
    dense = torch.randn((n, k), device="cuda", generator=g) * 0.02
    x = torch.randn((m, k), device="cuda", generator=g).half()
    for quant in ("int4_g128", "int4_g256"):
        w = pack_weight_device(dense, quant)
        full = dequantize_device(w, torch.float32).double()
        v = to_tiled(w) if tiled else w
        for scales in (w.scales.half(), w.scales.float()):
            assert torch.equal(scales.double(), w.scales.double())
            for epilogue in (0, 1, 2) if n % 128 == 0 else (0, 1):
                res = torch.randn((m, n), device="cuda", generator=g).half() if epilogue == 1 else None
                kw = dict(bits=4, group_size=w.group_size, epilogue=epilogue, tiled=tiled)
                assert ops.qgemv_plan(m, n, k, workspace=False, **kw)["tensor_memory"]
                y = ops.qgemv(x, v.packed_values, scales, None, n=n, k=k, residual=res, **kw)
                want = x.double() @ full.T
                if epilogue == 2:
                    want = torch.nn.functional.silu(want[:, :n // 2]) * want[:, n // 2:]
                if epilogue == 1:
                    want = want + res.double()
                assert float((y.double() - want).norm() / want.norm()) <= 2.8e-4, (quant, scales.dtype, epilogue)
    assert int(_lib.load().cacheir_b200_device_status(1)) == 0
