"""The streaming int4 product (up to 32 rows) against float64 products of the dequantised weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(m, n, k, tiled, quants, kernel, error=2.8e-4):
    from cacheir_b200 import _lib, ops
    from cacheir_b200.quantization import dequantize_device, pack_weight_device, to_tiled

    g = torch.Generator(device="cuda").manual_seed(m * 31 + n + k)
    dense = torch.randn((n, k), device="cuda", generator=g) * 0.02
    x = torch.randn((m, k + 8), device="cuda", generator=g).half()[:, :k]            # rows of a wider buffer
    for quant in quants:
        for odd_zero in (False, True) if quant == "int4_awq" else (False,):
            w = pack_weight_device(dense, quant)
            if odd_zero:                                   # zero points that are no small integers
                w.zero_points[::3] += 0.25
                w.zero_points[1] = -1500.0
            full = dequantize_device(w, torch.float32).double() if not odd_zero else \
                (torch.stack([w.packed_values & 15, w.packed_values >> 4], dim=2).view(n, k).double() - w.zero_points.double()[:, None]) * w.scales.double()[:, None]
            for epilogue in (0, 1, 2):
                paired = tiled and epilogue == 2 and quant == "int4_awq"
                if epilogue == 2 and n % (128 if paired else 256 if kernel == "stream" else 32):
                    continue
                v = to_tiled(w, paired=paired) if tiled else w
                n_out = n // 2 if epilogue == 2 else n
                res = torch.randn((m, n_out), device="cuda", generator=g).half() if epilogue == 1 else None
                kw = dict(bits=4, group_size=v.group_size or 0, epilogue=epilogue, tiled=tiled, paired=paired)
                plan = ops.qgemv_plan(m, n, k, workspace=False, **kw)
                assert plan["kernel"] == kernel
                y = ops.qgemv(x, v.packed_values, v.scales, v.zero_points, n=n, k=k, residual=res, **kw)
                want = x.double() @ full.T
                if epilogue == 2:
                    want = torch.nn.functional.silu(want[:, :n_out]) * want[:, n_out:]
                if epilogue == 1:
                    want = want + res.double()
                err = float((y.double() - want).norm() / want.norm())
                # (a zero point of -1500 makes its row outweigh all others: then a single rounding counts, at most 2^-11)
                assert err <= (2.0 ** -11 if odd_zero else error), (quant, epilogue, odd_zero, err)
    assert int(_lib.load().cacheir_b200_device_status(1)) == 0
    return plan


SHARES = [(5, 2176, 2048, "int4_awq", 1, 2), (8, 1900, 1536, "int4_awq", 2, 3), (3, 1920, 2048, "int4_awq", 2, 4), (8, 6144, 2560, "int4_awq", 4, 2),
          (5, 2176, 4096, "int4_awq", 4, 6), (8, 1400, 4096, "int4_awq", 4, 8), (9, 380, 1536, "int4_g128", 1, 3), (31, 256, 4096, "int4_g128", 1, 8),
          (17, 5632, 512, "int4_g128", 2, 1), (24, 2432, 1024, "int4_g128", 2, 2), (31, 768, 4096, "int4_g128", 2, 8), (17, 1024, 4096, "int4_g128", 2, 6),
          (31, 5632, 1024, "int4_g128", 4, 2), (17, 3060, 1536, "int4_g128", 4, 3), (31, 2100, 2048, "int4_g256", 4, 4), (9, 1408, 4096, "int4_g128", 4, 8)]


# every share of the rows and of K that the choice can take (row groups, CTAs along K), with fewer rows than the last band holds
@pytest.mark.parametrize("m, n, k, quant, row_groups, split", SHARES)
def test_stream_gemv_shares(m, n, k, quant, row_groups, split):
    plan = _check(m, n, k, True, (quant,), "stream")
    assert (plan["row_groups"], plan["split"]) == (row_groups, split)


# many weight rows in row order: several rounds of tiles, chunks of x, groups of two blocks, half a tile of gate rows at the end
@pytest.mark.parametrize("m, n, k, quant", [(1, 9472, 14336, "int4_g128"), (7, 9504, 14336, "int4_awq"), (3, 9600, 512, "int4_g256"), (8, 20000, 1280, "int4_awq"),
                                            (5, 40032, 384, "int4_g128")])
def test_many_weight_rows_in_row_order(m, n, k, quant):
    """As below, and the sums carry a constant of 1024 per code, about 256 times the products, that leaves at the end of every block: 2^-24 each,
    over up to 112 blocks 1.6e-4 beside the 2.8e-4."""
    _check(m, n, k, False, (quant,), "stream_rows", error=3.3e-4)


# edges: one k block (k groups without work), a k split over a cluster, bands and 32-row shares that are not full, rows that do not
# fill the eight columns of an MMA, the largest row counts of each form, many and few weight rows (every share size)
@pytest.mark.parametrize("tiled", [True, False])
@pytest.mark.parametrize("m, n, k", [(1, 128, 128), (2, 2048, 2048), (3, 256, 512), (8, 1280, 8192), (7, 9600, 256), (9, 512, 640), (16, 768, 2048),
                                     (17, 256, 1152), (32, 1536, 4096), (31, 4096, 384), (5, 320, 1280)])
def test_stream_gemv(m, n, k, tiled):
    """Products of exact fp16 integers are summed in float32 (2^-24 each) and rounded to fp16 once: 2^-11 / sqrt(3) of the result's
    root mean square is 2.8e-4."""
    from cacheir_b200 import _lib, ops
    from cacheir_b200.quantization import dequantize_device, pack_weight_device, to_tiled

    g = torch.Generator(device="cuda").manual_seed(m * 31 + n + k)
    dense = torch.randn((n, k), device="cuda", generator=g) * 0.02
    x = torch.randn((m, k + 8), device="cuda", generator=g).half()[:, :k]            # rows of a wider buffer
    for quant in ("int4_g128", "int4_awq") if m <= 8 else ("int4_g128",):
        for odd_zero in (False, True) if quant == "int4_awq" else (False,):
            w = pack_weight_device(dense, quant)
            if odd_zero:                                   # zero points that are no small integers
                w.zero_points[::3] += 0.25
                w.zero_points[1] = -1500.0
            full = dequantize_device(w, torch.float32).double() if not odd_zero else \
                (torch.stack([w.packed_values & 15, w.packed_values >> 4], dim=2).view(n, k).double() - w.zero_points.double()[:, None]) * w.scales.double()[:, None]
            for epilogue in (0, 1, 2):
                paired = tiled and epilogue == 2 and quant == "int4_awq"
                if epilogue == 2 and n % (128 if paired else 256):
                    continue
                v = to_tiled(w, paired=paired) if tiled else w
                n_out = n // 2 if epilogue == 2 else n
                res = torch.randn((m, n_out), device="cuda", generator=g).half() if epilogue == 1 else None
                ws = torch.zeros(ops.qgemv_workspace_bytes(m, k), device="cuda", dtype=torch.uint8)
                y = ops.qgemv(x, v.packed_values, v.scales, v.zero_points, bits=4, n=n, k=k, group_size=v.group_size or 0, epilogue=epilogue, residual=res,
                              workspace=ws, tiled=tiled, paired=paired)
                want = x.double() @ full.T
                if epilogue == 2:
                    want = torch.nn.functional.silu(want[:, :n_out]) * want[:, n_out:]
                if epilogue == 1:
                    want = want + res.double()
                err = float((y.double() - want).norm() / want.norm())
                # (a zero point of -1500 makes its row outweigh all others: then a single rounding counts, at most 2^-11)
                assert err <= (2.0 ** -11 if odd_zero else 2.8e-4), (quant, epilogue, odd_zero, err)
    assert int(_lib.load().cacheir_b200_device_status(1)) == 0
