"""Which kernel a call takes, asked through the library's plan queries: no GPU, nothing is launched."""
import pytest


@pytest.mark.parametrize("rows", [1, 8, 9, 32, 33, 100])
@pytest.mark.parametrize("group", [128, 256])
def test_paired_tiles_of_group_wise_codes_are_refused(rows, group):
    """Group scales lie in the weight's own row order: no kernel reads them for tiles that pair gate and up rows."""
    from cacheir_b200 import ops
    from cacheir_b200._lib import CacheIRB200Error

    for workspace in (False, True):
        with pytest.raises(CacheIRB200Error):
            ops.qgemv_plan(rows, 512, 512, bits=4, group_size=group, epilogue=ops.EPI_SWIGLU, tiled=True, paired=True, workspace=workspace)


# clusters of CTAs along K that a B200 runs at once (a cluster lives in one GPC), at one CTA per SM
AT_ONCE = {1: 148, 2: 74, 3: 44, 4: 33, 6: 20, 8: 15}


@pytest.mark.parametrize("n, k", [(512, 512), (1024, 4096), (1536, 6144), (2048, 2048), (2048, 8192), (2048, 11264), (2560, 2560), (3072, 3072), (4096, 14336),
                                  (4608, 8192), (5120, 5120), (5632, 2048), (6144, 4096), (8448, 2048), (9344, 4096)])
def test_streaming_products_split_into_clusters_that_run_at_once(n, k):
    """Sixteen clusters of eight CTAs take two turns, and with them twice the time."""
    from cacheir_b200 import ops

    for rows in (1, 4, 8, 9, 16, 17, 32) if k <= 8192 else (1, 4, 8):
        plan = ops.qgemv_plan(rows, n, k, bits=4, group_size=128 if k <= 8192 else 0, tiled=True, workspace=False)
        assert plan["kernel"] == "stream"
        clusters, split = -(-n // (32 * plan["row_groups"])), plan["split"]
        assert split == 1 or clusters <= AT_ONCE[split] * (2 if plan["row_groups"] == 1 else 1), (rows, plan)
        assert k // 128 // split >= 4


@pytest.mark.parametrize("t,n,k,tokens", [(1153, 1024, 8192, 0), (1001, 4096, 512, 0), (768, 6144, 512, 0), (1537, 8192, 8192, 0), (767, 14336, 2048, 0),
                                          (2048, 14336, 2048, 256), (1153, 22016, 1024, 256), (1001, 6144, 2048, 128)])
def test_dense_products_take_the_faster_form(t, n, k, tokens):
    """Single CTAs were 1.2 to 1.35 times faster than pairs on the first four, pairs 1.1 to 1.6 times on the last three."""
    from cacheir_b200 import _lib

    assert _lib.load_group("ragged").cacheir_b200_dense_pair_tokens(t, n, k, 1) == tokens
