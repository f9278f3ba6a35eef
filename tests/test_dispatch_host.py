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
