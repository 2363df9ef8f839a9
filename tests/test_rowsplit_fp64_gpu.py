"""The split of block rows over lane groups (rowsplit.cu) on both sides of its
FP64 limits: 150, 400 (rows of three blocks and more) and 640 rows (of eight)
for 25 x 25 and 27 x 27 blocks, 16 and 24 rows per SM for 9 x 9 ones.  Check and
tolerances as in test_rowsplit_gpu.py."""
import pytest

import test_rowsplit_gpu as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,n,lo,hi", [(27, 150, 1, 2), (27, 151, 1, 2), (27, 399, 4, 6), (27, 400, 4, 6),
                                       (27, 639, 9, 12), (27, 640, 9, 12), (25, 150, 1, 1), (25, 399, 3, 6),
                                       (25, 639, 9, 10), (25, 641, 9, 10)])
def test_wide_blocks(ctx, b, n, lo, hi):
    base.test_split_rows(ctx, b, n, lo, hi)


@pytest.mark.parametrize("per_sm", [16, 24])
@pytest.mark.parametrize("more", [0, 1])
def test_blocks_of_9(ctx, per_sm, more):
    import torch
    base.test_split_rows(ctx, 9, per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more, 9, 12)
