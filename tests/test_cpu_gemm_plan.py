"""Which tile width a GEMM takes (the library's rule, without a GPU): tiles of 384 columns follow sizes, not one width of the models."""
import pytest

from context_parallelism_b200 import _native as nv
from context_parallelism_b200.ops.gemm import EPI_BF16, EPI_F32, EPI_F32_ACC


def _width(M, N, K, epi):
    return nv.lib().cpb_gemm_plan(M, N, K, epi, 0) >> 16


@pytest.mark.parametrize("epi", [EPI_BF16, EPI_F32_ACC])
def test_one_column_of_384(epi):
    for N in (264, 320, 344, 376, 384):                               # one such column, two of the next width
        for M, K in ((4096, 50304), (50304, 4096), (1250, 50304), (16384, 2048), (4096, 8192), (128256, 4096)):
            assert _width(M, N, K, epi) == 384
        # A that L2 holds; few K blocks; items that leave a third of the pairs idle; a split that narrower tiles do without
        for M, K in ((4096, 4096), (65536, 1024), (65536, 2048), (20360, 2056), (12000, 4096), (8192, 4096), (8192, 8192)):
            assert _width(M, N, K, epi) < 384
    assert all(_width(M, N, K, epi) < 384 for N in (192, 256, 392, 768) for M, K in ((4096, 50304), (50304, 4096)))
    assert all(_width(4096, N, 50304, EPI_F32) < 384 for N in (264, 384))
