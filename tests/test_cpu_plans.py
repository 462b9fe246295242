"""Which kernel the library takes for which sizes (its rules, without a GPU)."""
import pytest

from context_parallelism_b200 import _native as nv
from context_parallelism_b200.ops.gemm import EPI_BF16, EPI_F32, EPI_F32_ACC


def _width(M, N, K, epi):
    return nv.lib().cpb_gemm_plan(M, N, K, epi, 0) >> 16


@pytest.mark.parametrize("epi", [EPI_BF16, EPI_F32_ACC])
def test_one_column_of_384(epi):
    """Tiles of 384 columns follow sizes, not one width of the models."""
    for N in (264, 320, 344, 376, 384):                               # one such column, two of the next width
        for M, K in ((4096, 50304), (50304, 4096), (1250, 50304), (16384, 2048), (4096, 8192), (128256, 4096), (30000, 2056), (33000, 1536)):
            assert _width(M, N, K, epi) == 384
        # A that L2 holds; few K blocks; items that leave a third of the pairs idle; a split that narrower tiles do without
        for M, K in ((4096, 4096), (65536, 960), (20360, 2048), (24000, 3072), (12000, 3072), (8192, 4096), (8192, 8192)):
            assert _width(M, N, K, epi) < 384
        # rows off a 128-byte line, waves half full
        assert _width(20360, N, 2056, EPI_BF16) == (384 if N > 320 else 192) and _width(42000, N, 4104, EPI_BF16) == 384
    assert all(_width(M, N, K, epi) < 384 for N in (192, 256, 392, 768) for M, K in ((4096, 50304), (50304, 4096)))
    assert all(_width(4096, N, 50304, EPI_F32) < 384 for N in (264, 384))


def test_four_ctas_per_sm():
    """head_dim 64: many CTAs go to the kernel with four per SM; a long causal sequence of few K/V heads needs more of them."""
    f = nv.lib().cpb_flash_fwd_plan
    four = [(64, 300, 300, 32, 8, 1, 0), (40, 1024, 1024, 32, 8, 1, 0), (3, 8192, 8192, 32, 8, 1, 0), (1, 24576, 24576, 32, 8, 1, 0), (1, 32768, 32768, 32, 8, 1, 0),
            (4, 20480, 20480, 8, 8, 1, 0), (1, 20480, 20480, 32, 8, 0, 0), (1, 20000, 40000, 32, 8, 1, 1)]
    two = [(1, 8192, 8192, 32, 8, 1, 0), (1, 16384, 16384, 32, 8, 0, 0), (1, 18944, 18944, 32, 8, 1, 0), (1, 20480, 20480, 32, 8, 1, 0),
           (2, 20480, 20480, 16, 4, 1, 0), (1, 22000, 22000, 30, 10, 1, 0)]
    for sizes, kernel in ((four, 2), (two, 0)):
        assert all(f(*s[:5], 64, *s[5:]) == kernel for s in sizes)
    assert f(1, 32768, 32768, 4, 1, 128, 1, 0) == 1 and f(1, 4096, 4096, 32, 8, 128, 1, 0) == 0
