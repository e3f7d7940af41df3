"""Dense GEMM tiles of 512 rows: two row blocks that share a tile's B, with two accumulators up to 128 columns and one beyond;
one and several tiles per CTA pair, ragged rows, columns and K blocks, a row block that lies beyond A altogether."""
import pytest

from clpeak_b200 import native as N
from tests.gpu_util import gemm_plan
from tests.test_gpu_gemm_tiles import check_every_element, elements_of

pytestmark = pytest.mark.gpu

# (tile width, several tiles per pair, (m, n, bytes of K))
PLANS = [(64, True, (21608, 168, 1024)), (128, True, (6845, 1200, 128)), (96, True, (12912, 400, 272)), (160, False, (305, 9928, 2576)), (160, True, (14827, 792, 3216)),
         (192, False, (326, 11992, 2960)), (192, True, (11357, 1064, 1808)), (224, False, (12317, 392, 5008)), (224, True, (6150, 3656, 1552))]


@pytest.mark.parametrize("tile_n,several,shape", PLANS)
@pytest.mark.parametrize("dtype", [N.DT_I8, N.DT_BF16, N.DT_F16, N.DT_E4M3, N.DT_E5M2, N.DT_TF32])
def test_every_plan(K, cuda, dtype, tile_n, several, shape):
    m, n, k_bytes = shape
    assert gemm_plan(K, dtype, m, n, elements_of(dtype, k_bytes)) == (tile_n, 1, 1)
    pairs = cuda.cuda.get_device_properties(0).multi_processor_count // 2
    assert (-(-m // 512) * -(-n // tile_n) > pairs) == several
    check_every_element(K, cuda, dtype, m, n, k_bytes)


def test_narrow_tiles_where_rows_are_not_whole_sectors(K):
    """Rows of an odd multiple of 16 bytes: short sums only.  The e4m3 shapes took 12.9 and 13.7 us in 96-wide tiles, 11.6 and 12.4 in large ones."""
    for n, k_bytes, tile_n in ((13928, 784, 0), (13680, 816, 0), (13928, 800, 96), (13680, 896, 96)):
        assert gemm_plan(K, N.DT_E4M3, 270, n, k_bytes)[0] == tile_n
    assert gemm_plan(K, N.DT_BF16, 12912, 400, 136) == (96, 1, 1)
