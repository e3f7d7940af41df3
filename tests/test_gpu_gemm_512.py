"""Dense GEMM tiles of 512 rows: two row blocks that share a tile's B, with two accumulators up to 128 columns and one beyond;
one and several tiles per CTA pair, ragged rows, columns and K blocks, a row block that lies beyond A altogether."""
import pytest

from clpeak_b200 import native as N
from tests.gpu_util import gemm_plan
from tests.test_gpu_gemm_tiles import check_every_element, elements_of

pytestmark = pytest.mark.gpu

# (tile width, several tiles per pair, (m, n, bytes of K))
PLANS = [(96, True, (12912, 400, 272)), (160, False, (305, 9928, 2576)), (160, True, (14827, 792, 3216)),
         (192, False, (326, 11992, 2960)), (192, True, (11357, 1064, 1808)), (224, False, (12317, 392, 5008)), (224, True, (6150, 3656, 1552))]


@pytest.mark.parametrize("tile_n,several,shape", PLANS)
@pytest.mark.parametrize("dtype", [N.DT_I8, N.DT_BF16, N.DT_TF32])
def test_every_plan(K, cuda, dtype, tile_n, several, shape):
    m, n, k_bytes = shape
    assert gemm_plan(K, dtype, m, n, elements_of(dtype, k_bytes)) == (tile_n, 1, 1)
    pairs = cuda.cuda.get_device_properties(0).multi_processor_count // 2
    assert (-(-m // 512) * -(-n // tile_n) > pairs) == several
    check_every_element(K, cuda, dtype, m, n, k_bytes)
