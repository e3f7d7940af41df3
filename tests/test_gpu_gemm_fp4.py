"""Block-scaled GEMM: the arrangement of the scale factors and the shapes where its tiles can go wrong."""
import ctypes as C

import pytest

from clpeak_b200 import native as N
from tests.gpu_util import dev_empty, gemm_plan, stream_ptr, sync
from tests.test_gpu_gemm import make_nvfp4_operand

pytestmark = pytest.mark.gpu


def run(K, cuda, dtype, m, n, k, a, sfa, b, sfb, alpha, ws, pad=4096):
    c = cuda.full((m * n + pad,), 0x7FC0, dtype=cuda.int16, device="cuda")
    status = dev_empty(1, cuda.int32)
    args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), d_sfa=sfa, d_sfb=sfb,
                      alpha=alpha, d_workspace=ws.data_ptr(), workspace_bytes=ws.numel(), d_status=status.data_ptr())
    K.clpk_gemm(C.byref(args), stream_ptr())
    sync()
    assert int(status.item()) == 0, "a device-side wait timed out"
    assert bool((c[m * n:] == 0x7FC0).all()), "the kernel wrote beyond C"
    assert not bool((c[:m * n] == 0x7FC0).any()), "some of C was never written"
    return c[:m * n]


def workspace(K, cuda, dtype, m, n, k):
    need = C.c_size_t(0)
    K.clpk_gemm_workspace_bytes(dtype, m, n, k, C.byref(need))
    return cuda.full((need.value,), 0xFF, dtype=cuda.uint8, device="cuda")


@pytest.mark.parametrize("dtype", [N.DT_NVF4, N.DT_MXF4])
@pytest.mark.parametrize("m,n,k", [(1, 8, 256), (130, 264, 2304), (300, 200, 4096)])
def test_scales_at_any_word_alignment(K, cuda, dtype, m, n, k):
    """Scale arrays need only be aligned to 4 bytes; the packed blocks, and so C, are the same."""
    a, sfa, ta, _ = make_nvfp4_operand(K, cuda, m, k, 40, dtype)
    b, sfb, tb, _ = make_nvfp4_operand(K, cuda, n, k, 41, dtype)
    results = []
    for offset in (0, 4, 8, 12):
        moved = []
        for sf in (sfa, sfb):
            t = cuda.empty(sf.numel() + 16, dtype=cuda.uint8, device="cuda")
            t[offset:offset + sf.numel()] = sf
            moved.append(t)
        ws = workspace(K, cuda, dtype, m, n, k)
        c = run(K, cuda, dtype, m, n, k, a, moved[0].data_ptr() + offset, b, moved[1].data_ptr() + offset, ta * tb, ws)
        results.append((ws, c))
    for ws, c in results[1:]:
        assert bool((ws == results[0][0]).all()) and bool((c == results[0][1]).all())


# Row-major scales are arranged by the multiplication itself up to four waves of 256 x 256 tiles, and by a launch of their own
# beyond, and for long NVFP4 sums from the second wave on.  One to nine K blocks (units hold two or four); 64- and 128-wide tiles
# whose last block of rows has no neighbour; 256-wide ones with one accumulator, one to four waves of them; K split.
@pytest.mark.parametrize("m,n,k", [(64, 64, 256), (130, 72, 768), (520, 328, 1280), (300, 1160, 2304), (2048, 2048, 2048), (2000, 2056, 512),
                                   (2200, 2304, 1792), (4096, 4096, 1024), (4100, 4616, 256), (600, 7000, 5376), (458, 1176, 6400), (300, 136, 11008)])
@pytest.mark.parametrize("dtype,offset", [(N.DT_NVF4, 0), (N.DT_NVF4, 4), (N.DT_MXF4, 0), (N.DT_MXF4, 4), (N.DT_MXF4, 8)])
def test_scales_arranged_on_the_way_and_in_front(K, cuda, dtype, offset, m, n, k):
    g = cuda.Generator(device="cuda").manual_seed(m + n + k)
    a, b = (cuda.randint(0, 256, (rows * k // 2,), dtype=cuda.uint8, device="cuda", generator=g) for rows in (m, n))
    block = 16 if dtype == N.DT_NVF4 else 32
    base = 0x30 if dtype == N.DT_NVF4 else 0x78                     # 0.5 ... 15, or 2^-7 ... 2^8
    sfa, sfb = (cuda.randint(base, base + 16 if dtype == N.DT_MXF4 else base + 0x28, (rows * k // block + offset,), dtype=cuda.uint8, device="cuda",
                             generator=g)[offset:] for rows in (m, n))
    in_front, on_the_way = workspace(K, cuda, dtype, m, n, k), workspace(K, cuda, dtype, m, n, k)
    args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_sfa=sfa.data_ptr(), d_sfb=sfb.data_ptr(), d_workspace=in_front.data_ptr(),
                      workspace_bytes=in_front.numel())
    K.clpk_gemm_pack_scales(C.byref(args), stream_ptr())
    want = run(K, cuda, dtype, m, n, k, a, None, b, None, 0.25, in_front)
    got = run(K, cuda, dtype, m, n, k, a, sfa.data_ptr(), b, sfb.data_ptr(), 0.25, on_the_way)
    assert bool((got == want).all()), "the same sums in the same order"
    assert bool((on_the_way == in_front).all()), "the workspace holds the arranged scales afterwards"


# both sides of each line: four waves of 74 tiles of 256 x 256; NVFP4 sums of more than 40 K blocks over all waves, in the first wave only
# where a scale array is not aligned to a K block's words
@pytest.mark.parametrize("launches,dtype,offset,m,n,k",
                         [(1, N.DT_NVF4, 0, 2048, 2048, 2048), (1, N.DT_NVF4, 0, 2048, 2048, 16384), (2, N.DT_NVF4, 4, 2048, 2048, 16384),
                          (1, N.DT_NVF4, 4, 2048, 2048, 10240), (1, N.DT_NVF4, 0, 2304, 2304, 5120), (2, N.DT_NVF4, 0, 2304, 2304, 5376),
                          (1, N.DT_NVF4, 0, 4352, 4352, 2560), (2, N.DT_NVF4, 0, 4352, 4352, 2816), (2, N.DT_NVF4, 0, 4352, 4608, 256),
                          (1, N.DT_NVF4, 0, 64, 64, 256), (1, N.DT_MXF4, 0, 2304, 2304, 5376), (1, N.DT_MXF4, 4, 2048, 2048, 16384),
                          (1, N.DT_MXF4, 4, 4352, 4352, 16384), (2, N.DT_MXF4, 0, 4352, 4608, 256)])
def test_launches_of_a_call_with_row_major_scales(K, cuda, launches, dtype, offset, m, n, k):
    if cuda.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the waves are those of 148 SMs")
    block = 16 if dtype == N.DT_NVF4 else 32
    a, b, sfa, sfb = (cuda.zeros(size, dtype=cuda.uint8, device="cuda") for size in (m * k // 2, n * k // 2, m * k // block + offset, n * k // block + offset))
    c, status, ws = cuda.zeros(m * n, dtype=cuda.int16, device="cuda"), cuda.zeros(1, dtype=cuda.int32, device="cuda"), workspace(K, cuda, dtype, m, n, k)
    args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), d_sfa=sfa.data_ptr() + offset,
                      d_sfb=sfb.data_ptr() + offset, alpha=1.0, d_workspace=ws.data_ptr(), workspace_bytes=ws.numel(), d_status=status.data_ptr())
    K.clpk_gemm(C.byref(args), stream_ptr())
    sync()
    graph, stream, nodes = cuda.cuda.CUDAGraph(keep_graph=True), cuda.cuda.Stream(), C.c_size_t(0)
    with cuda.cuda.graph(graph, stream=stream):
        K.clpk_gemm(C.byref(args), stream.cuda_stream)
    assert C.CDLL("libcuda.so.1").cuGraphGetNodes(C.c_void_p(graph.raw_cuda_graph()), None, C.byref(nodes)) == 0
    assert nodes.value == launches


def decoded(cuda, dtype, q, sf, rows, k):
    """The operand's values in fp64."""
    codes = cuda.stack((q & 15, q >> 4), dim=-1).view(rows, k).long()
    mags = cuda.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=cuda.float64, device="cuda")
    values = mags[codes & 7] * cuda.where(codes >= 8, -1.0, 1.0)
    block = 16 if dtype == N.DT_NVF4 else 32
    scale = sf.view(cuda.float8_e4m3fn).double() if dtype == N.DT_NVF4 else cuda.exp2(sf.double() - 127)
    return values * scale.view(rows, k // block).repeat_interleave(block, dim=1)


# one stage; 64-wide tiles in both halves of a scale block, with ragged last tiles; K split in four with ranges of unequal
# length; several tiles per CTA pair; whole tiles (PLANS below names the tiles)
@pytest.mark.parametrize("m,n,k", [(1, 8, 256), (64, 64, 256), (200, 200, 512), (384, 480, 256), (95, 352, 8960), (300, 136, 11008),
                                   (350, 416, 3328), (458, 1176, 6400), (2656, 120, 16384), (72, 1136, 13568), (8404, 216, 1024),
                                   (6976, 544, 5376), (512, 512, 2048)])
@pytest.mark.parametrize("dtype", [N.DT_NVF4, N.DT_MXF4])
def test_every_element(K, cuda, dtype, m, n, k):
    check_every_element(K, cuda, dtype, m, n, k)


# every tile with K whole, in two and in four: a 64-wide tile uses half of a block of B's scale factors, a 256-wide one
# two blocks in one box, 48 tensor-memory columns and five stages; and several tiles per CTA pair
PLANS = [(64, 1, 1, (33, 144, 256)), (128, 1, 1, (33, 5456, 768)), (64, 1, 2, (795, 2344, 256)), (128, 1, 2, (883, 4648, 256)),
         (64, 2, 1, (33, 1072, 3072)), (128, 2, 1, (34, 2128, 5376)), (256, 2, 1, (34, 4808, 8448)), (256, 2, 1, (512, 2304, 8192)),
         (64, 4, 1, (33, 128, 2816)), (128, 4, 1, (35, 1016, 5888)), (256, 4, 1, (33, 2136, 12288)), (256, 4, 1, (512, 1024, 16384)),
         (0, 1, 1, (2048, 5000, 1024))]


@pytest.mark.parametrize("tile_n,splits,tiles_per_pair,shape", PLANS)
@pytest.mark.parametrize("dtype", [N.DT_NVF4, N.DT_MXF4])
def test_every_plan(K, cuda, dtype, tile_n, splits, tiles_per_pair, shape):
    m, n, k = shape
    assert gemm_plan(K, dtype, m, n, k) == (tile_n, splits, 0)
    if tile_n:
        pairs = cuda.cuda.get_device_properties(0).multi_processor_count // 2
        assert (splits == 1 and -(-m // 256) * -(-n // tile_n) > pairs) == (tiles_per_pair > 1)
    check_every_element(K, cuda, dtype, m, n, k)


# an A of a few rows and tiles for most of the chip: many pairs asking for the same lines made small tiles up to 1.3 times
# slower than the large kernel's; half the pairs, or more rows, and they are faster
@pytest.mark.parametrize("tile_n,shape", [(0, (9, 9336, 14592)), (0, (1, 9128, 12032)), (0, (28, 6680, 4352)), (128, (2, 4456, 3328)),
                                          (128, (64, 6680, 4352)), (64, (9, 1024, 1536))])
def test_operands_of_a_few_rows(K, cuda, tile_n, shape):
    assert gemm_plan(K, N.DT_NVF4, *shape)[0] == tile_n
    check_every_element(K, cuda, N.DT_NVF4, *shape)


def check_every_element(K, cuda, dtype, m, n, k):
    a, sfa, ta, _ = make_nvfp4_operand(K, cuda, m, k, 40, dtype)
    b, sfb, tb, _ = make_nvfp4_operand(K, cuda, n, k, 41, dtype)
    alpha, ws = ta * tb, workspace(K, cuda, dtype, m, n, k)
    c = run(K, cuda, dtype, m, n, k, a, sfa.data_ptr(), b, sfb.data_ptr(), alpha, ws)
    fa, fb = decoded(cuda, dtype, a, sfa, m, k), decoded(cuda, dtype, b, sfb, n, k)
    want = alpha * (fa @ fb.T)
    # K roundings of the accumulator (truncating adder: one ulp each), one of alpha, one of the bf16 result
    tol = (k + 1) * 2.0 ** -23 * alpha * (fa.abs() @ fb.abs().T) + 2.0 ** -8 * want.abs() + 1e-30
    worst = float(((c.view(cuda.bfloat16).double().view(m, n) - want).abs() / tol).max())
    assert worst <= 1.0, f"worst error over all of C is {worst:.3g}x the stated tolerance"
    again = run(K, cuda, dtype, m, n, k, a, None, b, None, alpha, ws)       # scales already arranged
    assert bool((again == c).all()), "partial sums are added in a fixed order: the same bits every time"
