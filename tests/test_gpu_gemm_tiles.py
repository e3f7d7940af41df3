"""GEMM shapes that do not fill the chip with 512 x 256 tiles: narrower tiles, K split over the CTA pairs of a cluster,
several tiles per pair.  Every element of C against the fp64 product of the same operands."""
import ctypes as C

import pytest

from clpeak_b200 import native as N
from tests.gpu_util import dev_empty, gemm_plan, stream_ptr, sync
from tests.test_gpu_gemm import WIDE_OUT, make_gemm_operands

pytestmark = pytest.mark.gpu


def as_f64(cuda, dtype, q, rows, k):
    view = {N.DT_BF16: cuda.bfloat16, N.DT_F16: cuda.float16, N.DT_E4M3: cuda.float8_e4m3fn, N.DT_E5M2: cuda.float8_e5m2,
            N.DT_TF32: cuda.float32, N.DT_I8: cuda.int8}[dtype]
    return q.view(view).double().view(rows, k)


def run_into(K, cuda, dtype, m, n, k, d_a, d_b, alpha, pad=4096):
    canary = 0x7FC00000 if dtype in WIDE_OUT else 0x7FC0
    c = cuda.full((m * n + pad,), canary, dtype=cuda.int32 if dtype in WIDE_OUT else cuda.int16, device="cuda")
    status = dev_empty(1, cuda.int32)
    args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=d_a.data_ptr(), d_b=d_b.data_ptr(), d_c=c.data_ptr(), alpha=alpha,
                      d_status=status.data_ptr())
    K.clpk_gemm(C.byref(args), stream_ptr())
    sync()
    assert int(status.item()) == 0, "a device-side wait timed out"
    assert bool((c[m * n:] == canary).all()), "the kernel wrote beyond C"
    assert not bool((c[:m * n] == canary).any()), "some of C was never written"
    return c[:m * n]


# (m, n, bytes of K): one K block and less; a ragged last block in each stage position; K split in two and four with
# ranges of unequal length; ragged last tiles; several tiles per CTA pair (PLANS below names the tiles)
@pytest.mark.parametrize("m,n,k_bytes", [
    (1, 8, 16), (64, 64, 128), (129, 40, 144), (256, 96, 400), (300, 304, 4816), (64, 64, 32768), (200, 208, 9008),
    (512, 256, 1024), (1000, 1016, 528), (1288, 544, 12448), (2072, 3488, 928), (1024, 1024, 2048), (700, 904, 6000),
    (64, 11984, 1872), (8192, 3000, 1024), (16384, 72, 256), (120, 2008, 3232)])
@pytest.mark.parametrize("dtype", [N.DT_I8, N.DT_BF16, N.DT_F16, N.DT_E4M3, N.DT_E5M2, N.DT_TF32])
def test_every_element(K, cuda, dtype, m, n, k_bytes):
    check_every_element(K, cuda, dtype, m, n, k_bytes)


def elements_of(dtype, k_bytes):
    return k_bytes // (4 if dtype == N.DT_TF32 else 2 if dtype in (N.DT_BF16, N.DT_F16) else 1)


def check_every_element(K, cuda, dtype, m, n, k_bytes):
    k = elements_of(dtype, k_bytes)
    d_a, d_b = make_gemm_operands(K, cuda, dtype, m, n, k)
    alpha = 1.0 if dtype == N.DT_I8 else 0.75
    c = run_into(K, cuda, dtype, m, n, k, d_a, d_b, alpha)
    fa, fb = as_f64(cuda, dtype, d_a, m, k), as_f64(cuda, N.DT_E4M3 if dtype == N.DT_E5M2 else dtype, d_b, n, k)
    want = fa @ fb.T
    if dtype == N.DT_I8:
        assert bool((c.view(m, n) == want.to(cuda.int32)).all())           # |sums| < 2^24: exact in both
    else:
        got = c.view(cuda.float32 if dtype == N.DT_TF32 else cuda.bfloat16).double().view(m, n)
        want *= alpha
        # K roundings of the accumulator (truncating adder: one ulp each), one of alpha, one of the bf16 result
        tol = (k + 1) * 2.0 ** -23 * alpha * (fa.abs() @ fb.abs().T) + (0.0 if dtype == N.DT_TF32 else 2.0 ** -8) * want.abs() + 1e-30
        worst = float(((got - want).abs() / tol).max())
        assert worst <= 1.0, f"worst error over all of C is {worst:.3g}x the stated tolerance"
    again = run_into(K, cuda, dtype, m, n, k, d_a, d_b, alpha)
    assert bool((again == c).all()), "partial sums are added in a fixed order: the same bits every time"


# every tile width with K whole, in two and in four, and with several tiles per CTA pair: an odd number of 32-column
# chunks (96, 160, 224) is shared unevenly between the two epilogue warps of a quarter and between the pairs of a cluster.
# Ragged tiles, K blocks and ranges throughout.
PLANS = [(32, 1, 1, (75, 80, 528)), (64, 1, 1, (69, 2848, 560)), (96, 1, 1, (102, 4968, 528)), (128, 1, 1, (68, 7776, 576)),
         (160, 1, 1, (288, 5632, 528)), (192, 1, 1, (818, 3288, 544)), (224, 1, 1, (257, 7176, 544)), (256, 1, 1, (9690, 256, 544)),
         (64, 1, 2, (9715, 168, 128)), (96, 1, 2, (9922, 264, 2160)), (128, 1, 2, (5295, 792, 528)), (160, 1, 2, (336, 9672, 528)),
         (192, 1, 2, (1034, 5216, 544)), (224, 1, 2, (632, 10360, 528)), (256, 1, 2, (628, 11080, 576)),
         (32, 2, 1, (65, 560, 2544)), (64, 2, 1, (65, 1472, 3920)), (96, 2, 1, (64, 2376, 3728)), (128, 2, 1, (67, 3248, 4848)),
         (160, 2, 1, (70, 4848, 4768)), (192, 2, 1, (66, 5352, 6048)), (224, 2, 1, (71, 7352, 5808)), (256, 2, 1, (70, 7568, 7840)),
         (32, 4, 1, (68, 64, 1872)), (64, 4, 1, (69, 496, 2864)), (96, 4, 1, (67, 1152, 3344)), (128, 4, 1, (67, 1528, 5472)),
         (160, 4, 1, (69, 2256, 5616)), (192, 4, 1, (72, 2408, 8864)), (224, 4, 1, (67, 3232, 8480)), (256, 4, 1, (64, 3400, 12656))]


@pytest.mark.parametrize("tile_n,splits,tiles_per_pair,shape", PLANS)
@pytest.mark.parametrize("dtype", [N.DT_I8, N.DT_BF16, N.DT_TF32])
def test_every_plan(K, cuda, dtype, tile_n, splits, tiles_per_pair, shape):
    m, n, k_bytes = shape
    assert gemm_plan(K, dtype, m, n, elements_of(dtype, k_bytes)) == (tile_n, splits, 0)
    pairs = cuda.cuda.get_device_properties(0).multi_processor_count // 2
    assert (splits == 1 and -(-m // 256) * -(-n // tile_n) > pairs) == (tiles_per_pair > 1)
    check_every_element(K, cuda, dtype, m, n, k_bytes)


def test_plans_that_no_kernel_takes_are_refused(K):
    out = [C.c_uint32(0) for _ in range(2)]
    for args in ((N.DT_BF16, 0, 8, 8), (N.DT_MXF4_B64, 64, 64, 256), (99, 64, 64, 256)):
        with pytest.raises(N.ClpkError) as e:
            K.clpk_gemm_plan(*args, C.byref(out[0]), C.byref(out[1]), None)
        assert e.value.code == N.ERR_BAD_ARG


def test_aligned_launches_on_two_streams(K, cuda):
    """GEMMs whose producers meet once per wave, back to back on two streams and over more launches than there are wave
    counters: whoever holds the SMs, the bits are those of a launch by itself, and the counters are zero again."""
    m, n, k = 8192, 8192, 256
    d_a, d_b = make_gemm_operands(K, cuda, N.DT_BF16, m, n, k)
    want = run_into(K, cuda, N.DT_BF16, m, n, k, d_a, d_b, 1.0).clone()
    assert K.raw("clpk_gemm_last_launch_aligned")() == 1
    streams = [cuda.cuda.Stream() for _ in range(2)]
    out = [dev_empty(m * n, cuda.int16) for _ in streams]
    status = [dev_empty(1, cuda.int32) for _ in streams]
    sync()
    for _ in range(20):
        for s, c, st in zip(streams, out, status):
            args = N.GemmArgs(dtype=N.DT_BF16, m=m, n=n, k=k, d_a=d_a.data_ptr(), d_b=d_b.data_ptr(), d_c=c.data_ptr(), alpha=1.0,
                              d_status=st.data_ptr())
            K.clpk_gemm(C.byref(args), s.cuda_stream)
    sync()
    for c, st in zip(out, status):
        assert int(st.item()) == 0 and bool((c == want).all())
    assert wave_state(K)[0] == 0, "a counter did not come back to zero"


def wave_state(K):
    counters_set, dropouts = C.c_uint32(99), C.c_uint32(99)
    K.clpk_gemm_wave_state(C.byref(counters_set), C.byref(dropouts), stream_ptr())
    return counters_set.value, dropouts.value


def test_producers_meet_and_leave_the_counters_at_zero(K, cuda):
    """More launches than there are counters, each with the chip to itself: no producer gives up waiting for the others, and
    after each launch every counter is zero again -- one left above zero would let the producers of the launch that gets
    it next pass unmet, which no result shows."""
    m, n, k = 8192, 8192, 256
    d_a, d_b = make_gemm_operands(K, cuda, N.DT_BF16, m, n, k)
    c, status = dev_empty(m * n, cuda.int16), dev_empty(1, cuda.int32)
    args = N.GemmArgs(dtype=N.DT_BF16, m=m, n=n, k=k, d_a=d_a.data_ptr(), d_b=d_b.data_ptr(), d_c=c.data_ptr(), alpha=1.0,
                      d_status=status.data_ptr())
    sync()
    before = wave_state(K)
    assert before[0] == 0
    for _ in range(40):
        K.clpk_gemm(C.byref(args), stream_ptr())
        assert K.raw("clpk_gemm_last_launch_aligned")() == 1
        assert wave_state(K) == before
