"""The fp32 GEMM on the tensor cores: every tile width and K split, edges of tiles and of chunks, and the numbers that three
bf16 pieces cannot hold."""
import ctypes as C

import pytest

from clpeak_b200 import native as N
from tests.gpu_util import dev_empty, gemm_plan, stream_ptr, sync

pytestmark = pytest.mark.gpu


def operands(K, cuda, m, n, k):
    out = []
    for rows, seed in ((m, 50), (n, 51)):
        f = dev_empty(rows * k, cuda.float32)
        K.clpk_fill_f32(f.data_ptr(), rows * k, seed, N.DIST_NORMAL, 0.0, 0.02, stream_ptr())
        out.append(f.view(rows, k))
    return out


def multiply(K, cuda, a, b, alpha=1.0):
    (m, k), n = a.shape, b.shape[0]
    c = cuda.full((m * n + 1024,), 7.0, dtype=cuda.float32, device="cuda")
    status = cuda.full((1,), 7, dtype=cuda.int32, device="cuda")
    args = N.GemmArgs(dtype=N.DT_F32, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), alpha=alpha, d_status=status.data_ptr())
    K.clpk_gemm(C.byref(args), stream_ptr())
    sync()
    assert int(status.item()) == 0
    assert bool((c[m * n:] == 7.0).all()), "the kernel wrote beyond C"
    return c[:m * n].view(m, n)


def worst(c, a, b, alpha=1.0):
    """Largest error in units of 2^-24 sum |a b|."""
    want, s_abs = alpha * (a.double() @ b.double().T), abs(alpha) * (a.double().abs() @ b.double().abs().T)
    return float(((c.double() - want).abs() / (2.0 ** -24 * s_abs + 1e-300)).max())


def bound(k):
    """One rounding per chunk of 32, one of alpha, and at most eight units for what an instruction cuts when it aligns its
    products (two per chunk cut a sum of full size, in a chunk that is a part of the sum)."""
    return -(-k // 32) + 9


# (tile width, K ranges) and a shape that takes them: ragged rows, columns and chunks, odd N, several tiles per pair
PLANS = [((32, 1), (2618, 67, 188)), ((32, 2), (2644, 65, 324)), ((32, 4), (1067, 65, 396)), ((64, 1), (67, 2381, 228)), ((64, 1), (2577, 829, 164)),
         ((64, 2), (2819, 73, 488)), ((64, 4), (1655, 67, 580)), ((96, 1), (273, 2387, 180)), ((96, 1), (1090, 1867, 164)), ((96, 2), (66, 2435, 816)),
         ((96, 4), (2914, 65, 604)), ((128, 1), (529, 2327, 172)), ((128, 1), (1544, 2051, 176)), ((128, 2), (264, 1629, 1848)), ((128, 4), (65, 1447, 1732))]


@pytest.mark.parametrize("plan,shape", PLANS)
def test_every_plan(K, cuda, plan, shape):
    assert gemm_plan(K, N.DT_F32, *shape) == (*plan, 2)
    a, b = operands(K, cuda, *shape)
    c = multiply(K, cuda, a, b, 0.75)
    assert worst(c, a, b, 0.75) <= bound(shape[2])
    assert bool((c == multiply(K, cuda, a, b, 0.75)).all()), "partial sums are added in a fixed order: the same bits every time"


@pytest.mark.parametrize("m,n,k", [(256, 128, 256), (257, 129, 260), (255, 127, 252), (128, 1000, 288), (1000, 131, 1028), (300, 202, 2044), (2000, 2001, 512)])
def test_edges(K, cuda, m, n, k):
    a, b = operands(K, cuda, m, n, k)
    assert worst(multiply(K, cuda, a, b), a, b) <= bound(k)


@pytest.mark.parametrize("shape", [(300, 200, 1024), (2000, 1500, 260)])
def test_infinities_nans_and_overflow(K, cuda, shape):
    """They reach what a product in 64 bits says they reach, and nothing else."""
    a, b = operands(K, cuda, *shape)
    a[3, 5], a[130, 0], a[131, 7], b[7, shape[2] - 1] = float("inf"), float("nan"), 3.4e38, float("-inf")
    a[200] = 1e30
    b[9] = 1e30                           # 1e60 overflows, 1e30 * 0.02 does not
    c = multiply(K, cuda, a, b)
    want = (a.double() @ b.double().T).float()
    finite = cuda.isfinite(want)
    assert bool((cuda.isfinite(c) == finite).all())
    assert bool((cuda.isnan(c) == cuda.isnan(want)).all()) and bool((c[~finite & ~cuda.isnan(want)] == want[~finite & ~cuda.isnan(want)]).all())
    s_abs = a.double().abs() @ b.double().abs().T
    assert bool(((c.double() - want.double()).abs()[finite] <= (shape[2] + 2) * 2.0 ** -24 * s_abs[finite]).all())


@pytest.mark.parametrize("shape", [(300, 200, 1024), (2000, 1500, 260)])
@pytest.mark.parametrize("small,large", [(2.0 ** -96, 2.0 ** 90), (2.0 ** -110, 2.0 ** 100), (2.0 ** -140, 2.0 ** 120)])
def test_small_magnitudes_keep_their_bits(K, cuda, shape, small, large):
    """Elements whose pieces at their own size would leave bf16's range; zeros stay zeros."""
    a, b = operands(K, cuda, *shape)
    a[5:9] *= small
    a[100] = 0.0
    b *= large
    b[11] = 0.0
    c = multiply(K, cuda, a, b)
    assert worst(c, a, b) <= shape[2] + 2
    assert bool((c[100] == 0.0).all()) and bool((c[:, 11] == 0.0).all())


@pytest.mark.parametrize("plan,shape", PLANS)
def test_one_small_element_at_every_row_of_a_tile(K, cuda, plan, shape):
    """One row of a tile holds zeros and one magnitude that bf16 pieces at their own size could not hold, the others N(0, 0.02);
    the other operand is near 2^100, so that the small element's products are ordinary numbers: every row of the tile, in the
    tile's halves that the two CTAs of a pair convert, in the first, a middle and the last chunk, with K split and not."""
    assert gemm_plan(K, N.DT_F32, *shape) == (*plan, 2)
    (m, n, k), tn = shape, plan[0]
    a, b = operands(K, cuda, *shape)
    smalls, columns = (2.0 ** -120, 1.375 * 2.0 ** -130, 1.25 * 2.0 ** -140), (0, k - 1, k // 2 + 1)
    failed = []
    # every row of B at every magnitude, every row of A at one of them
    for operand, other, tile, runs in ((b, a, tn, [(r, v) for r in range(tn) for v in range(3)]), (a, b, 256, [(r, r % 3) for r in range(256)])):
        saved = operand.clone()
        other *= 2.0 ** 100
        for r, v in runs:
            if r >= operand.shape[0]:
                continue
            rows = cuda.arange(r, operand.shape[0], tile, device="cuda")
            at, small = columns[(r + v) % 3], smalls[v]
            operand[rows] = 0.0
            operand[rows, at] = small
            c = multiply(K, cuda, a, b)
            got = (c[:, rows].T if operand is b else c[rows]).double()
            want = other[:, at].double() * float(cuda.tensor(small, dtype=cuda.float32))
            # one product, of which at most 2^-24 is left out, and a rounding of it and of alpha
            if not bool(((got - want).abs() <= 3 * 2.0 ** -24 * want.abs()).all()):
                failed.append(("B" if operand is b else "A", r, small))
            operand[rows] = saved[rows]
        other *= 2.0 ** -100
    assert not failed, f"{len(failed)} of the single elements are lost, the first: {failed[:5]}"


@pytest.mark.parametrize("exponents", [(-70, -70), (-60, -72), (-63, -75), (-40, -66)])
def test_results_near_the_end_of_the_range(K, cuda, exponents):
    """Products that fp32 holds only in part: K roundings to 2^-149 besides the relative ones."""
    m, n, k = 300, 200, 2044
    assert gemm_plan(K, N.DT_F32, m, n, k)[2] == 2
    a, b = operands(K, cuda, m, n, k)
    a *= 2.0 ** exponents[0]
    b *= 2.0 ** exponents[1]
    c = multiply(K, cuda, a, b)
    want, s_abs = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    assert bool(((c.double() - want).abs() <= (k + 2) * (2.0 ** -24 * s_abs + 2.0 ** -150)).all())


@pytest.mark.parametrize("exponents", [(-64, -64), (-68, -68), (-58, -70), (-100, -28), (-134, 0), (0, -134), (-120, 60), (60, -135)])
@pytest.mark.parametrize("plan,shape", [((32, 4), (300, 200, 2044)), ((128, 1), (1544, 2051, 176))])
def test_small_results_keep_their_bits(K, cuda, plan, shape, exponents):
    """Results and operands down to the last bits of fp32: the error of larger ones, and a rounding to 2^-149 for each K range and
    for alpha.  Zeros in their place would be hundreds of such units off."""
    assert gemm_plan(K, N.DT_F32, *shape) == (*plan, 2)
    a, b = (cuda.randn(rows, shape[2], generator=cuda.Generator(device="cuda").manual_seed(rows), device="cuda") for rows in shape[:2])
    a, b = (a.double() * 2.0 ** exponents[0]).float(), (b.double() * 2.0 ** exponents[1]).float()
    c = multiply(K, cuda, a, b, 0.75)
    want, s_abs = 0.75 * (a.double() @ b.double().T), 0.75 * (a.double().abs() @ b.double().abs().T)
    room = bound(shape[2]) * 2.0 ** -24 * s_abs + (plan[1] + 1) * 2.0 ** -150
    assert bool(((c.double() - want).abs() <= room).all()) and float((want.abs() / room).median()) > 20


def median_time(K, cuda, dtype, a, b, c, status):
    (m, k), n = a.shape, b.shape[0]
    args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), alpha=1.0, d_status=status.data_ptr())
    times = []
    for _ in range(7):
        start, end = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        for _ in range(3):
            K.clpk_gemm(C.byref(args), stream_ptr())
        end.record()
        sync()
        times.append(start.elapsed_time(end))
    return sorted(times)[3]


def test_small_numbers_and_zeros_cost_nothing(K, cuda):
    """A small element in every row of A, small results, half of A zeros: the time of ordinary operands, within a half."""
    n = 2048
    a, b = operands(K, cuda, n, n, n)
    c, status = dev_empty(n * n, cuda.float32), dev_empty(1, cuda.int32)
    one_small = a.clone()
    one_small[:, 7] = 2.0 ** -120
    ordinary = median_time(K, cuda, N.DT_F32, a, b, c, status)
    for x, y in ((one_small, b), (a * 2.0 ** -60, b * 2.0 ** -60), (a.clamp(min=0.0), b)):
        assert median_time(K, cuda, N.DT_F32, x, y, c, status) <= 1.5 * ordinary


def test_a_nan_costs_no_more_than_the_cuda_cores(K, cuda):
    """One NaN and nothing but NaNs at 4096^3: not the time of the CUDA-core kernel; results too large for the scaled pieces in every
    tile: within three times that."""
    n = 4096
    a, b = operands(K, cuda, n, n, n)
    c, status = dev_empty(n * n, cuda.float32), dev_empty(1, cuda.int32)
    cuda_cores = median_time(K, cuda, N.DT_F32_FFMA, a, b, c, status)
    one_in_a, one_in_b, all_of_a = a.clone(), b.clone(), cuda.full_like(a, float("nan"))
    one_in_a[77, 7] = one_in_b[1234, 4000] = float("nan")
    for x, y in ((one_in_a, b), (a, one_in_b), (all_of_a, b)):
        assert median_time(K, cuda, N.DT_F32, x, y, c, status) <= cuda_cores
    assert median_time(K, cuda, N.DT_F32, a * 2.0 ** 50, b * 2.0 ** 50, c, status) <= 3 * cuda_cores


@pytest.mark.parametrize("plan,shape", PLANS)
def test_sums_that_are_not_finite_in_every_plan(K, cuda, plan, shape):
    """Single infinities and NaNs in the first and the last rows and chunks, then results beyond 2^110 throughout: each output that
    is finite in 64 bits is, within fp32 rounding, and the others are infinite or NaN as there."""
    (m, n, k), (a, b) = shape, operands(K, cuda, *shape)
    a[m - 1, k - 1], a[3, 0], b[n - 1, 1], b[5, k - 2] = float("nan"), float("inf"), float("-inf"), float("nan")
    assert gemm_plan(K, N.DT_F32, m, n, k) == (*plan, 2)
    large = [t * 2.0 ** 61 for t in operands(K, cuda, *shape)]
    for x, y in ((a, b), large):
        c = multiply(K, cuda, x, y)
        want = x.double() @ y.double().T
        s_abs = x.double().abs() @ y.double().abs().T
        assert bool((cuda.isnan(c) == cuda.isnan(want)).all()) and bool((cuda.isinf(c) == cuda.isinf(want)).all())
        infinite, finite = cuda.isinf(want), cuda.isfinite(want)
        assert bool((c.double()[infinite] == want[infinite]).all())
        assert bool(((c.double() - want).abs()[finite] <= (k + 2) * 2.0 ** -24 * s_abs[finite]).all())


def test_wide_range_of_magnitudes(K, cuda):
    """Every element of its own binade between 2^-40 and 2^40: the error stays relative to the products."""
    m, n, k = 513, 260, 1000
    a, b = operands(K, cuda, m, n, k)
    for t, seed in ((a, 3), (b, 4)):
        g = cuda.Generator(device="cuda").manual_seed(seed)
        t *= 2.0 ** cuda.randint(-40, 41, t.shape, generator=g, device="cuda").float()
    assert worst(multiply(K, cuda, a, b), a, b) <= bound(k)


def test_the_cuda_cores_on_request(K, cuda):
    """DT_F32_FFMA: no tile of the tensor cores at any size, the same product within fp32 rounding."""
    m, n, k = 300, 202, 2044
    assert gemm_plan(K, N.DT_F32, m, n, k)[2] == 2 and gemm_plan(K, N.DT_F32_FFMA, m, n, k)[2] != 2
    a, b = operands(K, cuda, m, n, k)
    c, status = dev_empty(m * n, cuda.float32), dev_empty(1, cuda.int32)
    args = N.GemmArgs(dtype=N.DT_F32_FFMA, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), alpha=1.0, d_status=status.data_ptr())
    K.clpk_gemm(C.byref(args), stream_ptr())
    sync()
    assert worst(c.view(m, n), a, b) <= k + 2
