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


def multiply(K, cuda, a, b, alpha=1.0, dtype=N.DT_F32):
    (m, k), n = a.shape, b.shape[0]
    c = cuda.full((m * n + 1024,), 7.0, dtype=cuda.float32, device="cuda")
    status = cuda.full((1,), 7, dtype=cuda.int32, device="cuda")
    args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), alpha=alpha, d_status=status.data_ptr())
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
    """One rounding for each turn of 64 products, one for each of four K ranges that begins a turn of its own, one of alpha, one unit
    for the products that are left out, and two for each of the four instructions of a turn that cut a sum of full size."""
    return -(-k // 64) + 3 + 1 + 1 + 8


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


# whole tiles and chunks, one row, column and four k more, and one less, for each tile width
@pytest.mark.parametrize("tile_n,m,n,k", [(t, m + d, n + d, k + 4 * d) for t, m, n, k in
                                          [(32, 512, 128, 1024), (64, 512, 256, 1024), (64, 1024, 512, 512), (96, 512, 1536, 1024)]
                                          for d in (0, 1, -1)] + [(128, 2048, 2048, 96), (96, 2049, 2049, 100), (128, 2047, 2047, 92), (128, 2000, 2001, 64),
                                                                  (64, 1000, 131, 1028), (32, 300, 202, 2044)])
def test_edges(K, cuda, tile_n, m, n, k):
    plan = gemm_plan(K, N.DT_F32, m, n, k)
    assert (plan[0], plan[2]) == (tile_n, 2)
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
    """Products that fp32 holds only in part: a rounding to 2^-149 for each of the four K ranges and for alpha besides the relative ones,
    of results of which many are larger by far."""
    m, n, k = 300, 200, 2044
    assert gemm_plan(K, N.DT_F32, m, n, k) == (32, 4, 2)
    a, b = operands(K, cuda, m, n, k)
    a *= 2.0 ** exponents[0]
    b *= 2.0 ** exponents[1]
    c = multiply(K, cuda, a, b)
    want, s_abs = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    room = bound(k) * 2.0 ** -24 * s_abs + 5 * 2.0 ** -150
    assert bool(((c.double() - want).abs() <= room).all()) and float((want.abs() / room).max()) > 3, "zeros would pass"


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


@pytest.mark.parametrize("values", ["uniform", "magnitudes", "constant"])
@pytest.mark.parametrize("shape", [(2048, 2048, k) for k in (64, 96, 128, 256, 512, 1024, 4096)] + [(512, 512, 16384), (1024, 65, 1028)])
def test_sums_of_one_sign(K, cuda, shape, values):
    """What the tensor cores cut does not cancel there: sums come out low by 6 to 8.5e-8 of their size (2^-24 is 6e-8), whatever K.  The
    CUDA cores' error grows with K and is larger, but where they add eight or more short chains (1024 x 65 x 1028: 7.3 to 7.8e-8)."""
    assert gemm_plan(K, N.DT_F32, *shape)[2] == 2
    m, n, k = shape
    g = cuda.Generator(device="cuda").manual_seed(k)
    draw = {"uniform": lambda rows: cuda.rand(rows, k, generator=g, device="cuda"), "magnitudes": lambda rows: cuda.randn(rows, k, generator=g, device="cuda").abs(),
            # the largest products that are left out: all of one sign, 2^-24 of each
            "constant": lambda rows: cuda.full((rows, k), 1 + 2.0 ** -8 - 2.0 ** -17, device="cuda")}[values]
    a, b = draw(m), draw(n)
    want = a.double() @ b.double().T
    error = {dtype: float((multiply(K, cuda, a, b, dtype=dtype).double() - want).norm() / want.norm()) for dtype in (N.DT_F32, N.DT_F32_FFMA)}
    # roundings of up to 256 turns beside the cut: half a unit of a sum that grows evenly, as a random walk
    assert error[N.DT_F32] <= 1e-7 + 2.0 ** -25 * (k / 64) ** 0.5 / 3 ** 0.5
    if shape != (1024, 65, 1028):
        assert error[N.DT_F32] <= 1.01 * error[N.DT_F32_FFMA]


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
    assert worst(multiply(K, cuda, a, b, dtype=N.DT_F32_FFMA), a, b) <= k + 2
