"""fp32 / fp64 GEMM shapes that take the small tiles and the split of K: every element of C against the fp64 product."""
import ctypes as C

import numpy as np
import pytest

from clpeak_b200 import native as N
from tests.gpu_util import dev_empty, gemm_plan, stream_ptr, sync

pytestmark = pytest.mark.gpu


def operand(K, cuda, dtype, rows, k, seed):
    f = dev_empty(rows * k, cuda.float32)
    K.clpk_fill_f32(f.data_ptr(), rows * k, seed, N.DIST_NORMAL, 0.0, 0.02, stream_ptr())
    if dtype != N.DT_F64:
        return f
    d = dev_empty(rows * k, cuda.float64)
    K.clpk_convert_f32(d.data_ptr(), f.data_ptr(), rows * k, N.DT_F64, stream_ptr())
    return d


# fewer k blocks than groups and ranks could take; ranges and groups of unequal length; ragged tiles in both directions;
# N odd (no vector store); one and several CTAs per SM
@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (33, 65, 20), (64, 64, 16384), (129, 131, 36), (131, 102, 7688), (201, 73, 2828), (863, 251, 2456),
                                   (1315, 363, 956), (440, 434, 520), (64, 868, 1036), (719, 366, 688), (459, 349, 4636), (3720, 110, 596),
                                   (2254, 496, 464), (1024, 1024, 512), (97, 106, 5732), (719, 368, 6380), (64, 64, 4100)])
@pytest.mark.parametrize("dtype", [N.DT_F32, N.DT_F32_FFMA, N.DT_F64])
def test_every_element(K, cuda, dtype, m, n, k):
    check_every_element(K, cuda, dtype, m, n, k)


# (tile, K ranges, twice the K groups) and a shape that takes them
PLANS = [(N.DT_F32, (0, 1, 0), (1135, 1699, 36)), (N.DT_F32, (64, 1, 0), (52, 36, 64)), (N.DT_F32, (64, 2, 0), (42, 58, 128)),
         (N.DT_F32, (64, 4, 0), (127, 33, 256)), (N.DT_F32, (64, 8, 0), (94, 36, 512)), (N.DT_F32, (64, 8, 1), (64, 64, 16384)),
         (N.DT_F32_FFMA, (0, 1, 0), (1135, 1699, 36)), (N.DT_F32_FFMA, (0, 1, 0), (2048, 2048, 512)), (N.DT_F32_FFMA, (0, 1, 0), (2047, 2050, 516)),
         (N.DT_F32_FFMA, (64, 1, 0), (52, 36, 64)), (N.DT_F32_FFMA, (64, 1, 0), (4095, 366, 2456)), (N.DT_F32_FFMA, (64, 1, 1), (459, 863, 520)),
         (N.DT_F32_FFMA, (64, 2, 0), (42, 58, 128)), (N.DT_F32_FFMA, (64, 2, 1), (719, 366, 2456)), (N.DT_F32_FFMA, (64, 4, 0), (127, 33, 256)),
         (N.DT_F32_FFMA, (64, 4, 1), (64, 2048, 2456)), (N.DT_F32_FFMA, (64, 8, 0), (94, 36, 512)), (N.DT_F32_FFMA, (64, 8, 1), (64, 64, 16384)),
         (N.DT_F64, (32, 1, 0), (47, 70, 64)), (N.DT_F64, (32, 1, 1), (2287, 33, 512)), (N.DT_F64, (32, 4, 0), (68, 61, 512)),
         (N.DT_F64, (32, 8, 1), (64, 64, 16384)), (N.DT_F64, (64, 8, 0), (130, 197, 512))]


@pytest.mark.parametrize("dtype,plan,shape", PLANS)
def test_every_plan(K, cuda, dtype, plan, shape):
    assert gemm_plan(K, dtype, *shape) == plan
    check_every_element(K, cuda, dtype, *shape)


# short fp64 sums: shapes that 32-wide tiles made 1.1 to 2.5 times slower take the kernel with K whole, an odd N also in more CTAs than
# run at once, and shapes that small tiles serve best keep them
@pytest.mark.parametrize("tile,shape", [(0, (4153, 558, 6)), (0, (2888, 782, 2)), (0, (12879, 166, 12)), (0, (11657, 120, 14)), (0, (394, 15109, 38)),
                                        (0, (963, 955, 248)), (0, (12127, 1916, 10)), (0, (1674, 807, 4)), (32, (863, 251, 248)), (32, (64, 64, 128)),
                                        (0, (661, 6775, 24)), (32, (1481, 215, 40))])
def test_short_fp64_sums(K, cuda, tile, shape):
    assert gemm_plan(K, N.DT_F64, *shape)[0] == tile
    check_every_element(K, cuda, N.DT_F64, *shape)


# fp64 with K whole in 64 x 64 tiles: whole tiles, ragged ones with an even N and with an odd one (whose C goes through shared memory),
# sums of one block to more than the ring holds and with every remainder of a block's pieces
WHOLE = [(m, n, k) for m, n in ((640, 704), (641, 702), (639, 705), (7000, 2), (6401, 1), (63, 6402), (65, 6465)) for k in (2, 16, 18, 32, 46, 48, 50, 64)]
WHOLE += [(641, 702, 368), (639, 705, 368), (2048, 2048, 464), (2047, 2046, 466), (2046, 2047, 1042)]


@pytest.mark.parametrize("m,n,k", WHOLE)
def test_whole_fp64_tiles(K, cuda, m, n, k):
    assert gemm_plan(K, N.DT_F64, m, n, k) == (0, 1, 0)
    check_every_element(K, cuda, N.DT_F64, m, n, k)


# beside them, the same sizes with K split or in 32-wide tiles
@pytest.mark.parametrize("plan,shape", [((64, 2, 0), (641, 702, 464)), ((64, 2, 0), (639, 705, 464)), ((64, 2, 0), (65, 6465, 368)), ((32, 1, 0), (640, 704, 464)),
                                        ((32, 1, 0), (7000, 2, 96)), ((32, 2, 0), (6401, 1, 464)), ((32, 1, 0), (63, 6402, 464))])
def test_fp64_beside_whole_tiles(K, cuda, plan, shape):
    assert gemm_plan(K, N.DT_F64, *shape) == plan
    check_every_element(K, cuda, N.DT_F64, *shape)


def check_every_element(K, cuda, dtype, m, n, k):
    a, b = operand(K, cuda, dtype, m, k, 40), operand(K, cuda, dtype, n, k, 41)
    alpha, results = 0.75, []
    for _ in range(2):
        c = cuda.full((m * n + 1024,), float("nan"), dtype=a.dtype, device="cuda")
        status = cuda.full((1,), 7, dtype=cuda.int32, device="cuda")
        args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), alpha=alpha,
                          d_status=status.data_ptr())
        K.clpk_gemm(C.byref(args), stream_ptr())
        sync()
        assert int(status.item()) == 0
        assert bool(cuda.isnan(c[m * n:]).all()), "the kernel wrote beyond C"
        results.append(c[:m * n])
    assert bool((results[0] == results[1]).all()), "partial sums are added in a fixed order: the same bits every time"
    fa, fb = a.double().view(m, k), b.double().view(n, k)
    want, s_abs = alpha * (fa @ fb.T), alpha * (fa.abs() @ fb.abs().T)
    # K roundings of the accumulator and one of alpha; fp64: the reference sum rounds as often
    u = 2.0 ** -52 if dtype == N.DT_F64 else 2.0 ** -24
    worst = float(((results[0].double().view(m, n) - want).abs() / ((k + 2) * u * s_abs + 1e-300)).max())
    assert worst <= 1.0, f"worst error over all of C is {worst:.3g}x the stated tolerance"


@pytest.mark.parametrize("dtype", [N.DT_F32, N.DT_F32_FFMA])
def test_nan_and_infinity_stay_in_their_rows_and_columns(K, cuda, dtype):
    """Zero fill beyond K and beyond the operands must not meet them: 0 * inf would spread."""
    m, n, k = 70, 66, 1028
    a, b = operand(K, cuda, N.DT_F32, m, k, 1), operand(K, cuda, N.DT_F32, n, k, 2)
    a[3 * k + 5], b[7 * k + k - 1] = float("inf"), float("nan")
    c, status = dev_empty(m * n, cuda.float32), dev_empty(1, cuda.int32)
    args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), alpha=1.0, d_status=status.data_ptr())
    K.clpk_gemm(C.byref(args), stream_ptr())
    sync()
    bad = ~np.isfinite(c.view(m, n).cpu().numpy())
    assert bad[3].all() and bad[:, 7].all() and bad.sum() == m + n - 1
