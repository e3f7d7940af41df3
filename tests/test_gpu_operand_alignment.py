"""Operand kernels on pointers that are not aligned for their wide accesses: the same elements, and about the same time."""
import numpy as np
import pytest

from clpeak_b200 import native as N
from tests.gpu_util import assert_bits_equal, dev_empty, stream_ptr, sync, to_np

pytestmark = pytest.mark.gpu


def assert_about_as_fast(cuda, at_offset, offsets, factor, rounds=25, calls=4):
    """Best of many bursts on both sides, taken in turn: what else the machine does only adds time, and rarely to all of
    one side's."""
    best = {}
    for off in (0, *offsets):
        for _ in range(3):
            at_offset(off)
    for _ in range(rounds):
        for off in (0, *offsets):
            e0, e1 = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(calls):
                at_offset(off)
            e1.record()
            sync()
            best[off] = min(best.get(off, 1e9), e0.elapsed_time(e1) * 1e3 / calls)
    slow = {off: us for off, us in best.items() if us >= factor * best[0]}
    assert not slow, f"us at these offsets: {slow}; {best[0]:.1f} at none"


N_TIMED = 8192 * 4096              # two to three times the L2 in floats


@pytest.mark.parametrize("dist", [0, 1, 2])
@pytest.mark.parametrize("n", [3, 8, 13, 4100])
def test_fill_at_every_offset(K, orc, cuda, dist, n):
    want = orc.fill_f32(n, 31, dist, 0.5, 3.0)
    for offset in range(9):
        buf = cuda.full((n + offset + 8,), 77.0, dtype=cuda.float32, device="cuda")
        K.clpk_fill_f32(buf.data_ptr() + 4 * offset, n, 31, dist, 0.5, 3.0, stream_ptr())
        sync()
        got = to_np(buf)
        assert_bits_equal(got[offset:offset + n], want, "fill")
        assert np.all(got[:offset] == 77.0) and np.all(got[offset + n:] == 77.0), "the fill wrote outside its range"


@pytest.mark.parametrize("n", [5, 16, 29, 5000])
def test_fill_i8_at_every_offset(K, orc, cuda, n):
    want = orc.fill_i8(n, 9)
    for offset in range(17):
        buf = cuda.full((n + offset + 8,), 77, dtype=cuda.int8, device="cuda")
        K.clpk_fill_i8(buf.data_ptr() + offset, n, 9, stream_ptr())
        sync()
        got = to_np(buf)
        assert_bits_equal(got[offset:offset + n], want, "fill_i8")
        assert np.all(got[:offset] == 77) and np.all(got[offset + n:] == 77)


@pytest.mark.parametrize("n", [1, 6, 8, 15, 40, 32768, 32769, 70001])
def test_absmax_at_every_offset(K, orc, cuda, n):
    """The largest in the head, in the steps and at the very end, from every offset."""
    src = orc.fill_f32(n, 8, N.DIST_UNIFORM_PM1)
    buf = cuda.full((n + 32,), 50.0, dtype=cuda.float32, device="cuda")        # larger than all of the operand's own
    out = dev_empty(1, cuda.float32)
    for offset in range(9):
        for at in {0, min(5, n - 1), n // 2, n - 1}:
            x = src.copy()
            x[at] = -9.5
            buf.fill_(50.0)
            buf[offset:offset + n] = cuda.from_numpy(x).cuda()
            K.clpk_absmax_f32(out.data_ptr(), buf.data_ptr() + 4 * offset, n, stream_ptr())
            sync()
            assert float(out.item()) == 9.5, (offset, at)


# bits of an element; the source's offset decides the loads (32, 16 or 4 bytes), the destination's where the array is cut
@pytest.mark.parametrize("dtype,bits", [(N.DT_F16, 16), (N.DT_BF16, 16), (N.DT_E4M3, 8), (N.DT_E5M2, 8), (N.DT_I8, 8), (N.DT_TF32, 32),
                                        (N.DT_F64, 64), (N.DT_E2M1, 4)])
@pytest.mark.parametrize("n", [2, 8, 22, 2062])
def test_convert_at_every_pair_of_offsets(K, orc, cuda, dtype, bits, n):
    x = orc.fill_f32(n, 6, N.DIST_NORMAL, 0.0, 2.0)
    want = x.astype(np.float64) if dtype == N.DT_F64 else orc.convert_f32(x, dtype)
    want = np.ascontiguousarray(want).view(np.uint8).ravel()
    unit, size = max(bits // 8, 1), n * bits // 8
    src = cuda.empty(n + 16, dtype=cuda.float32, device="cuda")
    for src_offset in range(9):
        src.fill_(1e6)
        src[src_offset:src_offset + n] = cuda.from_numpy(x).cuda()
        for dst_offset in range(0, 32 // unit + 1):
            first = unit * dst_offset
            buf = cuda.full((first + size + 64,), 0x5A, dtype=cuda.uint8, device="cuda")
            K.clpk_convert_f32(buf.data_ptr() + first, src.data_ptr() + 4 * src_offset, n, dtype, stream_ptr())
            sync()
            got = to_np(buf)
            assert np.array_equal(got[first:first + size], want), (src_offset, dst_offset)
            assert np.all(got[:first] == 0x5A) and np.all(got[first + size:] == 0x5A), "the conversion wrote outside its range"


BLOCK = {N.DT_MXF4: 32, N.DT_MXF4_B64: 64, N.DT_NVF4: 16, N.DT_NVF4_B32: 32}


@pytest.mark.parametrize("dtype", list(BLOCK))
@pytest.mark.parametrize("rows,cols", [(1, 64), (7, 192), (33, 320)])
def test_quantize_at_every_pair_of_offsets(K, orc, cuda, dtype, rows, cols):
    n, ts = rows * cols, 1.0 if dtype in (N.DT_MXF4, N.DT_MXF4_B64) else float(np.float32(2.5e-4))
    x = orc.fill_f32(n, 6, N.DIST_NORMAL).reshape(rows, cols)
    x[0, :64] = 0.0                                                 # a warp that takes the divisions
    want_packed, want_scales = orc.quantize_fp4(x, dtype, ts)
    src, scales = cuda.empty(n + 16, dtype=cuda.float32, device="cuda"), dev_empty(n // BLOCK[dtype], cuda.uint8)
    for src_offset in range(9):
        src.fill_(1e6)
        src[src_offset:src_offset + n] = cuda.from_numpy(x.ravel()).cuda()
        for first in range(9):
            packed = cuda.full((first + n // 2 + 16,), 0x5A, dtype=cuda.uint8, device="cuda")
            K.clpk_quantize_fp4(packed.data_ptr() + first, scales.data_ptr(), src.data_ptr() + 4 * src_offset, rows, cols, dtype, ts, stream_ptr())
            sync()
            got = to_np(packed)
            assert_bits_equal(got[first:first + n // 2], want_packed.ravel(), "fp4 codes")
            assert_bits_equal(to_np(scales), want_scales.ravel(), "fp4 scales")
            assert np.all(got[:first] == 0x5A) and np.all(got[first + n // 2:] == 0x5A)


# cut at the first aligned address it is the same work; one element at a time took 1.8 to 4 times as long
@pytest.mark.parametrize("dist", [0, 1, 2])
def test_fill_is_as_fast_from_any_offset(K, cuda, dist):
    d = dev_empty(N_TIMED + 8, cuda.float32)
    assert_about_as_fast(cuda, lambda off: K.clpk_fill_f32(d.data_ptr() + 4 * off, N_TIMED, 3, dist, 0.0, 1.0, stream_ptr()), (1, 4), 1.3)


def test_fill_i8_is_as_fast_from_any_offset(K, cuda):
    d = dev_empty(N_TIMED + 16, cuda.int8)
    assert_about_as_fast(cuda, lambda off: K.clpk_fill_i8(d.data_ptr() + off, N_TIMED, 3, stream_ptr()), (1, 8), 1.3)


# a small array is one CTA's, which took five times the time (a burst of launches as fast as the host issues them, so with
# more room than the others); a large one took three times
@pytest.mark.parametrize("n,factor", [(32768, 2.5), (N_TIMED, 1.3)])
def test_absmax_is_as_fast_from_any_offset(K, cuda, n, factor):
    src, out = dev_empty(n + 8, cuda.float32), dev_empty(1, cuda.float32)
    src.zero_()
    assert_about_as_fast(cuda, lambda off: K.clpk_absmax_f32(out.data_ptr(), src.data_ptr() + 4 * off, n, stream_ptr()), (1, 4), factor,
                         calls=40 if n < N_TIMED else 4)


# the loads are narrower where source and destination are not aligned at once; one element at a time took 3 to 5 times as long
@pytest.mark.parametrize("dtype,bits", [(N.DT_BF16, 16), (N.DT_E4M3, 8), (N.DT_TF32, 32), (N.DT_F64, 64), (N.DT_E2M1, 4)])
def test_convert_is_nearly_as_fast_from_any_offset(K, cuda, dtype, bits):
    src, dst = dev_empty(N_TIMED + 16, cuda.float32), dev_empty(N_TIMED * bits // 8 + 64, cuda.uint8)
    src.zero_()
    unit = max(bits // 8, 1)

    def convert(offsets):
        src_offset, dst_offset = offsets or (0, 0)
        K.clpk_convert_f32(dst.data_ptr() + unit * dst_offset, src.data_ptr() + 4 * src_offset, N_TIMED, dtype, stream_ptr())

    assert_about_as_fast(cuda, convert, ((1, 0), (4, 0), (0, 1), (3, 1)), 1.6)


# narrower loads and stores (2.5 times at most); one thread per scale block, every quotient computed twice, took 5 to 12 times as long
@pytest.mark.parametrize("dtype", list(BLOCK))
def test_quantize_is_nearly_as_fast_from_any_offset(K, cuda, dtype):
    src, packed, scales = dev_empty(N_TIMED + 16, cuda.float32), dev_empty(N_TIMED // 2 + 16, cuda.uint8), dev_empty(N_TIMED // 16, cuda.uint8)
    K.clpk_fill_f32(src.data_ptr(), N_TIMED + 16, 3, N.DIST_NORMAL, 0.0, 0.02, stream_ptr())

    def quantize(offsets):
        src_offset, dst_offset = offsets or (0, 0)
        K.clpk_quantize_fp4(packed.data_ptr() + dst_offset, scales.data_ptr(), src.data_ptr() + 4 * src_offset, 4096, N_TIMED // 4096, dtype, 2e-5,
                            stream_ptr())

    assert_about_as_fast(cuda, quantize, ((1, 0), (4, 0), (0, 4), (0, 1), (3, 1)), 3.5)
