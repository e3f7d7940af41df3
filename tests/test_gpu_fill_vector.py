"""The eight-at-a-time operand kernels where they can go wrong: lengths around a step, pointers that are not aligned for
the wide accesses, special values, and the shared-divisor quotients against the oracle's IEEE divisions."""
import numpy as np
import pytest

from clpeak_b200 import native as N
from tests.gpu_util import assert_bits_equal, dev_empty, stream_ptr, sync, to_np

pytestmark = pytest.mark.gpu


def at_offset(cuda, a: np.ndarray, offset: int):
    """A device copy of `a` that starts `offset` elements into an aligned buffer (and the buffer, which must live)."""
    t = cuda.from_numpy(np.ascontiguousarray(a))
    buf = cuda.empty(a.size + offset + 16, dtype=t.dtype, device="cuda")
    buf[offset:offset + a.size] = t.cuda()
    return buf, buf.data_ptr() + offset * a.itemsize


@pytest.mark.parametrize("dist", [0, 1, 2])
@pytest.mark.parametrize("n,offset", [(7, 0), (8, 0), (9, 0), (4099, 0), (4099, 1), (64, 4)])
def test_fill_lengths_and_alignment(K, orc, cuda, dist, n, offset):
    buf = cuda.full((n + offset + 8,), 77.0, dtype=cuda.float32, device="cuda")
    K.clpk_fill_f32(buf.data_ptr() + 4 * offset, n, 31, dist, 0.5, 3.0, stream_ptr())
    sync()
    got = to_np(buf)
    assert_bits_equal(got[offset:offset + n], orc.fill_f32(n, 31, dist, 0.5, 3.0), "fill")
    assert np.all(got[:offset] == 77.0) and np.all(got[offset + n:] == 77.0), "the fill wrote outside its range"


def test_normal_deviates_over_their_whole_range(K, orc, cuda):
    """2^25 deviates take 98 % of the 2^23 radii and 87 % of the 2^24 angles there are."""
    n = 1 << 25
    d = dev_empty(n, cuda.float32)
    K.clpk_fill_f32(d.data_ptr(), n, 5, N.DIST_NORMAL, 0.0, 1.0, stream_ptr())
    sync()
    assert_bits_equal(to_np(d), orc.fill_f32(n, 5, N.DIST_NORMAL), "normal deviates")


@pytest.mark.parametrize("seed,at", [(1884646, 641), (7288700, 535), (6692669, 556), (4960922, 3392)])
@pytest.mark.parametrize("offset", [0, 5])
def test_fill_where_a_carry_reaches_bit_30(K, orc, cuda, seed, at, offset):
    """Consecutive elements share what stands above bit 30 of the generator's first step, until element `at` of these seeds:
    in the middle of a step, its last element, and its first one."""
    mask = (1 << 64) - 1

    def mix(z):
        z = (z + 0x9E3779B97F4A7C15) & mask
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        return z ^ (z >> 31)
    assert (mix(seed) + 0x9E3779B97F4A7C15 + at) % (1 << 30) == 0
    n = at + 300
    d, q = dev_empty(n + 8, cuda.float32), dev_empty(n + 8, cuda.int8)
    for dist in (N.DIST_UNIFORM01, N.DIST_UNIFORM_PM1, N.DIST_NORMAL):
        K.clpk_fill_f32(d.data_ptr() + 4 * offset, n, seed, dist, 0.25, 2.0, stream_ptr())
        sync()
        assert_bits_equal(to_np(d)[offset:offset + n], orc.fill_f32(n, seed, dist, 0.25, 2.0), "fill")
    K.clpk_fill_i8(q.data_ptr() + offset, n, seed, stream_ptr())
    sync()
    assert_bits_equal(to_np(q)[offset:offset + n], orc.fill_i8(n, seed), "fill_i8")


@pytest.mark.parametrize("n", [(1 << 22) - 8, 1 << 22, (1 << 22) + 1031, (1 << 22) + 2048])
def test_fill_with_one_and_two_steps_per_thread(K, orc, cuda, n):
    d = cuda.full((n + 8,), 77.0, dtype=cuda.float32, device="cuda")
    for dist in (N.DIST_UNIFORM01, N.DIST_NORMAL):
        K.clpk_fill_f32(d.data_ptr(), n, 3, dist, 0.0, 1.0, stream_ptr())
        sync()
        got = to_np(d)
        assert_bits_equal(got[:n], orc.fill_f32(n, 3, dist), "fill")
        assert np.all(got[n:] == 77.0)


@pytest.mark.parametrize("n,offset", [(15, 0), (16, 0), (33, 0), (5000, 3)])
def test_fill_i8_lengths_and_alignment(K, orc, cuda, n, offset):
    buf = cuda.full((n + offset + 8,), 77, dtype=cuda.int8, device="cuda")
    K.clpk_fill_i8(buf.data_ptr() + offset, n, 9, stream_ptr())
    sync()
    got = to_np(buf)
    assert_bits_equal(got[offset:offset + n], orc.fill_i8(n, 9), "fill_i8")
    assert np.all(got[:offset] == 77) and np.all(got[offset + n:] == 77)


def saturate_infinities(codes: np.ndarray, x: np.ndarray):
    """e2m1 codes of the oracle, with infinities at the largest magnitude: its nearest-value search has no answer there."""
    codes, x = codes.ravel(), x.ravel()
    for i in np.flatnonzero(np.isinf(x)):
        shift = 4 * (i & 1)
        codes[i // 2] = (codes[i // 2] & (0xF0 >> shift)) | ((15 if x[i] < 0 else 7) << shift)
    return codes


def special_values(orc, n, scale):
    src = orc.fill_f32(n, 6, N.DIST_NORMAL, 0.0, scale)
    odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-42, -1e-42, 3.4e38, -3.4e38, 1e-30], dtype=np.float32)
    src[: odd.size] = odd
    src[-3:] = [np.inf, -0.0, 2.5]
    return src


@pytest.mark.parametrize("dtype,unit", [(N.DT_F16, 2), (N.DT_BF16, 2), (N.DT_E4M3, 1), (N.DT_E5M2, 1), (N.DT_I8, 1), (N.DT_TF32, 4),
                                        (N.DT_F64, 8), (N.DT_E2M1, 1)])
@pytest.mark.parametrize("n,src_offset,dst_offset", [(40, 0, 0), (1046, 0, 0), (1046, 1, 0), (1046, 0, 1)])
def test_convert_lengths_and_alignment(K, cuda, orc, dtype, unit, n, src_offset, dst_offset):
    src = special_values(orc, n, 2.0)
    if dtype in (N.DT_E4M3, N.DT_E5M2, N.DT_I8, N.DT_E2M1):
        src[np.isnan(src)] = 1.0                                    # a NaN's code is not part of these formats' contract
    if dtype == N.DT_E2M1:
        src[np.isfinite(src) & (np.abs(src) > 1e30)] = -1e9         # the oracle's distances in fp64 all round to one value there
    out_bytes = n // 2 if dtype == N.DT_E2M1 else n * unit
    keep, p_src = at_offset(cuda, src, src_offset)
    buf = cuda.full((out_bytes + unit * dst_offset + 32,), 0x5A, dtype=cuda.uint8, device="cuda")
    K.clpk_convert_f32(buf.data_ptr() + unit * dst_offset, p_src, n, dtype, stream_ptr())
    sync()
    got, first = to_np(buf), unit * dst_offset
    body = np.ascontiguousarray(got[first:first + out_bytes])
    if dtype == N.DT_F64:
        want = src.astype(np.float64)
        assert np.array_equal(body.view(np.float64), want, equal_nan=True)
    else:
        want = np.ascontiguousarray(orc.convert_f32(src, dtype)).view(np.uint8).ravel()
        if dtype == N.DT_E2M1:
            want = saturate_infinities(want, src)
        nan = np.repeat(np.isnan(src), unit) if dtype != N.DT_E2M1 else np.zeros(out_bytes, bool)
        assert np.array_equal(body[~nan], want[~nan])
    assert np.all(got[:first] == 0x5A) and np.all(got[first + out_bytes:] == 0x5A)


@pytest.mark.parametrize("n,offset", [(1, 0), (7, 0), (4097, 1), (32768, 0), (32769, 0), (1 << 20, 0), ((1 << 22) + 5, 2)])
def test_absmax_lengths(K, cuda, orc, n, offset):
    src = orc.fill_f32(n, 8, N.DIST_NORMAL)
    src[n // 2] = -9.5
    src[-1] = np.nan if n > 1 else -9.5                             # ignored, as fmaxf does
    keep, p_src = at_offset(cuda, src, offset)
    out = cuda.full((1,), 1e9, dtype=cuda.float32, device="cuda")
    K.clpk_absmax_f32(out.data_ptr(), p_src, n, stream_ptr())
    sync()
    assert float(out.item()) == 9.5


@pytest.mark.parametrize("n,offset", [(25 << 20, 0), ((25 << 20) + 1, 0), ((25 << 20) + 4099, 3)])
def test_absmax_of_arrays_beyond_the_cache(K, cuda, n, offset):
    """From 100 MiB on the array is read from its end, by a kernel of its own: the largest magnitude is found wherever it lies."""
    src = cuda.zeros(n + offset, dtype=cuda.float32, device="cuda")
    K.clpk_fill_f32(src.data_ptr(), n + offset, 8, N.DIST_UNIFORM_PM1, 0.0, 1.0, stream_ptr())
    out = cuda.empty(1, dtype=cuda.float32, device="cuda")
    for at in (None, 0, 1, 8, n // 2, n - 8193, n - 9, n - 2, n - 1):
        if at is not None:
            src[offset + at] = -2.0 - at / n
        want = float(src[offset:].abs().max())
        out.fill_(1e9)
        K.clpk_absmax_f32(out.data_ptr(), src.data_ptr() + 4 * offset, n, stream_ptr())
        assert float(out.item()) == want
        if at is not None:
            src[offset + at] = float("nan")                         # ignored, as fmaxf does
            K.clpk_absmax_f32(out.data_ptr(), src.data_ptr() + 4 * offset, n, stream_ptr())
            assert float(out.item()) < want
            src[offset + at] = 0.0


BLOCK = {N.DT_MXF4: 32, N.DT_MXF4_B64: 64, N.DT_NVF4: 16, N.DT_NVF4_B32: 32}


@pytest.mark.parametrize("dtype", list(BLOCK))
@pytest.mark.parametrize("ts,scale", [(1.0, 1.0), (2.9e-5, 0.02), (0.3337, 40.0), (1e-30, 1e-28), (1.7e25, 3e27), (1e-4, 1e-30)])
def test_quantize_ties_and_special_blocks(K, orc, cuda, dtype, ts, scale):
    rows, cols = 64, 1024
    if dtype in (N.DT_MXF4, N.DT_MXF4_B64):
        ts = 1.0
    x = orc.fill_f32(rows * cols, 12, N.DIST_NORMAL, 0.0, scale)
    ties = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0], dtype=np.float32) * np.float32(ts)
    x = x.reshape(rows, cols)
    for r in range(1, 9):                                           # values on and beside the ties, under several scales
        s = np.float32(2.0 ** (r - 4) * (1 + r / 8))
        x[r, ::2] = np.resize(ties * s, cols // 2)
        x[r, 1::2] = np.nextafter(np.resize(ties * s, cols // 2), np.float32(np.inf if r & 1 else -np.inf))
    x[9] = 0.0
    x[10, ::3] = -0.0
    if dtype in (N.DT_NVF4, N.DT_NVF4_B32):                         # an infinite block has no ue8m0 scale
        x[11, 5], x[11, 100] = np.inf, -np.inf
    x[11, 200], x[11, 300] = 1e-42, -1e-42
    x[12, :16] = np.float32(1e-25)
    x = np.ascontiguousarray(x)
    want_packed, want_scales = orc.quantize_fp4(x, dtype, float(np.float32(ts)))
    want_packed = saturate_infinities(want_packed, x)
    for src_offset, dst_offset in ((0, 0), (1, 0), (0, 1)):         # aligned; the source, the codes not
        keep, p_src = at_offset(cuda, x.ravel(), src_offset)
        packed = dev_empty(rows * cols // 2 + 8, cuda.uint8)
        scales = dev_empty(rows * cols // BLOCK[dtype], cuda.uint8)
        K.clpk_quantize_fp4(packed.data_ptr() + dst_offset, scales.data_ptr(), p_src, rows, cols, dtype, float(np.float32(ts)), stream_ptr())
        sync()
        assert_bits_equal(to_np(scales), want_scales.ravel(), "fp4 scales")
        assert_bits_equal(to_np(packed)[dst_offset:dst_offset + rows * cols // 2], want_packed.ravel(), "fp4 codes")


@pytest.mark.parametrize("dtype", [N.DT_NVF4, N.DT_MXF4])
def test_quantize_generated_operands(K, orc, cuda, dtype):
    """Four million ordinary values under the usual tensor scale: every rounding of the shared-divisor quotients."""
    rows, cols = 2048, 2048
    x = orc.fill_f32(rows * cols, 40, N.DIST_NORMAL, 0.0, 0.02)
    ts = float(np.float32(np.abs(x).max()) / np.float32(6.0 * 448.0)) if dtype == N.DT_NVF4 else 1.0
    want_packed, want_scales = orc.quantize_fp4(x.reshape(rows, cols), dtype, ts)
    src = cuda.from_numpy(x).cuda()
    packed, scales = dev_empty(rows * cols // 2, cuda.uint8), dev_empty(rows * cols // BLOCK[dtype], cuda.uint8)
    K.clpk_quantize_fp4(packed.data_ptr(), scales.data_ptr(), src.data_ptr(), rows, cols, dtype, ts, stream_ptr())
    sync()
    assert_bits_equal(to_np(scales), want_scales.ravel(), "fp4 scales")
    assert_bits_equal(to_np(packed), want_packed.ravel(), "fp4 codes")


@pytest.mark.parametrize("rows,cols", [(25600, 1024), (409, 65600)])
@pytest.mark.parametrize("dtype", list(BLOCK))
def test_quantize_operands_beyond_the_cache(K, orc, cuda, dtype, rows, cols):
    """From 100 MiB on kernels of their own read the source as lines that leave the cache first, the MX kinds from its end."""
    x = orc.fill_f32(rows * cols, 40, N.DIST_NORMAL, 0.0, 0.02)
    ts = float(np.float32(np.abs(x).max()) / np.float32(6.0 * 448.0)) if dtype in (N.DT_NVF4, N.DT_NVF4_B32) else 1.0
    x[rows * cols - 70:rows * cols - 3], x[:64:3], x[4096:4160] = 0.0, -0.0, np.float32(1e-42)
    want_packed, want_scales = orc.quantize_fp4(x.reshape(rows, cols), dtype, ts)
    src = cuda.from_numpy(x).cuda()
    packed, scales = dev_empty(rows * cols // 2, cuda.uint8), dev_empty(rows * cols // BLOCK[dtype], cuda.uint8)
    K.clpk_quantize_fp4(packed.data_ptr(), scales.data_ptr(), src.data_ptr(), rows, cols, dtype, ts, stream_ptr())
    sync()
    assert_bits_equal(to_np(scales), want_scales.ravel(), "fp4 scales")
    assert_bits_equal(to_np(packed), want_packed.ravel(), "fp4 codes")


def test_operand_kernels_under_each_others_tails(K, orc, cuda):
    """fill -> absmax -> quantise -> fill again into the same buffer, back to back: each kernel may start before the one in
    front of it has ended, and has to wait for it before it reads or overwrites its data."""
    rows, cols = 512, 2048
    n = rows * cols
    f, top = dev_empty(n, cuda.float32), dev_empty(16, cuda.float32)
    packed = [dev_empty(n // 2, cuda.uint8) for _ in range(8)]
    scales = [dev_empty(n // 16, cuda.uint8) for _ in range(8)]
    halves = [dev_empty(n, cuda.bfloat16) for _ in range(8)]
    for i in range(8):
        K.clpk_fill_f32(f.data_ptr(), n, 60 + i, N.DIST_NORMAL, 0.0, 0.02, stream_ptr())
        K.clpk_absmax_f32(top.data_ptr() + 4 * i, f.data_ptr(), n, stream_ptr())
        K.clpk_quantize_fp4(packed[i].data_ptr(), scales[i].data_ptr(), f.data_ptr(), rows, cols, N.DT_NVF4, 4e-5, stream_ptr())
        K.clpk_convert_f32(halves[i].data_ptr(), f.data_ptr(), n, N.DT_BF16, stream_ptr())
    sync()
    for i in range(8):
        want = orc.fill_f32(n, 60 + i, N.DIST_NORMAL, 0.0, 0.02)
        assert float(top[i].item()) == float(np.abs(want).max())
        want_packed, want_scales = orc.quantize_fp4(want.reshape(rows, cols), N.DT_NVF4, float(np.float32(4e-5)))
        assert_bits_equal(to_np(packed[i]), want_packed.ravel(), "fp4 codes")
        assert_bits_equal(to_np(scales[i]), want_scales.ravel(), "fp4 scales")
        assert_bits_equal(to_np(halves[i].view(cuda.int16)), orc.convert_f32(want, N.DT_BF16), "bf16")
