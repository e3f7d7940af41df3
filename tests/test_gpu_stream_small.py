"""Stream kernels where their launches change shape (slots owned or shared, tiles dealt or claimed) and under each other's
tails: every kernel may start before the one in front of it in the stream has ended."""
import ctypes as C

import numpy as np
import pytest

from clpeak_b200 import native as N
from tests.gpu_util import dev_empty, stream_ptr, sync

pytestmark = pytest.mark.gpu

TILE, SLOTS, ROUNDS = 8192, 4096, 8          # of the 256-bit read kernel


def checksum(parts):
    return int(np.bitwise_xor.reduce(parts.cpu().numpy().view(np.uint32)))


@pytest.mark.parametrize("n_bytes", [TILE * (SLOTS - 1) + 16, TILE * SLOTS, TILE * SLOTS + TILE + 48, TILE * SLOTS * ROUNDS,
                                     TILE * (SLOTS * ROUNDS + 1) + 16])
def test_wide_read_at_its_edges(K, cuda, n_bytes):
    n = n_bytes // 4
    src = dev_empty(n, cuda.float32)
    K.clpk_fill_f32(src.data_ptr(), n, 3, N.DIST_UNIFORM01, 0.0, 1.0, stream_ptr())
    parts = cuda.full((SLOTS,), 0x5A5A5A5A, dtype=cuda.int32, device="cuda")       # every slot is written by the call
    want = int(np.bitwise_xor.reduce(src.cpu().numpy().view(np.uint32)))
    for _ in range(2):
        K.clpk_stream_read(N.STREAM_WIDE, src.data_ptr(), n_bytes, parts.data_ptr(), stream_ptr())
        assert checksum(parts) == want


@pytest.mark.parametrize("variant", list(N.STREAM_VARIANTS))
@pytest.mark.parametrize("n", [4, 2052, 1 << 16, (1 << 20) + 12, 148 * 8192 * 4, 148 * 8192 * 4 + 8192, 1 << 23])
def test_dependent_kernels_back_to_back(K, cuda, variant, n):
    """b <- copy of (b + 1.5 c), eight times, with a read of every intermediate: each kernel needs all of the one before."""
    a, b, c = (dev_empty(n, cuda.float32) for _ in range(3))
    for t, seed in ((b, 1), (c, 2)):
        K.clpk_fill_f32(t.data_ptr(), n, seed, N.DIST_UNIFORM01, 0.0, 1.0, stream_ptr())
    want_b, one = b.clone(), c.clone()
    grid = C.c_int(0)
    K.clpk_stream_read_grid(variant, C.byref(grid))
    parts = [cuda.full((grid.value,), -1, dtype=cuda.int32, device="cuda") for _ in range(8)]
    sync()
    for p in parts:
        K.clpk_stream_triad(variant, a.data_ptr(), b.data_ptr(), c.data_ptr(), 1.5, n, stream_ptr())
        K.clpk_stream_copy(variant, b.data_ptr(), a.data_ptr(), 4 * n, stream_ptr())
        K.clpk_stream_read(variant, b.data_ptr(), 4 * n, p.data_ptr(), stream_ptr())
    status = C.c_uint32(0)
    K.clpk_stream_status(C.byref(status), stream_ptr())
    for p in parts:
        want_b = want_b + one * 1.5
        assert checksum(p) == int(np.bitwise_xor.reduce(want_b.cpu().numpy().view(np.uint32)))
    assert bool((b == want_b).all())


def test_the_launches_can_be_captured(K, cuda):
    """Operands, a small GEMM with scales to arrange and a stream pass as one graph, replayed on new contents."""
    rows = cols = 256
    n = rows * cols
    f, top = dev_empty(n, cuda.float32), dev_empty(1, cuda.float32)
    q, sf, c = dev_empty(n // 2, cuda.uint8), dev_empty(n // 16, cuda.uint8), dev_empty(n, cuda.bfloat16)
    ws, st, out = dev_empty(2 * n // 16, cuda.uint8), dev_empty(1, cuda.int32), dev_empty(n, cuda.float32)
    parts = dev_empty(SLOTS, cuda.int32)
    single = N.GemmArgs(dtype=N.DT_F32, m=rows, n=rows, k=cols, d_a=f.data_ptr(), d_b=f.data_ptr(), d_c=out.data_ptr(), alpha=1.0, d_status=st.data_ptr())
    scaled = N.GemmArgs(dtype=N.DT_NVF4, m=rows, n=rows, k=cols, d_a=q.data_ptr(), d_b=q.data_ptr(), d_c=c.data_ptr(), d_sfa=sf.data_ptr(),
                        d_sfb=sf.data_ptr(), alpha=1.0, d_workspace=ws.data_ptr(), workspace_bytes=ws.numel(), d_status=st.data_ptr())

    def run(s):
        K.clpk_fill_f32(f.data_ptr(), n, 17, N.DIST_NORMAL, 0.0, 0.02, s)
        K.clpk_absmax_f32(top.data_ptr(), f.data_ptr(), n, s)
        K.clpk_quantize_fp4(q.data_ptr(), sf.data_ptr(), f.data_ptr(), rows, cols, N.DT_NVF4, 3e-5, s)
        K.clpk_gemm(C.byref(scaled), s)
        K.clpk_gemm(C.byref(single), s)
        K.clpk_stream_read(N.STREAM_WIDE, out.data_ptr(), 4 * n, parts.data_ptr(), s)

    run(stream_ptr())
    sync()
    want = [t.clone() for t in (f, top, q, sf, c, out, parts)]
    stream = cuda.cuda.Stream()
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph, stream=stream):
        run(stream.cuda_stream)
    for _ in range(3):
        for t in (f, top, q, sf, c, out, parts):
            t.zero_()
        graph.replay()
        sync()
        assert all(bool((t == w).all()) for t, w in zip((f, top, q, sf, c, out, parts), want))
