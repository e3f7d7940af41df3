"""Block-scaled GEMM: the arrangement of the scale factors and the shapes where its tiles can go wrong."""
import ctypes as C

import pytest

from clpeak_b200 import native as N
from tests.gpu_util import dev_empty, stream_ptr, sync
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
