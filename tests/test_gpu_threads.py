"""Calls from several host threads at once, each on a stream of its own: nothing that belongs to a kernel as a whole may
depend on the shape of one call."""
import ctypes as C
import threading

import pytest

from clpeak_b200 import native as N
from tests.gpu_util import gemm_plan, sync

pytestmark = pytest.mark.gpu


# pairs of shapes that take the same kernel and ask for different amounts of shared memory, because one gives an SM
# one CTA and the other two: 64 x 64 tiles in fp32, 32 x 32 and 64 x 64 tiles in fp64
@pytest.mark.parametrize("dtype,one,two", [(N.DT_F32_FFMA, (52, 36, 64), (2479, 194, 64)), (N.DT_F32, (52, 36, 64), (2479, 194, 64)), (N.DT_F64, (47, 70, 64), (41, 2373, 64)),
                                           (N.DT_F64, (130, 197, 512), (1344, 33, 512))])
def test_gemms_of_different_shapes_from_two_threads(K, cuda, dtype, one, two):
    if dtype == N.DT_F32_FFMA:
        assert gemm_plan(K, dtype, *one) == gemm_plan(K, dtype, *two) == (64, 1, 0)
    real = cuda.float64 if dtype == N.DT_F64 else cuda.float32
    start, refused, outputs = threading.Barrier(2), [], []

    def work(shape):
        m, n, k = shape
        cuda.cuda.set_device(0)
        stream = cuda.cuda.Stream()
        # whole numbers whose sums fit the significand: every order of the sum gives the same bits
        a, b = (cuda.randint(-8, 8, (rows, k), device="cuda").to(real) for rows in (m, n))
        c, status = cuda.full((m, n), float("nan"), dtype=real, device="cuda"), cuda.zeros(1, dtype=cuda.int32, device="cuda")
        args = N.GemmArgs(dtype=dtype, m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(), alpha=1.0,
                          d_status=status.data_ptr())
        sync()
        start.wait(60)
        for _ in range(5000):
            try:
                K.clpk_gemm(C.byref(args), stream.cuda_stream)
            except N.ClpkError as e:
                refused.append(f"{shape}: {e}")
        stream.synchronize()
        outputs.append((c, (a.double() @ b.double().T).to(real), status))

    threads = [threading.Thread(target=work, args=(shape,)) for shape in (one, two)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not refused, f"{len(refused)} of 10000 calls refused, the first: {refused[0]}"
    assert len(outputs) == 2
    for got, want, status in outputs:
        assert bool((got == want).all()) and int(status.item()) == 0
