"""Calls past ctypes answer as the ctypes wrapper does: plain arguments, arguments that only ctypes converts, and those it refuses.
Nothing is launched: no element, a NULL buffer, or no such type."""
import ctypes as C
import os
import sysconfig
import threading

import numpy as np
import pytest

from clpeak_b200 import build
from clpeak_b200 import native as N

FAST = N._calls()
pytestmark = pytest.mark.skipif(FAST is None, reason="built without the interpreter's headers")

ARRAY = (N.GemmArgs * 2)()
FILL = "clpk_fill_f32"
CALLS = [(FILL, (0, 0, 1, 2, 0.0, 1.0, None)), (FILL, (None, 5, 1, 2, 0.0, 1.0, 0)), (FILL, (None, 5, 1, 7, 0.0, 1.0, 0)),
         (FILL, (0, 0, 2 ** 64 - 1, 2, 0.0, 1.0, 0)), (FILL, (2 ** 64 - 1, 0, 2 ** 63, 2, 0.0, 1.0, 0)), (FILL, (0, 0, 2 ** 70, 2, 0.0, 1.0, 0)),
         (FILL, (0, 0, -1, 2, 0.0, 1.0, 0)), (FILL, (-1, 0, 1, 2, 0.0, 1.0, 0)), (FILL, (0, 0, 1, 2 ** 31, 0.0, 1.0, 0)),
         (FILL, (0, 0, 1, -1, 0.0, 1.0, 0)), (FILL, (0, 0, 1, 2 ** 32 + 2, 0.0, 1.0, 0)), (FILL, (0, 0, 1, True, 0.0, 1.0, 0)),
         (FILL, (0, 0, 1, 2, 0, 1, 0)), (FILL, (0, 0, 1, 2, 1e300, float("nan"), 0)), (FILL, (0, 0, 1, 2.0, 0.0, 1.0, 0)),
         (FILL, (0, 0.0, 1, 2, 0.0, 1.0, 0)), (FILL, (0, 0, 1, 2, "0", 1.0, 0)), (FILL, (0, np.int64(0), 1, 2, 0.0, 1.0, 0)),
         (FILL, (0, 0, 1, 2, np.float32(0), 1.0, 0)), (FILL, (C.c_void_p(0), C.c_uint64(0), 1, C.c_int(2), C.c_float(0), 1.0, C.c_void_p(0))),
         (FILL, (0, 0, 1)), (FILL, ()), (FILL, (b"", 0, 1, 2, 0.0, 1.0, 0)), (FILL, ([], 0, 1, 2, 0.0, 1.0, 0)),
         ("clpk_fill_i8", (0, 0, 1, 0)), ("clpk_fill_i8", (0, 5, 1, 0)), ("clpk_convert_f32", (0, 0, 0, N.DT_BF16, 0)),
         ("clpk_convert_f32", (0, 0, 0, 99, 0)), ("clpk_quantize_fp4", (0, 0, 0, 4, 64, N.DT_NVF4, 1.0, 0)),
         ("clpk_quantize_fp4", (0, 0, 0, 4, 64, N.DT_NVF4, 1, 0)), ("clpk_absmax_f32", (None, None, 0, None)),
         ("clpk_stream_read", (99, 0, 0, 0, 0)), ("clpk_stream_copy", (99, 0, 0, 0, 0)), ("clpk_stream_triad", (99, 0, 0, 0, 1.5, 0, 0)),
         ("clpk_gemm", (C.byref(N.GemmArgs()), 0)), ("clpk_gemm", (N.GemmArgs(), 0)), ("clpk_gemm", (None, 0)), ("clpk_gemm", (C.byref(ARRAY), 0)),
         ("clpk_gemm", (C.byref(ARRAY[1]), None)), ("clpk_gemm", (C.pointer(ARRAY[0]), 0)), ("clpk_gemm", (C.byref(C.c_int()), 0)),
         ("clpk_gemm", (0, 0)), ("clpk_gemm_pack_scales", (C.byref(N.GemmArgs(dtype=N.DT_BF16)), 0)),
         ("clpk_gemm_pack_scales", (C.byref(N.GemmArgs(dtype=N.DT_NVF4, m=1, n=1, k=100)), 0))]


def outcome(f, args):
    try:
        return f(*args)
    except Exception as e:                                          # noqa: BLE001: whatever either raises
        return type(e), str(e)


@pytest.mark.parametrize("name,args", CALLS)
def test_the_same_answer_as_through_ctypes(K, name, args):
    assert type(getattr(K, name)) is not type(outcome)              # not the Python wrapper
    assert outcome(getattr(K, name), args) == outcome(lambda *a: K.call(name, *a), args)


@C.CFUNCTYPE(C.c_int, C.POINTER(N.GemmArgs), C.c_void_p)
def tells_m(args, stream):
    return args[0].m if args else -1


def test_the_structure_that_a_byref_names(K):
    """A byref may carry an offset: what it passes then is not the structure that it refers to."""
    array = (N.GemmArgs * 3)(*(N.GemmArgs(m=m) for m in (5, 6, 7)))
    inside = N.GemmArgs.from_buffer(array, C.sizeof(N.GemmArgs))
    named = [(C.byref(array[0]), 5), (C.byref(array[0], 0), 5), (C.byref(array[0], C.sizeof(N.GemmArgs)), 6), (C.byref(array[1]), 6),
             (C.byref(array[1], C.sizeof(N.GemmArgs)), 7), (C.byref(array[1], -C.sizeof(N.GemmArgs)), 5), (C.byref(array[2], -C.sizeof(N.GemmArgs)), 6),
             (C.byref(inside), 6), (C.byref(inside, C.sizeof(N.GemmArgs)), 7), (C.pointer(array[2]), 7),
             (C.byref(N.GemmArgs(m=9)), 9), (N.GemmArgs(m=9), 9), (None, -1)]
    call = K._checked("clpk_gemm", tells_m)
    for args, m in named:
        with pytest.raises(N.ClpkError) as e:
            call(args, None)
        assert e.value.code == m
    with pytest.raises(C.ArgumentError):
        call(C.byref(array, C.sizeof(N.GemmArgs)), None)


def test_which_structures_go_past_ctypes():
    went = []
    call = FAST.bind("clpk_gemm", C.cast(tells_m, C.c_void_p).value, lambda *a: went.append("ctypes"), went.append, C.byref, type(C.byref(C.c_int())), N.GemmArgs)
    array = (N.GemmArgs * 2)(N.GemmArgs(m=5), N.GemmArgs(m=6))
    for args in (C.byref(array[1]), C.byref(N.GemmArgs(m=7)), C.byref(array[0], C.sizeof(N.GemmArgs)), array[0]):
        call(args, None)
    assert went == [6, 7, "ctypes", "ctypes"]


def test_errors_of_several_threads_at_once(K):
    wrong = []

    def work(what, text):
        for _ in range(300):
            got = outcome(getattr(K, what[0]), what[1])
            if got[0] is not N.ClpkError or text not in got[1]:
                wrong.append(got)
    threads = [threading.Thread(target=work, args=a) for a in (((FILL, (None, 5, 1, 2, 0.0, 1.0, 0)), "d_dst is NULL"),
                                                               ((FILL, (1, 5, 1, 9, 0.0, 1.0, 0)), "unknown distribution 9"))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_an_extension_of_another_interpreter_is_not_loaded(tmp_path, monkeypatch):
    for name in ("_clpk_calls.so", "_clpk_calls.cpython-39-x86_64-linux-gnu.so", "_clpk_calls.abi3.so"):
        (tmp_path / name).write_bytes(b"not for this one")
    monkeypatch.setattr(N, "LIB_DIR", tmp_path)
    assert N._calls.__wrapped__() is None


@pytest.mark.parametrize("headers", [False, True])
def test_an_extension_of_older_sources_does_not_stay(tmp_path, monkeypatch, headers):
    old = tmp_path / ("_clpk_calls" + sysconfig.get_config_var("EXT_SUFFIX"))
    old.write_bytes(b"older than its sources")
    os.utime(old, (0, 0))
    monkeypatch.setattr(build, "LIB", tmp_path)
    if not headers:
        monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
        assert build.build_calls() is None and not old.exists()
    else:
        assert build.build_calls() == old and old.read_bytes()[:4] == b"\x7fELF"
        built = old.stat().st_mtime_ns
        assert build.build_calls() == old and old.stat().st_mtime_ns == built
