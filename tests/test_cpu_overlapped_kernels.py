"""Kernels that may start under the tail of the kernel before them in the stream, by their source: they wait, and nothing
that they read is promised to stay the same while they run.

A `const __restrict__` parameter lets the compiler read through the read-only path, whose data may not change during the
kernel's lifetime -- and that lifetime begins while the kernel before may still be writing.  The cache-hint intrinsics
(__ldcs and the like) come with no documented order against the wait either.  Both are shown here and not on a GPU:
a run proves nothing about what a compiler may do."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "clpeak_b200" / "csrc"
WAITS = re.compile(r"\b(griddep_wait|join_stream|join_previous_launch)\s*\(")
LOADS = re.compile(r"\b__ld(g|cs|cg|ca|lu|cv)\s*\(")


def matching(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced source")


def kernels():
    """name -> (parameters, body) of every __global__ function."""
    out = {}
    for path in sorted(CSRC.rglob("*.cu")) + sorted(CSRC.rglob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            head = re.compile(r"(?:__launch_bounds__|__cluster_dims__)\s*\(").search(text, m.end(), m.end() + 120)
            at = m.end()
            while head:
                at = matching(text, head.end() - 1, "()") + 1
                head = re.compile(r"\s*(?:void\s+)?(?:__launch_bounds__|__cluster_dims__)\s*\(").match(text, at)
            name = re.compile(r"(\w+)\s*\(").search(text, at)
            close = matching(text, name.end() - 1, "()")
            body = text.index("{", close)
            out[name.group(1)] = (text[name.end():close], text[body:matching(text, body, "{}") + 1])
    return out


KERNELS = kernels()
OVERLAPPED = sorted(name for name, (_, body) in KERNELS.items() if WAITS.search(body))


def test_the_parser_finds_the_kernels():
    assert {"fill_f32_kernel", "stream_triad_wide", "sgemm_kernel", "gemm_kernel", "gemm_tiles_kernel", "pack_scales_kernel"} <= set(OVERLAPPED)
    assert "pointer_chase_kernel" in KERNELS and "pointer_chase_kernel" not in OVERLAPPED


def test_every_kernel_launched_behind_another_waits():
    launched = set()
    for path in CSRC.rglob("*.cu"):
        text = path.read_text()
        launched |= set(re.findall(r"\blaunch_(?:behind|simt|clusters)\(\s*(?:\w+ \? )?(\w+)[<,]", text))
    assert len(launched) >= 17 and {"gemm_tiles_kernel", "gemm_f32_kernel"} <= launched and launched <= set(OVERLAPPED), launched - set(OVERLAPPED)


@pytest.mark.parametrize("name", OVERLAPPED)
def test_nothing_is_promised_to_stay_the_same(name):
    params, body = KERNELS[name]
    assert "__restrict__" not in params
    assert not LOADS.search(body)
