"""The waits of the fp32 kernel's teams that take turns.  A wait on an mbarrier's parity tells the last two phases apart, no
more: it ends a round too early where the phase before the one waited for is not complete.  So whoever waits must have waited for that
phase too, or for something that comes after it.  Shown on the CPU: a run on a GPU would need a late load to show it."""
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
NAMES = ("raw_stages", "conv_stages", "accs")
GROUPS = 2                                       # of converters, and issuing warps


@pytest.fixture(scope="module")
def rings():
    """width -> the numbers of its stages and barriers, as a compiler evaluates the kernel's source"""
    source = (ROOT / "clpeak_b200" / "csrc" / "clpk_gemm_f32.cuh").read_text()
    tile = re.search(r"constexpr uint32_t kF32M = .*?\ntemplate <uint32_t TN> struct F32Tile \{.*?\n\};\n", source, re.S).group(0)
    show = "".join(f'std::printf("%u %u {n} %u\\n", TN, kF32Groups, F32Tile<TN>::{n});' for n in NAMES) + \
        "".join(f'std::printf("%u %u {n} %u\\n", TN, kF32Groups, {n});' for n in ("kF32Bars",))
    out = ROOT / "tests" / "_build"
    out.mkdir(exist_ok=True)
    (out / "f32_tile.cpp").write_text(f"#include <cstddef>\n#include <cstdint>\n#include <cstdio>\n{tile}"
                                      f"template <uint32_t TN> void show() {{ {show} }}\nint main() {{ show<32>(); show<64>(); show<96>(); show<128>(); }}\n")
    subprocess.run(["g++", "-std=c++17", "-o", str(out / "f32_tile"), str(out / "f32_tile.cpp")], check=True)
    found = {}
    for line in subprocess.run([str(out / "f32_tile")], check=True, capture_output=True, text=True).stdout.splitlines():
        width, groups, name, value = line.split()
        assert int(groups) == GROUPS
        found.setdefault(int(width), {})[name] = int(value)
    return found


def waits(t, chunks_of_a_tile, tiles):
    """(team, kind of event, number of the event waited for) in each team's order"""
    chunk = turn = 0
    for _ in range(tiles):
        for first in range(0, chunks_of_a_tile, 2):
            of_turn = range(chunk, chunk + min(2, chunks_of_a_tile - first))
            for c in of_turn:
                yield f"converters {c % GROUPS}", "raw", c
                yield f"converters {c % GROUPS}", "emptied", c - t["conv_stages"]
            yield f"issuer {turn % GROUPS}", "accumulator", turn - t["accs"]
            for c in of_turn:
                yield f"issuer {turn % GROUPS}", "converted", c
            chunk, turn = of_turn[-1] + 1, turn + 1


def too_early(t, chunks_of_a_tile, bars):
    """waits of which nothing says that the phase before theirs is complete"""
    known, wrong = set(), []
    for team, kind, event in waits(t, chunks_of_a_tile, 40):
        before = event - bars[kind]
        # a group converts, and arrives for, its chunks in order, and all accumulators are given back in order; what an issuing warp
        # has had consumed, and loads, are known one by one
        later = range(before, event, GROUPS) if kind == "converted" else range(before, event) if kind == "accumulator" else (before,)
        if before >= 0 and not any((team, kind, e) in known for e in later):
            wrong.append((team, kind, event))
        known.add((team, kind, event))
    return wrong


@pytest.mark.parametrize("width", [32, 64, 96, 128])
def test_no_wait_can_end_a_round_too_early(rings, width):
    t = rings[width]
    bars = {"raw": t["raw_stages"], "emptied": t["kF32Bars"], "converted": t["kF32Bars"], "accumulator": t["accs"]}
    for chunks_of_a_tile in range(1, 40):
        assert not too_early(t, chunks_of_a_tile, bars)


def test_one_barrier_for_each_of_an_odd_number_of_stages_would_not_do():
    def kinds(raw, conv, accs):
        bars = {"raw": raw, "emptied": conv, "converted": conv, "accumulator": accs}
        return {kind for n in range(1, 12) for _, kind, _ in too_early({"raw_stages": raw, "conv_stages": conv, "accs": accs}, n, bars)}
    assert kinds(5, 5, 2) == {"raw", "emptied", "converted"} and kinds(7, 4, 3) == {"raw", "converted"} and kinds(8, 6, 4) == set()
