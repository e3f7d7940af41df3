"""bench.py's line on standard output: short enough to be kept whole by whoever keeps the end of an output, with every
key that a reader of the headline needs; the rest goes to the details and nothing is lost."""
import json

import bench

LIMIT = 2800            # characters

KEYS = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline", "dtype", "data",
        "config", "roofline", "cpu_baseline", "e2e", "gpu_launches", "clocks")


def full_line():
    """A line as main() puts it together, every number at full length and the rows as many as they are."""
    x = 1234.5678901234567
    clocks = {"sm_mhz": x, "sm_max_mhz": x, "reasons": ["sw_power_cap", "sync_boost", "applications_clocks_setting"], "samples": 1234, "power_w": x}
    rows = {f"gemm_kind_{i}_16384": {"TFLOPS": x, "ms": x, "ms_rounds": [x] * 6, "note": "n" * 200, "sustained": dict(clocks)} for i in range(60)}
    variants = {"read": "wide", "copy": "wide", "triad": "wide"}
    kernels = {k: {"ms": x, "GBps": x, "frac_of_spec_8TBps": x} for k in variants}
    return {
        "metric": bench.METRIC, "value": x, "unit": bench.UNIT, "n_gpus": 8, "steps": 20, "warmup": 5, "ms_per_step": x, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": "w" * 90, "bytes_per_array": 1 << 33, "algorithmic_bytes_per_step": 6 << 33, "variants": variants, "l2": "l" * 70,
                   "parallelism": "replicas x8, no collective"},
        "kernels": kernels,
        "roofline": {"bound": "hbm", "kernel": "stream_triad_wide", "achieved": x, "peak": x, "peak_source": "s" * 60, "unit": "GB/s", "frac": x,
                     "frac_of_spec": x, "traffic": {"read": x, "write": x, "source": "t" * 100}},
        "cpu_baseline": {"value": x, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "s" * 90, "rows": rows, "other_reference_cpu_rows": rows,
                         "reference_cuda_kernels_on_this_gpu": rows},
        "e2e": {"value": x, "unit": bench.UNIT, "h2d_bytes_per_step": 1 << 34, "d2h_bytes_per_step": 1 << 14, "steps": 10, "ms_per_step": x,
                "host_buffer": "pinned 12345 MiB chunk reused"},
        "e2e_plugin": {"devices": rows}, "gpu_launches": 60, "clocks": clocks, "read_checksum": 1 << 31,
        "verified_at_full_size": {"read_checksum_equals_xor_of_all_words": True, "copy_equals_source_bitwise": True,
                                  "triad_equals_b_plus_s_times_c_bitwise": True, "elements_per_array": 1 << 31, "all_ranks": True},
        "rows": rows, "spec_peaks_per_gpu": bench.SPEC,
    }


def test_the_headline_is_short_and_complete():
    line = full_line()
    assert len(json.dumps(line)) > 40_000
    headline, details = bench.split_line(line)
    assert len(json.dumps(headline)) < LIMIT, len(json.dumps(headline))
    assert set(KEYS) <= set(headline) and headline["value"] == line["value"] and headline["e2e"] == line["e2e"]
    assert headline["cpu_baseline"]["kind"] == "port" and "rows" not in headline["cpu_baseline"]


def test_nothing_is_lost():
    line = full_line()
    headline, details = bench.split_line(line)
    base = dict(headline["cpu_baseline"], **details.pop("cpu_baseline"))
    assert dict(headline, **details, cpu_baseline=base) == line


def test_a_line_without_rows_or_baseline():
    line = dict(full_line(), rows=None, cpu_baseline=None, e2e_plugin=None)
    headline, details = bench.split_line(line)
    assert headline["cpu_baseline"] is None and details["rows"] is None and "cpu_baseline" not in details
