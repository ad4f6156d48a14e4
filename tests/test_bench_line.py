"""The printed line of bench.py's default run: every key of the contract, and
short enough for a reader that keeps the end of a log only -- whatever the
nested records hold."""
import json

import bench


def _line(buckets=10, text=400):
    note = "n" * text
    err = [{"d1": [0.0, 1.0], "count": 123456789, "max_abs": 0.00037049687807666487,
            "rms_abs": 3.910825465525674e-05} for _ in range(buckets)]
    mode = {"options_per_s": 262345678901.2345, "max_abs": 0.00056123456789, "rms_abs": 3.612345678e-05,
            "buckets": err}
    clocks = {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 9, "window_samples": 6,
              "window_s": 0.0671234}
    base = {"value": 310631989.6795044, "unit": "options/s", "cores": 16, "kind": "port",
            "sample": "10000000 options x 100 passes (of 100) of the same book, static partition over 16 "
                      "threads, 3.22 s", "note": note}
    tune = {"vec_per_thread": 1, "block": 128, "blocks_per_sm": 4, "load_path": 7, "pdl": 1, "resident_32nds": 10}
    return {
        "metric": bench.METRIC, "value": 302467890123.4567, "unit": "options/s", "n_gpus": 1, "steps": 20,
        "warmup": 5, "ms_per_step": 3.3061234567, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded book, reference config distributions)",
        "config": bench.map_config(bench.N_OPTIONS, bench.NUM_RUNS, 1), "tune": tune,
        "roofline": {"bound": "hbm", "achieved": 8468.123456789, "peak": 6790.7, "unit": "GB/s",
                     "frac": 1.2470123456789, "peak_source": "measured", "traffic": None, "traffic_note": note,
                     "bytes_per_launch": 280000000, "avg_launch_us": 33.061234567, "l2_assisted": True,
                     "l2_bytes": 135528448, "prefix_bytes": 42352576, "note": note},
        "accuracy": {"max_abs_vs_fp64": 4.07123456789e-05, "rms_abs_vs_fp64": 3.61234567e-06, "gate": 1e-4},
        "e2e": {"value": 288756959042.715, "unit": "options/s", "h2d_bytes_per_step": 240000000,
                "d2h_bytes_per_step": 40000000, "ms_per_step": 3.463119999999975,
                "mode": "pipelined bsg_price_soa(BSG_ASYNC, pinned host arrays) + bsg_synchronize",
                "synchronous": {"value": 210756959042.715, "ms_per_step": 4.763119999999975}},
        "gpu_launches": 2000, "clocks": clocks,
        "repeats": {"values": [302467890123.4567] * 3, "note": note, "spread": 0.0002123456789},
        "roofline_2p28": {"workload": note, "value": 2.606123456789e11, "frac": 1.0941234567, "ms_per_step": 103.0123,
                          "max_abs_vs_fp64": 4.71234567e-05, "gpu_launches": 300, "tune": tune, "clocks": clocks},
        "batch": {"workload": note, "value": 2.554123456e11, "roofline": {"frac": 1.0731234567, "bound": "hbm"},
                  "speedup_vs_plain": 5.0912345678, "bit_identical": True, "gpu_launches": 300, "clocks": clocks},
        "serve": {"workload": note, "trace": {m: {"p99_ms": 0.2201234567, "options_per_s": 1.9012345678e9}
                                              for m in ("batched", "plain")},
                  "host_link": {"h2d_GBps": 211.123456789},
                  "throughput_at_equal_p99": [{"p99_bound_ms": b, "batched_options_per_s": 5.1412345e9,
                                               "plain_options_per_s": 2.34123456e8, "ratio": 28.1123456,
                                               "batched_rate_per_s": 5e4, "plain_note": note}
                                              for b in (0.5, 1.0, 2.0)], "sweep": {"batched": err, "plain": err}},
        "swaptions": {"workload": note, "value": 2.6312345678e10, "ms_per_step": 4.8612345678, "gpu_launches": 3,
                      "vs_oracle": {"max_rel_price_diff": 8.9123456e-15, "note": note}, "cpu_baseline": base},
        "precision": {"workload": note, "modes": {m: mode for m in ("fast", "sfu_ref", "libm_ref")}, "note": note},
        "fp64": {"workload": note, "value": 36580615149.77613, "max_rel_vs_cpu_fp64": 33.95476584328323,
                 "max_rel_above_1e-6_of_max_s_k": 1.1031606907609629e-10,
                 "max_diff_over_max_s_k": 8.505145105559493e-16, "cpu_baseline": base},
        "io": {"workload": note, "parse": {"speedup": 39.71979310453595, "bit_identical": True},
               "write": {"speedup": 43.806362026673895, "byte_identical": True}},
        "cpu_baseline": base,
    }


def test_the_line_is_short_and_whole():
    line = _line()
    assert len(json.dumps(line)) > 3000
    text = bench.printed_line(line)
    assert len(text) <= bench.LINE_LIMIT < 3000 and "\n" not in text
    got = json.loads(text)
    assert set(got) == set(line)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks", "tune"):
        assert got[key] == line[key] or key == "clocks"
    assert got["clocks"]["reasons"] == [] and got["clocks"]["sm_mhz"] == 2070.0
    assert got["e2e"]["h2d_bytes_per_step"] == 240000000 and abs(got["e2e"]["value"] / line["e2e"]["value"] - 1) < 1e-5
    assert abs(got["roofline"]["frac"] - line["roofline"]["frac"]) < 1e-5
    assert got["cpu_baseline"]["sample"] == line["cpu_baseline"]["sample"]
    # every nested record is there with its figures
    assert got["batch"]["speedup_vs_plain"] and got["serve"]["equal_p99"][1][3] == 28.1123
    assert got["precision"]["fast_max_abs"] and got["io"]["parse_speedup"]
    assert line["roofline"]["note"]  # the caller's own is left as it was


def test_records_give_way_to_the_limit():
    line = _line()
    line["tune"]["note"] = "x" * 400
    got = json.loads(bench.printed_line(line))
    assert len(bench.printed_line(line)) <= bench.LINE_LIMIT
    assert got["io"] == "in --records" and got["value"] == line["value"]


def test_a_record_that_failed_says_so():
    line = _line()
    line["serve"] = {"error": "BsgError: no"}
    assert json.loads(bench.printed_line(line))["serve"] == {"error": "BsgError: no"}
