"""The benchmark's line on standard output: every key that its readers need, and short enough to
survive where only the last 3,000 characters of the output are kept."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))


def test_line_is_short_and_complete():
    import bench
    figure = 123456.78901234567
    ties = {k: 8388608 for k in ("prim_mismatch", "prim_mismatch_exact_tie", "prim_mismatch_loose_tie",
                                 "prim_mismatch_not_tie", "valid_mismatch")}
    err = {"max": figure * 1e-12}
    load = {"load_of_batched_peak": 0.8, "p50_ms": figure, "p99_ms": figure, "by_kind": {"cp": {"p50_ms": figure}},
            "slowest_1pct": [{"kind": "cp", "n": 949, "latency_ms": figure}] * 400}
    line = {"metric": bench.METRIC, "value": figure, "unit": "Mqueries/s", "n_gpus": 8, "steps": 20, "warmup": 5,
            "ms_per_step": figure, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic",
            "config": {"workload": bench.WORKLOAD, "variant": "auto+morton", "queries_per_rank": 1 << 24,
                       "parallelism": "replicated scene, 8 query shard(s)", "l2": "flushed between steps",
                       "streams": "a step's closest points and rays on two streams, the rays at lower priority"},
            "plain_exact_mqps": figure, "quantised_wide8_mqps": figure, "quantised_wide16_mqps": figure,
            "quantised_wide8_vs_plain": figure, "quantised_wide16_vs_plain": figure, "tuned_vs_plain": figure,
            "parity": {"tuned": {"cp": ties, "ray": ties}}, "fp64_error": {"cp3d_exact": err, "ray3d_exact": err},
            "roofline": {"bound": "hbm", "achieved": figure, "peak": figure, "unit": "GB/s", "frac": figure,
                         "traffic": figure, "kernel": "cp3d_coherent", "peak_source": "measured on this kind of GPU",
                         "note": "x" * 4000, "l2": {"peak": figure, "frac": figure}, "binding": {"a": "y" * 4000}},
            "cpu_baseline": {"value": figure, "unit": "Mqueries/s", "cores": 192, "kind": "port", "sample": "z" * 2000},
            "e2e": {"value": figure, "unit": "Mqueries/s", "ms_per_step": figure, "h2d_bytes_per_step": 301989888,
                    "d2h_bytes_per_step": 905969664, "lanes": 2, "host_records_match": True, "note": "w" * 2000},
            "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 12345},
            "gpu_launches": 80, "serving_c4": {"batched": {"loads": [load]}},
            "silhouette_c2": {"coherent": {"mqueries_per_s": figure}, "fp64_error": {"sil3d_exact": err}},
            "closest_point_2d_c0": {"fp64_error": {"cp2d": err, "ray2d": err, "sil2d": err}},
            "batched_c3": {"batched_graph": {"mqueries_per_s": figure}, "batched_vs_tuned_per_scene": figure}}
    line["summary"] = bench.summary(line)
    text = json.dumps(bench.headline(line))
    assert len(json.dumps(line)) > 20_000 and len(text) < 3000, len(text)
    got = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert k in got, k
    assert got["value"] == figure and got["e2e"]["h2d_bytes_per_step"] == 301989888
    assert got["e2e"]["d2h_bytes_per_step"] == 905969664 and got["clocks"]["sm_mhz"] == 1965.0


def test_line_without_optional_parts():
    import bench
    got = bench.headline({"metric": "m", "value": 1.0, "e2e": None, "roofline": None, "cpu_baseline": None, "summary": {}})
    assert got["e2e"] is None and got["value"] == 1.0
