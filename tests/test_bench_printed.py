"""The line bench.py prints from a full record: every key of the contract,
the headline numbers unrounded, and short enough (under 5 000 characters) to
be kept whole by a log's tail, however long the record's tables are."""
import importlib.util
import json
import os

from common import ROOT

CONTRACT = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
            "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e",
            "gpu_launches", "clocks", "roofline", "cpu_baseline")


def _bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def _record(metric, workload):
    x = 12345.678901234567
    long = {f"variant {i}": {"kernel_us": x, "text": "what this row says " * 4} for i in range(40)}
    return {
        "metric": metric, "value": x, "unit": "evals/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 1e3 / x, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32", "data": "synthetic",
        "config": {"workload": workload, "precision": "a sentence on the form's precision " * 6,
                   "events_per_rank": {"data": 1100000, "mc": 1000000}, "l2": "flushed " * 20,
                   "parallelism": "single GPU"},
        "plain_f64": {"value": x, "unit": "evals/s", "ms_per_step": x, "speedup": x},
        "fp32_recompute": long, "cached_variants": long, "hessian": long, "host": long,
        "e2e": {"value": x, "unit": "evals/s", "h2d_bytes_per_step": 128,
                "d2h_bytes_per_step": 136, "call": "FCN.nll_grad(x) with x a host numpy vector"},
        "roofline": {"bound": "hbm", "achieved": x, "peak": x, "unit": "GB/s", "frac": 0.7123456789,
                     "peak_kind": "measured", "kernel": "a kernel's name and what it does " * 2,
                     "launch_us": x, "traffic": x, "traffic_source": "where from " * 9,
                     "plain_f64_kernel": long},
        "gpu_launches": 20, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": [],
                                       "samples": 40},
        "check": {"dnll": x, "grad_max_rel": 1e-8, "nll_mixed": x},
        "setup_s": {"dataset": x}, "engine": long,
    }


def test_printed_line():
    b = _bench()
    line = _record(b.METRIC, b.WORKLOAD)
    line["workloads"] = {n: b._compact(_record(w[4], w[5])) for n, w in b.WORKLOADS.items()
                         if n != "lc2pkpi"}
    sv = {k: 12345.678901234567 for k in
          ("n_fits", "evals", "seconds", "evals_per_s", "latency_p50_s", "latency_p99_s",
           "mean_evals_per_fit", "errors", "converged", "events_total", "pool_tiles", "pool_gb",
           "budget_gb", "batches", "mean_requests_per_batch", "launch_seconds")}
    line["serving"] = {"metric": "m", "unit": "evals/s", "workload": "w" * 300,
                       "saturated": dict(sv, tuning=[1] * 200, driver="native"),
                       "arrivals_over_1s": dict(sv, tuning=[1] * 200, driver="native")}
    line["cpu_baseline"] = {"value": 1.3, "unit": "evals/s", "cores": 16, "kind": "port",
                            "sample": "what was run and how long it took " * 8}
    text = json.dumps(b._printed(line))
    assert len(text) < 5000 < 15000 < len(json.dumps(line))
    d = json.loads(text)
    for k in CONTRACT:
        assert k in d, k
    assert d["value"] == line["value"] and d["ms_per_step"] == line["ms_per_step"]
    assert d["config"] == line["config"] and d["gpu_launches"] == 20
    assert d["roofline"]["frac"] == 0.712346 and d["clocks"]["reasons"] == []
    assert set(d["workloads"]) == set(b.WORKLOADS) - {"lc2pkpi"}
    assert all(w["value"] == 12345.7 and w["clocks"]["sm_mhz"] == 1965.0
               for w in d["workloads"].values())
    # a workload that failed, no extras, other ranks' shape
    line["workloads"] = {"error": "RuntimeError('x')"}
    assert json.loads(json.dumps(b._printed(line)))["workloads"] == line["workloads"]
    del line["workloads"], line["serving"], line["cpu_baseline"], line["clocks"]
    assert "value" in b._printed(line)
