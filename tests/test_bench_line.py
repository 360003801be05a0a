"""bench.py's JSON line stays a few KB long whatever the records of the other
configurations hold (per-channel errors of a thousand channels made it 53 KB,
more than a reader of the last lines of output takes), with the measurement's
own figures unchanged."""
import json

import bench


def record():
    errors = {"channels": 1024, "min": -133.7, "median": -132.8, "max": -132.17, "nonfinite_channels": 0,
              "per_channel": [-132.12 - 0.001 * i for i in range(1024)]}
    form = {"latency_ms": {"p50": 0.22695350000390135, "p99": 0.23625539999727613, "max": 1.7963960000315637},
            "deadline_ms": 16 / 3, "block_bytes": 1039032320, "device_bytes": 1569794048, "error_db_vs_fp64": errors}
    tuner = [{"levels": [[128 << i, 1] for i in range(8)], "mean_ms": 0.0347, "max_ms": 0.28} for _ in range(30)]
    fit = {"sizes": [1, 2, 4], "us": [16.38, 26.62, 43.04], "fixed_us": 8.2, "what": "x" * 90}
    return {
        "metric": bench.METRIC, "value": 1.6212792946669161, "unit": "GSamples/s", "n_gpus": 1, "steps": 20,
        "warmup": 5, "ms_per_step": 0.020211199950426816, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic", "config": bench.config_dict(128),
        "gpu_launches": 42, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []},
        "e2e": {"value": 0.61, "unit": "GSamples/s", "h2d_bytes_per_step": 131072, "d2h_bytes_per_step": 131072,
                "what": "y" * 300},
        "roofline": {"bound": "hbm", "achieved": 3783.8, "peak": 6545.0, "frac": 0.578, "tiling": [32, 8, 4],
                     "size_floor": {"us": 16.38, "gbs": 4048.0, "grids_us": {str(i): 1.0 for i in range(6)},
                                    "fit": fit}},
        "cpu_baseline": {"value": 0.06, "unit": "GSamples/s", "cores": 16, "kind": "port", "sample": "s"},
        "configs": {"cfg1": {"channels": 2, "latency_ms": {"p50": 0.0276, "p99": 0.0354},
                             "error_db_vs_fp64": [-133.2, -133.2]},
                    "cfg3": {"channels": 1024, **{s: dict(form) for s in ("fp32", "fp24", "fp16", "bf16")}},
                    "cfg4": {"channels": 256, "autotuner": tuner, "fp32": dict(form), "fp16": dict(form)},
                    "cfg5": {s: {"latency_ms": {"p99": 1.2}, "deadline_misses": 0} for s in ("fp32", "fp24")}},
    }


def test_line_is_short_and_keeps_the_figures():
    r = record()
    assert len(json.dumps(r)) > 40000
    text = json.dumps(bench.stdout_line(r))
    assert "\n" not in text and len(text) < 4500
    d = json.loads(text)
    assert set(d) == set(r)
    for k in ("metric", "unit", "n_gpus", "steps", "warmup", "higher_is_better", "scaling", "vs_baseline", "dtype",
              "data", "config", "gpu_launches", "clocks", "cpu_baseline"):
        assert d[k] == r[k], k
    for k in ("value", "ms_per_step"):
        assert abs(d[k] - r[k]) <= 1e-6 * r[k]
    assert {k: d["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step")} == \
        {k: r["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step")}
    assert d["configs"]["cfg3"]["fp24"]["error_db_vs_fp64"] == {"max": -132.17, "nonfinite_channels": 0}
    assert d["configs"]["cfg4"]["fp32"]["latency_ms"]["p99"] == 0.2362554
