"""The printed line of bench.py stays short enough to be kept whole."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

CONTRACT = {"metric": "m", "value": 1 / 3, "unit": "solves/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 291.98842366536456, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic", "config": {"workload": "w" * 200, "n_unknowns": 8402},
            "e2e": {"value": 2.5, "unit": "solves/s", "h2d_bytes_per_step": 2262064304, "d2h_bytes_per_step": 1443388944},
            "gpu_launches": 5844, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}}


def record(requests):
    leg = {"value": 2.4, "per_request": [["h", 9955, 4, 30.0, 0.1, 0.2, 4, 0]] * requests, "how": "x" * 500,
           "phase_ms": {"p%d" % k: k / 7 for k in range(requests // 4)}}
    roof = {"kernel": "k" * 90, "bound": "tensor", "achieved": 908.8359458018093, "peak": 1954.3, "unit": "TFLOP/s",
            "frac": 0.4650442336395688, "ms": 134.19856029376388, "traffic": {"case": "c" * 300}, "note": "n" * 300}
    legs = ("serving", "batched", "transient", "retarded", "rcs", "incidence", "far_precision", "mixed")
    return dict(CONTRACT, **{k: leg for k in legs}, rooflines=[roof] * 12, roofline=roof)


def test_line_is_short_and_keeps_the_contract():
    for requests in (0, 40, 4000):
        out = bench.printed(record(requests))
        line = json.dumps(out)
        assert len(line) <= bench.LINE_BYTES
        back = json.loads(line)
        for k, v in CONTRACT.items():
            assert back[k] == v or abs(back[k] - v) <= 1e-5 * abs(v)
        assert back["roofline"]["frac"] == 0.465044
    assert bench.printed(record(40))["serving"]["value"] == 2.4
