"""The benchmark's line stays short enough to be read from the end of its output."""
import json

import bench


def test_line_is_short_and_detail_is_whole():
    variant = {"solves_per_s": 25354.0123456789, "ms_per_step": 40.4, "steps": 20, "stages": {"x" * 40: 1.0 / 3}, "note": "n" * 600}
    line = {"metric": bench.METRIC, "value": 25354.0, "unit": "solves/s", "ms_per_step": 40.4, "dtype": "d" * 200,
            "config": bench.config_dict(10680, 7200, 1), "e2e": {"value": 1.0}, "roofline": {"note": "r" * 1200},
            "variants": {f"variant_{i:02d}_with_a_long_name": dict(variant) for i in range(25)},
            "parity_vs_oracle": {"a": "b" * 2000}, "c2_eval": {"a": "b" * 2000}}
    short, detail = bench.split_line(line)
    assert len(json.dumps(short)) < 8000
    assert short["value"] == line["value"] and short["config"] == line["config"] and short["roofline"] == line["roofline"]
    assert short["variants"]["variant_03_with_a_long_name"] == {"solves_per_s": 25354.0123456789, "ms_per_step": 40.4}
    assert detail == {k: line[k] for k in ("variants", "parity_vs_oracle", "c2_eval")}
