"""bench.py's line: short enough for what a log's tail keeps, whatever the entries behind it hold."""
import json

import bench


def test_headline_fits_a_log_tail():
    text = "x" * 400
    entry = {"value": 1234567890.123456789, "unit": "points/s of a kind", "ms_per_step": 3.14159265358979, "config": text,
             "roofline": {"note": text}, "clocks": {"reasons": []}}
    e2e = {"value": 3.7e8 / 3, "unit": "points/s", "h2d_bytes_per_step": 16384, "d2h_bytes_per_step": 8589934592,
           "path": text[:120], "other": {"staged": dict(entry), "drop_in": dict(entry)}, "link": dict(entry)}
    line = {"metric": "m", "value": 1e10 / 3, "e2e": e2e, "clocks": {"sm_mhz": 2070.0, "reasons": []},
            "cpu_as_shipped": dict(entry), "roofline": {"frac": 1.0 / 3}, "gpu_launches": 20,
            "configs": {"c%d" % k: dict(entry) for k in range(8)}}
    line["configs"]["c8"] = {"error": text}
    short, details = bench.headline(line)
    assert len(json.dumps(short)) < 1500
    assert short["value"] == 3333330000.0 and short["e2e"]["value"] == 123333000.0 and short["gpu_launches"] == 20
    assert short["e2e"]["h2d_bytes_per_step"] == 16384 and short["e2e"]["d2h_bytes_per_step"] == 8589934592
    assert short["configs"]["c3"] == {"value": 1234570000.0, "unit": "points/s", "ms": 3.14159}
    assert details["configs"]["c3"] == entry and details["configs"]["c8"]["error"] == text
    assert details["e2e"]["other"]["drop_in"] == entry and details["cpu_as_shipped"] == entry
    assert "other" in line["e2e"] and "configs" in line  # the caller's line stays whole


def test_headline_without_configurations():
    line = {"metric": "m", "value": 2.5, "e2e": {"value": 1.0}, "config": {"n": 1 << 40}}
    assert bench.headline(line) == (line, {})
