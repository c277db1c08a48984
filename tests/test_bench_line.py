"""The line that the bench prints: the headline keys whole, the variants cut to
their figures, a few kilobytes however long the record is."""
import json

import bench


def test_the_line_is_short_and_keeps_the_headline():
    history = [1e-7] * 1000
    record = {"metric": "m", "value": 1.23456789012e10, "e2e": {"value": 1.0123456789e10, "note": "x" * 500},
              "clocks": {"sm_mhz": 2070.0}, "gpu_launches": 42,
              "roofline": {"bound": "integer pipes", "frac": 0.123456789, "note": "y"},
              "variants": {"mixed": {"value": 2.3456789e10, "roofline": {"frac": 1}, "clocks": {}},
                           "serving": [{"lambda_per_s": 50, "p50_ms": 1.23456789, "accuracy": {"cases": history,
                                                                                               "within_bar": True}}],
                           "precision_sweep": {"worst_rel_l2_u": 1e-8, "runs": [{"rel_l2_u_every": history}] * 6}}}
    line = json.dumps(bench.brief(record))
    assert len(line) < 1000 and "\n" not in line
    back = json.loads(line)
    assert back["value"] == record["value"] and back["e2e"] == {"value": 1.0123456789e10}
    assert back["clocks"] == record["clocks"] and back["gpu_launches"] == 42
    assert back["variants"]["mixed"] == {"value": 2.34568e10}
    assert back["variants"]["serving"] == [{"lambda_per_s": 50, "p50_ms": 1.23457, "accuracy": {"within_bar": True}}]
    assert back["variants"]["precision_sweep"] == {"worst_rel_l2_u": 1e-8}
