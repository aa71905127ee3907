"""What the benchmark reports when training broke while it ran."""
import json

import pytest

import bench


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_no_rate_is_reported_beside_a_loss_that_is_not_finite(bad):
    good = {"value": 10.0, "mfu": 0.5, "loss": 7.0, "e2e_loss": 0.8, "e2e": {"value": 9.0, "unit": "tokens/s"}}
    assert bench.without_broken_runs(good) == good
    late = bench.without_broken_runs({**good, "e2e_loss": bad})
    assert late["value"] == 10.0 and late["e2e"]["value"] is None and "not finite" in late["e2e"]["unavailable"]
    early = bench.without_broken_runs({**good, "loss": bad, "e2e_loss": bad})
    assert early["value"] is None and early["mfu"] is None and "not finite" in early["unavailable"]
    for r in (late, early):
        json.loads(json.dumps(r, allow_nan=False))
