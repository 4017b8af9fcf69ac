"""The autotuner leaves a setting at the library's default unless another value
is faster by more than two runs of one value differ; the committed settings
follow that rule on their own measurements."""
import json

import pytest

from delta2_gb300 import autotune


@pytest.mark.parametrize("ms, want", [
    ({0: 0.6653, 1: 0.6752, 2: 0.6445, 3: 0.6431, 4: 0.656}, 2),
    ({0: 1.0, 2: 1.0, 3: 0.98}, 3),
    ({0: 0.9, 1: 0.8}, 1),
    ({2: 1.0, 3: 2.0}, 2)])
def test_first_iters_prefers_the_default_on_a_tie(ms, want):
    assert autotune.choose_first_iters(ms) == want


def test_committed_settings_follow_the_rules():
    with open(autotune.DEFAULT_OUT) as f:
        res = json.load(f)
    ms = {int(k): v for k, v in res["measurements"]["ccd_ms_per_step_by_ee_first_iters"].items()}
    assert res["settings"]["ee_first_iters"] == autotune.choose_first_iters(ms)
    totals = {}
    for key, t in res["measurements"]["pile_seconds_by_grid_min_parts"].items():
        v = int(key.split("/")[1])
        totals[v] = totals.get(v, 0.0) + t
    assert res["settings"]["grid_min_parts"] == autotune.choose_grid_threshold(totals)
