"""The direct path's batched host arithmetic equals the per-pair formulas, whatever shape the points have."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from acoustic_agent_b200 import direct
from acoustic_agent_b200.directivity import source_directivity


@pytest.mark.parametrize("model", ["omni", "cardioid", {"type": "dipole", "orientation_deg": 33.0},
                                   {"type": "focused", "elevation_deg": -20.0}])
@pytest.mark.parametrize("pairs", [0, 1, 37])
def test_distances_and_gains_equal_the_single_pair(model, pairs):
    rng = np.random.default_rng(pairs)
    points = rng.normal(size=(pairs, 2, 3)) * 5.0
    if pairs > 1:
        points[1, 1] = points[1, 0]                       # coincident
        points[2, 1] = points[2, 0] + [1e-13, 0.0, 0.0]   # closer than the directivity's limit
    emitter = source_directivity(model)
    distances, gains = direct._distances_and_gains(points, emitter)
    assert distances == [float(np.linalg.norm(s - t)) for s, t in points]
    assert gains == [direct.directivity_gain(t - s, emitter) for s, t in points]


@pytest.mark.parametrize("column", [False, True])
def test_unoccluded_results_take_any_point_shape(column):
    cfg = SimpleNamespace(direct_occlusion=False, min_distance_m=0.3, c=343.0)
    pairs = [([0.0, 0.0, 1.0], [2.0, 1.0, 1.5]), ((1.0, 1.0, 1.0), (1.0, 1.0, 1.1))]
    want = direct.direct_results(None, None, pairs, cfg, "cardioid")
    shaped = [(np.reshape(s, (3, 1)) if column else np.asarray(s), np.reshape(t, (3, 1)) if column else t)
              for s, t in pairs]
    with np.testing.suppress_warnings() as quiet:
        quiet.filter(DeprecationWarning)
        got = direct.direct_results(None, None, shaped, cfg, "cardioid")
    for a, b in zip(want, got):
        assert a["band_gains"] == b["band_gains"] and a["distance_m"] == b["distance_m"]
        assert a["occlusion"] == 1.0 and a["occlusion_surface"] is None
        np.testing.assert_array_equal(b["transmission"], np.ones(6))
    assert want[0]["transmission"].base is None and direct.direct_results(None, None, [], cfg) == []
