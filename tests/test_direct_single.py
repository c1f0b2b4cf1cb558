"""One pair's direct sound costs no more on the host than the formulas themselves, and equals them.

The queries are answered by a stand-in, so only the host's part is timed: the shortest of many runs against the per-pair
formulas, restated here, with half of their time to spare.
"""
from __future__ import annotations

import math
import time
from types import SimpleNamespace

import numpy as np
import pytest

from acoustic_agent_b200 import _lib, bands, direct
from acoustic_agent_b200.directivity import source_directivity

CONFIG = SimpleNamespace(direct_occlusion=True, direct_occlusion_mode="volumetric", direct_occlusion_radius_m=0.1,
                         direct_occlusion_samples=32, direct_transmission=True, num_transmission_rays=4,
                         min_distance_m=1.0, c=343.0)
TABLES = SimpleNamespace(names=("wall", "shelf"))
RECORD = np.dtype([("occlusion", "<f8"), ("transmission", "<f8", (6,)), ("occlusion_surface", "<i4"), ("reserved", "<i4")])


def answer(scene, tables, queries, count, *, samples, stream=None):
    records = np.zeros(count, dtype=RECORD)
    for k in range(count):
        q = queries[k]
        share = (q.source[0] * 7.0 + q.listener[1] * 3.0 + q.radius + q.max_layers) % 1.0
        records[k]["occlusion"] = 1.0 if share > 0.7 else share
        records[k]["transmission"] = share * np.arange(6)
        records[k]["occlusion_surface"] = int(share * 3.0) - 1
    return records


def one_by_one(pairs):
    emitter, out = source_directivity("cardioid"), []
    for source, listener in pairs:
        src, lst = np.asarray(source, dtype=float), np.asarray(listener, dtype=float)
        distance = float(np.linalg.norm(src - lst))
        gain = direct.directivity_gain(lst - src, emitter)
        attenuation = 1.0 / max(distance, CONFIG.min_distance_m)
        air = np.asarray([math.exp(-a * distance) for a in bands.AIR_ABSORPTION_NP_PER_M], dtype=float)
        occlusion, transmission, surface = 1.0, np.ones(6, dtype=float), None
        if distance > 1e-6:
            queries = (_lib.ACDirectQuery * 1)()
            queries[0] = direct.make_query(src, lst, CONFIG)
            record = direct.run_queries(None, TABLES, queries, 1, samples=32)[0]
            occlusion, index = float(record["occlusion"]), int(record["occlusion_surface"])
            surface = TABLES.names[index] if index >= 0 else None
            if occlusion < 1.0:
                transmission = np.asarray(record["transmission"], dtype=float)
        out.append({"distance_m": distance, "delay_s": distance / CONFIG.c, "distance_attenuation": attenuation,
                    "air_absorption": air, "occlusion": occlusion, "transmission": transmission,
                    "occlusion_surface": surface, "source_directivity_gain": gain,
                    "band_gains": {band: float(gain * attenuation * air[i] * (occlusion + (1.0 - occlusion) * transmission[i]))
                                   for i, band in enumerate(bands.FREQUENCY_BANDS)}})
    return out


@pytest.mark.parametrize("pairs", [1, 2, 3, 40])
def test_results_equal_the_single_pair(monkeypatch, pairs):
    monkeypatch.setattr(direct, "run_queries", answer)
    points = np.random.default_rng(pairs).uniform(0.0, 6.0, (pairs, 2, 3))
    if pairs > 2:
        points[1, 1] = points[1, 0]   # no query
    for got, want in zip(direct.direct_results(None, TABLES, list(points), CONFIG, "cardioid"), one_by_one(points)):
        assert got.keys() == want.keys()
        for key, value in want.items():
            if isinstance(value, np.ndarray):
                np.testing.assert_array_equal(got[key], value)
            else:
                assert got[key] == value and type(got[key]) is type(value), key


def test_one_pair_costs_no_more_than_its_formulas(monkeypatch):
    records = answer(None, TABLES, [direct.make_query(np.ones(3), 2.0 * np.ones(3), CONFIG)], 1, samples=1)
    monkeypatch.setattr(direct, "run_queries", lambda *args, **kw: records)
    pair = [(np.asarray([1.0, 2.0, 1.5]), np.asarray([3.0, 1.0, 1.2]))]

    def shortest(call, best=1.0):
        for _ in range(400):
            start = time.perf_counter()
            call()
            best = min(best, time.perf_counter() - start)
        return best

    batched, alone = [], []
    for _ in range(5):
        batched.append(shortest(lambda: direct.direct_results(None, TABLES, pair, CONFIG, "cardioid")))
        alone.append(shortest(lambda: one_by_one(pair)))
    assert min(batched) <= 1.5 * min(alone)
