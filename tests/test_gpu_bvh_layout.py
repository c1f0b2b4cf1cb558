"""The float32 traversal BVH's node layouts cull the same rays wherever the scene lies.

The binary layout holds centres and half extents, the four-wide one bounds; both are conservative, so every leaf size
and width must give the same hits and the same fixed-point sums, close to the origin and hundreds of metres away, where
float32 coordinates are coarse.
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import runtime, scene, workloads  # noqa: E402


@pytest.mark.parametrize("shift", [0.0, 60.0, 420.0, 2000.0])
def test_bvh_layouts_agree_far_from_the_origin(shift):
    w = workloads.apartment(21, rooms=6)
    spec = dict(w.spec)
    move = lambda p: [float(p[0]) + shift, float(p[1]) - shift]   # noqa: E731
    spec["corners"] = [tuple(move(c)) for c in spec["corners"]]
    spec["surface_segments"] = [dict(s, a=move(s["a"]), b=move(s["b"])) for s in spec["surface_segments"]]
    spec["objects"] = [dict(o, position=move(o["position"])) for o in spec["objects"]]
    arrays = scene.compile_scene(spec)
    src, lst = (np.asarray([*move(p), p[2]]) for p in (w.sources[0], w.listeners[0]))
    t = runtime.TraceSpec(source=src, listener=lst, num_rays=5000, num_bounces=30, num_bins=100, bin_duration=0.01,
                          speed_of_sound=343.0, max_path_length=343.0, direct_delay=0.01, use_bvh=True, seed=5)
    want = None
    for width, leaf in ((4, 1), (2, 1), (2, 2), (2, 8)):
        dev = runtime.DeviceScene(arrays, traversal="bvh", bvh_leaf=leaf, bvh_width=width)
        assert dev.bvh_width == width
        b = runtime.trace(dev, t, record_rays=True)
        torch.cuda.synchronize()
        got = [v.cpu().numpy() for v in (b.ray_surfaces, b.hit_counts, b.contrib_counts, b.echogram_fx,
                                         b.surface_energy_fx)]
        want = got if want is None else want
        for a, e in zip(got, want):
            np.testing.assert_array_equal(a, e)
        dev.close()
