"""The float64 tracer's kernels give the same rays and sums.

A launch takes exact or sifted loops, the reference's walk or the sifted one, by its rays, its scenes' surfaces and its
kind; a caller's grid leaves the warps full.  The sums are integers and the arithmetic is the reference's, so there is no
tolerance.
"""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import runtime, scene, workloads  # noqa: E402


def arrays_of(boxes):
    if boxes == "apartment":
        return scene.compile_scene(workloads.apartment(21, rooms=2).spec)
    side = 6.0 if boxes <= 18 else 11.0
    corners = [(0.0, 0.0), (side, 0.0), (side, side - 1.0), (0.0, side - 1.0)]
    objects = workloads._place_boxes(np.random.default_rng(3), corners, boxes, [(1.0, 1.0), (4.0, 3.0)], side=(0.3, 1.2))
    spec = {"corners": corners, "height": 3.0, "materials": workloads._uniform_materials(), "objects": objects}
    return scene.compile_scene(workloads.with_surface_materials(spec, 4, scattering=(0.05, 0.5)))


def spec_of(rays, tree, **kw):
    return runtime.TraceSpec(source=(1.0, 1.0, 1.5), listener=(4.0, 3.0, 1.6), num_rays=rays, num_bounces=15, num_bins=60,
                             bin_duration=0.005, speed_of_sound=343.0, max_path_length=0.3 * 343.0, direct_delay=0.01,
                             use_bvh=tree, seed=7, precision="float64", **kw)


def words(b):
    return [v.cpu().numpy() for v in (b.echogram_fx, b.hit_counts, b.contrib_counts, b.surface_energy_fx, b.counters[:4])]


# surfaces on both sides of the rule's limits (12, 24 and 64) and rays on both sides of its limits per warp
@pytest.mark.parametrize("boxes", [0, 6, 8, 16, 20, 50, "apartment"])
@pytest.mark.parametrize("rays", [1000, 3000, 12000, 50000])
def test_every_launch_gives_the_same_sums(boxes, rays):
    dev = runtime.DeviceScene(arrays_of(boxes))
    want = {}
    for tree in (False, True):   # full warps on the caller's grid: another kernel or split than the launch's own
        want[tree] = words(runtime.trace(dev, spec_of(rays, tree, grid_blocks=300)))
        for a, e in zip(words(runtime.trace(dev, spec_of(rays, tree))), want[tree]):
            np.testing.assert_array_equal(a, e, err_msg=f"single, tree {tree}")
    other = spec_of(500, True, energy_scale=2.0 ** 40)
    for kinds in ((False, False), (True, True), (False, True)):
        jobs = [(dev, spec_of(rays, k), runtime.TraceBuffers.allocate(dev.num_surfaces, 60, torch.device("cuda", 0)))
                for k in kinds]
        jobs.append((dev, replace(other, use_bvh=kinds[1]),
                     runtime.TraceBuffers.allocate(dev.num_surfaces, 60, torch.device("cuda", 0))))
        runtime.trace_batch(jobs, runtime.BatchWorkspace(torch.device("cuda", 0)))
        torch.cuda.synchronize()
        for (_, s, b) in jobs[:2]:
            for a, e in zip(words(b), want[bool(s.use_bvh)]):
                np.testing.assert_array_equal(a, e, err_msg=f"batch {kinds}, tree {s.use_bvh}")
    dev.close()
