"""A room of at most 16 walls and boxes that AUTO gives a tree takes every stack depth.

AUTO scans such a room in a launch whose stack is too shallow for its tree, so a depth chosen for the launch's other
scenes, or for none, never refuses it.  Scan and tree find the same hits, so there is no tolerance.
"""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import runtime, scene, workloads  # noqa: E402

DEVICE = torch.device("cuda", 0) if torch.cuda.is_available() else None


def room(boxes):
    corners = [(0.0, 0.0), (6.0, 0.0), (6.0, 5.0), (0.0, 5.0)]
    objects = workloads._place_boxes(np.random.default_rng(3), corners, boxes, [(1.0, 1.0), (4.0, 3.0)], side=(0.3, 1.2))
    spec = {"corners": corners, "height": 3.0, "materials": workloads._uniform_materials(), "objects": objects}
    return scene.compile_scene(workloads.with_surface_materials(spec, 4, scattering=(0.05, 0.5)))


def spec(**kw):
    return runtime.TraceSpec(source=(1.0, 1.0, 1.5), listener=(4.0, 3.0, 1.6), num_rays=3000, num_bounces=40, num_bins=100,
                             bin_duration=0.01, speed_of_sound=343.0, max_path_length=343.0, direct_delay=0.01,
                             use_bvh=True, seed=7, **kw)


def words(b):
    return [v.cpu().numpy() for v in (b.echogram_fx, b.hit_counts, b.contrib_counts, b.surface_energy_fx, b.counters[:4])]


def assert_same(got, want, what):
    for a, e in zip(words(got), want):
        np.testing.assert_array_equal(a, e, err_msg=str(what))


def allocate(dev):
    return runtime.TraceBuffers.allocate(dev.num_surfaces, 100, DEVICE)


@pytest.mark.parametrize("boxes", [1, 12])
def test_every_depth_traces_the_room_as_the_scan_does(boxes):
    arrays = room(boxes)
    scan = runtime.DeviceScene(arrays, traversal="scan")
    want = words(runtime.trace(scan, spec()))
    dev = runtime.DeviceScene(arrays)
    assert dev.traversal == "hybrid" and np.count_nonzero(np.asarray(arrays.arrays["kinds"]) != 1) <= 16
    for entries in (1, dev.bvh_stack_need - 1, dev.bvh_stack_need, runtime.MAX_STACK_ENTRIES):
        assert_same(runtime.trace(dev, spec(stack_entries=entries)), want, ("single", entries))
        buffers = [allocate(dev), allocate(dev)]
        runtime.trace_batch([(dev, spec(), b) for b in buffers], runtime.BatchWorkspace(DEVICE), stack_entries=entries)
        for b in buffers:
            assert_same(b, want, ("batch", entries))
        service = runtime.TraceService(0, capacity=64, stack_entries=entries)
        b = allocate(dev)
        waiting = set(service.submit([(dev, spec(), b)]))
        while waiting:
            waiting.difference_update(service.poll())
        assert_same(b, want, ("service", entries))
        service.close()
        chosen = runtime.DeviceScene(arrays, stack_entries=entries)   # a depth chosen for the scene
        assert_same(runtime.trace(chosen, spec()), want, ("scene", entries))
        chosen.close()
    for bad in (-1, runtime.MAX_STACK_ENTRIES + 1):
        with pytest.raises(ValueError, match="stack_entries"):
            runtime.trace(dev, spec(stack_entries=bad))
    scan.close()
    dev.close()


def test_a_tree_that_the_caller_chose_still_needs_its_depth():
    dev = runtime.DeviceScene(room(12), traversal="hybrid")
    with pytest.raises(ValueError, match="stack_entries"):
        runtime.trace(dev, spec(stack_entries=dev.bvh_stack_need - 1))
    dev.close()


def test_the_room_leaves_the_depth_of_a_launch_to_its_other_scenes():
    w = workloads.apartment(21, rooms=2)
    house = runtime.DeviceScene(scene.compile_scene(w.spec), traversal="bvh")
    need = house.bvh_stack_need
    house.close()
    house = runtime.DeviceScene(scene.compile_scene(w.spec), traversal="bvh", stack_entries=need)
    small = runtime.DeviceScene(room(12))
    assert runtime.launch_stack_entries([house, small]) == need
    jobs = [(house, replace(spec(), source=w.sources[0], listener=w.listeners[0]), allocate(house)),
            (small, spec(), allocate(small))]
    runtime.trace_batch(jobs, runtime.BatchWorkspace(DEVICE))
    for dev, s, b in jobs:
        assert_same(b, words(runtime.trace(dev, s)), dev.traversal)
    house.close()
    small.close()
