"""The boxes' tree of a room culls conservatively for rays that start on the room's far walls.

A node test's roundings grow with the coordinates of the ray as well as the box's, so boxes near the coordinate origin in
a hall of kilometres need a pad for the hall.  The tree over walls and boxes is padded for both; for rays from one end of
the hall that graze the boxes' edges the hits must agree.
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import runtime, scene, workloads  # noqa: E402
from oracle import oracle  # noqa: E402

RAYS, BOUNCES = 400_000, 2


@pytest.mark.parametrize("reach", [300.0, 4000.0, 16000.0])
def test_boxes_near_the_origin_of_a_long_hall(reach):
    corners = [(-reach, -reach), (reach, -reach), (reach, reach), (-reach, reach)]
    objects = [{"type": "shelf", "position": [4.0 * (k % 12) - 23.0, 7.0 * (k // 12) - 41.0], "rotation": 0.0,
                "size": [0.4 + 0.01 * k, 0.6, 60.0], "z": 30.0} for k in range(144)]
    spec = {"corners": corners, "height": 60.0, "materials": workloads._uniform_materials(), "objects": objects}
    arrays = scene.compile_scene(workloads.with_surface_materials(spec, 4, scattering=(0.05, 0.5)))
    rng = np.random.default_rng(int(reach))
    listener = np.asarray([0.95 * reach, -0.4 * reach, 25.0])
    a = arrays.arrays
    boxes = np.nonzero(np.asarray(a["kinds"]) == 2)[0]
    pick = rng.choice(boxes, RAYS)
    edge = np.asarray(a["box_center"])[pick] + rng.choice([-1.0, 1.0], (RAYS, 2)) * np.asarray(a["box_half"])[pick]
    aim = np.c_[edge + rng.normal(0.0, 1e-7 * reach, (RAYS, 2)), rng.uniform(5.0, 55.0, RAYS)] - listener
    directions = (aim / np.linalg.norm(aim, axis=1, keepdims=True)).astype(np.float32)
    _, bank, _, _ = oracle.workspace(1, 0, 0)
    workspace = (torch.as_tensor(directions, device="cuda"), torch.ones((BOUNCES, RAYS), device="cuda"),
                 torch.zeros((BOUNCES, RAYS), dtype=torch.int32, device="cuda"))   # specular reflections
    want = None
    for traversal in ("bvh", "hybrid"):
        dev = runtime.DeviceScene(arrays, traversal=traversal)
        assert dev.traversal == traversal
        b = runtime.trace(dev, runtime.TraceSpec(
            source=(0.3 * reach, 0.2 * reach, 30.0), listener=listener, num_rays=RAYS, num_bounces=BOUNCES, num_bins=10,
            bin_duration=1.0, speed_of_sound=343.0, max_path_length=1e7, direct_delay=0.1, use_bvh=True,
            rng="reference", seed=5), record_rays=True, workspace=workspace)
        torch.cuda.synchronize()
        got = b.ray_surfaces.cpu().numpy()
        assert np.isin(got, boxes).sum() > RAYS // 4
        want = got if want is None else want
        np.testing.assert_array_equal(got, want)
        dev.close()
