"""The float64 kernel's quick tests never change a ray: hits and counts equal the oracle's.

Quotients by approximate reciprocals settle only what is clear, so the cases are those that are not: directions along
the axes and almost along them, rays at wall ends, box edges, the floor's outline and the ceiling's rim, few rays (a
warp's lanes partly unused) and more than one warp's worth, BVH walk and linear loop.  The reference's operations decide
each ray, so the hit sequences are equal; the tolerance on the sums is that of the fixed-point words (1e-9 relative).
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import runtime, scene, workloads  # noqa: E402
from oracle import oracle  # noqa: E402

BOUNCES = 12


def directions(arrays, listener, count: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    axes = np.concatenate([np.eye(3), -np.eye(3)])
    tilted = axes + 10.0 ** rng.uniform(-17, -2, (6, 1)) * rng.choice([-1.0, 1.0], (6, 3))
    low, high = np.asarray(arrays["bvh_bounds_min"], float), np.asarray(arrays["bvh_bounds_max"], float)
    pick = rng.integers(0, low.shape[0], count)
    corner = np.where(rng.integers(0, 2, (count, 3)) == 1, high[pick], low[pick])
    aimed = corner - np.asarray(listener, float) + rng.choice([0.0, 1e-9, -1e-6, 1e-3], (count, 1))
    free = rng.normal(size=(count, 3))
    d = np.concatenate([axes, tilted, aimed, free])
    d = d[np.linalg.norm(d, axis=1) > 1e-6]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(d[rng.permutation(len(d))[:count]])


@pytest.mark.parametrize("use_bvh", [True, False])
@pytest.mark.parametrize("room", ["shoebox", "u_furnished", "apartment"])
@pytest.mark.parametrize("rays", [1, 33, 700])
def test_float64_hits_equal_the_oracle(room, use_bvh, rays):
    w = {"shoebox": lambda: workloads.shoebox(3), "u_furnished": lambda: workloads.u_furnished(3, channels=1),
         "apartment": lambda: workloads.apartment(3, rooms=6)}[room]()
    compiled = scene.compile_scene(w.spec)
    arrays = compiled.arrays
    src, lst = np.asarray(w.sources[0], float), np.asarray(w.listeners[0], float)
    rng = np.random.default_rng(rays)
    _, bank, _, _ = oracle.workspace(1, 0, 0)
    d = directions(arrays, lst, rays, 100 + rays)
    u = rng.uniform(size=(BOUNCES, rays))
    idx = rng.integers(0, bank.shape[0], (BOUNCES, rays)).astype(np.int32)
    common = dict(num_bins=60, c=343.0)
    want = oracle.trace(arrays, source=src, listener=lst, directions=d, diffuse_bank=bank, diffuse_random=u,
                        diffuse_indices=idx, bin_dur=0.01, max_path_len=200.0, direct_delay=0.004, use_bvh=use_bvh,
                        record_rays=True, **common)
    spec = runtime.TraceSpec(source=src, listener=lst, num_rays=rays, num_bounces=BOUNCES, num_bins=60,
                             bin_duration=0.01, speed_of_sound=343.0, max_path_length=200.0, direct_delay=0.004,
                             use_bvh=use_bvh, precision="float64", rng="reference", seed=1)
    dev = runtime.DeviceScene(compiled)
    cuda = tuple(torch.as_tensor(v, device="cuda").contiguous() for v in (d, u, idx))
    b = runtime.trace(dev, spec, record_rays=True, workspace=cuda)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(b.ray_surfaces.cpu().numpy(), want["ray_surfaces"])
    np.testing.assert_array_equal(b.hit_counts.cpu().numpy(), want["hit_counts"])
    np.testing.assert_array_equal(b.contrib_counts.cpu().numpy(), want["contrib_counts"])
    np.testing.assert_allclose(runtime.fixed_to_float64(b.echogram_fx, b.scale.value), want["echogram"], rtol=1e-9,
                               atol=1e-12 * float(np.max(want["echogram"])))
    dev.close()
