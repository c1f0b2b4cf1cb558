"""Batch jobs with copies of their accumulators give the sums of the same job traced alone.

A small room's job gets copies up to 32 KB of accumulators (2 * 6 * bins words, five times that with ambisonics, and four
per surface); 48 bins with ambisonics and 300 without lie below that limit, 90 and 400 above it.  The sums are integers,
so there is no tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import runtime, scene, workloads  # noqa: E402

OUTPUTS = ("echogram_fx", "ambisonic_fx", "hit_counts", "contrib_counts", "surface_energy_fx", "echogram", "ambisonic",
           "surface_energy")


@pytest.mark.parametrize("room", ["shoebox", "u_room"])
@pytest.mark.parametrize("ambisonics,few,many", [(True, 48, 90), (False, 300, 400)])
@pytest.mark.parametrize("rays", [2048, 2049, 20011])
def test_copies_give_the_sums_of_a_single_trace(room, ambisonics, few, many, rays):
    w = workloads.shoebox(5) if room == "shoebox" else workloads.u_furnished(5, channels=1)
    device = torch.device("cuda", 0)
    dev = runtime.DeviceScene(scene.compile_scene(w.spec))
    words = lambda bins: 12 * bins * (5 if ambisonics else 1) + 4 * dev.num_surfaces   # noqa: E731
    assert 8 * words(few) <= 32 * 1024 < 8 * words(many)

    def spec(bins, seed):
        return runtime.TraceSpec(source=w.sources[0], listener=w.listeners[0], num_rays=rays, num_bounces=25,
                                 num_bins=bins, bin_duration=0.005, speed_of_sound=343.0, max_path_length=0.2 * 343.0,
                                 direct_delay=0.004, use_bvh=True, render_ambisonics=ambisonics, seed=seed)

    jobs = []
    for bins, seed in ((few, 9), (many, 9), (few, 10), (7, 11)):
        b = runtime.TraceBuffers.allocate(dev.num_surfaces, bins, device, ambisonics=ambisonics)
        for name in OUTPUTS:
            if getattr(b, name) is not None:
                getattr(b, name).fill_(-7)
        jobs.append((dev, spec(bins, seed), b))
    workspace = runtime.BatchWorkspace(device)
    for _ in range(2):   # the second launch finds the first one's sums in the workspace
        runtime.trace_batch(jobs, workspace)
    torch.cuda.synchronize()
    for k, (_, s, got) in enumerate(jobs):
        want = runtime.trace(dev, s)
        torch.cuda.synchronize()
        for name in OUTPUTS:
            if getattr(want, name) is not None:
                np.testing.assert_array_equal(getattr(got, name).cpu().numpy(), getattr(want, name).cpu().numpy(),
                                              err_msg=f"job {k}, {name}")
        np.testing.assert_array_equal(got.counters.cpu().numpy()[:4], want.counters.cpu().numpy()[:4])
        assert got.contrib_counts.sum().item() > 0
    dev.close()
