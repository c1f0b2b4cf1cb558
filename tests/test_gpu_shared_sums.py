"""A trace's sums do not depend on where they are accumulated.

Single traces with few bins add up in each block's shared memory, larger ones in global memory; batch jobs with few bins
use several copies of their accumulators.  All of them are the same integer sums, so the same rays binned at the same
bin length must give the same words, on both sides of each limit.
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import runtime, scene, workloads  # noqa: E402


def words(buffers, bins):
    out = {"echogram_fx": buffers.echogram_fx[:, :bins], "echogram": buffers.echogram[:, :bins],
           "hits": buffers.hit_counts, "contributions": buffers.contrib_counts, "energy_fx": buffers.surface_energy_fx,
           "energy": buffers.surface_energy, "counters": buffers.counters[:4]}
    if buffers.ambisonic_fx is not None:
        out["ambisonic_fx"] = buffers.ambisonic_fx[:, :, :bins]
        out["ambisonic"] = buffers.ambisonic[:, :, :bins]
    return {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("room", ["shoebox", "u_room"])
@pytest.mark.parametrize("ambisonics", [False, True])
@pytest.mark.parametrize("rays", [1, 700, 20011])
def test_sums_are_the_same_in_shared_memory_in_copies_and_in_the_outputs(room, ambisonics, rays):
    w = workloads.shoebox(5) if room == "shoebox" else workloads.u_furnished(5, channels=1)
    arrays = scene.compile_scene(w.spec)
    dev = runtime.DeviceScene(arrays)
    S = arrays.num_surfaces
    # the most bins whose accumulators fit 40 KB of shared memory (16 bytes per cell, 8 more per surface)
    limit = (40 * 1024 - 24 * S) // (16 * 6 * (4 if ambisonics else 1))

    def spec(bins, **kw):
        return runtime.TraceSpec(source=w.sources[0], listener=w.listeners[0], num_rays=rays, num_bounces=25,
                                 num_bins=bins, bin_duration=0.005, speed_of_sound=343.0, max_path_length=0.35 * 343.0,
                                 direct_delay=0.004, use_bvh=True, render_ambisonics=ambisonics, seed=9,
                                 energy_scale=2.0 ** 60, **kw)

    want = None
    for bins in (3000, limit + 1, limit, 100):    # every deposit falls into the first 100 bins of 5 ms
        b = runtime.trace(dev, spec(bins))
        torch.cuda.synchronize()
        got = words(b, 100)
        want = got if want is None else want
        for key, value in want.items():
            np.testing.assert_array_equal(got[key], value, err_msg=f"{key}, {bins} bins")
    assert want["contributions"].sum() > 0 or rays == 1
    # a batch of the same job, with copies of its accumulators (100 bins) and without (3000), beside another job
    for bins in (100, 3000):
        buffers = [runtime.TraceBuffers.allocate(S, n, torch.device("cuda", 0), ambisonics=ambisonics) for n in (bins, 37)]
        jobs = [(dev, spec(bins), buffers[0]), (dev, spec(37), buffers[1])]
        for buf in buffers:
            for t in (buf.echogram_fx, buf.hit_counts, buf.contrib_counts, buf.surface_energy_fx):
                t.fill_(-7)
        runtime.trace_batch(jobs, runtime.BatchWorkspace(torch.device("cuda", 0)))
        torch.cuda.synchronize()
        got = words(buffers[0], 100)
        for key, value in want.items():
            np.testing.assert_array_equal(got[key], value, err_msg=f"{key}, batch, {bins} bins")
    dev.close()
