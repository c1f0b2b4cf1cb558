"""A batch workspace of one job list serves every part of it.

Copies of the accumulators, which only few jobs of few scenes get, may make a part's best size larger than the whole
list's; the part is then traced without them.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import _lib, runtime, scene, workloads  # noqa: E402


@pytest.mark.parametrize("staged", [True, False])
@pytest.mark.parametrize("ambisonics", [False, True])
def test_a_part_of_the_list_fits_the_lists_workspace(staged, ambisonics):
    device, lib, keep = torch.device("cuda", 0), _lib.load(), []
    rooms = [workloads.shoebox(30 + k) for k in range(6)]
    scenes = [runtime.DeviceScene(scene.compile_scene(w.spec)) for w in rooms]
    specs = [runtime.TraceSpec(source=w.sources[0], listener=w.listeners[0], num_rays=40000, num_bounces=20, num_bins=40,
                               bin_duration=0.005, speed_of_sound=343.0, max_path_length=0.2 * 343.0, direct_delay=0.004,
                               use_bvh=True, render_ambisonics=ambisonics and k != 1, seed=k)
             for k, w in enumerate(rooms)]
    buffers = [runtime.TraceBuffers.allocate(s.num_surfaces, 40, device, ambisonics=ambisonics) for s in scenes]
    jobs = (_lib.ACJob * len(rooms))()
    for k in range(len(rooms)):
        jobs[k].scene = scenes[k].handle.value
        jobs[k].params = runtime.params_struct(specs[k], device, keep)
        jobs[k].outputs = buffers[k].outputs_struct()
    cfg, size = _lib.ACBatchConfig(), ctypes.c_size_t()
    _lib.check(lib.ac_batch_workspace_size(jobs, len(rooms), ctypes.byref(cfg), ctypes.byref(size)), "size")
    ws = torch.empty(size.value, dtype=torch.uint8, device=device)
    staging = torch.empty(size.value, dtype=torch.uint8, pin_memory=True) if staged else None
    stream = torch.cuda.current_stream(device)
    for part in (1, 2, 4, 6):   # one, two, four scenes (one of them without ambisonics: a launch of its own), all
        _lib.check(lib.ac_trace_batch(jobs, part, ctypes.byref(cfg), ctypes.c_void_p(ws.data_ptr()), ws.numel(),
                                      ctypes.c_void_p(staging.data_ptr() if staged else None),
                                      ctypes.c_void_p(stream.cuda_stream)), "ac_trace_batch")
        torch.cuda.synchronize()
        for k in range(part):
            want = runtime.trace(scenes[k], specs[k])
            torch.cuda.synchronize()
            for name in ("echogram_fx", "hit_counts", "contrib_counts", "surface_energy_fx"):
                np.testing.assert_array_equal(getattr(buffers[k], name).cpu().numpy(), getattr(want, name).cpu().numpy(),
                                              err_msg=f"{part} jobs, job {k}, {name}")
            if specs[k].render_ambisonics:
                np.testing.assert_array_equal(buffers[k].ambisonic_fx.cpu().numpy(), want.ambisonic_fx.cpu().numpy())
    rc = lib.ac_trace_batch(jobs, len(rooms), ctypes.byref(cfg), ctypes.c_void_p(ws.data_ptr()), 256, None,
                            ctypes.c_void_p(stream.cuda_stream))
    assert rc != 0   # too small for the tables themselves
    for s in scenes:
        s.close()
