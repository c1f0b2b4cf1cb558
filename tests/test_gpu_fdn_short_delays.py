"""FDN designs with short delay lines: the short steps against the oracle, and their time against long delays.

A step of 16 samples needs delays of 144, one of 14 meets the shortest that is accepted.  The operation order is the
reference's, so there is no tolerance.  The time per sample of short steps may be at most 1.8 times that of long ones
(1.6 is 79 cycles, a network with a barrier every 32 samples, against 49; a step of 8 took 4 times).
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import _lib, late_reverb, runtime  # noqa: E402


def batch(shortest, allpass, lengths):
    design = late_reverb.design(16000, 7, (0.9, 0.8, 0.7, 0.6, 0.5, 0.4))
    delays = [shortest + 53 * l for l in range(16)]
    outs = [torch.full((max(n, 1),), float("nan"), dtype=torch.float64, device="cuda") for n, _ in lengths]
    jobs = (_lib.ACFdnJob * len(lengths))()
    for job, out, (n, preroll) in zip(jobs, outs, lengths):
        job.absorptive[:] = np.asarray(design.absorptive, dtype=np.float64).reshape(-1).tolist()
        job.tone[:] = np.asarray(design.tone, dtype=np.float64).reshape(-1).tolist()
        job.delays[:] = delays
        job.allpass_delays[:] = list(allpass)
        job.num_samples, job.preroll, job.out = n, preroll, out.data_ptr()
    return design, np.asarray(delays), jobs, outs


@pytest.mark.parametrize("shortest,allpass", [(128, (33, 34, 35, 36)), (143, oracle.FDN_ALLPASS),
                                              (144, oracle.FDN_ALLPASS), (144, (33, 64, 65, 4096)),
                                              (169, oracle.FDN_ALLPASS), (287, (40, 41, 42, 43))])
def test_short_steps_match_the_oracle(shortest, allpass):
    lengths = [(n, p) for p in (0, 5) for n in (1, 13, 14, 15, 16, 17, 27, 28, 29, 32, 143, 144, 911)]
    design, delays, jobs, outs = batch(shortest, allpass, lengths)
    runtime.fdn_impulse(jobs, len(lengths), runtime.FdnWorkspace(torch.device("cuda")))
    torch.cuda.synchronize()
    want = oracle.fdn_impulse(delays, design.absorptive, 1000, np.asarray(allpass), design.tone)
    for (n, preroll), out in zip(lengths, outs):
        np.testing.assert_array_equal(out.cpu().numpy(), want[preroll:preroll + n])


@pytest.mark.parametrize("impulses", [8, 444])
def test_short_delays_cost_little_more_than_long_ones(impulses):
    workspace = runtime.FdnWorkspace(torch.device("cuda"))

    def milliseconds(shortest):
        _, _, jobs, outs = batch(shortest, oracle.FDN_ALLPASS, [(16000, 0)] * impulses)
        times = []
        for _ in range(8):
            start, stop = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            runtime.fdn_impulse(jobs, impulses, workspace)
            stop.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(stop))
        return min(times[3:])

    reference = milliseconds(576)
    for shortest in (128, 144, 287):
        assert milliseconds(shortest) <= 1.8 * reference, shortest
