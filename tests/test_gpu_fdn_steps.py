"""The FDN kernel at every step size and at the edges of its steps, against the oracle bit for bit.

The launch picks its step from the batch's shortest delay line and all-pass and from the number of impulses; each case
sits on one side of a limit of that rule.  The operation order is the reference's, so there is no tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import _lib, late_reverb, runtime  # noqa: E402


@pytest.mark.parametrize("shortest,allpass", [(128, oracle.FDN_ALLPASS), (287, oracle.FDN_ALLPASS),
                                              (288, oracle.FDN_ALLPASS), (575, oracle.FDN_ALLPASS),
                                              (576, oracle.FDN_ALLPASS), (900, (63, 341, 441, 556)),
                                              (900, (33, 64, 65, 4096)), (200, (33, 34, 35, 36))])
@pytest.mark.parametrize("crowd", [False, True])
def test_fdn_steps_match_the_oracle(shortest, allpass, crowd):
    design = late_reverb.design(16000, 7, (0.9, 0.8, 0.7, 0.6, 0.5, 0.4))
    delays = [shortest + 53 * l for l in range(16)]
    lengths = [(1, 0), (0, 40), (31, 1), (64, 0), (129, 62), (700, 300), (33, 1000)]   # (samples, preroll)
    count = torch.cuda.get_device_properties(0).multi_processor_count + 1 if crowd else len(lengths)
    outs, jobs = [], (_lib.ACFdnJob * count)()
    for k in range(count):
        n, pre = lengths[k % len(lengths)]
        outs.append(torch.full((max(n, 1),), float("nan"), dtype=torch.float64, device="cuda"))
        jobs[k].absorptive[:] = np.asarray(design.absorptive, dtype=np.float64).reshape(-1).tolist()
        jobs[k].tone[:] = np.asarray(design.tone, dtype=np.float64).reshape(-1).tolist()
        jobs[k].delays[:] = delays
        jobs[k].allpass_delays[:] = list(allpass)
        jobs[k].num_samples, jobs[k].preroll, jobs[k].out = n, pre, outs[k].data_ptr()
    runtime.fdn_impulse(jobs, count, runtime.FdnWorkspace(torch.device("cuda")))
    torch.cuda.synchronize()
    want = oracle.fdn_impulse(np.asarray(delays), design.absorptive, max(n + p for n, p in lengths),
                              np.asarray(allpass), design.tone)
    for k in range(count):
        n, pre = lengths[k % len(lengths)]
        np.testing.assert_array_equal(outs[k].cpu().numpy()[:n], want[pre:pre + n])
