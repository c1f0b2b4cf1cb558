"""The block-pipelined crossover filter at the edges of its steps and of its block shapes.

Every sample is compared with the oracle's band synthesis bit for bit (the filter keeps the reference's operation
order, so there is no tolerance): signals shorter than, equal to and just past a step of 32 or 64 samples, batches that
fill the wide blocks unevenly, and batches on both sides of the rule that picks the block shape.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import _lib, bands, late_reverb, runtime  # noqa: E402

FS = 16000
LENGTHS = (1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 257, 300, 511, 640)


@pytest.mark.parametrize("count_of", [lambda sms: 1, lambda sms: 16, lambda sms: 2 * sms, lambda sms: 2 * sms + 1,
                                      lambda sms: 2 * sms + 3])
def test_filter_matches_the_oracle_at_step_edges(count_of):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count = count_of(sms)
    rng = np.random.default_rng(count)
    dev = torch.device("cuda", 0)
    jobs, host = [], []
    for k in range(count):
        n = LENGTHS[(k * 7) % len(LENGTHS)] if count > 1 else 640
        echo = rng.uniform(0.0, 1e-3, (6, n)).astype(np.float32)     # one sample per bin: any length
        white = rng.uniform(-1.0, 1.0, n)
        air = bands.air_gain_table(n, 1, FS, 0.004, 343.0)
        out = torch.full((6, n), float("nan"), dtype=torch.float32, device=dev)
        jobs.append(runtime.SynthJob(torch.as_tensor(echo, device=dev), out, FS, 1.0 / FS, 1, 0.004, 343.0, "reference",
                                     torch.as_tensor(white, device=dev), torch.as_tensor(air, device=dev)))
        host.append((echo, white))
    runtime.synthesize_batch(jobs, runtime.SynthBatchWorkspace(dev))
    torch.cuda.synchronize()
    for job, (echo, white) in zip(jobs, host):
        want = oracle.synthesize(echo, fs=FS, bin_dur=1.0 / FS, direct_delay=0.004, c=343.0, white=white)
        np.testing.assert_array_equal(job.out.cpu().numpy(), want)


@pytest.mark.parametrize("rirs", [1, 2, 299])
def test_single_shape_synthesis_equals_the_ragged_one(rirs):
    rng = np.random.default_rng(rirs)
    dev = torch.device("cuda", 0)
    bins, bin_s = 5, 0.0021                                          # 34 samples per bin, 170 samples
    echo = torch.as_tensor(rng.uniform(0.0, 1e-3, (rirs, 6, bins)).astype(np.float32), device=dev)
    n = bins * bands.samples_per_bin(bin_s, FS)
    delays = torch.full((rirs,), 0.003, dtype=torch.float64, device=dev)
    p = runtime.synth_params(rirs, bins, bin_s, FS, 343.0, rng_mode="philox", seed=9, direct_delays=delays)
    one = runtime.synthesize(echo, p, runtime.SynthWorkspace(dev))
    out = torch.empty(rirs, 6, n, dtype=torch.float32, device=dev)
    runtime.synthesize_batch([runtime.SynthJob(echo[k], out[k], FS, bin_s, 9, 0.003) for k in range(rirs)],
                             runtime.SynthBatchWorkspace(dev))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(one.cpu().numpy(), out.cpu().numpy())


def test_late_tail_band_split_is_the_same_in_wide_blocks():
    """Tails on both sides of the block-shape rule: a large ragged batch equals each of its tails alone."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count = 2 * sms + 5
    rng = np.random.default_rng(4)
    dev = torch.device("cuda", 0)
    lengths = [200 + 37 * (k % 5) for k in range(count)]
    traced = [torch.as_tensor(rng.normal(0.0, 1e-2, (6, n)), device=dev) for n in lengths]

    def jobs(indices):
        return [late_reverb.LateReverbJob(traced[k], torch.empty(6, lengths[k], device=dev),
                                          torch.empty(6, lengths[k], device=dev), FS, k % 3,
                                          (0.5, 0.5, 0.4, 0.4, 0.3, 0.3), 0.001, 0.006, 0.25) for k in indices]

    r = late_reverb.LateReverbRenderer(0)
    batch = jobs(range(count))
    stats, _, _ = r.render(batch)
    picks = [0, 1, 5, 6, count // 2, count - 2, count - 1]
    alone = jobs(picks)
    for k, job in zip(picks, alone):
        s, _, _ = r.render([job])
        torch.cuda.synchronize()
        np.testing.assert_array_equal(batch[k].out.cpu().numpy(), job.out.cpu().numpy())
        np.testing.assert_array_equal(batch[k].component.cpu().numpy(), job.component.cpu().numpy())
        np.testing.assert_array_equal(stats[k].cpu().numpy()[:, :_lib.AC_LATE_STATS], s[0].cpu().numpy())
