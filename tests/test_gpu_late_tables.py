"""The late tails' job tables take what a caller's own designs say, and refuse what does not fit their fields."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import late_reverb  # noqa: E402

FS, N = 16000, 4000


class Delayed(late_reverb.FdnDesign):
    """A network that is heard from its first sample on."""

    @property
    def preroll(self) -> int:
        return 0


def job(seed=3, **kw):
    traced = torch.zeros((6, N), dtype=torch.float64, device="cuda")
    traced[:, :2000] = 1e-3
    out = torch.zeros((6, N), dtype=torch.float32, device="cuda")
    return late_reverb.LateReverbJob(traced, out, torch.zeros_like(out), FS, seed, [0.5] * 6, kw.pop("bin", 0.001),
                                     kw.pop("transition", 0.1), **kw)


def test_a_designs_own_preroll_counts():
    renderer = late_reverb.LateReverbRenderer(0)
    d = late_reverb.design(FS, 3, [0.5] * 6)
    own = Delayed(d.delays, d.absorptive, d.tone, d.allpass)
    first, second, third = job(), job(), job()
    renderer.render([first, second], designs=[own, d])
    renderer.render([third])
    torch.cuda.synchronize()
    np.testing.assert_array_equal(second.component.cpu().numpy(), third.component.cpu().numpy())
    assert not torch.equal(first.component, second.component)


@pytest.mark.parametrize("field,value", [("delays", np.asarray([211])), ("absorptive", np.ones((1, 1, 1))),
                                         ("tone", np.ones((1, 1))), ("allpass", (225,))])
def test_fields_of_another_size_are_refused(field, value):
    renderer = late_reverb.LateReverbRenderer(0)
    d = replace(late_reverb.design(FS, 3, [0.5] * 6), **{field: value})
    with pytest.raises(ValueError):
        renderer.render([job(), job()], designs=[d, d])


def test_an_energy_bin_of_a_day_is_longer_than_the_signal():
    renderer = late_reverb.LateReverbRenderer(0)
    want, got = job(bin=1.0), job(bin=2.0 ** 32 / FS + 1.0)
    renderer.render([want])
    renderer.render([got])
    torch.cuda.synchronize()
    np.testing.assert_array_equal(got.out.cpu().numpy(), want.out.cpu().numpy())
