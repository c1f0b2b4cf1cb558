"""The median search of large nodes on keys that leave all, half or none of a chunk's surfaces after a digit.

A pass lists a chunk's surfaces once at most half of them still share the median's digits, so the cases are keys whose
digits split a chunk exactly in half or one surface to either side of it, that part only in their last byte, or that
tie on one axis and part on the next; sizes have last chunks of one surface and of all 1,024.  The tree is the host
restatement's, bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import _lib, bvh  # noqa: E402

KEYS = ("bounds_min", "bounds_max", "start", "count", "escape", "primitives")


def keys(kind: str, n: int) -> np.ndarray:
    i = np.arange(n)
    lo = np.zeros((n, 3))
    if kind in ("half", "more", "fewer"):   # of every 1,024 surfaces: x = 1 but for 512, 511 or 513 of them
        other = {"half": 512, "more": 511, "fewer": 513}[kind]
        lo[:, 0] = np.where(i % 1024 < other, 1.0 + 2.0 ** -9 * (1 + i % 7), 1.0)
        lo[:, 1] = (i * 7919 % n) * 1e-7
    elif kind == "last":                    # neighbouring doubles
        lo[:, 0] = 1.0 + (i * 7919 % 251) * 2.0 ** -52
    else:                                   # the widest axis ties, the next ones decide
        lo[:, 0] = (i % 3) * 100.0
        lo[:, 1] = (i * 31 % 17) * 1.0
        lo[:, 2] = (i * 7919 % n) * 1e-3
    return lo


@pytest.mark.parametrize("kind", ["half", "more", "fewer", "last", "chain"])
@pytest.mark.parametrize("n", [2049, 3073, 4096, 5121, 70001])
def test_median_search_equals_the_host_build(n, kind):
    lo = keys(kind, n)
    tree, want = bvh.build_bvh(lo, lo, leaf_size=3), _lib.build_bvh(lo, lo, 3)
    for k in KEYS:
        np.testing.assert_array_equal(np.asarray(tree[k]), np.asarray(want[k]), err_msg=k)
