"""The shared-memory subtree build at the sizes where its sorts change shape, array by array.

A thread holds two or four places, a warp's blocks have 64 or 128, and longer strides cross warps; a node of an odd
count leaves a place of padding in its block.  Each size runs with spread keys, with ties on every axis (the order then
comes from the parents' axes and the surface index) and with all boxes the same, at leaf sizes 1, 4 and 255.  Sizes
above 2,048 build subtrees below large nodes, whose order starts from their parents' axes.  The tree is the host
restatement's, bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from acoustic_agent_b200 import _lib, bvh  # noqa: E402

KEYS = ("bounds_min", "bounds_max", "start", "count", "escape", "primitives", "node_count", "leaf_count", "max_depth")


@pytest.mark.parametrize("kind", ["spread", "ties", "same"])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 31, 33, 63, 64, 65, 127, 129, 255, 257, 511, 513, 1023, 1024, 1025, 2047,
                               2048, 2050, 3001, 4099, 1 << 18])
def test_subtrees_equal_the_host_build(n, kind):
    rng = np.random.default_rng(n)
    if kind == "spread":
        lo = rng.normal(size=(n, 3)) * np.array([1e-3, 1.0, 1e3])
        size = rng.uniform(0.0, 1.0, (n, 3))
    elif kind == "ties":
        lo = rng.integers(-2, 3, (n, 3)).astype(np.float64) * 0.5
        size = np.zeros((n, 3))
        lo[rng.random((n, 3)) < 0.1] = -0.0
    else:
        lo, size = np.tile([1.0, -2.0, 0.0], (n, 1)), np.ones((n, 3))
    for leaf in (1, 4, 255):
        tree, want = bvh.build_bvh(lo, lo + size, leaf_size=leaf), _lib.build_bvh(lo, lo + size, leaf)
        for k in KEYS:
            np.testing.assert_array_equal(np.asarray(tree[k]), np.asarray(want[k]), err_msg=f"{k}, leaf {leaf}")
