"""Levels of more rows than a 32-bit product of row and shared-memory row bytes holds: the slab
kernel against the streaming kernel."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_slab_of_many_rows(cuda):
    import flowfilter_b200 as ffb

    H, W = 1_800_001, 5  # 2,048 bytes a row of a top level: 2^31 at 1,048,576 rows, 2^32 at 2,097,152
    rng = np.random.default_rng(1)
    frames = rng.integers(0, 256, (2, H, W), dtype=np.uint8)
    out = []
    for path in (1, 3):
        f = ffb.FlowFilter(H, W)
        f.maxflow, f.gamma, f.smoothIterations = 2.0, 5.0, 1
        f.setTuningState([(path, 0)])
        assert ("fused" if path == 1 else "slab") in f.tuning()
        for x in frames:
            f.loadImage(x)
            f.compute()
        out.append((f.getFlow(), f.getImage()))
        del f
    for a, b in zip(*out):
        assert np.array_equal(a, b)
