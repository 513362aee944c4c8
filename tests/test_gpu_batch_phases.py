"""Batches on both sides of the pixel line between slab and streaming phases, which depends on
their smoothing iterations: every stream's results are those of the stream alone."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(9, 1), (11, 1), (17, 2), (19, 2), (26, 3), (27, 3), (27, 5)])
def test_streams_around_the_line(cuda, n, S):
    """n streams of 640x480 with 2 levels: n * 0.307 M pixels in phase B, against 3, 5.5 and 8 M."""
    import flowfilter_b200 as ffb

    b = ffb.BatchFlowFilter([(480, 640, 2)] * n)
    alone = ffb.PyramidalFlowFilter(480, 640, 2)
    for f in [alone] + [b.stream(i) for i in range(n)]:
        f.maxflow, f.gamma, f.smoothIterations = 4.0, [10.0, 40.0], [S, 2]
    frames = cuda.from_numpy(np.random.default_rng(n).integers(0, 256, (3, 480, 640), dtype=np.uint8)).cuda()
    for x in frames:
        b.step(b.pack([x] * n))
        alone.loadImage(x)
        alone.computeAsync()
    flow, image = alone.flowTensor(), alone.imageTensor()
    for i in range(n):
        assert cuda.equal(b.stream(i).flowTensor(), flow) and cuda.equal(b.stream(i).imageTensor(), image), i
