"""Batched steps queued on alternating streams without a wait: each follows the one before."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STREAMS = [(480, 640, 2), (61, 77, 1), (333, 500, 3), (720, 1280, 3)]


def alone_and_batch(ffb):
    alone, batch = [ffb.PyramidalFlowFilter(*s) for s in STREAMS], ffb.BatchFlowFilter(STREAMS)
    for i, (_, _, levels) in enumerate(STREAMS):
        for f in (alone[i], batch.stream(i)):
            f.gamma = [10.0, 20.0, 40.0][:levels] if levels > 1 else 10.0
            f.smoothIterations = [2, 1, 3][:levels] if levels > 1 else 2
            f.maxflow = 4.0
    return alone, batch


@pytest.mark.parametrize("limit", [-1, 200000])
def test_steps_on_alternating_streams(cuda, limit):
    import flowfilter_b200 as ffb

    T = 24
    alone, batch = alone_and_batch(ffb)
    batch.setTuning(limit)
    rng = np.random.default_rng(8)
    frames = [[cuda.from_numpy(rng.integers(0, 256, s[:2], dtype=np.uint8)).cuda() for s in STREAMS] for _ in range(4)]
    packed = [batch.pack(x) for x in frames]
    sides = [cuda.cuda.Stream() for _ in range(3)]
    cuda.cuda.synchronize()
    for t in range(T):
        batch.step(packed[t % 4], sides[t % 3])
    cuda.cuda.synchronize()
    for i, f in enumerate(alone):
        for t in range(T):
            f.loadImage(frames[t % 4][i])
            f.computeAsync()
        assert np.array_equal(batch.stream(i).getFlow(), f.getFlow()), i
        assert np.array_equal(batch.stream(i).getImage(), f.getImage()), i
