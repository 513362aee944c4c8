"""A batched step whose first phase streams its large levels and runs the others (small ones, and
ones beyond the streaming kernel's smoothing passes) by the slab kernel beside them, or by the
tile kernel where a pixel limit is set, against the streams alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (height, width, levels, gamma, smooth, maxflow, border): 8.3 M pixels of levels 0 in phase A
STREAMS = [(1080, 1920, 3, [5.0, 9.0, 20.0], [1, 2, 3], 4.0, 3)] * 4 + [
    (61, 77, 1, [4.0], [1], 6.0, 3), (5, 3, 1, [4.0], [2], 1.0, 0), (240, 321, 1, [8.0], [4], 4.0, 2),
    (200, 333, 3, [8.0, 8.0, 9.0], [6, 1, 2], 4.0, 40), (720, 1280, 1, [10.0], [5], 3.0, 3)]


@pytest.mark.parametrize("limit", [-1, 200000])
def test_levels_beside_match_streams_alone(cuda, limit):
    import flowfilter_b200 as ffb

    torch = cuda
    rng = np.random.default_rng(3)
    alone = [ffb.PyramidalFlowFilter(*s[:3]) for s in STREAMS]
    batch = ffb.BatchFlowFilter([s[:3] for s in STREAMS])
    batch.setTuning(limit)
    for i, s in enumerate(STREAMS):
        for f in (alone[i], batch.stream(i)):
            f.gamma = s[3] if s[2] > 1 else s[3][0]
            f.smoothIterations = s[4] if s[2] > 1 else s[4][0]
            f.maxflow, f.propagationBorder = s[5], s[6]
        alone[i].setFused(0)  # per-stage kernels
    assert batch.launches() == 4  # ingest with pyramid, a streaming launch per phase, the levels beside
    for t in range(4):
        frames = [torch.from_numpy(rng.integers(0, 256, s[:2], dtype=np.uint8)).cuda() for s in STREAMS]
        batch.step(batch.pack(frames))
        for f, x in zip(alone, frames):
            f.loadImage(x)
            f.computeAsync()
        for i, f in enumerate(alone):
            assert np.array_equal(batch.stream(i).getFlow(), f.getFlow()), (i, t)
            assert np.array_equal(batch.stream(i).getImage(), f.getImage()), (i, t)
