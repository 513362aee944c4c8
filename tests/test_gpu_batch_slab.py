"""Batched steps whose phases run the slab kernel: uneven sizes, iterations beyond the streaming
kernel's and levels of both classes, against the streams alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (height, width, levels, gamma, smooth, maxflow, border)
MIXES = [
    [(480, 640, 2, [10.0, 50.0], [4, 1], 4.0, 3), (61, 77, 1, [4.0], [1], 6.0, 3), (5, 3, 1, [4.0], [2], 1.0, 0)],
    [(500, 421, 3, [5.0, 9.0, 20.0], [1, 2, 6], 7.0, 2)] * 2 + [(130, 1283, 2, [8.0, 8.0], [3, 3], 3.0, 40)],
    [(33, 129, 2, [8.0, 8.0], [2, 2], 2.0, 3)],
]


@pytest.mark.parametrize("mix", range(len(MIXES)))
def test_slab_phases_match_streams_alone(cuda, mix):
    import flowfilter_b200 as ffb

    torch = cuda
    rng = np.random.default_rng(mix)
    streams = MIXES[mix]
    alone = [ffb.PyramidalFlowFilter(*s[:3]) for s in streams]
    batch = ffb.BatchFlowFilter([s[:3] for s in streams])
    for i, s in enumerate(streams):
        for f in (alone[i], batch.stream(i)):
            f.gamma = s[3] if s[2] > 1 else s[3][0]
            f.smoothIterations = s[4] if s[2] > 1 else s[4][0]
            f.maxflow, f.propagationBorder = s[5], s[6]
        alone[i].setFused(0)  # per-stage kernels
    for t in range(5):
        frames = [torch.from_numpy(rng.integers(0, 256, s[:2], dtype=np.uint8)).cuda() for s in streams]
        batch.step(batch.pack(frames))
        for f, x in zip(alone, frames):
            f.loadImage(x)
            f.computeAsync()
        for i, f in enumerate(alone):
            assert np.array_equal(batch.stream(i).getFlow(), f.getFlow()), (i, t)
            assert np.array_equal(batch.stream(i).getImage(), f.getImage()), (i, t)
