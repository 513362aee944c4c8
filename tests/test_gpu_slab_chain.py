"""A slab top level starts beside the pyramid kernel before it, and the level after it beside
both: frames issued back to back, with every kernel the level after it may run, end in the
per-stage kernels' states, bit for bit."""

from __future__ import annotations

import pytest

from test_gpu_slab import frames_of, same, states

pytestmark = pytest.mark.gpu

STAGE, STREAM, TILE, SLAB = 0, 1, 2, 3


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("path", [STAGE, STREAM, TILE, SLAB])
@pytest.mark.parametrize("H,W,levels", [(96, 130, 2), (480, 640, 2), (400, 500, 3), (333, 421, 4)])
def test_back_to_back_frames(cuda, H, W, levels, path, graphs):
    import flowfilter_b200 as ffb

    clip = [cuda.from_numpy(x).cuda() for x in frames_of(H, W, 6, H + levels)]
    out = []
    for tuned in (False, True):
        f = ffb.PyramidalFlowFilter(H, W, levels)
        f.maxflow = 4.0
        f.gamma = [8.0, 20.0, 30.0, 40.0][:levels]
        f.smoothIterations = [1, 2, 1, 2][:levels]
        f.setGraphs(graphs)
        f.setTuningState([(STAGE, 0)] * levels)
        if tuned:
            state = [(SLAB, 0)] * levels
            state[levels - 2] = (path, 0)
            f.setTuningState(state)
        for t in range(30):
            f.loadImage(clip[t % len(clip)])
            f.compute()
        out.append(states(f, levels))
    assert same(*out)
