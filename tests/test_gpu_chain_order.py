"""The order that chained kernels give by themselves: a slab top level that starts beside the
pyramid kernel, the level after it beside both, and frames queued one after the other without a
wait between them."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_slab import SLAB, frames_of
from test_gpu_stream_order import fresh_filters, oracle_states

pytestmark = pytest.mark.gpu

STAGE, STREAM, TILE = 0, 1, 2


@pytest.mark.parametrize("tuning", [(SLAB, 1), (SLAB, 0), (TILE, 0)])
def test_fresh_chained_filters_agree(cuda, tuning):
    fresh_filters(tuning, 300)


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("path", [STAGE, STREAM, TILE, SLAB])
@pytest.mark.parametrize("top", [TILE, SLAB])
@pytest.mark.parametrize("H,W,levels", [(96, 130, 2), (240, 320, 2), (333, 421, 3)])
def test_frames_queued_without_a_wait(cuda, H, W, levels, top, path, graphs):
    """Frames queued on one stream, every fourth on a new image and the others on the same one (so
    that a frame's kernels follow the last one's directly): the flow of each, copied on the same
    stream, and the last state of every level are the oracle's."""
    import flowfilter_b200 as ffb
    from test_gpu_stream_order import configure

    T, every = 24, 4
    clip = frames_of(H, W, T // every, H + levels)
    dev = [cuda.from_numpy(x).cuda() for x in clip]
    want = oracle_states([clip[t // every] for t in range(T)], levels, 3)
    f = ffb.PyramidalFlowFilter(H, W, levels)
    configure(f, levels)
    f.setGraphs(graphs)
    state = [(SLAB, 0)] * levels
    state[levels - 2], state[levels - 1] = (path, 0), (top, 0)
    f.setTuningState(state)
    flows = {}
    for t in range(T):
        if t % every == 0:
            f.loadImage(dev[t // every])
        f.computeAsync()
        if t % 5 == 2:
            flows[t] = f.flowTensor().clone()
    cuda.cuda.synchronize()
    for t, y in flows.items():
        assert np.array_equal(y.cpu().numpy(), want[t][0]), t
    got = [f.levelState(l, k) for l in range(levels) for k in (0, 2, 3 if l < levels - 1 else 1)]
    for i, (a, b) in enumerate(zip(got, want[-1])):
        assert np.array_equal(a, b), i
