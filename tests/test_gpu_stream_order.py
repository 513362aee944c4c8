"""The filters' own buffers are cleared and filled in the order of the streams that use them,
whatever the default stream is doing; and the same frames give the same states in fresh filters."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from test_gpu_slab import frames_of

pytestmark = pytest.mark.gpu

BUSY = 60_000_000  # clock cycles the default stream spins: about 30 ms


def configure(f, levels, oracle=False):
    gamma, smooth = [8.0, 20.0, 30.0][:levels], [3, 1, 2][:levels]
    if oracle:
        f.set_gammas(gamma)
        f.set_smooths(smooth)
        f.set_max_flow(2.0)
        f.set_propagation_border(3)
    else:
        f.gamma, f.smoothIterations, f.maxflow, f.propagationBorder = gamma, smooth, 2.0, 3


def oracle_states(clip, levels, border):
    f = O.Filter.pyramidal(*clip[0].shape, levels)
    configure(f, levels, True)
    f.set_propagation_border(border)
    out = []
    for x in clip:
        f.load(x)
        f.compute()
        out.append([f.level_state(l, k) for l in range(levels) for k in (0, 2, 3 if l < levels - 1 else 1)])
    return out


@pytest.mark.parametrize("graphs", [False, True])
def test_scratch_is_cleared_before_the_frame_that_makes_it(cuda, graphs):
    """Per-stage levels allocate their scratch in their first frame: with the default stream
    busy, frames on another stream still end in the oracle's state."""
    import flowfilter_b200 as ffb

    H, W, levels, T = 120, 161, 3, 40
    clip = frames_of(H, W, T, 2)
    dev = [cuda.from_numpy(x).cuda() for x in clip]
    want = oracle_states(clip, levels, 3)[-1]
    side = cuda.cuda.Stream()
    f = ffb.PyramidalFlowFilter(H, W, levels)
    configure(f, levels)
    f.setGraphs(graphs)
    f.setTuningState([(0, 0)] * levels)
    cuda.cuda.synchronize()
    cuda.cuda._sleep(BUSY)
    with cuda.cuda.stream(side):
        for x in dev:
            f.loadImage(x)
            f.computeAsync()
    cuda.cuda.synchronize()
    got = [f.levelState(l, k) for l in range(levels) for k in (0, 2, 3 if l < levels - 1 else 1)]
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_staging_images_are_cleared_before_the_upload(cuda):
    """The pipelined host path makes its staging images in its first call: with the default
    stream busy, every frame's flow is that of the blocking loop."""
    import flowfilter_b200 as ffb

    H, W, levels, T = 120, 161, 2, 30
    clip = frames_of(H, W, T, 3)
    flows = []
    for pipelined in (False, True):
        f = ffb.PyramidalFlowFilter(H, W, levels)
        configure(f, levels)
        out = [cuda.zeros((H, W, 2)).pin_memory().numpy() for _ in clip]
        side = cuda.cuda.Stream()
        cuda.cuda.synchronize()
        if pipelined:
            pinned = [cuda.from_numpy(x).pin_memory().numpy() for x in clip]
            cuda.cuda.synchronize()
            cuda.cuda._sleep(BUSY)
            for x, y in zip(pinned, out):
                f.processAsync(x, y, side)
            f.synchronize()
        else:
            for x, y in zip(clip, out):
                f.loadImage(x)
                f.compute()
                f.getFlow(y)
        cuda.cuda.synchronize()
        flows.append([y.copy() for y in out])
    for t, (a, b) in enumerate(zip(*flows)):
        assert np.array_equal(a, b), t


def fresh_filters(tuning, n):
    """The first frames of n fresh filters, whose scratch, pyramid and top level are all made in
    the same few microseconds: every state field has to equal the oracle's in each of them."""
    import flowfilter_b200 as ffb

    H, W, levels = 100, 227, 2
    clip = frames_of(H, W, 2, 5)
    want = oracle_states(clip, levels, 40)
    names = [(l, k) for l in range(levels) for k in (0, 2, 3 if l < levels - 1 else 1)]
    for i in range(n):
        f = ffb.PyramidalFlowFilter(H, W, levels)
        configure(f, levels)
        f.propagationBorder = 40
        f.setTuningState([tuning] * levels)
        for t, x in enumerate(clip):
            f.loadImage(x)
            f.compute()
            for (l, k), w in zip(names, want[t]):
                got = f.levelState(l, k)
                if not np.array_equal(got, w):
                    rows = np.unique(np.nonzero(got != w)[0])
                    pytest.fail(f"filter {i}, frame {t}: level {l} field {k} differs in {len(rows)} rows: {rows[:8]}")


def test_fresh_per_stage_filters_agree(cuda):
    fresh_filters((0, 0), 300)
