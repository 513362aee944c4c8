"""Stage functions queued one after the other, each reading what the one before has just
written: no result is that of an earlier pass over the same buffers."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from test_gpu_slab import frames_of

pytestmark = pytest.mark.gpu

H, W, ROUNDS = 300, 420, 60


@pytest.mark.parametrize("dtype", ["u8", "f32"])
def test_pyramid_model_update_smooth(cuda, dtype):
    from flowfilter_b200 import stages

    clip = frames_of(H, W, 4, 9)
    if dtype == "f32":
        clip = [x.astype(np.float32) / 255 for x in clip]
    dev = [cuda.from_numpy(x).cuda() for x in clip]
    flow = cuda.randn((H // 2, W // 2, 2), generator=cuda.Generator(device="cuda").manual_seed(1), device="cuda")
    old = cuda.rand((H // 2, W // 2), generator=cuda.Generator(device="cuda").manual_seed(2), device="cuda")
    want = []
    for x in clip:
        small = O.pyramid_down(x)
        a0, grad = O.image_model(small)
        f = O.propagate(flow.cpu().numpy(), 3, 3)
        u, i = O.update(a0, grad, old.cpu().numpy(), f, 0.01, 2.0)
        want.append([small, a0, grad, u, i, O.smooth(u, 2)])
    got = []
    for n in range(ROUNDS):
        small = stages.pyramid_down(dev[n % 4])
        a0, grad = stages.image_model(small)
        f = stages.propagate(flow, 3, 3)
        u, i = stages.update(a0, grad, old, f, 0.01, 2.0)
        out = [small, a0, grad, u, i, stages.smooth(u, 2)]
        if n >= ROUNDS - 4:  # the others give their memory to the next round
            got.append((n % 4, out))
    cuda.cuda.synchronize()
    for k, out in got:
        for j, (a, b) in enumerate(zip(out, want[k])):
            assert np.array_equal(a.cpu().numpy(), b), (k, j)


@pytest.mark.parametrize("depth", [1, 4])
def test_lax_wendroff_over_several_launches(cuda, depth):
    """40 iterations take three launches, each reading what the one before has just written, of
    images that change from call to call."""
    from flowfilter_b200 import LaxWendroffPropagator
    from make_reference_fixtures import lw_inputs

    pairs = [lw_inputs(H, W, depth, s) for s in range(3)]
    flow = pairs[0][0]
    want = [O.lax_wendroff(flow, x, 40) for _, x in pairs]
    imgs = [cuda.from_numpy(x).cuda() for _, x in pairs]
    lw = LaxWendroffPropagator(cuda.from_numpy(flow).cuda(), imgs[0])
    lw.iterations = 40
    for n in range(ROUNDS):
        lw.setInputImage(imgs[n % 3])
        lw.compute()
        if n % 7 < 3:
            assert np.array_equal(lw.getPropagatedImage().cpu().numpy(), want[n % 3]), n
