"""Levels on both sides of the pixel line from which the streaming kernel is the default, which
depends on N and S: the kernel chosen, and its states against the per-stage kernels'."""

from __future__ import annotations

import pytest

from test_gpu_slab import frames_of, same

pytestmark = pytest.mark.gpu

# (height, width, delta, N, S, kernel)
LINES = [(900, 990, True, 1, 1, "slab"), (900, 1010, True, 1, 1, "fused"), (1200, 1570, True, 4, 2, "slab"),
         (1200, 1601, True, 4, 2, "fused"), (1500, 1990, True, 4, 4, "slab"), (1500, 2010, True, 4, 4, "fused"),
         (1000, 1349, False, 2, 1, "slab"), (1000, 1351, False, 2, 1, "fused"), (1500, 1610, False, 2, 2, "slab"),
         (1500, 1620, False, 2, 2, "fused"), (2160, 3840, False, 3, 4, "fused"), (2160, 3840, True, 2, 3, "fused")]


@pytest.mark.parametrize("H,W,delta,N,S,kernel", LINES)
def test_default_kernel_of_large_levels(cuda, H, W, delta, N, S, kernel):
    import flowfilter_b200 as ffb

    # a delta level is level 0 of a pyramid, whose image rows every kernel takes at any width
    clip = [cuda.from_numpy(x).cuda() for x in frames_of(H, W, 2, N + S)]
    out = []
    for fused in (2, 0):
        f = ffb.PyramidalFlowFilter(H, W, 2) if delta else ffb.FlowFilter(H, W)
        f.maxflow = float(N)
        f.gamma, f.smoothIterations = ([10.0, 20.0], [S, 1]) if delta else (10.0, S)
        f.setFused(fused)
        assert f"level 0: {kernel if fused else 'per-stage'}" in f.tuning()
        for x in clip:
            f.loadImage(x)
            f.compute()
        out.append([f.levelState(0, k) for k in ((0, 2, 3) if delta else (0, 1, 2))])
    assert same(*out)
