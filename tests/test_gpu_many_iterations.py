"""Levels of more iterations than the timed configurations: the default kernel follows the cost of
the slab kernel's halo, and every choice gives the per-stage kernels' states."""

from __future__ import annotations

import pytest

from test_gpu_slab import frames_of, same, states

pytestmark = pytest.mark.gpu

# (height, width, delta, N, S, kernel): both sides of each line of the rule
CHOICES = [
    (240, 320, True, 4, 2, "slab"), (239, 320, True, 4, 2, "tile"), (240, 320, True, 8, 4, "tile"),
    (280, 400, True, 8, 4, "slab"), (240, 320, True, 10, 8, "slab"), (120, 160, False, 4, 4, "slab"),
    (120, 160, False, 8, 4, "tile"), (150, 200, False, 8, 4, "slab"), (512, 512, True, 8, 8, "slab"),
    (512, 512, True, 10, 12, "per-stage"), (512, 512, True, 10, 15, "per-stage"), (512, 512, True, 20, 8, "per-stage"),
    (480, 640, False, 4, 12, "slab"), (480, 640, False, 20, 8, "per-stage"), (480, 640, False, 28, 12, "per-stage"),
]


@pytest.mark.parametrize("H,W,delta,N,S,kernel", CHOICES)
def test_default_kernel(cuda, H, W, delta, N, S, kernel):
    import flowfilter_b200 as ffb

    clip = [cuda.from_numpy(x).cuda() for x in frames_of(H, W, 3, N + S)]
    coarse = cuda.randn((H // 2, W // 2, 2), generator=cuda.Generator(device="cuda").manual_seed(4), device="cuda")
    out = []
    for fused in (2, 0):
        img = cuda.zeros((H, W), dtype=cuda.uint8, device="cuda")
        f = ffb.DeltaFlowFilter(img, coarse) if delta else ffb.FlowFilter(H, W)
        f.maxflow, f.smoothIterations, f.gamma = float(N), S, 10.0
        f.setFused(fused)
        assert (kernel if fused else "per-stage") in f.tuning()
        got = []
        for x in clip:
            if delta:
                img.copy_(x)
            else:
                f.loadImage(x)
            f.compute()
            got += [f.levelState(0, k) for k in ((0, 2, 3) if delta else (0, 1, 2))]
        out.append(got)
    assert same(*out)


@pytest.mark.parametrize("levels,maxflow,smooth", [(1, 20.0, [8]), (2, 10.0, [15, 1]), (2, 8.0, [6, 12])])
def test_differentiable_forward(cuda, levels, maxflow, smooth):
    """The frame forward of many iterations, with and without a tape, is that of the stage nodes."""
    from flowfilter_b200 import diff

    H, W = 180, 260
    g = cuda.Generator(device="cuda").manual_seed(levels)
    frames = cuda.rand((2, 2, H, W), generator=g, device="cuda")
    flows = []
    for per_stage, grad in ((True, False), (False, False), (False, True)):
        f = diff.DiffPyramidalFlowFilter(H, W, levels, [0.01, 0.02][:levels], smooth, maxflow=maxflow)
        f.per_stage = per_stage
        with cuda.set_grad_enabled(grad):
            flows.append(f(frames).detach())
    assert cuda.equal(flows[0], flows[1]) and cuda.equal(flows[0], flows[2])


def test_no_memory_for_scratch(cuda):
    """Levels that run per stage by default, because it is faster, run the slab kernel where their
    scratch cannot be allocated; levels that are asked to run per stage fail."""
    import flowfilter_b200 as ffb
    from flowfilter_b200 import _lib

    clip = frames_of(480, 640, 2, 1)
    out = []
    for fail in (False, True):
        f = ffb.FlowFilter(480, 640)
        f.maxflow, f.smoothIterations, f.gamma = 20.0, 8, 10.0
        assert "per-stage" in f.tuning()
        if fail:
            _lib.lib().ff_debug_fail_allocation_after(2)
        try:
            for x in clip:
                f.loadImage(x)
                f.compute()
        finally:
            _lib.lib().ff_debug_fail_allocation_after(-1)
        assert ("slab" if fail else "per-stage") in f.tuning()
        out.append([f.levelState(0, k) for k in (0, 1, 2)])
    assert same(*out)
    f = ffb.FlowFilter(480, 640)
    f.setFused(0)
    f.loadImage(clip[0])
    _lib.lib().ff_debug_fail_allocation_after(2)
    try:
        with pytest.raises(_lib.FFError):
            f.compute()
    finally:
        _lib.lib().ff_debug_fail_allocation_after(-1)
