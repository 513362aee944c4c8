"""Inference of one differentiable filter on several streams at once: each has its own scratch."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [1, 2])
def test_streams_at_once(cuda, levels):
    from flowfilter_b200 import diff

    H, W, B, T = 256, 300, 4, 8
    f = diff.DiffPyramidalFlowFilter(H, W, levels, [0.01, 0.02][:levels], [2, 3][:levels], maxflow=4.0)
    g = cuda.Generator(device="cuda").manual_seed(levels)
    clips = [cuda.rand((B, T, H, W), generator=g, device="cuda") for _ in range(3)]
    sides = [cuda.cuda.Stream() for _ in clips]
    with cuda.no_grad():
        want = [f(x).clone() for x in clips]
        cuda.cuda.synchronize()
        for _ in range(5):
            got = []
            for x, s in zip(clips, sides):
                with cuda.cuda.stream(s):
                    got.append(f(x))
            cuda.cuda.synchronize()
            assert all(cuda.equal(a, b) for a, b in zip(got, want))
