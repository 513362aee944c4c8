"""The frame driver's propagation adjoint at the edges of its windows (64 columns in float32, 32
in float64, two halo columns on inner sides) and row runs, with every border: the frame node's
gradients against the per-stage nodes' (one adjoint launch per sub-step)."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_diff import float_frames, sequence_loss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("border", [0, 1, 3])
@pytest.mark.parametrize("H,W", [(4, 4), (9, 62), (16, 64), (21, 65), (30, 67), (130, 124), (37, 187)])
def test_propagation_adjoint_at_window_edges(cuda, H, W, border, dtype):
    """Both run the same forward, so the same upwind branches; the gradients differ by the
    order of their sums.  Tolerance: about 100 roundings on the way through three frames of
    two levels, each at most a few times the largest gradient: 2^-24 * 1000 of it in float32,
    2^-53 * 1000 in float64."""
    import flowfilter_b200.diff as dm

    B, T = 2, 3
    dt = getattr(cuda, dtype)
    frames = cuda.from_numpy(float_frames(B, T, H, W, H + W).astype(np.float64)).to("cuda", dt)
    proj = cuda.from_numpy(np.random.default_rng(5).normal(0, 1, (B, T, H, W, 2))).to("cuda", dt)
    res = []
    for per_stage in (False, True):
        f = dm.DiffPyramidalFlowFilter(H, W, 2, [3.0, 12.0], [1, 2], maxflow=4.0, border=border, dtype=dt,
                                       checkpoint_every=2)
        f.per_stage = per_stage
        x = frames.clone().requires_grad_(True)
        flows = f(x)
        sequence_loss(flows, proj).backward()
        res.append((flows.detach().cpu().numpy(), x.grad.cpu().numpy()))
    np.testing.assert_array_equal(res[0][0], res[1][0])
    eps = 2.0 ** (-24 if dtype == "float32" else -53)
    a, b = res[0][1], res[1][1]
    assert np.isfinite(b).all() and np.abs(a - b).max() <= 1000 * eps * np.abs(b).max()
