"""ff_diff_frame_infer through the C ABI: the optional copy of the top level's unsmoothed flow,
which the Python layer asks for with one level only."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu


def run(torch, name, flt, frames, dtype, fu_shift, workspace):
    """Two frames by ``name``; the state, and the top's unsmoothed flow in a buffer that starts
    ``fu_shift`` elements into an allocation (None: not asked for)."""
    from flowfilter_b200 import diff as dm
    from flowfilter_b200._lib import call

    d, B = (1 if dtype == torch.float64 else 0), frames.shape[0]
    g = dm._geom(flt, B)
    ws = dm._workspace(workspace, d, g, frames)
    ws.fill_(float("nan"))  # nothing may be read from it that the call has not written
    empty = [torch.zeros((B, h, w) + c, dtype=dtype, device="cuda") for h, w in flt.shapes for c in ((2,), (), (2,))]
    gamma, weights = flt.gamma.detach(), flt.weights.detach()
    h, w = flt.shapes[-1]
    fu = None if fu_shift is None else torch.zeros(fu_shift + B * h * w * 2, dtype=dtype, device="cuda")[fu_shift:]
    state, out = empty, []
    for t in range(2):
        new = [torch.empty_like(x) for x in empty]
        frame = frames[:, t].contiguous()
        tail = [dm._p(ws), dm._stream()]
        if name == "ff_diff_frame_forward":
            tail.insert(0, None)  # y_out
        call(name, d, ctypes.byref(g), int(t == 0), dm._p(frame), dm._p(gamma), dm._p(weights), dm._ptrs(state),
             dm._ptrs(new), dm._p(fu), *tail)
        state = new
        out += [x.clone() for x in new] + ([fu.clone()] if fu is not None else [])
    return out


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("levels,H,W", [(1, 33, 45), (2, 40, 132), (3, 61, 83)])
@pytest.mark.parametrize("fu_shift", [0, 1, 2])
def test_unsmoothed_flow_changes_nothing_else(cuda, levels, H, W, dtype, fu_shift):
    """Every output equals the taped forward's, and the state that of a call without fu_out, bit
    for bit, wherever fu_out starts."""
    from flowfilter_b200 import diff as dm

    dt = getattr(cuda, dtype)
    flt = dm.DiffPyramidalFlowFilter(H, W, levels, [0.01, 0.02, 0.03][:levels], [2, 1, 3][:levels], maxflow=3.0, dtype=dt)
    g = cuda.Generator(device="cuda").manual_seed(W + levels)
    frames = cuda.rand((2, 2, H, W), generator=g, device="cuda", dtype=dt)
    infer = ("ff_diff_frame_infer", flt, frames, dt)
    with_fu = run(cuda, *infer, fu_shift, "ff_diff_frame_infer_bytes")
    without = run(cuda, *infer, None, "ff_diff_frame_infer_bytes")
    taped = run(cuda, "ff_diff_frame_forward", flt, frames, dt, fu_shift, "ff_diff_frame_tape_bytes")
    assert all(cuda.equal(a, b) for a, b in zip(with_fu, taped)) and len(with_fu) == len(taped)
    state = [x for i, x in enumerate(with_fu) if i % (3 * levels + 1) != 3 * levels]
    assert all(cuda.equal(a, b) for a, b in zip(state, without)) and len(state) == len(without)
