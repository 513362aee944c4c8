"""Stage calls of the C ABI whose output shares memory with an input whose rows lie closer than
their length (one row for all: pitch 0): in place, as any other overlap."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

H, W, N = 60, 200, 3


def p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("row", [0, 17, H - 1])
def test_one_input_row_inside_the_output(cuda, row):
    from flowfilter_b200._lib import call, lib

    rng = np.random.default_rng(row)
    line = rng.normal(0, 1, (W, 2)).astype(np.float32)
    full = np.ascontiguousarray(np.broadcast_to(line, (H, W, 2)))
    stream = ctypes.c_void_p(cuda.cuda.current_stream().cuda_stream)
    ws = cuda.empty(lib().ff_stage_propagate_payload_workspace_size(H, W), dtype=cuda.uint8, device="cuda")
    for _ in range(20):
        out = cuda.zeros((H, W, 2), device="cuda")
        out[row] = cuda.from_numpy(line)
        call("ff_stage_propagate", p(out[row]), 0, H, W, N, 2, p(out), W * 8, p(ws), stream)
        assert np.array_equal(out.cpu().numpy(), O.propagate(full, N, 2))
        out.zero_()
        out[row] = cuda.from_numpy(line)
        call("ff_stage_smooth", p(out[row]), 0, H, W, N, p(out), W * 8, p(ws), stream)
        assert np.array_equal(out.cpu().numpy(), O.smooth(full, N))
