"""Stage functions on padded rows that end with the memory they lie in: the padding after the
last row is not there, and what lies beside the rows does not matter."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def exact_rows(torch, values, pitch, channels):
    """A view of ``values`` with rows ``pitch`` pixels apart in a block of 2 MB multiples that ends
    with its last pixel; NaN between the rows."""
    H, W = values.shape[:2]
    n = ((H - 1) * pitch + W) * channels
    block = torch.full(((n + (1 << 19) - 1) // (1 << 19) * (1 << 19),), float("nan"), device="cuda")
    size, stride = (H, W) + (channels,) * (channels > 1), (pitch * channels,) + (channels,) * (channels > 1) + (1,)
    # the last pixel at the end, the start moved down to 32 bytes (4 pixels are one access)
    view = block.as_strided(size, stride, (block.numel() - n) // 8 * 8)
    view.copy_(torch.from_numpy(values))
    return view


@pytest.mark.parametrize("H,W,pitch", [(9, 13, 16), (40, 130, 132), (33, 255, 256), (20, 126, 136), (12, 5, 8)])
@pytest.mark.parametrize("n", [1, 4])
def test_rows_without_padding_after_the_last(cuda, H, W, pitch, n):
    from flowfilter_b200 import stages

    rng = np.random.default_rng(W + n)
    f, v = (rng.normal(0, 1, (H, W, 2)).astype(np.float32) for _ in range(2))
    s = rng.random((H, W), dtype=np.float32)
    flow, vec, sca = exact_rows(cuda, f, pitch, 2), exact_rows(cuda, v, pitch, 2), exact_rows(cuda, s, pitch, 1)
    assert np.array_equal(stages.propagate(flow, n, 1).cpu().numpy(), O.propagate(f, n, 1))
    got = [t.cpu().numpy() for t in stages.propagate_payload(flow, sca, vec, n, 1)]
    assert all(np.array_equal(x, y) for x, y in zip(got, O.propagate_payload(f, s, v, n, 1)))
    assert np.array_equal(stages.smooth(flow, n).cpu().numpy(), O.smooth(f, n))
    a0, grad = (t.cpu().numpy() for t in stages.image_model(sca))
    wa, wg = O.image_model(s)
    assert np.array_equal(a0, wa) and np.array_equal(grad, wg)
