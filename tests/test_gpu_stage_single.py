"""One propagation iteration on rows that do not allow four pixels at a time, on both sides of the
size from which it runs as two passes."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(307, 651), (308, 651), (767, 651), (770, 651), (1000, 652)])
@pytest.mark.parametrize("n", [1, 2])
def test_single_iteration(cuda, H, W, n):
    from flowfilter_b200 import stages

    rng = np.random.default_rng(H)
    f, v = (rng.normal(0, 1, (H, W, 2)).astype(np.float32) for _ in range(2))
    s = rng.random((H, W), dtype=np.float32)
    dev = [cuda.from_numpy(x).cuda() for x in (f, s, v)]
    assert np.array_equal(stages.propagate(dev[0], n, 2).cpu().numpy(), O.propagate(f, n, 2))
    got = [t.cpu().numpy() for t in stages.propagate_payload(*dev, n, 2)]
    assert all(np.array_equal(a, b) for a, b in zip(got, O.propagate_payload(f, s, v, n, 2)))
