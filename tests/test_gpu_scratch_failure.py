"""A per-stage filter whose scratch cannot be allocated: the frame fails whole, and computed
again it is the frame of a filter that never failed."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_slab import frames_of, same, states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [1, 2, 3])
def test_frame_after_a_failed_one(cuda, levels):
    import flowfilter_b200 as ffb
    from flowfilter_b200 import _lib

    lib = _lib.lib()
    clip = frames_of(64, 90, 3, levels)

    def make():
        f = ffb.PyramidalFlowFilter(64, 90, levels)
        f.maxflow = 4.0
        f.setFused(0)
        return f

    ref = make()
    want = []
    for x in clip:
        ref.loadImage(x)
        ref.compute()
        want.append(states(ref, levels))
    n = 0
    while True:
        f = make()
        f.loadImage(clip[0])
        lib.ff_debug_fail_allocation_after(n)
        try:
            f.compute()
        except _lib.FFError as e:
            assert e.status == _lib.FF_ERR_OUT_OF_MEMORY
        else:
            break
        finally:
            lib.ff_debug_fail_allocation_after(-1)
        for t, x in enumerate(clip):
            f.loadImage(x)
            f.compute()
            assert same(states(f, levels), want[t]), (n, t)
        n += 1
    assert n == 4 + 9 * (levels - 1)  # the scratch fields of a top level and of each delta level
