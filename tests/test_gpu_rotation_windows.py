"""The Lax-Wendroff kernel at the edges of its windows (64 columns, less an even halo on inner
sides) and row bands, against the oracle: bit for bit, since both round the same operations."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from make_reference_fixtures import lw_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,d,it", [
    (16, 64, 1, 1),      # one full window, one band
    (17, 65, 4, 1),      # one column and one row beyond
    (33, 96, 1, 16),     # the deepest halo of one launch: windows 32 columns apart
    (40, 97, 4, 15),     # an odd halo, rounded up
    (700, 121, 1, 4),    # windows 56 apart: one pixel in the last, many bands
    (301, 2050, 4, 3),   # more windows than multiprocessors' worth of bands
    (2500, 31, 1, 2),    # narrower than a window
])
def test_window_and_band_edges(cuda, h, w, d, it):
    from flowfilter_b200 import LaxWendroffPropagator

    flow, img = lw_inputs(h, w, d, h + 3 * w + it)
    flow_t = cuda.from_numpy(flow).cuda()
    img_t = cuda.from_numpy(img).cuda()
    lw = LaxWendroffPropagator(flow_t, img_t)
    lw.iterations = it
    lw.compute()
    np.testing.assert_array_equal(lw.getPropagatedImage().cpu().numpy(), O.lax_wendroff(flow, img, it))
