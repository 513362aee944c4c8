"""What a call uploads or clears is in place when it returns, for streams that are not ordered
after the default stream."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_gpu_batch_streams import STREAMS, alone_and_batch

pytestmark = pytest.mark.gpu

BUSY = 60_000_000  # clock cycles the default stream spins: about 30 ms


def test_tables_of_a_first_batched_step(cuda):
    import flowfilter_b200 as ffb

    rng = np.random.default_rng(4)
    frames = [cuda.from_numpy(rng.integers(0, 256, s[:2], dtype=np.uint8)).cuda() for s in STREAMS]
    side = cuda.cuda.Stream()
    for _ in range(5):
        alone, batch = alone_and_batch(ffb)
        packed = batch.pack(frames)
        cuda.cuda.synchronize()
        cuda.cuda._sleep(BUSY)
        for _ in range(4):  # the second and third step build a table each
            batch.step(packed, side)
        cuda.cuda.synchronize()
        for i, f in enumerate(alone):
            for _ in range(4):
                f.loadImage(frames[i])
                f.computeAsync()
            assert np.array_equal(batch.stream(i).getFlow(), f.getFlow()), i


@pytest.mark.parametrize("how", ["copy", "device copy", "set"])
def test_buffers_of_the_c_abi(cuda, how):
    import flowfilter_b200 as ffb
    from flowfilter_b200._lib import call

    H, W = 480, 640
    a, b = ctypes.c_void_p(), ctypes.c_void_p()
    pitch = ctypes.c_size_t()
    new = np.random.default_rng(6).integers(0, 256, (H, W), dtype=np.uint8)
    old = np.zeros_like(new)
    want = ffb.FlowFilter(H, W)
    want.loadImage(new if how != "set" else np.full_like(new, 7))
    want.compute()
    for p in (a, b):
        call("ff_malloc_pitch", ctypes.byref(p), ctypes.byref(pitch), W, H)
    try:
        call("ff_memcpy2d", a, pitch, old.ctypes.data_as(ctypes.c_void_p), W, W, H, 0)
        call("ff_memcpy2d", b, pitch, new.ctypes.data_as(ctypes.c_void_p), W, W, H, 0)
        side = cuda.cuda.Stream()
        f = ffb.FlowFilter(H, W)
        cuda.cuda.synchronize()
        cuda.cuda._sleep(BUSY)
        if how == "copy":
            call("ff_memcpy2d", a, pitch, new.ctypes.data_as(ctypes.c_void_p), W, W, H, 0)
        elif how == "device copy":
            call("ff_memcpy2d", a, pitch, b, pitch, W, H, 2)
        else:
            call("ff_memset2d", a, pitch, 7, W, H)
        call("ff_filter_load_image_device_async", f._h, a, pitch, ctypes.c_void_p(side.cuda_stream))
        f.computeAsync(side)
        cuda.cuda.synchronize()
        assert np.array_equal(f.getImage(), want.getImage())
    finally:
        for p in (a, b):
            call("ff_free", p)
