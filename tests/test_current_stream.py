"""The handle of the current stream, with and without the torch functions that give it alone."""

from __future__ import annotations

import sys
import types

import pytest


@pytest.mark.parametrize("initialised,private,want", [(True, True, 7), (True, False, 5), (False, True, 5)])
def test_current_stream(monkeypatch, initialised, private, want):
    from flowfilter_b200 import _lib

    fake = types.ModuleType("torch")
    fake.cuda = types.SimpleNamespace(is_initialized=lambda: initialised,
                                      current_stream=lambda: types.SimpleNamespace(cuda_stream=5))
    fake._C = types.SimpleNamespace()
    if private:
        fake._C._cuda_getDevice = lambda: 1
        fake._C._cuda_getCurrentRawStream = lambda device: 6 + device
    monkeypatch.setitem(sys.modules, "torch", fake)
    assert _lib.current_stream() == want
